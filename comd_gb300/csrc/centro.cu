// centro.cu -- centrosymmetry parameter of every atom
// (AtomVisualize::computeCentrosymmetry, src-viz/AtomVisualize.c:399-672), a
// headless kernel over the link cells.
//
// One thread per atom of the compacted atom list (64 per CTA).  The
// neighbour scan visits the atom's own box (box-relative differences), then
// the 26 adjacent boxes in x-outer, z-inner order, wrapped once per axis with
// the periodic offset rounded to float (AtomVisualize.c:458-505), and keeps
// up to 12 candidates: the next free entry while fewer than 12 are held, then
// the first entry of largest r^2 is replaced unless the candidate's r^2 is
// larger.  All of it in FP64 with the reference's operation order (this
// translation unit is built without FMA contraction); r^2 values are
// compared as the integer images of non-negative doubles.
//
// The parameter is the minimum over the 10395 pairings of the 12 vectors of
// the sum of |r_a + r_b|^2, accumulated in a float over the pairs in the
// order of their lower index (testCentro, :560-664).  The 66 pair terms are
// rounded to FP32 once; a depth-first search over the pairings (the lowest
// unpaired vector paired first, as the visualiser's loops pair them) finds
// the least plain-FP32 sum, cutting every branch whose partial sum already
// reaches the best complete one (partial sums of non-negative terms never
// decrease, so the cut loses nothing; the greedy pairing gives the first
// bound).  A second search visits the pairings whose FP32 sum lies within
// 4e-6 of that least and sums them exactly as testCentro does (double terms,
// each partial sum rounded to float).  Both sums round at most six float
// additions of non-negative terms, so each is within 12 units of 2^-24 of
// the exact sum: a pairing outside the window cannot be the reference's
// minimum, and the result is the reference's value bit for bit.
// APPROX_CENTROSYM's greedy pairing (:528-557) is the `approx` variant.
#include <algorithm>

#include "sim.h"

using namespace cg;
using namespace cgapi;

namespace {

constexpr int NPAIR = 66;
constexpr int CT = 64;  // threads (atoms) per CTA

// index of the pair a < b among the 66, row by row
__device__ __forceinline__ int pidx(int a, int b) { return 11 * a - (a * (a - 1)) / 2 + b - a - 1; }

__device__ __forceinline__ long long key(double rsq) { return __double_as_longlong(rsq); }

// |a + b|^2 of two held vectors, the reference's order
__device__ __forceinline__ double pair_term(const double (*v)[3][CT], int a, int b, int t) {
  const double x = __dadd_rn(v[a][0][t], v[b][0][t]);
  const double y = __dadd_rn(v[a][1][t], v[b][1][t]);
  const double z = __dadd_rn(v[a][2][t], v[b][2][t]);
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// Depth-first over the pairings: the lowest unpaired entry is paired next,
// with its partners in index order.  A branch whose partial FP32 sum reaches
// `bound` (STRICT) or exceeds it is cut.  leaf(sum, nn, pp) gets every
// pairing kept; its pairs are (nn[l], pp[l]), l = 0..5, lower index first.
template <bool STRICT, class Leaf>
__device__ __forceinline__ void pairing_dfs(const float (*p)[CT], int t, const float &bound,
                                            Leaf &&leaf) {
  int nn[6], pp[6];
  float acc[6];
  int used = 1, lvl = 0;
  nn[0] = 0;
  pp[0] = 0;
  acc[0] = 0.0f;
  while (true) {
    int q = pp[lvl] + 1;
    while (q < 12 && (used >> q & 1)) q++;
    if (q >= 12) {  // this level's partners are done
      used &= ~(1 << nn[lvl]);
      if (lvl == 0) break;
      lvl--;
      used &= ~(1 << pp[lvl]);
      continue;
    }
    pp[lvl] = q;
    const float a = __fadd_rn(acc[lvl], p[pidx(nn[lvl], q)][t]);
    if (STRICT ? a >= bound : a > bound) continue;
    if (lvl == 5) {
      leaf(a, nn, pp);
      continue;
    }
    used |= 1 << q;
    lvl++;
    acc[lvl] = a;
    const int n = __ffs(~used) - 1;
    nn[lvl] = n;
    pp[lvl] = n;
    used |= 1 << n;
  }
}

// the FP32 extent of every box's atoms (relative to its centre): lo, then hi;
// without bounds when a position is not a number, and nothing in an empty box
__global__ void __launch_bounds__(256) box_extent_kernel(Slots s, int nboxes, float4 *ext) {
  const int b = blockIdx.x * 256 + threadIdx.x;
  if (b >= nboxes) return;
  const float inf = __int_as_float(0x7f800000);
  float4 lo = make_float4(inf, inf, inf, 0.f), hi = make_float4(-inf, -inf, -inf, 0.f);
  const int n = s.natoms[b];
  for (int k = 0; k < n; k++) {
    const float4 q = __ldg(s.pos32 + b * CG_MAXATOMS + k);
    if (!(q.x + q.y + q.z == q.x + q.y + q.z)) {
      lo = make_float4(-inf, -inf, -inf, 0.f);
      hi = make_float4(inf, inf, inf, 0.f);
      break;
    }
    lo = make_float4(fminf(lo.x, q.x), fminf(lo.y, q.y), fminf(lo.z, q.z), 0.f);
    hi = make_float4(fmaxf(hi.x, q.x), fmaxf(hi.y, q.y), fmaxf(hi.z, q.z), 0.f);
  }
  ext[2 * b] = lo;
  ext[2 * b + 1] = hi;
}

// how far p (a coordinate) lies outside [lo + f, hi + f], by the operations of
// the candidates' test: no atom of the box gives a smaller |(q - p) + f|
__device__ __forceinline__ float outside(float lo, float hi, float p, float f) {
  return fmaxf(fmaxf((lo - p) + f, -((hi - p) + f)), 0.f);
}

__global__ void __launch_bounds__(CT) centro_kernel(Geom g, Slots s, const double *dcenter,
                                                    const int *atom_slot, int ntot, int approx,
                                                    float slack, const float4 *ext,
                                                    double *out) {
  // per thread (column t): held vectors, their r^2 (integer images) and the
  // pair terms rounded to FP32.  Warps run the scan and the pairing phases
  // at different times with no barrier between them, so no array is shared
  // between the phases.
  __shared__ double v[12][3][CT];
  __shared__ long long vk[12][CT];
  __shared__ float p32[NPAIR][CT];
  const int t = threadIdx.x;
  const int a = blockIdx.x * CT + t;
  if (a >= ntot) return;
  const int io = atom_slot[a];
  const int b = io >> 6, i = io & 63;
  const int ni = s.natoms[b];
  const RepGeo &R = rep_of(g, b);
  const int nx = R.nbx[0], ny = R.nbx[1], nz = R.nbx[2];
  const int lb = b - R.box0;
  const int bz = lb / (nx * ny), by = (lb - bz * nx * ny) / nx, bx = lb - bz * nx * ny - by * nx;
  const d4 ri = s.r[io];
  int nb = 0, kmax = 0;
  long long rmax = 0;
  auto offer = [&](double dx, double dy, double dz) {
    const double rsq =
        __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    const long long kk = key(rsq);
    int i1;
    if (nb < 12) {
      i1 = nb++;
    } else {
      if (kk > rmax) return;
      i1 = kmax;
    }
    v[i1][0][t] = dx;
    v[i1][1][t] = dy;
    v[i1][2][t] = dz;
    vk[i1][t] = kk;
    if (nb == 12) {  // first entry of largest r^2
      kmax = 0;
      rmax = vk[0][t];
      for (int k = 1; k < 12; k++)
        if (vk[k][t] > rmax) {
          kmax = k;
          rmax = vk[k][t];
        }
    }
  };
  // Candidates past the largest of twelve held are refused by the FP64 test in
  // `offer`; an FP32 test in front of it (box-centred positions; est < cut
  // holds for every candidate that `offer` would take, the FP32 distance
  // erring by less than `own` and 1e-6 of it) refuses nearly all of them first,
  // and whole boxes by their extent.  Within a box every thread runs on to its
  // next candidate that passes, so that the insertions of a warp's threads,
  // the expensive part, happen together.  At 256,000 atoms 1.95 ms where an
  // FP64 test of every candidate took 3.64; one loop over all candidates,
  // whose box changes diverge, took 3.31.
  const double cxi = __dadd_rn(dcenter[3 * b + 0], ri.x);
  const double cyi = __dadd_rn(dcenter[3 * b + 1], ri.y);
  const double czi = __dadd_rn(dcenter[3 * b + 2], ri.z);
  const float4 pi = __ldg(s.pos32 + io);
  const float own = slack + 1e-6f * (fabsf(pi.x) + fabsf(pi.y) + fabsf(pi.z));
  float cut = 3.0e38f;  // est must be below it
  // the candidates of box b2 with corner offset e (own box: relative)
  auto scan = [&](int b2, int nj, bool same, double ex, double ey, double ez, float fx, float fy,
                  float fz) {
    int j = 0;
    while (true) {
      bool got = false;
      for (; j < nj; j++) {
        const float4 q = __ldg(s.pos32 + b2 * CG_MAXATOMS + j);
        const float tx = (q.x - pi.x) + fx, ty = (q.y - pi.y) + fy, tz = (q.z - pi.z) + fz;
        // (not >=: a NaN goes on to the exact test)
        got = !(tx * tx + ty * ty + tz * tz >= cut) && !(same && j == i);
        if (got) break;
      }
      if (!got) break;
      const d4 rj = s.r[b2 * CG_MAXATOMS + j];
      j++;
      if (same)
        offer(__dsub_rn(rj.x, ri.x), __dsub_rn(rj.y, ri.y), __dsub_rn(rj.z, ri.z));
      else
        offer(__dsub_rn(__dadd_rn(ex, rj.x), cxi), __dsub_rn(__dadd_rn(ey, rj.y), cyi),
              __dsub_rn(__dadd_rn(ez, rj.z), czi));
      if (nb == 12) {
        // est < (r + e)^2, e the FP32 vector's error: slack for the box offset,
        // and roundings of the atom's own position and of the distance
        const float r2 = __double2float_ru(__longlong_as_double(rmax));
        const float r = sqrtf(r2), e = own + 1e-6f * r;
        cut = (r2 + e * (2.0f * r + e) + 1e-30f) * 1.000001f;
      }
    }
  };
  scan(b, ni, true, 0.0, 0.0, 0.0, 0.f, 0.f, 0.f);
  for (int cell = 0; cell < 27; cell++) {  // x-outer, z-inner
    if (cell == 13) continue;
    float ox = 0.0f, oy = 0.0f, oz = 0.0f;
    int qx = bx + cell / 9 - 1, qy = by + cell / 3 % 3 - 1, qz = bz + cell % 3 - 1;
    if (qx < 0) { qx = nx - 1; ox = __double2float_rn(-R.bounds[0]); }
    if (qx >= nx) { qx = 0; ox = __double2float_rn(R.bounds[0]); }
    if (qy < 0) { qy = ny - 1; oy = __double2float_rn(-R.bounds[1]); }
    if (qy >= ny) { qy = 0; oy = __double2float_rn(R.bounds[1]); }
    if (qz < 0) { qz = nz - 1; oz = __double2float_rn(-R.bounds[2]); }
    if (qz >= nz) { qz = 0; oz = __double2float_rn(R.bounds[2]); }
    const int b2 = R.box0 + qz * nx * ny + qy * nx + qx;
    const double ex = __dadd_rn((double)ox, dcenter[3 * b2 + 0]);
    const double ey = __dadd_rn((double)oy, dcenter[3 * b2 + 1]);
    const double ez = __dadd_rn((double)oz, dcenter[3 * b2 + 2]);
    const float fx = (float)(ex - dcenter[3 * b + 0]), fy = (float)(ey - dcenter[3 * b + 1]),
                fz = (float)(ez - dcenter[3 * b + 2]);
    // a box whose atoms all fail the test is passed over whole
    const float4 lo = __ldg(ext + 2 * b2), hi = __ldg(ext + 2 * b2 + 1);
    const float gx = outside(lo.x, hi.x, pi.x, fx), gy = outside(lo.y, hi.y, pi.y, fy),
                gz = outside(lo.z, hi.z, pi.z, fz);
    if (gx * gx + gy * gy + gz * gz >= cut) continue;
    scan(b2, s.natoms[b2], false, ex, ey, ez, fx, fy, fz);
  }
  double c = 1000.0;
  if (nb >= 12) {
    if (approx) {
      // greedy pairing; a vector with r^2 = 0 counts as paired
      int paired = 0;
      for (int q = 0; q < 12; q++) paired |= (vk[q][t] > 0 ? 0 : 1) << q;
      c = 0.0;
      for (int j = 0; j < 11; j++) {
        if (paired >> j & 1) continue;
        double summin = 1000.0;
        int kmin = -1;
        for (int k = j + 1; k < 12; k++) {
          if (paired >> k & 1) continue;
          const double sum = pair_term(v, j, k, t);
          if (sum < summin) {
            kmin = k;
            summin = sum;
          }
        }
        c = __dadd_rn(c, summin);
        paired |= 1 << j;
        if (kmin >= 0) paired |= 1 << kmin;
      }
    } else {
      for (int x = 0, k = 0; x < 12; x++)
        for (int y = x + 1; y < 12; y++, k++) p32[k][t] = __double2float_rn(pair_term(v, x, y, t));
      // first bound: the greedy pairing's FP32 sum (a complete pairing)
      float best = 0.0f;
      for (int used = 0, step = 0; step < 6; step++) {
        const int n = __ffs(~used) - 1;
        used |= 1 << n;
        int qb = -1;
        float pb = 0.0f;
        for (int q = n + 1; q < 12; q++)
          if (!(used >> q & 1) && (qb < 0 || p32[pidx(n, q)][t] < pb)) {
            qb = q;
            pb = p32[pidx(n, q)][t];
          }
        used |= 1 << qb;
        best = __fadd_rn(best, pb);
      }
      pairing_dfs<true>(p32, t, best, [&](float sum, const int *, const int *) { best = sum; });
      const float window = __fadd_rn(best, __fmul_rn(best, 4e-6f)) + 1e-37f;
      pairing_dfs<false>(p32, t, window, [&](float, const int *nn, const int *pp) {
        float e = 0.0f;  // testCentro
        for (int l = 0; l < 6; l++)
          e = __double2float_rn(__dadd_rn((double)e, pair_term(v, nn[l], pp[l], t)));
        if ((double)e < c) c = (double)e;
      });
    }
  }
  out[io] = c;
}

// min / max over the replica's atoms (minCentro from 1000, maxCentro from 0),
// into range[0] and range[1], which hold those two: the values are not
// negative, so their bits are ordered as they are.  (One CTA over all boxes
// took 342 us at 256,000 atoms.)
__global__ void __launch_bounds__(256)
    centro_range_kernel(Slots s, const int *atom_slot, const double *c, int a0, int na,
                        unsigned long long *range) {
  double lo = 1000.0, hi = 0.0;
  for (int a = a0 + blockIdx.x * 256 + threadIdx.x; a < a0 + na; a += gridDim.x * 256) {
    const double x = c[atom_slot[a]];
    lo = x < lo ? x : lo;
    hi = x > hi ? x : hi;
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(range, (unsigned long long)__double_as_longlong(lo));
    atomicMax(range + 1, (unsigned long long)__double_as_longlong(hi));
  }
}

}  // namespace

extern "C" {

int comdgb_sim_centrosymmetry(comdgb_sim *h, int r, int approx, double *out, double *cmin,
                              double *cmax) {
  if (!h) return set_err(COMDGB_ERR_ARG, "null handle");
  if (r < 0 || r >= h->nrep) return set_err(COMDGB_ERR_ARG, "replica %d of %d", r, h->nrep);
  CK(cudaSetDevice(h->device));
  int err = 0;
  if (!h->centro) {
    double *c = dalloc<double>((size_t)h->nslots + 2, &err);
    float4 *x = dalloc<float4>(2 * (size_t)h->g.nboxes, &err);
    if (!err) {
      h->centro = track(h, c);
      h->centro_ext = track(h, x);
    } else {
      cudaGetLastError();
      cudaFree(c);
      cudaFree(x);
    }
    if (err) return set_err(COMDGB_ERR_NOMEM, "centrosymmetry buffer");
  }
  cudaStream_t st = h->stream;
  CK(cudaMemsetAsync(h->centro, 0, sizeof(double) * (size_t)h->nslots, st));  // empty slots 0
  const RepGeo &R = h->reps[r];
  double range[2] = {1000.0, 0.0};
  CK(cudaMemcpyAsync(h->centro + h->nslots, range, sizeof range, cudaMemcpyHostToDevice, st));
  if (h->ntot > 0) {
    // the error that the box offsets (up to two widths) bring to an FP32 vector
    double width = 0.0;
    for (const RepGeo &q : h->reps)
      for (int j = 0; j < 3; j++) width = std::max(width, q.boxsize[j]);
    const float slack = (float)(1.7320508 * 16.0 / 16777216.0 * 2.0 * width);
    launch_pos32_atoms(h->g, h->s, h->atom_slot, h->ntot, st);
    box_extent_kernel<<<(h->g.nboxes + 255) / 256, 256, 0, st>>>(h->s, h->g.nboxes,
                                                                 h->centro_ext);
    centro_kernel<<<(h->ntot + CT - 1) / CT, CT, 0, st>>>(h->g, h->s, h->dcenter, h->atom_slot,
                                                           h->ntot, approx, slack,
                                                           h->centro_ext, h->centro);
    centro_range_kernel<<<2 * h->sms, 256, 0, st>>>(
        h->s, h->atom_slot, h->centro, R.a0, R.na,
        reinterpret_cast<unsigned long long *>(h->centro + h->nslots));
  }
  CK(cudaGetLastError());
  if (out)
    CK(cudaMemcpyAsync(out, h->centro + (size_t)R.box0 * CG_MAXATOMS,
                       sizeof(double) * (size_t)R.nb * CG_MAXATOMS, cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(range, h->centro + h->nslots, sizeof range, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (cmin) *cmin = range[0];
  if (cmax) *cmax = range[1];
  return 0;
}

}  // extern "C"
