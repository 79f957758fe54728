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
// formed in FP32 once; a depth-first search over the pairings (the lowest
// unpaired vector paired first, as the visualiser's loops pair them) cuts every
// branch whose partial FP32 sum is past a window above the least complete one
// so far (partial sums of non-negative terms never decrease, so the cut loses
// nothing; the greedy pairing gives the first window), and the pairings it
// keeps are summed exactly as testCentro does (double terms, each partial sum
// rounded to float).  The window holds the reference's minimum: with m the
// largest component, an FP32 component of r_a + r_b is off by at most d =
// 2^-22 m, so the FP32 sum F of a pairing and its exact sum T differ by at
// most 2 d sqrt(18 T) + 18 d^2 + 6e-7 T; the reference's sum is within 12 units
// of 2^-24 of T.  A pairing with the least reference sum thus has an F of at
// most F' + 18.5 d sqrt(F') + 340 d^2 + 3e-6 F', F' any pairing's; the window
// is wider than that.  The result is the reference's value bit for bit.
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

struct V3 {
  double x, y, z;
};
// |a + b|^2 of two held vectors, the reference's order
__device__ __forceinline__ double pair_term(const V3 &a, const V3 &b) {
  const double x = __dadd_rn(a.x, b.x), y = __dadd_rn(a.y, b.y), z = __dadd_rn(a.z, b.z);
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// Depth-first over the pairings from level L (pairs formed) on: the lowest
// unpaired entry is paired next, with its partners in index order.  A branch
// whose partial sum exceeds `bound` is cut.  leaf(sum, pairs) gets every pairing
// kept, pair l in bits 8 l: its lower index, then its higher.
template <int L, class P, class Leaf>
__device__ __forceinline__ void pairing_dfs(P &&p, int used, float acc, unsigned long long pairs,
                                            const float &bound, Leaf &&leaf) {
  const int n = __ffs(~used) - 1;
  for (int m = ~used & 0xfff & ~(1 << n); m != 0; m &= m - 1) {
    const int q = __ffs(m) - 1;
    const float a = __fadd_rn(acc, p(pidx(n, q)));
    if (a > bound) continue;
    const unsigned long long with = pairs | (unsigned long long)(n | q << 4) << (8 * L);
    if constexpr (L == 5) leaf(a, with);
    else pairing_dfs<L + 1>(p, used | 1 << n | 1 << q, a, with, bound, leaf);
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

// What bounds the exact variant is latency in divergent code: 12 of 32 lanes
// active, and as many warps as shared memory holds.  So a thread keeps there
// only the r^2 and the candidate's number of its held vectors, and later the
// 66 terms in the place of the r^2 (288 bytes a thread; with the vectors it was
// 648, and nine warps an SM), and the exact sums wait until its search is over,
// when the warp forms them together.  256,000 atoms: 1,947 us -> 1,230 us
// (1,383 with 80 registers and 24 warps an SM).
template <bool APPROX>
__global__ void __launch_bounds__(CT) centro_kernel(Geom g, Slots s, const double *dcenter,
                                                    const int *atom_slot, int ntot, float slack,
                                                    const float4 *ext, double *out) {
  // A thread's column t: 33 of 8 bytes (the twelve r^2 as integer images, later
  // the terms in pairs) and the held candidates' numbers.  Warps run the scan
  // and the pairing phases at different times with no barrier between them:
  // the columns of two threads share no byte.
  __shared__ uint2 col[APPROX ? 12 : (NPAIR + 1) / 2][CT];
  __shared__ unsigned short held[12][CT];  // cell * 64 + atom
  __shared__ double vs[APPROX ? 36 : 1][APPROX ? CT : 1];
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
  auto held_rsq = [&](int k) {
    const uint2 r = col[k][t];
    return (long long)((unsigned long long)r.y << 32 | r.x);
  };
  auto offer = [&](const V3 &d, int number) {
    const double rsq =
        __dadd_rn(__dadd_rn(__dmul_rn(d.x, d.x), __dmul_rn(d.y, d.y)), __dmul_rn(d.z, d.z));
    const long long kk = key(rsq);
    int i1;
    if (nb < 12) {
      i1 = nb++;
    } else {
      if (kk > rmax) return;
      i1 = kmax;
    }
    col[i1][t] = make_uint2((unsigned)kk, (unsigned)(kk >> 32));
    held[i1][t] = (unsigned short)number;
    if (nb == 12) {  // first entry of largest r^2
      kmax = 0;
      rmax = held_rsq(0);
#pragma unroll
      for (int k = 1; k < 12; k++) {
        const long long r = held_rsq(k);
        if (r > rmax) {
          kmax = k;
          rmax = r;
        }
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
  // box and corner of cell (x-outer, z-inner; 13 is the own box), wrapped once
  // per axis with the periodic offset rounded to float
  auto corner = [&](int cell, V3 &e) {
    float ox = 0.0f, oy = 0.0f, oz = 0.0f;
    int qx = bx + cell / 9 - 1, qy = by + cell / 3 % 3 - 1, qz = bz + cell % 3 - 1;
    if (qx < 0) { qx = nx - 1; ox = __double2float_rn(-R.bounds[0]); }
    if (qx >= nx) { qx = 0; ox = __double2float_rn(R.bounds[0]); }
    if (qy < 0) { qy = ny - 1; oy = __double2float_rn(-R.bounds[1]); }
    if (qy >= ny) { qy = 0; oy = __double2float_rn(R.bounds[1]); }
    if (qz < 0) { qz = nz - 1; oz = __double2float_rn(-R.bounds[2]); }
    if (qz >= nz) { qz = 0; oz = __double2float_rn(R.bounds[2]); }
    const int b2 = R.box0 + qz * nx * ny + qy * nx + qx;
    e = V3{__dadd_rn((double)ox, dcenter[3 * b2 + 0]), __dadd_rn((double)oy, dcenter[3 * b2 + 1]),
           __dadd_rn((double)oz, dcenter[3 * b2 + 2])};
    return b2;
  };
  // the vector to atom j of box b2
  auto vector = [&](int b2, int j, bool same, const V3 &e) {
    const d4 rj = s.r[b2 * CG_MAXATOMS + j];
    if (same) return V3{__dsub_rn(rj.x, ri.x), __dsub_rn(rj.y, ri.y), __dsub_rn(rj.z, ri.z)};
    return V3{__dsub_rn(__dadd_rn(e.x, rj.x), cxi), __dsub_rn(__dadd_rn(e.y, rj.y), cyi),
              __dsub_rn(__dadd_rn(e.z, rj.z), czi)};
  };
  auto held_vector = [&](int k) {
    const int number = held[k][t], cell = number >> 6;
    V3 e;
    const int b2 = cell == 13 ? b : corner(cell, e);
    return vector(b2, number & 63, cell == 13, e);
  };
  const float4 pi = __ldg(s.pos32 + io);
  const float own = slack + 1e-6f * (fabsf(pi.x) + fabsf(pi.y) + fabsf(pi.z));
  float cut = 3.0e38f;  // est must be below it
  // the candidates of a cell: box b2, corner e (own box: relative)
  auto scan = [&](int cell, int b2, int nj, const V3 &e, float fx, float fy, float fz) {
    const bool same = cell == 13;
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
      offer(vector(b2, j, same, e), cell * 64 + j);
      j++;
      if (nb == 12) {
        // est < (r + e)^2, e the FP32 vector's error: slack for the box offset,
        // and roundings of the atom's own position and of the distance
        const float r2 = __double2float_ru(__longlong_as_double(rmax));
        const float r = sqrtf(r2), err = own + 1e-6f * r;
        cut = (r2 + err * (2.0f * r + err) + 1e-30f) * 1.000001f;
      }
    }
  };
  scan(13, b, ni, V3{0.0, 0.0, 0.0}, 0.f, 0.f, 0.f);
  for (int cell = 0; cell < 27; cell++) {  // x-outer, z-inner
    if (cell == 13) continue;
    V3 e;
    const int b2 = corner(cell, e);
    const float fx = (float)(e.x - dcenter[3 * b + 0]), fy = (float)(e.y - dcenter[3 * b + 1]),
                fz = (float)(e.z - dcenter[3 * b + 2]);
    // a box whose atoms all fail the test is passed over whole
    const float4 lo = __ldg(ext + 2 * b2), hi = __ldg(ext + 2 * b2 + 1);
    const float gx = outside(lo.x, hi.x, pi.x, fx), gy = outside(lo.y, hi.y, pi.y, fy),
                gz = outside(lo.z, hi.z, pi.z, fz);
    if (gx * gx + gy * gy + gz * gz >= cut) continue;
    scan(cell, b2, s.natoms[b2], e, fx, fy, fz);
  }
  double c = 1000.0;
  if (nb >= 12) {
    if constexpr (APPROX) {
      for (int k = 0; k < 12; k++) {
        const V3 d = held_vector(k);
        vs[3 * k][t] = d.x;
        vs[3 * k + 1][t] = d.y;
        vs[3 * k + 2][t] = d.z;
      }
      auto v = [&](int k) { return V3{vs[3 * k][t], vs[3 * k + 1][t], vs[3 * k + 2][t]}; };
      // greedy pairing; a vector with r^2 = 0 counts as paired
      int paired = 0;
      for (int q = 0; q < 12; q++) paired |= (held_rsq(q) > 0 ? 0 : 1) << q;
      c = 0.0;
      for (int j = 0; j < 11; j++) {
        if (paired >> j & 1) continue;
        double summin = 1000.0;
        int kmin = -1;
        for (int k = j + 1; k < 12; k++) {
          if (paired >> k & 1) continue;
          const double sum = pair_term(v(j), v(k));
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
      float x[12], y[12], z[12], most = 0.0f;
#pragma unroll
      for (int k = 0; k < 12; k++) {
        const V3 d = held_vector(k);
        x[k] = (float)d.x;
        y[k] = (float)d.y;
        z[k] = (float)d.z;
        most = fmaxf(most, fmaxf(fabsf(x[k]), fmaxf(fabsf(y[k]), fabsf(z[k]))));
      }
      float low = 0.0f;
#pragma unroll
      for (int i = 0, k = 0; i < 12; i++)
#pragma unroll
        for (int j = i + 1; j < 12; j++, k++) {
          const float sx = x[i] + x[j], sy = y[i] + y[j], sz = z[i] + z[j];
          const float term = fmaf(sz, sz, fmaf(sy, sy, sx * sx));
          if (k & 1) col[k >> 1][t] = make_uint2(__float_as_uint(low), __float_as_uint(term));
          low = term;
        }
      const unsigned *terms = &col[0][t].x;
      auto p = [&](int k) { return __uint_as_float(terms[(k >> 1) * (2 * CT) + (k & 1)]); };
      // first bound: the greedy pairing's FP32 sum (a complete pairing)
      float best = 0.0f;
      for (int used = 0, step = 0; step < 6; step++) {
        const int n = __ffs(~used) - 1;
        used |= 1 << n;
        int qb = -1;
        float pb = 0.0f;
        for (int q = n + 1; q < 12; q++)
          if (!(used >> q & 1) && (qb < 0 || p(pidx(n, q)) < pb)) {
            qb = q;
            pb = p(pidx(n, q));
          }
        used |= 1 << qb;
        best = __fadd_rn(best, pb);
      }
      const float d = most * 0x1p-22f;
      auto window = [&](float f) { return f * 1.000005f + d * (24.0f * sqrtf(f) + 600.0f * d) + 1e-37f; };
      float bound = window(best), kept = 0.0f;
      unsigned long long pending = 0;
      auto exact = [&](unsigned long long pairs) {  // testCentro
        float e = 0.0f;
        for (int l = 0; l < 6; l++) {
          const int pair = (int)(pairs >> (8 * l)) & 255;
          e = __double2float_rn(
              __dadd_rn((double)e, pair_term(held_vector(pair & 15), held_vector(pair >> 4))));
        }
        if ((double)e < c) c = (double)e;
      };
      // one pairing is kept for later, those that may be as good (the one kept
      // or the new one) are summed at once
      pairing_dfs<0>(p, 0, 0.0f, 0ull, bound, [&](float sum, unsigned long long pairs) {
        if (sum < best) {
          best = sum;
          bound = window(best);
        }
        if (pending != 0 && !(kept > bound)) exact(pairs);
        else {
          pending = pairs;
          kept = sum;
        }
      });
      if (pending != 0) exact(pending);
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
    const unsigned n = (h->ntot + CT - 1) / CT;
    if (approx)
      centro_kernel<true><<<n, CT, 0, st>>>(h->g, h->s, h->dcenter, h->atom_slot, h->ntot, slack,
                                            h->centro_ext, h->centro);
    else
      centro_kernel<false><<<n, CT, 0, st>>>(h->g, h->s, h->dcenter, h->atom_slot, h->ntot, slack,
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
