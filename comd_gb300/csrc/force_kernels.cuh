// force_kernels.cuh -- list builds (both precisions) and the mixed-precision
// link-cell force kernels; the FP64 passes are in force64.cuh.
//
// Work decomposition (full pairs: every atom sums over all its neighbours,
// so per-atom sums need no atomics and are deterministic):
//   nbr_build   one CTA per box.  The box's stencil entries (27 neighbour
//               boxes with the reference's multiplicity) are staged from HBM
//               into shared memory; each warp tests atoms of the box against
//               32 candidates per iteration, compacting hits with a ballot
//               into the atom's neighbour list (uint16 codes: entry index
//               << 6 | slot).  The passes test r2 <= rc2 (eam.c:521,
//               ljForce.c:193) again.
//   eam_pass1   one thread per atom over its list: pair phi, phi', rho
//               (eam.c:484-549), then F(rho) and F'(rho) fused in
//               (eam.c:576-594).
//   eam_pass2   one thread per atom: (F'_i + F'_j) rho'(r) dr/r and the
//               x-x stress (eam.c:595-653), r2 < rc2.
//   lj_pass     one thread per atom: the 12-6 terms of ljForce.c:151-215.
// Atoms whose neighbour count exceeds the list capacity fall back to a
// direct scan of their stencil, so results never depend on the capacity.
#pragma once

#include "common.cuh"
#include "poly64.cuh"

namespace cg {

enum { EVAL_TABLE = 0, EVAL_CHEBY = 1 };
constexpr int PASS_THREADS = 256;  // CTA size of the EAM passes

struct ForceArgs {
  Geom g;
  Slots s;
  EntryTab et;
  const int *atom_slot;  // [ntot] slot of the a-th atom (box order)
  const int *box_start;  // [nboxes+1] first atom index of each box
  int ntot;
  uint16_t *nbr;         // [ntot*cap]
  int *nbr_n;            // [ntot] list length (> cap: overflowed)
  int *npair;            // [ntot] neighbours within the cutoff (written by the passes)
  int cap;
  // FP64: positions in fixed point and F'(rho) by slot (the bits of three
  // 64-bit integers; w), their unit, and in that of their squares the width of the
  // range from FX_NEAR in which a pair is surely within the cutoff, and the
  // least r^2 that is surely beyond it
  d4 *fx;
  FxUnit fxu;
  u64 fx_span, fx_far;
  double *atom_stress;   // [ntot] per-atom share of the scalar stress
  int *status;
  Persist pl;            // persistent lists keyed by id (FP64)
  ForceOrder fo;         // persistent lists in force order (mixed; fo.list != nullptr)
  // force order, a step sequence: the velocity-Verlet coefficients of the
  // update the force pass makes when ST_FUSE is set (p -= vv_dt f, r += vv_c p)
  double vv_dt, vv_c;
  cudaGraphConditionalHandle cond;  // the rebuild section that follows that update (0: none)
  // force order, a force call whose results go straight to an attached host
  // simflat_t (device pointers of its registered f, rho, fi; slot-indexed),
  // or null
  double *host_f, *host_rho, *host_fi;
};

// Stencil entry of box jb seen from box b when both stencils are the full
// 27 boxes in getNeighborBoxes order (periodic, nbx >= 3): (dx+1)*9 +
// (dy+1)*3 + (dz+1) with the minimum-image box difference; -1 when the boxes
// are not neighbours (then the atoms are farther apart than a box, i.e.
// beyond the cutoff).
__device__ __forceinline__ int stencil_entry(const Geom &g, int b, int jb) {
  const int ci = __ldg(g.boxc + b), cj = __ldg(g.boxc + jb);
  const RepGeo &R = rep_of(g, b);
  int e = 0;
#pragma unroll
  for (int ax = 0; ax < 3; ax++) {
    int d = ((cj >> (10 * ax)) & 1023) - ((ci >> (10 * ax)) & 1023);
    if (d > 1) d -= R.nbx[ax];
    else if (d < -1) d += R.nbx[ax];
    if (d > 1 || d < -1) return -1;
    e = e * 3 + d + 1;
  }
  return e;
}

// Box offset of a stencil entry: FP64 value, or FP32 hi + lo parts.
template <class T>
struct BoxOff;
template <>
struct BoxOff<double> {
  double x, y, z;
};
template <>
struct BoxOff<float> {
  float x, y, z, lx, ly, lz;
};

template <class T>
struct PrecT;

template <>
struct PrecT<double> {
  typedef DSum Acc;
  static __device__ __forceinline__ void pos(const Slots &s, int slot, double &x, double &y,
                                             double &z) {
    d4 v = s.r[slot];
    x = v.x; y = v.y; z = v.z;
  }
  static __device__ __forceinline__ BoxOff<double> drbox(const EntryTab &et, int idx) {
    d4 v = et.dr64[idx];
    return BoxOff<double>{v.x, v.y, v.z};
  }
  static __device__ __forceinline__ double fi(const Slots &s, int slot) { return s.fi[slot]; }
};

template <>
struct PrecT<float> {
  // every per-atom sum Kahan-compensated: forces, energy, density, stress
  typedef KSum Acc;
  static __device__ __forceinline__ void pos(const Slots &s, int slot, float &x, float &y,
                                             float &z) {
    float4 v = __ldg(s.pos32 + slot);
    x = v.x; y = v.y; z = v.z;
  }
  static __device__ __forceinline__ BoxOff<float> drbox(const EntryTab &et, int idx) {
    float4 h = __ldg(et.dr32 + 2 * idx), l = __ldg(et.dr32 + 2 * idx + 1);
    return BoxOff<float>{h.x, h.y, h.z, l.x, l.y, l.z};
  }
  static __device__ __forceinline__ float fi(const Slots &s, int slot) {
    return __ldg(s.fi32 + slot);
  }
};

// FP64: dr = drbox + r_i - r_j as the reference forms it, r2 with fused sums
// (two FP64 operations and two roundings fewer per pair)
__device__ __forceinline__ double pair_r2(const BoxOff<double> &o, double xi, double yi,
                                          double zi, double xj, double yj, double zj, double &dx,
                                          double &dy, double &dz) {
  dx = (o.x + xi) - xj;
  dy = (o.y + yi) - yj;
  dz = (o.z + zi) - zj;
  return fma(dz, dz, fma(dy, dy, dx * dx));
}

// FP32: coordinates are relative to the box centre (|x| <= boxsize/2) and
// the box offset is added as hi + lo, so dr carries only its own rounding
__device__ __forceinline__ float pair_r2(const BoxOff<float> &o, float xi, float yi, float zi,
                                         float xj, float yj, float zj, float &dx, float &dy,
                                         float &dz) {
  dx = ((xi - xj) + o.x) + o.lx;
  dy = ((yi - yj) + o.y) + o.ly;
  dz = ((zi - zj) + o.z) + o.lz;
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// Visit every stencil candidate of atom (b, i) directly (overflow path).
// fn(j_slot, dx, dy, dz, r2) is called for candidates with r2 <= rc2.
template <class T, class F>
__device__ void scan_stencil(const ForceArgs &A, int b, int i, T xi, T yi, T zi, T rc2, F &&fn) {
  int ne = A.et.n[b];
  for (int e = 0; e < ne; e++) {
    int jb = A.et.box[b * CG_NNBR + e];
    BoxOff<T> bo = PrecT<T>::drbox(A.et, b * CG_NNBR + e);
    int nj = A.s.natoms[jb];
    for (int k = 0; k < nj; k++) {
      if (jb == b && k == i) continue;
      int js = jb * CG_MAXATOMS + k;
      T xj, yj, zj, dx, dy, dz;
      PrecT<T>::pos(A.s, js, xj, yj, zj);
      T r2 = pair_r2(bo, xi, yi, zi, xj, yj, zj, dx, dy, dz);
      if (r2 > rc2) continue;
      fn(js, dx, dy, dz, r2);
    }
  }
}

// Visit the atom's neighbour list (or its stencil when the list overflowed).
// Entries a hair past the cutoff are among them: the passes test r2 again.
// VEC: read eight codes per 16-byte load and unroll over them (light
// passes: independent gathers in flight); otherwise one copy of the pair
// code in the loop (heavy passes: instruction cache).
template <class T, bool VEC = false, class F>
__device__ __forceinline__ void for_each_neighbor(const ForceArgs &A, int a, int b, int i, T xi,
                                                  T yi, T zi, T rc2, F &&fn) {
  const int n = A.nbr_n[a];
  if (n > A.cap) {
    scan_stencil<T>(A, b, i, xi, yi, zi, rc2, fn);
    return;
  }
  const int ebase = b * CG_NNBR;
  auto visit = [&](uint32_t code) {
    const int e = code >> 6, k = code & 63;
    const int js = __ldg(A.et.box + ebase + e) * CG_MAXATOMS + k;
    T xj, yj, zj, dx, dy, dz;
    BoxOff<T> bo = PrecT<T>::drbox(A.et, ebase + e);
    PrecT<T>::pos(A.s, js, xj, yj, zj);
    T r2 = pair_r2(bo, xi, yi, zi, xj, yj, zj, dx, dy, dz);
    fn(js, dx, dy, dz, r2);
  };
  if (VEC) {
    const uint16_t *lst = A.nbr + (size_t)a * A.cap;
    for (int t0 = 0; t0 < n; t0 += 8) {
      const uint4 pk = *reinterpret_cast<const uint4 *>(lst + t0);
      const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (t0 + u < n) visit((w[u >> 1] >> ((u & 1) * 16)) & 0xffffu);
    }
  } else {
    const uint32_t *lst = reinterpret_cast<const uint32_t *>(A.nbr + (size_t)a * A.cap);
#pragma unroll 1
    for (int t = 0; t < n; t++) visit((__ldg(lst + (t >> 1)) >> ((t & 1) * 16)) & 0xffffu);
  }
}

// ---------------------------------------------------------------------------
// neighbour-list build: a CTA per box at a time, a warp per two or more of its
// atoms
// ---------------------------------------------------------------------------
#define NB_THREADS 128
#define NB_TILE 768  // candidates staged at a time (27 boxes of 64 are 1,728)

// The stencil entries of box b (warp 0): boxes, box offsets, candidate offsets
// and, in s_code, each entry's stencil index (the passes take the box offset
// from it).  SORT: by neighbour box (ties by entry), so that every list comes
// out in ascending neighbour slot -- atoms in force order are in box order,
// and lanes of a warp then walk the position array together.  The lanes take
// the entries in the order that an interior box's come out in; only where the
// boxes wrap are they ranked.
template <bool SORT>
__device__ __forceinline__ int stage_entries(const ForceArgs &A, int b, int *s_box, int *s_off,
                                             BoxOff<float> *s_dr, int *s_code) {
  const int ne = A.et.n[b];
  if (threadIdx.x < 32) {
    const int l = threadIdx.x;
    const bool in = l < ne;
    const int e = SORT && ne == CG_NNBR ? (l % 3) * 9 + ((l / 3) % 3) * 3 + l / 9 : l;
    const int jb = in ? A.et.box[b * CG_NNBR + e] : 0x7fffffff;
    int rank = l;
    if (SORT) {
      const int before = __shfl_up_sync(0xffffffffu, jb, 1);
      if (!__all_sync(0xffffffffu, l == 0 || !in || before < jb)) {
        rank = 0;
        for (int q = 0; q < ne; q++) {
          const int jq = __shfl_sync(0xffffffffu, jb, q), eq = __shfl_sync(0xffffffffu, e, q);
          rank += jq < jb || (jq == jb && eq < e);
        }
      }
    }
    if (in) {
      s_box[rank] = jb;
      s_dr[rank] = PrecT<float>::drbox(A.et, b * CG_NNBR + e);
      s_code[rank] = e;
      // (more than 64 only in a reported overflow)
      s_off[rank + 1] = min(A.s.natoms[jb], CG_MAXATOMS);
    }
    __syncwarp();
    int x = in ? s_off[l + 1] : 0;
    for (int o = 1; o < 32; o <<= 1) {  // inclusive scan
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (l >= o) x += y;
    }
    if (in) s_off[l + 1] = x;
    if (l == 0) s_off[0] = 0;
  }
  __syncthreads();
  return ne;
}

// force-order entry code of stencil entry e = (dx+1)*9 + (dy+1)*3 + (dz+1)
// (periodic, nbx >= 3): the three box differences as 2-bit fields d+1 at
// bits 0, 2 and 4
__device__ __forceinline__ int fo_code(int e) {
  return (e / 9) | (((e / 3) % 3) << 2) | ((e % 3) << 4);
}

// FP32: candidates staged as (x - drbox, y - drbox, z - drbox, key) in the
// centre box's frame, padded to whole 32-candidate chunks with far-away
// sentinels.  A warp tests NA atoms against every chunk it loads and appends
// the hits of each to its list at once: the ballot's bits below the lane give
// the place.  The cutoff of the build (rc2b)
// is widened by more than the FP32 distances err (list_cutoff in api.cu), so
// the list holds every pair that the passes accept with their exact dr.  The
// FP64 simulations use the same build on FP32 copies of their positions: an
// FP64 test of every candidate, 12 operations for each of seven candidates
// per neighbour, took 1,785 us for the lists of 256,000 atoms.
// Bound by the instructions issued.  Parking the ballots in shared memory and
// finding the h-th set bit (__fns) for full-warp stores took more of them
// than the tests: 270 us for those lists, 129 now (65% of the issue slots).
#define NB_ATOMS 2                 // atoms tested per candidate load
// Modes: LIST_STEP writes the per-step list (uint16 codes); LIST_ID (runs
// only when a rebuild is due) writes neighbour ids into the atom's id-keyed
// row and records its position; LIST_FO (also only when due) writes the
// transposed force-order list and the atom's force-order record.
enum { LIST_STEP = 0, LIST_ID = 1, LIST_FO = 2 };

template <int MODE>
__device__ __forceinline__ bool build_skipped(const ForceArgs &A) {
  return MODE != LIST_STEP && !*(volatile const int *)(A.status + ST_REBUILD);
}

// row of atom i of box b: list storage, count slot and capacity
template <int MODE>
__device__ __forceinline__ int build_row(const ForceArgs &A, int b, int i) {
  const int slot = b * CG_MAXATOMS + i;
  if (MODE == LIST_ID) {
    const int idi = A.s.id[slot];
    A.pl.rref[idi] = world64(A.g, b, A.s.r[slot]);
    return idi;
  }
  const int a = A.box_start[b] + i;
  if (MODE == LIST_FO) {
    const float4 p = A.s.pos32[slot];
    const int id = A.s.id[slot];
    A.fo.ref[a] = make_float4(p.x, p.y, p.z, __int_as_float(b));
    A.fo.id[a] = id;
    A.fo.of_id[id] = a;
    A.fo.slot[a] = slot;
    A.fo.pos[a] = p;
  }
  return a;
}

template <int MODE>
__device__ __forceinline__ int build_cap(const ForceArgs &A) {
  return MODE == LIST_ID ? A.pl.vcap : MODE == LIST_FO ? A.fo.vcap : A.cap;
}

template <int MODE>
__device__ __forceinline__ void build_count(const ForceArgs &A, int row, int total) {
  if (MODE == LIST_ID) A.pl.vcount[row] = total;
  else if (MODE == LIST_FO) A.fo.n[row] = total;
  else A.nbr_n[row] = total;
  // persistent lists: counted for the lists being built (rebuild_done makes
  // it the current lists' count)
  if (total > build_cap<MODE>(A))
    atomicAdd(A.status + (MODE == LIST_STEP ? ST_NBR_OVERFLOW : ST_OVF_BUILD), 1);
}

// a candidate's key: what its list entry holds (LIST_STEP: bit 16 set in the
// atom's own box)
template <int MODE>
__device__ __forceinline__ int build_key(const ForceArgs &A, int jb, int e, int k, bool own) {
  if (MODE == LIST_ID) return A.s.id[jb * CG_MAXATOMS + k];
  // force order: with periodic nbx >= 3 the entry index is the code
  if (MODE == LIST_FO) return (int)(((unsigned)(A.box_start[jb] + k) << 6) | fo_code(e));
  return (own ? 1 << 16 : 0) | (e << 6) | k;
}

// The lists of the atoms of box b (not empty): NT threads (the CTA), NA atoms
// tested per candidate load, the shared arrays of the kernel.
template <int MODE, int NT, int NA>
__device__ __forceinline__ void build_box32(const ForceArgs &A, float rc2b, int b, float4 *cand,
                                            int *s_cnt, int *s_box, int *s_off, int *s_code,
                                            BoxOff<float> *s_dr) {
  static_assert(NA % 2 == 0, "atoms are tested in pairs");
  const int ni = min(A.s.natoms[b], CG_MAXATOMS);
  const int ne = stage_entries<MODE != LIST_ID>(A, b, s_box, s_off, s_dr, s_code);
  const int ncand = s_off[ne];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t below = (1u << lane) - 1u;
  const int cap = build_cap<MODE>(A);
  const int a0 = MODE == LIST_ID ? 0 : A.box_start[b];
  // the lists of the box's rows: offsets below are of 32 bits
  uint16_t *step = MODE == LIST_STEP ? A.nbr + (size_t)a0 * cap : nullptr;
  uint32_t *fo = MODE == LIST_FO ? A.fo.list + (size_t)(a0 >> 5) * 32 * cap : nullptr;
  for (int base = 0; base < ncand; base += NB_TILE) {
    const int nc = min(NB_TILE, ncand - base), nchunk = (nc + 31) >> 5;
    if (base > 0) __syncthreads();  // the tile before is done with
    // 16 threads an entry
    for (int e = threadIdx.x >> 4; e < ne; e += NT / 16) {
      const int jb = s_box[e], off = s_off[e], end = min(s_off[e + 1], base + nc);
      const BoxOff<float> o = s_dr[e];
      for (int c = max(off, base) + (threadIdx.x & 15); c < end; c += 16) {
        const float4 q = __ldg(A.s.pos32 + jb * CG_MAXATOMS + (c - off));
        // negated, so the test below is one packed add per axis: pa + (-c)
        // rounds exactly as pa - c
        cand[c - base] =
            make_float4(-((q.x - o.x) - o.lx), -((q.y - o.y) - o.ly), -((q.z - o.z) - o.lz),
                        __int_as_float(build_key<MODE>(A, jb, s_code[e], c - off, jb == b)));
      }
    }
    for (int c = nc + threadIdx.x; c < (nchunk << 5); c += NT)
      cand[c] = make_float4(-1e18f, -1e18f, -1e18f, 0.f);
    __syncthreads();
    for (int i0 = NA * warp; i0 < ni; i0 += NA * (NT / 32)) {
      // (rows past the last only after an overflow)
      const int na = min(NA, MODE == LIST_ID ? ni - i0 : min(ni - i0, A.ntot - a0 - i0));
      if (na <= 0) break;
      // the atoms in pairs, one per half of the packed FP32x2 operations (two
      // pair tests per instruction; r^2 = dx*dx, + dy*dy, + dz*dz rounded as
      // fmaf(dz, dz, fmaf(dy, dy, dx * dx))); a missing atom is far away from
      // all candidates
      float2 px[NA / 2], py[NA / 2], pz[NA / 2];
      int cnt[NA], id[NA];
      bool far = false;  // an atom too far out for the margin (its stencil is scanned)
#pragma unroll
      for (int u = 0; u < NA; u++) {
        float4 p = make_float4(-1e18f, -1e18f, -1e18f, 0.f);
        cnt[u] = id[u] = 0;
        if (u < na) {
          const int slot = b * CG_MAXATOMS + i0 + u;
          p = __ldg(A.s.pos32 + slot);
          if (MODE == LIST_ID) id[u] = A.s.id[slot];
          if (base > 0) cnt[u] = s_cnt[i0 + u];
          far = far || p.w != 0.f;
        }
        (u & 1 ? px[u / 2].y : px[u / 2].x) = p.x;
        (u & 1 ? py[u / 2].y : py[u / 2].x) = p.y;
        (u & 1 ? pz[u / 2].y : pz[u / 2].x) = p.z;
      }
      // the candidate's place counted from atom i0, an atom u being none of
      // its own neighbours (it sits in every stencil entry of its own box)
      auto append = [&](int u, float r2, int key, int from) {
        const bool self = MODE == LIST_ID ? key == id[u] : from == u;
        const bool hit = r2 <= rc2b && !self;
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        const int h = cnt[u] + __popc(m & below);
        if (hit && h < cap) {
          if (MODE == LIST_ID) A.pl.vlist[(size_t)id[u] * cap + h] = key;
          else if (MODE == LIST_STEP) step[(i0 + u) * cap + h] = (uint16_t)key;
          else {
            const int row = (a0 & 31) + i0 + u;
            fo[((row >> 5) * cap + h) * 32 + (row & 31)] = (uint32_t)key;
          }
        }
        cnt[u] += __popc(m);
      };
      for (int q = 0; q < nchunk; q++) {
        const float4 cq = cand[(q << 5) + lane];
        const float2 cx = make_float2(cq.x, cq.x), cy = make_float2(cq.y, cq.y),
                     cz = make_float2(cq.z, cq.z);
        const int key = __float_as_int(cq.w);
        const int from = MODE == LIST_FO ? (int)((unsigned)key >> 6) - a0 - i0
                                         : (key & (1 << 16 | 63)) - (1 << 16) - i0;
#pragma unroll
        for (int u = 0; u < NA; u += 2) {
          const float2 dx = __fadd2_rn(px[u / 2], cx), dy = __fadd2_rn(py[u / 2], cy),
                       dz = __fadd2_rn(pz[u / 2], cz);
          float2 r2 = __fmul2_rn(dx, dx);
          r2 = __ffma2_rn(dy, dy, r2);
          r2 = __ffma2_rn(dz, dz, r2);
          append(u, r2.x, key, from);
          append(u + 1, r2.y, key, from);
        }
      }
      if (lane < na) {
        int mine = cnt[0];
#pragma unroll
        for (int u = 1; u < NA; u++) mine = lane == u ? cnt[u] : mine;
        s_cnt[i0 + lane] = mine;
        if (base + NB_TILE >= ncand) {
          const int row = build_row<MODE>(A, b, i0 + lane);
          build_count<MODE>(A, row, mine);
          if (MODE != LIST_FO && far && __ldg(A.s.pos32 + b * CG_MAXATOMS + i0 + lane).w != 0.f)
            (MODE == LIST_ID ? A.pl.vcount : A.nbr_n)[row] = cap + 1;
        }
      }
      __syncwarp();
    }
  }
}

// NT threads per CTA, NA atoms tested per candidate load.  A grid-stride
// loop over the boxes, the grid sized to the resident CTAs: a launch with no
// rebuild due (most steps, with skin lists) costs one check per resident
// CTA instead of one CTA per box.
template <int MODE, int NT = NB_THREADS, int NA = NB_ATOMS>
static __global__ void __launch_bounds__(NT) nbr_build32_kernel(ForceArgs A, float rc2b) {
  __shared__ __align__(16) float4 cand[NB_TILE];
  __shared__ int s_cnt[CG_MAXATOMS];
  __shared__ int s_box[CG_NNBR], s_off[CG_NNBR + 1], s_code[CG_NNBR];
  __shared__ BoxOff<float> s_dr[CG_NNBR];
  if (build_skipped<MODE>(A)) return;
  for (int b = blockIdx.x; b < A.g.nboxes; b += gridDim.x) {
    if (A.s.natoms[b] == 0) continue;
    build_box32<MODE, NT, NA>(A, rc2b, b, cand, s_cnt, s_box, s_off, s_code, s_dr);
    __syncthreads();  // the next box restages the shared arrays
  }
}

// The per-step list of every atom from its id-keyed skin list (LIST_ID),
// one warp per atom, 32 entries a round: the neighbour's current slot, its
// stencil entry as seen from the atom's box, an FP32 distance test (rc2b is
// widened as the build's, so no pair within the cutoff is lost) and a ballot
// to pack the codes.  The passes then walk the entries near the cutoff alone.
static __global__ void __launch_bounds__(NB_THREADS) nbr_cut_kernel(ForceArgs A, float rc2b) {
  const int a = (blockIdx.x * NB_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (a >= A.ntot) return;
  const int slot = A.atom_slot[a], b = slot >> 6, idi = A.s.id[slot];
  const int n = A.pl.vcount[idi];
  const float4 pi = __ldg(A.s.pos32 + slot);
  if (n > A.pl.vcap || pi.w != 0.f) {  // no skin list to go by: the passes scan
    if (lane == 0) A.nbr_n[a] = A.cap + 1;
    return;
  }
  const int *lst = A.pl.vlist + (size_t)idi * A.pl.vcap;
  uint16_t *out = A.nbr + (size_t)a * A.cap;
  int cnt = 0;
  for (int t0 = 0; t0 < n; t0 += 32) {
    bool hit = false;
    uint32_t code = 0;
    if (t0 + lane < n) {
      const int js = __ldg(A.pl.slot_of + __ldg(lst + t0 + lane));
      const int e = stencil_entry(A.g, b, js >> 6);
      if (e >= 0) {
        const float4 q = __ldg(A.s.pos32 + js);
        float dx, dy, dz;
        hit = pair_r2(PrecT<float>::drbox(A.et, b * CG_NNBR + e), pi.x, pi.y, pi.z, q.x, q.y, q.z,
                      dx, dy, dz) <= rc2b;
        code = (e << 6) | (js & 63);
      }
    }
    const uint32_t m = __ballot_sync(0xffffffffu, hit);
    const int pos = cnt + __popc(m & ((1u << lane) - 1u));
    if (hit && pos < A.cap) out[pos] = (uint16_t)code;
    cnt += __popc(m);
  }
  if (lane == 0) {
    A.nbr_n[a] = cnt;
    if (cnt > A.cap) atomicAdd(A.status + ST_NBR_OVERFLOW, 1);
  }
}

// ---------------------------------------------------------------------------
// EAM pass 1 (+ embedding): phi, phi', rho per pair; F, F' per atom
// ---------------------------------------------------------------------------
template <class T, int EVAL>
struct EamPot {
  Table<T> phi, rho, f;
  Cheb<T> ch;
  ChebLow32 chlo;  // FP32 only
  PairSeg seg;     // FP32 Chebyshev only
  PolyTables poly; // FP64 Chebyshev only
  TabPoly tpoly;   // FP64 tables only
  FoTab tab;       // FP32 tables only
  T rc2;
  bool same_grid;  // the tables of phi and rho have the same intervals
};

template <int EVAL>
__device__ __forceinline__ double cheb_series(const EamPot<double, EVAL> &P, int s, double x) {
  return cheb_eval64(P.ch.c[s], P.ch.a[s], P.ch.b[s], x);
}
// the reference coefficients for arguments below the re-expansion interval
// (never taken in practice; kept out of line so it costs no code in the loop)
static __device__ __noinline__ float cheb_low32(const ChebLow32 &L, int s, float x) {
  return cheb_eval32(L.c[s], L.a[s], L.ys[s], L.yo[s], x);
}

template <int EVAL>
__device__ __forceinline__ float cheb_series(const EamPot<float, EVAL> &P, int s, float x) {
  if (x >= P.chlo.lo[s]) return cheb_eval32(P.ch.c[s], P.ch.a[s], P.ch.ys[s], P.ch.yo[s], x);
  return cheb_low32(P.chlo, s, x);
}

// r and 1/r from r^2: rsqrt refined by one Newton step (about 1 ulp)
__device__ __forceinline__ void r_and_inv(float r2, float &r, float &inv) {
  float y = rsqrtf(r2);
  y = y * fmaf(-0.5f * r2, y * y, 1.5f);
  inv = y;
  r = r2 * y;
}

// phi, phi' and rho of one pair distance from the FP32 series: the three
// re-expanded series share the interval [lo, rc] and so one T_k recurrence
template <int EVAL>
__device__ __forceinline__ void cheb_pair32(const EamPot<float, EVAL> &P, float r, float &phi,
                                            float &dphi, float &rho) {
  if (P.chlo.pair_shared && r >= P.chlo.lo[0]) {
    cheb3_eval32(P.ch.c[0], P.ch.c[3], P.ch.c[1], P.ch.a[0], P.ch.ys[0], P.ch.yo[0], r, phi,
                 dphi, rho);
  } else if (!P.chlo.pair_shared) {
    phi = cheb_series(P, 0, r);
    dphi = cheb_series(P, 3, r);
    rho = cheb_series(P, 1, r);
  } else {
    phi = cheb_low32(P.chlo, 0, r);
    dphi = cheb_low32(P.chlo, 3, r);
    rho = cheb_low32(P.chlo, 1, r);
  }
}
template <class T, int EVAL>
__device__ __forceinline__ void eam_pair_terms(const EamPot<T, EVAL> &P, T r, T &phi, T &dphi,
                                               T &rho) {
  if (EVAL == EVAL_CHEBY) {
    cheb_pair32(P, r, phi, dphi, rho);
  } else {
    T drho;
    table_eval(P.phi, r, phi, dphi);
    table_eval(P.rho, r, rho, drho);
  }
}

template <class T, int EVAL>
__device__ __forceinline__ void eam_embed(const EamPot<T, EVAL> &P, T rho, T &F, T &dF) {
  if (EVAL == EVAL_CHEBY) {
    int k;
    double t;
    if (sizeof(T) == 8 && poly_at(P.poly.embed, (double)rho, k, t)) {
      F = (T)poly_col(P.poly.embed, EF_F, k, t);
      dF = (T)poly_col(P.poly.embed, EF_DF, k, t);
      return;
    }
    F = cheb_series(P, 2, rho);
    dF = cheb_series(P, 5, rho);
  } else {
    table_eval(P.f, rho, F, dF);
  }
}

template <class T, int EVAL>
__device__ __forceinline__ T eam_drho(const EamPot<T, EVAL> &P, T r) {
  if (EVAL == EVAL_CHEBY) return cheb_series(P, 4, r);
  T v, d;
  table_eval(P.rho, r, v, d);
  return d;
}

// Pair terms of one distance: phi, w = phi'(r)/r and rho.  The FP32
// Chebyshev path reads them from the segment table in shared memory (sm)
// and returns false for a distance below the table (or with no table): the
// caller then takes that pair from the series in a second, rare sweep, so
// the pair loop itself holds no call.
template <class T, int EVAL>
__device__ __forceinline__ bool eam_pair_w(const EamPot<T, EVAL> &P, const float4 *, T r2,
                                           T &phi, T &w, T &rho) {
  T r, inv_r, dphi;
  r_and_inv(r2, r, inv_r);
  eam_pair_terms<T, EVAL>(P, r, phi, dphi, rho);
  w = dphi * inv_r;
  return true;
}
static __device__ __forceinline__ bool eam_pair_w(const EamPot<float, EVAL_CHEBY> &P,
                                                  const float4 *sm, float r2, float &phi,
                                                  float &w, float &rho) {
  const float u = (r2 - P.seg.s_lo) * P.seg.inv_h;
  if (!(u >= 0.f)) return false;
  const int k = min((int)u, P.seg.n - 1);
  const float t = u - (float)k;
  const float4 cp = sm[k], cr = sm[P.seg.n + k];
  phi = seg_cubic(cp, t);
  w = P.seg.dscale * seg_dcubic(cp, t);
  rho = seg_cubic(cr, t);
  return true;
}
// the series for a pair below the table (Chebyshev only)
template <class T, int EVAL>
__device__ __forceinline__ void pair_w_series(const EamPot<T, EVAL> &, T, T &, T &, T &) {}
static __device__ __noinline__ void pair_w_series(const EamPot<float, EVAL_CHEBY> &P, float r2,
                                                  float &phi, float &w, float &rho) {
  float r, inv_r, dphi;
  r_and_inv(r2, r, inv_r);
  cheb_pair32(P, r, phi, dphi, rho);
  w = dphi * inv_r;
}
template <class T, int EVAL>
__device__ __forceinline__ bool below_seg(const EamPot<T, EVAL> &, T) {
  return false;
}
static __device__ __forceinline__ bool below_seg(const EamPot<float, EVAL_CHEBY> &P, float r2) {
  return !((r2 - P.seg.s_lo) * P.seg.inv_h >= 0.f);
}

// wr = (F'_i + F'_j) rho'(r) / r for one pair (fsum = F'_i + F'_j); the FP32
// Chebyshev path reads rho's cubic (sm holds the rho half of the table).
// false: below the table, as eam_pair_w.
template <class T, int EVAL>
__device__ __forceinline__ bool eam_embed_w(const EamPot<T, EVAL> &P, const float4 *, T r2,
                                            T fsum, T &wr) {
  T r, inv_r;
  r_and_inv(r2, r, inv_r);
  wr = fsum * eam_drho<T, EVAL>(P, r) * inv_r;
  return true;
}
static __device__ __forceinline__ bool eam_embed_w(const EamPot<float, EVAL_CHEBY> &P,
                                                   const float4 *sm, float r2, float fsum,
                                                   float &wr) {
  const float u = (r2 - P.seg.s_lo) * P.seg.inv_h;
  if (!(u >= 0.f)) return false;
  const int k = min((int)u, P.seg.n - 1);
  wr = fsum * (P.seg.dscale * seg_dcubic(sm[k], u - (float)k));
  return true;
}
template <class T, int EVAL>
__device__ __forceinline__ T embed_w_series(const EamPot<T, EVAL> &, T, T) {
  return T(0);
}
static __device__ __noinline__ float embed_w_series(const EamPot<float, EVAL_CHEBY> &P, float r2,
                                                    float fsum) {
  float r, inv_r;
  r_and_inv(r2, r, inv_r);
  return fsum * (cheb_series(P, 4, r) * inv_r);
}

template <class T, int EVAL>
__device__ __forceinline__ bool uses_seg(const EamPot<T, EVAL> &P) {
  return sizeof(T) == 4 && EVAL == EVAL_CHEBY && P.seg.n > 0;
}

// the segment table (nrec float4 from src) into shared memory, once per CTA
__device__ __forceinline__ void stage_seg(float4 *sm, const float4 *src, int nrec) {
  for (int q = threadIdx.x; q < nrec; q += blockDim.x) sm[q] = __ldg(src + q);
  __syncthreads();
}

// ---------------------------------------------------------------------------
// EAM pass 1: density, pair energy and pair force of one atom.  `visit`
// runs the atom's neighbour traversal with a pair functor.
// ---------------------------------------------------------------------------
template <class T>
struct Pass1Acc {
  typename PrecT<T>::Acc fx, fy, fz, ep, rh;
  int cnt;
  __device__ __forceinline__ void zero() {
    fx.zero(); fy.zero(); fz.zero(); ep.zero(); rh.zero();
    cnt = 0;
  }
  __device__ __forceinline__ void add(T phi, T w, T rho, T dx, T dy, T dz) {
    fx.add(w * dx);
    fy.add(w * dy);
    fz.add(w * dz);
    ep.add(phi / T(2.0));
    rh.add(rho);
  }
};

template <class T, int EVAL, class V>
__device__ __forceinline__ void eam_pass1_sum(const EamPot<T, EVAL> &P, const float4 *sm,
                                              Pass1Acc<T> &acc, V &&visit) {
  const T rc2 = P.rc2;
  bool low = false;
  visit([&](T, T dx, T dy, T dz, T r2) {
    if (r2 > rc2) return;
    acc.cnt++;
    T phi, w, rho;
    if (!eam_pair_w(P, sm, r2, phi, w, rho)) {
      low = true;
      return;
    }
    acc.add(phi, w, rho, dx, dy, dz);
  });
  if (low)  // pairs below the table: the series, in a second sweep
    visit([&](T, T dx, T dy, T dz, T r2) {
      if (r2 > rc2 || !below_seg(P, r2)) return;
      T phi, w, rho;
      pair_w_series(P, r2, phi, w, rho);
      acc.add(phi, w, rho, dx, dy, dz);
    });
}

// per-atom results of pass 1: F and F' fused in (eam.c:576-594)
template <class T, int EVAL>
__device__ __forceinline__ float eam_pass1_store(const ForceArgs &A, const EamPot<T, EVAL> &P,
                                                 Pass1Acc<T> &acc, int slot) {
  double rho_i = acc.rh.value();
  T F, dF;
  eam_embed<T, EVAL>(P, (T)rho_i, F, dF);
  d4 fo;
  fo.x = acc.fx.value();
  fo.y = acc.fy.value();
  fo.z = acc.fz.value();
  fo.w = acc.ep.value() + (double)F;
  A.s.f[slot] = fo;
  A.s.rho[slot] = rho_i;
  A.s.fi[slot] = (double)dF;
  if (sizeof(T) == 4) A.s.fi32[slot] = (float)dF;
  return (float)dF;
}

// grid-stride over the compact atoms; the grid is sized to the resident CTAs
// so each CTA stages the segment table once
template <class T, int EVAL>
__global__ void __launch_bounds__(PASS_THREADS)
    eam_pass1_kernel(ForceArgs A, const __grid_constant__ EamPot<T, EVAL> P) {
  extern __shared__ float4 seg_sm[];
  if (uses_seg(P)) stage_seg(seg_sm, P.seg.p1, 2 * P.seg.n);
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < A.ntot; a += gridDim.x * blockDim.x) {
    const int slot = A.atom_slot[a];
    const int b = slot >> 6, i = slot & 63;
    T xi, yi, zi;
    PrecT<T>::pos(A.s, slot, xi, yi, zi);
    Pass1Acc<T> acc;
    acc.zero();
    eam_pass1_sum(P, seg_sm, acc, [&](auto &&fn) {
      for_each_neighbor<T>(A, a, b, i, xi, yi, zi, P.rc2,
                                        [&](int, T dx, T dy, T dz, T r2) { fn(T(0), dx, dy, dz, r2); });
    });
    eam_pass1_store(A, P, acc, slot);
    A.npair[a] = acc.cnt;
  }
}

// ---------------------------------------------------------------------------
// EAM pass 2: embedding force and stress
// ---------------------------------------------------------------------------
template <class T>
struct Pass2Acc {
  typename PrecT<T>::Acc fx, fy, fz, sx;
  __device__ __forceinline__ void zero() { fx.zero(); fy.zero(); fz.zero(); sx.zero(); }
  __device__ __forceinline__ void add(T wr, T dx, T dy, T dz) {
    fx.add(wr * dx);
    fy.add(wr * dy);
    fz.add(wr * dz);
    sx.add(wr * dx * dx);
  }
};

// visit(fn) calls fn(F'_j, dx, dy, dz, r2) per neighbour
template <class T, int EVAL, class V>
__device__ __forceinline__ void eam_pass2_sum(const EamPot<T, EVAL> &P, const float4 *sm, T fii,
                                              Pass2Acc<T> &acc, V &&visit) {
  const T rc2 = P.rc2;
  bool low = false;
  visit([&](T fj, T dx, T dy, T dz, T r2) {
    if (r2 >= rc2) return;
    T wr;
    if (!eam_embed_w(P, sm, r2, fii + fj, wr)) {
      low = true;
      return;
    }
    acc.add(wr, dx, dy, dz);
  });
  if (low)
    visit([&](T fj, T dx, T dy, T dz, T r2) {
      if (r2 >= rc2 || !below_seg(P, r2)) return;
      acc.add(embed_w_series(P, r2, fii + fj), dx, dy, dz);
    });
}

template <class T>
__device__ __forceinline__ void eam_pass2_store(const ForceArgs &A, Pass2Acc<T> &acc, int slot,
                                                int a) {
  d4 fo = A.s.f[slot];
  fo.x += acc.fx.value();
  fo.y += acc.fy.value();
  fo.z += acc.fz.value();
  A.s.f[slot] = fo;
  A.atom_stress[a] = acc.sx.value();
}

template <class T, int EVAL>
__global__ void __launch_bounds__(PASS_THREADS)
    eam_pass2_kernel(ForceArgs A, const __grid_constant__ EamPot<T, EVAL> P) {
  extern __shared__ float4 seg_sm[];
  if (uses_seg(P)) stage_seg(seg_sm, P.seg.p1 + P.seg.n, P.seg.n);
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < A.ntot; a += gridDim.x * blockDim.x) {
    const int slot = A.atom_slot[a];
    const int b = slot >> 6, i = slot & 63;
    T xi, yi, zi;
    PrecT<T>::pos(A.s, slot, xi, yi, zi);
    Pass2Acc<T> acc;
    acc.zero();
    eam_pass2_sum(P, seg_sm, PrecT<T>::fi(A.s, slot), acc, [&](auto &&fn) {
      for_each_neighbor<T, true>(A, a, b, i, xi, yi, zi, P.rc2,
                                 [&](int js, T dx, T dy, T dz, T r2) {
                                   fn(PrecT<T>::fi(A.s, js), dx, dy, dz, r2);
                                 });
    });
    eam_pass2_store(A, acc, slot, a);
  }
}

// ---------------------------------------------------------------------------
// Force-order passes (mixed precision, persistent lists)
// ---------------------------------------------------------------------------
constexpr int FO1_THREADS = 512;  // pass 1 (density): 2 CTAs of 64 registers per SM

// list lines fetched ahead, unroll of the list walk and pass 2's register
// cap (chosen by measurement; -D overrides for sweeps).  Pass 2 (the force
// pass, five compensated sums) runs with CTAs of 128 to 512 threads; its
// register count follows the cap, not the CTA size.
#ifndef COMDGB_FO_PREFETCH
#define COMDGB_FO_PREFETCH 4
#endif
#ifndef COMDGB_FO1_UNROLL
#define COMDGB_FO1_UNROLL 4  // pass 1 (and LJ)
#endif
#ifndef COMDGB_FO2_UNROLL
#define COMDGB_FO2_UNROLL 2  // pass 2
#endif
#ifndef COMDGB_FO2F_MAXNREG  // the force pass without energies (OBS = false)
#define COMDGB_FO2F_MAXNREG 64
#endif
#ifndef COMDGB_FO2_MAXNREG
#define COMDGB_FO2_MAXNREG 64
#endif
// 1: the density pass writes the entries within the cutoff (the cut list)
// and the force pass walks them; 0: the force pass walks the skin list
#ifndef COMDGB_FO_CUT
#define COMDGB_FO_CUT 1
#endif
constexpr int FO_PREFETCH = COMDGB_FO_PREFETCH;
constexpr int FO1_UNROLL = COMDGB_FO1_UNROLL, FO2_UNROLL = COMDGB_FO2_UNROLL;
constexpr int FO1_BATCH = 4, FO2_BATCH = 4;  // entries loaded before the first is used

__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// The box sizes of the pair offsets of force-order atom `slot`'s replica:
// FP32 hi + lo, the y and z ones pre-scaled by 1/4 and 1/16 (their code
// fields are read in place, x 4 and x 16, exactly).  MULTI: a batch of
// replicas (the box size comes from the atom's replica); else replica 0's
// sizes are kernel-parameter constants (no registers held).
struct FoFrame {
  float hx, hy, hz, lx, ly, lz;
};
template <bool MULTI>
__device__ __forceinline__ FoFrame fo_frame(const ForceArgs &A, int slot) {
  FoFrame f{A.g.hi0[0], A.g.hi0[1], A.g.hi0[2], A.g.lo0[0], A.g.lo0[1], A.g.lo0[2]};
  if (MULTI) {
    const RepGeo &R = rep_of(A.g, slot >> 6);
    f = FoFrame{R.hi[0], R.hi[1], R.hi[2], R.lo[0], R.lo[1], R.lo[2]};
  }
  f.hy *= 0.25f, f.ly *= 0.25f, f.hz *= 0.0625f, f.lz *= 0.0625f;
  return f;
}

// dr of list entry p = j << 6 | (dz+1) << 4 | (dy+1) << 2 | (dx+1) between
// the atom at pi and its neighbour at q: (pi - q) - d * boxsize.  A field
// f * 2^s in place, OR-ed into the bits of 2^23, is the float 2^23 + f *
// 2^s: subtracted from 2^23 + 2^s it gives -d * 2^s exactly.
__device__ __forceinline__ float fo_dr(const FoFrame &f, uint32_t p, float4 pi, float4 q,
                                       float &dx, float &dy, float &dz) {
  const float ex = 8388609.0f - __int_as_float(0x4B000000 | (int)(p & 0x3u));
  const float ey = 8388612.0f - __int_as_float(0x4B000000 | (int)(p & 0xCu));
  const float ez = 8388624.0f - __int_as_float(0x4B000000 | (int)(p & 0x30u));
  dx = fmaf(ex, f.lx, fmaf(ex, f.hx, pi.x - q.x));
  dy = fmaf(ey, f.ly, fmaf(ey, f.hy, pi.y - q.y));
  dz = fmaf(ez, f.lz, fmaf(ez, f.hz, pi.z - q.z));
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// the transposed row of force-order atom a in a list of capacity vcap
__device__ __forceinline__ size_t fo_row(int a, int vcap) {
  return (size_t)(a >> 5) * vcap * 32 + (a & 31);
}

// Visit n entries of the list `lst` (a force-order list: skin or cut) of
// force-order atom a at FP32 position pi: fn(fj, dx, dy, dz, r2) for every
// entry, the neighbours' positions being pj's: with NEED_FI fo.pf and fj is
// F'(rho_j) (its w), else fj is unspecified.  n > vcap (the skin list
// overflowed): the stencil of the atom's current slot is scanned instead.
template <bool NEED_FI, bool MULTI, int UNROLL, class F>
__device__ __forceinline__ void fo_walk(const ForceArgs &A, const uint32_t *list, int n, int a,
                                        int slot, float4 pi, const float4 *pj, float rc2,
                                        F &&fn) {
  if (n > A.fo.vcap) {
    const float4 p = __ldg(A.s.pos32 + slot);
    scan_stencil<float>(A, slot >> 6, slot & 63, p.x, p.y, p.z, rc2,
                        [&](int js, float dx, float dy, float dz, float r2) {
                          fn(NEED_FI ? __ldg(A.s.fi32 + js) : 0.f, dx, dy, dz, r2);
                        });
    return;
  }
  const FoFrame fr = fo_frame<MULTI>(A, slot);
  const uint32_t *lst = list + fo_row(a, A.fo.vcap);
  if constexpr (NEED_FI && UNROLL > 1) {
    // the force pass: a batch's entries and gathers before its first pair (at
    // 4M atoms, 4 a batch: 575 us against 604 unrolled by two with the
    // Chebyshev tables, 650 against 895 with the table potential; 2 a batch
    // 660 and 742, 6 a batch 627 and 672)
    for (int t0 = 0; t0 < n; t0 += FO2_BATCH) {
      uint32_t p[FO2_BATCH];
      float4 q[FO2_BATCH];
#pragma unroll
      for (int u = 0; u < FO2_BATCH; u++) {
        if (t0 + u + FO_PREFETCH < n) prefetch_l1(lst + (size_t)(t0 + u + FO_PREFETCH) * 32);
        p[u] = __ldg(lst + (size_t)min(t0 + u, n - 1) * 32);
      }
#pragma unroll
      for (int u = 0; u < FO2_BATCH; u++) q[u] = __ldg(pj + (p[u] >> 6));
#pragma unroll
      for (int u = 0; u < FO2_BATCH; u++) {
        float dx, dy, dz;
        const float r2 = fo_dr(fr, p[u], pi, q[u], dx, dy, dz);
        if (t0 + u < n) fn(q[u].w, dx, dy, dz, r2);
      }
    }
  } else {
    // the warp's list lines stream from HBM: pull line t + FO_PREFETCH into L1
    // while line t is used (within this atom's list only)
#pragma unroll UNROLL
    for (int t = 0; t < n; t++) {
      if (t + FO_PREFETCH < n) prefetch_l1(lst + (size_t)(t + FO_PREFETCH) * 32);
      const uint32_t p = __ldg(lst + (size_t)t * 32);
      const float4 q = __ldg(pj + (p >> 6));
      float dx, dy, dz;
      const float r2 = fo_dr(fr, p, pi, q, dx, dy, dz);
      fn(q.w, dx, dy, dz, r2);
    }
  }
}

// the skin list of force-order atom a
template <bool NEED_FI, bool MULTI, int UNROLL = FO2_UNROLL, class F>
__device__ __forceinline__ void fo_for_each(const ForceArgs &A, int a, int slot, float4 pi,
                                            const float4 *pj, float rc2, F &&fn) {
  fo_walk<NEED_FI, MULTI, UNROLL>(A, A.fo.list, A.fo.n[a], a, slot, pi, pj, rc2, fn);
}

// ---------------------------------------------------------------------------
// Force-order EAM (mixed precision, persistent lists): the density pass with
// the embedding fused in, then the force pass.  The reference's pass 1
// (eam.c:484-549) computes phi, phi' and rho per pair and pass 3
// (eam.c:595-653) rho'; here the density pass needs rho alone, and the
// force pass takes phi (the pair energy), phi' and rho' together, so every
// per-atom force component is one compensated sum.  The pass criteria stay
// the reference's: phi, phi' and rho for r^2 <= rc^2, the embedding force
// and stress for r^2 < rc^2.
// ---------------------------------------------------------------------------

// The passes' pair functions in shared memory, COPIES interleaved copies of
// every record (record q of copy c at q * COPIES + c; lane l reads copy l mod
// COPIES through `sm`, its own first record): the Chebyshev potential's
// cubics (PairSeg), or the table potential's interval coefficients (FoTab:
// one 16-byte record a pair, 48 KB for the 3,000 intervals of the Cu tables;
// COPIES = 0 reads them from global memory, for CTAs too small to be worth
// the staging).  At 282,000 atoms the table potential's passes took 88 + 97
// us reading two 32-byte records a pair from global memory, 66 + 63 us so (with
// the batched gathers).

// density pass: rho
template <int COPIES>
__device__ __forceinline__ void stage_rho(float4 *sm, const EamPot<float, EVAL_CHEBY> &P) {
  if (P.seg.n <= 0) return;
  for (int q = threadIdx.x; q < P.seg.n1 * COPIES; q += blockDim.x)
    sm[q] = __ldg(P.seg.rho1 + q / COPIES);
  __syncthreads();
}
template <int COPIES>
__device__ __forceinline__ void stage_rho(float4 *sm, const EamPot<float, EVAL_TABLE> &P) {
  if (COPIES == 0 || P.tab.n <= 0) return;
  for (int q = threadIdx.x; q < P.tab.n; q += blockDim.x) sm[q] = __ldg(P.tab.rho + q);
  __syncthreads();
}
// force pass: phi'/r and rho'/r (Chebyshev: 2 n2 records, then with OBS the n
// phi cubics, one copy), or phi' and rho' (table)
template <int COPIES, bool OBS>
__device__ __forceinline__ void stage_force(float4 *sm, const EamPot<float, EVAL_CHEBY> &P) {
  const PairSeg &S = P.seg;
  if (S.n <= 0) return;
  const int m = 2 * S.n2 * COPIES;
  for (int q = threadIdx.x; q < m; q += blockDim.x) sm[q] = __ldg(S.dcub + q / COPIES);
  if (OBS)
    for (int q = threadIdx.x; q < S.n; q += blockDim.x) sm[m + q] = __ldg(S.p1 + q);
  __syncthreads();
}
template <int COPIES, bool OBS>
__device__ __forceinline__ void stage_force(float4 *sm, const EamPot<float, EVAL_TABLE> &P) {
  if (COPIES == 0 || P.tab.n <= 0) return;
  for (int q = threadIdx.x; q < P.tab.n; q += blockDim.x) sm[q] = __ldg(P.tab.der + q);
  __syncthreads();
}
// this lane's copy
template <int EVAL, int COPIES>
__device__ __forceinline__ const float4 *fo_copy(const float4 *sm) {
  return EVAL == EVAL_CHEBY && COPIES > 1 ? sm + (threadIdx.x & (COPIES - 1)) : sm;
}

// interval and offset of r in the table, as table_eval
__device__ __forceinline__ int fo_interval(const FoTab &t, float r, float &u) {
  if (r < t.x0) r = t.x0;
  else if (r > t.xn) r = t.xn;
  const float v = (r - t.x0) * t.invDx;
  const float fl = fmaxf(fminf(floorf(v), (float)(t.n - 1)), 0.f);
  u = v - fl;
  return (int)fl;
}

// rho(r) of one pair distance.  false: below the pair table (the series, in
// a second sweep)
template <int COPIES>
static __device__ __forceinline__ bool fo_rho(const EamPot<float, EVAL_TABLE> &P,
                                              const float4 *sm, float r2, float &rho) {
  float r, inv_r, v, d;
  r_and_inv(r2, r, inv_r);
  if (P.tab.n > 0) {
    const int i = fo_interval(P.tab, r, v);
    const float4 c = COPIES == 0 ? __ldg(P.tab.rho + i) : sm[i];
    rho = fmaf(v, fmaf(v, c.z, c.y), c.x);
  } else {
    table_eval(P.rho, r, rho, d);
  }
  return true;
}
// (n1 segments of the same range as the force pass's table, so "below the
// table" is below_seg's test)
template <int COPIES>
static __device__ __forceinline__ bool fo_rho(const EamPot<float, EVAL_CHEBY> &P,
                                              const float4 *sm, float r2, float &rho) {
  const float u = (r2 - P.seg.s_lo) * P.seg.inv_h1;
  if (!(u >= 0.f)) return false;
  const int k = min((int)u, P.seg.n1 - 1);
  rho = seg_cubic(sm[k * COPIES], u - (float)k);
  return true;
}
template <int EVAL>
__device__ __forceinline__ float fo_rho_series(const EamPot<float, EVAL> &, float) {
  return 0.f;
}
static __device__ __noinline__ float fo_rho_series(const EamPot<float, EVAL_CHEBY> &P, float r2) {
  float r, inv_r;
  r_and_inv(r2, r, inv_r);
  return cheb_series(P, 1, r);
}

// phi (OBS only), phi'(r)/r and rho'(r)/r of one pair distance.  false: below
// the pair table
template <bool OBS, int COPIES>
static __device__ __forceinline__ bool fo_pair(const EamPot<float, EVAL_TABLE> &P,
                                               const float4 *sm, const float4 *, float r2,
                                               float &phi, float &wphi, float &wrho) {
  float r, inv_r, dphi, v, drho;
  r_and_inv(r2, r, inv_r);
  if (P.tab.n > 0) {
    const int i = fo_interval(P.tab, r, v);
    const float4 d = COPIES == 0 ? __ldg(P.tab.der + i) : sm[i];
    dphi = fmaf(v, d.y, d.x);
    drho = fmaf(v, d.w, d.z);
    if (OBS) {
      const float4 c = __ldg(P.tab.phi + i);
      phi = fmaf(v, fmaf(v, c.z, c.y), c.x);
    }
  } else {
    table_eval(P.phi, r, phi, dphi);
    table_eval(P.rho, r, v, drho);
  }
  wphi = dphi * inv_r;
  wrho = drho * inv_r;
  return true;
}
// (two conflict-free 16-byte shared loads per pair, the phi cubic a third
// only when the energy is summed)
template <bool OBS, int COPIES>
static __device__ __forceinline__ bool fo_pair(const EamPot<float, EVAL_CHEBY> &P,
                                               const float4 *sm, const float4 *phi_sm, float r2,
                                               float &phi, float &wphi, float &wrho) {
  const float d = r2 - P.seg.s_lo;
  float u = d * P.seg.inv_h2;
  if (!(u >= 0.f)) return false;
  if (COMDGB_SEG2_RUNS > 1 && u >= (float)P.seg.n2a)
    u = fmaf(r2 - P.seg.s2b, P.seg.inv_h2b, (float)P.seg.n2a);
  const int k = min((int)u, P.seg.n2 - 1);
  const float t = u - (float)k;
  wphi = seg_cubic(sm[(2 * k) * COPIES], t);
  wrho = seg_cubic(sm[(2 * k + 1) * COPIES], t);
  if (OBS) {
    const float u1 = d * P.seg.inv_h;
    const int k1 = min((int)u1, P.seg.n - 1);
    phi = seg_cubic(phi_sm[k1], u1 - (float)k1);
  }
  return true;
}

// the series for a pair below the table (FP32 Chebyshev only)
template <int EVAL>
__device__ __forceinline__ void fo_pair_series(const EamPot<float, EVAL> &, float, float &,
                                               float &, float &) {}
static __device__ __noinline__ void fo_pair_series(const EamPot<float, EVAL_CHEBY> &P, float r2,
                                                   float &phi, float &wphi, float &wrho) {
  float r, inv_r, dphi, rho;
  r_and_inv(r2, r, inv_r);
  cheb_pair32(P, r, phi, dphi, rho);
  wphi = dphi * inv_r;
  wrho = cheb_series(P, 4, r) * inv_r;
}

// per-atom results of the density pass: F and F' fused in (eam.c:576-594)
template <int EVAL, bool OBS>
__device__ __forceinline__ void fo_density_store(const ForceArgs &A,
                                                 const EamPot<float, EVAL> &P, const KSum &rh,
                                                 int a, int slot, float4 pi, int cnt, int ncut) {
  const double rho_i = rh.value();
  float F, dF;
  eam_embed<float, EVAL>(P, (float)rho_i, F, dF);
  if (OBS) {  // the host-visible rho, F' and the embedding energy
    A.s.rho[slot] = rho_i;
    A.s.fi[slot] = (double)dF;
    A.fo.emb[a] = F;
    if (A.host_rho) {
      A.host_rho[slot] = rho_i;
      A.host_fi[slot] = (double)dF;
    }
  }
  A.s.fi32[slot] = dF;
  A.fo.pf[a] = make_float4(pi.x, pi.y, pi.z, dF);
  A.fo.ncut[a] = ncut;
  A.npair[a] = cnt;
}

#ifdef COMDGB_FO1_MAXNREG  // sweep variant: a register cap instead of the launch bound
#define FO1_BOUNDS __maxnreg__(COMDGB_FO1_MAXNREG)
#else
#define FO1_BOUNDS __launch_bounds__(FO1_THREADS, 2)
#endif

// Density pass: rho_i = sum of rho(r_ij) over the skin list within the
// cutoff, F(rho_i) and F'(rho_i); the entries within the cutoff are written
// to the cut list for the force pass.  OBS: a force call whose results the
// caller can read (see the force pass); otherwise only what the force pass
// needs is stored.
template <int EVAL, bool MULTI, bool OBS>
__global__ void FO1_BOUNDS
    fo_eam_pass1_kernel(ForceArgs A, const __grid_constant__ EamPot<float, EVAL> P) {
  extern __shared__ float4 seg_sm[];
  stage_rho<RHO_COPIES>(seg_sm, P);
  const float4 *rho_sm = fo_copy<EVAL, RHO_COPIES>(seg_sm);
  const float rc2 = P.rc2;
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < A.ntot; a += gridDim.x * blockDim.x) {
    const int slot = A.fo.slot[a];
    const float4 pi = A.fo.pos[a];
    const int n = A.fo.n[a];
    KSum rh;
    rh.zero();
    int cnt = 0;
    if (n > A.fo.vcap) {  // overflowed skin list: the stencil, no cut list
      fo_walk<false, MULTI, 1>(A, A.fo.list, n, a, slot, pi, A.fo.pos, rc2,
                               [&](float, float, float, float, float r2) {
                                 if (r2 > rc2) return;
                                 cnt++;
                                 float rho;
                                 if (!fo_rho<RHO_COPIES>(P, rho_sm, r2, rho)) rho = fo_rho_series(P, r2);
                                 rh.add(rho);
                               });
      fo_density_store<EVAL, OBS>(A, P, rh, a, slot, pi, cnt, A.fo.vcap + 1);
      continue;
    }
    const FoFrame fr = fo_frame<MULTI>(A, slot);
    const size_t row = fo_row(a, A.fo.vcap);
    const uint32_t *lst = A.fo.list + row;
    uint32_t *cut = A.fo.cut + row;
    bool low = false;
    if (EVAL == EVAL_TABLE) {
      // batches: the entries and the neighbours' positions of a whole batch are
      // loaded before the first is used.  (The table's evaluation keeps the
      // compiler from doing so in an unrolled loop: 1,047 us a pass at 4M
      // atoms against 720; the Chebyshev pass takes 579 us unrolled, 589 so.)
      for (int t0 = 0; t0 < n; t0 += FO1_BATCH) {
        uint32_t p[FO1_BATCH];
        float4 q[FO1_BATCH];
#pragma unroll
        for (int u = 0; u < FO1_BATCH; u++) {
          if (t0 + u + FO_PREFETCH < n) prefetch_l1(lst + (size_t)(t0 + u + FO_PREFETCH) * 32);
          p[u] = __ldg(lst + (size_t)min(t0 + u, n - 1) * 32);
        }
#pragma unroll
        for (int u = 0; u < FO1_BATCH; u++) q[u] = __ldg(A.fo.pos + (p[u] >> 6));
#pragma unroll
        for (int u = 0; u < FO1_BATCH; u++) {
          float dx, dy, dz;
          const float r2 = fo_dr(fr, p[u], pi, q[u], dx, dy, dz);
          if (r2 > rc2 || t0 + u >= n) continue;
          if (COMDGB_FO_CUT) cut[(size_t)cnt * 32] = p[u];
          cnt++;
          float rho;
          if (fo_rho<RHO_COPIES>(P, rho_sm, r2, rho)) rh.add(rho);
          else low = true;
        }
      }
    } else {
#pragma unroll FO1_UNROLL
      for (int t = 0; t < n; t++) {
        if (t + FO_PREFETCH < n) prefetch_l1(lst + (size_t)(t + FO_PREFETCH) * 32);
        const uint32_t p = __ldg(lst + (size_t)t * 32);
        const float4 q = __ldg(A.fo.pos + (p >> 6));
        float dx, dy, dz;
        const float r2 = fo_dr(fr, p, pi, q, dx, dy, dz);
        if (r2 > rc2) continue;
        if (COMDGB_FO_CUT) cut[(size_t)cnt * 32] = p;
        cnt++;
        float rho;
        if (fo_rho<RHO_COPIES>(P, rho_sm, r2, rho)) rh.add(rho);
        else low = true;
      }
    }
    if (low)  // pairs below the table: the series, in a second sweep
      fo_walk<false, MULTI, 1>(A, A.fo.list, n, a, slot, pi, A.fo.pos, rc2,
                               [&](float, float, float, float, float r2) {
                                 if (r2 <= rc2 && below_seg(P, r2)) rh.add(fo_rho_series(P, r2));
                               });
    fo_density_store<EVAL, OBS>(A, P, rh, a, slot, pi, cnt, cnt);
  }
}

// force pass: the per-atom sums
// (OBS: also the pair energy and the embedding stress)
template <bool OBS>
struct ForceSums {
  KSum fx, fy, fz, ep, sx;
  __device__ __forceinline__ void zero() {
    fx.zero(); fy.zero(); fz.zero();
    if (OBS) {
      ep.zero();
      sx.zero();
    }
  }
  // phi and w = phi'/r for r^2 <= rc^2; we = (F'_i + F'_j) rho'/r, zero
  // unless r^2 < rc^2
  __device__ __forceinline__ void add(float phi, float wphi, float we, float dx, float dy,
                                      float dz) {
    const float w = wphi + we;
    fx.add(w * dx);
    fy.add(w * dy);
    fz.add(w * dz);
    if (OBS) {
      ep.add(phi);
      sx.add(we * dx * dx);
    }
  }
};

constexpr int FO2_MAX_THREADS = 512;  // the force pass runs with 128, 256 (default) or 512

// the force of slot into the attached host array (real4 per slot)
__device__ __forceinline__ void fo_host_f(const ForceArgs &A, int slot, const d4 &f) {
  double *h = A.host_f + 4 * (size_t)slot;
  h[0] = f.x;
  h[1] = f.y;
  h[2] = f.z;
  h[3] = f.w;
}

// The end of a force-order force call inside a step sequence: with ST_FUSE
// set (fuse), atom a's velocity step with the force just summed and the two
// position half steps around the step boundary, as one multiply-add each
// (the arithmetic of the mixed-precision middle-part update), and its
// tracking record; else its FP32 force record for the velocity step that
// follows.  Safe inside the pass: the other atoms of the pass read the
// positions that a kernel before it stored in pf (EAM: the density pass, LJ:
// fo_lj_settle_kernel), never r, p, fo.pos or pos32.
__device__ __forceinline__ void fo_force_end(const ForceArgs &A, int a, int slot, bool fuse,
                                             float fx, float fy, float fz) {
  if (!fuse) {
    A.fo.force[a] = make_float4(fx, fy, fz, 0.f);
    return;
  }
  d4 p = A.s.p[slot];
  p.x = fma(-A.vv_dt, (double)fx, p.x);
  p.y = fma(-A.vv_dt, (double)fy, p.y);
  p.z = fma(-A.vv_dt, (double)fz, p.z);
  A.s.p[slot] = p;
  d4 r = A.s.r[slot];
  r.x = fma(p.x, A.vv_c, r.x);
  r.y = fma(p.y, A.vv_c, r.y);
  r.z = fma(p.z, A.vv_c, r.z);
  A.s.r[slot] = r;
  if (a == 0) cond_pending(A.cond, A.status);
  const int b = slot >> 6;
  fo_track_at(A.g, A.fo, b, a, r, centred32(rep_of(A.g, b), r.x, r.y, r.z), A.status,
              A.cond);
}

// Force pass: f_i = sum over the cut list of (phi'(r) + (F'_i + F'_j)
// rho'(r)) dr/r, the per-atom energy 1/2 sum phi + F(rho_i) and the
// embedding x-x stress (eam.c:534-545, 644-649; f is +grad U as in the
// reference).
// Every force call ends with fo_force_end: the FP32 force record in force
// order, or inside a step sequence (ST_FUSE) the next step's velocity and
// position update made right here.  OBS: also the slot arrays' f with the
// per-atom energy, and the stress -- a force call whose results the caller
// can read (a force call, the one ending nTimeSteps).  The force calls
// inside a step sequence are not OBS: the next force call overwrites their
// energies and stress before anything can read them (the reference's
// nTimeSteps ends with its own computeForce, timestep.c:137).
template <int EVAL, bool MULTI, bool OBS>
__global__ void __maxnreg__(OBS ? COMDGB_FO2_MAXNREG : COMDGB_FO2F_MAXNREG)
    fo_eam_pass2_kernel(ForceArgs A, const __grid_constant__ EamPot<float, EVAL> P) {
  extern __shared__ float4 seg_sm[];
  stage_force<FORCE_COPIES, OBS>(seg_sm, P);
  const float4 *dcub_sm = fo_copy<EVAL, FORCE_COPIES>(seg_sm);
  const float4 *phi_sm = seg_sm + 2 * SEG2_N * FORCE_COPIES;
  const float rc2 = P.rc2;
  const bool fuse = !OBS && *(volatile const int *)(A.status + ST_FUSE);
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < A.ntot; a += gridDim.x * blockDim.x) {
    const int slot = A.fo.slot[a];
    const float4 pi = A.fo.pf[a];
    const float fii = pi.w;
    const int n = COMDGB_FO_CUT ? A.fo.ncut[a] : A.fo.n[a];
    ForceSums<OBS> acc;
    acc.zero();
    bool low = EVAL == EVAL_CHEBY && P.seg.n == 0;  // no table: the series for all
    const uint32_t *list = COMDGB_FO_CUT ? A.fo.cut : A.fo.list;
    if (!low)
      fo_walk<true, MULTI, FO2_UNROLL>(A, list, n, a, slot, pi, A.fo.pf, rc2,
                                       [&](float fj, float dx, float dy, float dz, float r2) {
        if (r2 > rc2) return;
        float phi, wphi, wrho;
        if (!fo_pair<OBS, FORCE_COPIES>(P, dcub_sm, phi_sm, r2, phi, wphi, wrho)) {
          low = true;
          return;
        }
        const float we = r2 < rc2 ? (fii + fj) * wrho : 0.f;
        acc.add(phi, wphi, we, dx, dy, dz);
      });
    // pairs below the table: the series, in a second sweep, an entry at a time
    // (its calls gain nothing from a batch: 5.85 ms a step of 4 M atoms with
    // the series for every pair, 6.13 in batches and after an empty first sweep)
    if (low)
      fo_walk<true, MULTI, 1>(A, list, n, a, slot, pi, A.fo.pf, rc2,
                              [&](float fj, float dx, float dy, float dz, float r2) {
        if (r2 > rc2 || !below_seg(P, r2)) return;
        float phi, wphi, wrho;
        fo_pair_series(P, r2, phi, wphi, wrho);
        const float we = r2 < rc2 ? (fii + fj) * wrho : 0.f;
        acc.add(phi, wphi, we, dx, dy, dz);
      });
    const float fx = acc.fx.valuef(), fy = acc.fy.valuef(), fz = acc.fz.valuef();
    fo_force_end(A, a, slot, fuse, fx, fy, fz);
    if (OBS) {
      d4 fo;
      fo.x = fx;
      fo.y = fy;
      fo.z = fz;
      fo.w = 0.5 * acc.ep.value() + (double)__ldg(A.fo.emb + a);
      A.s.f[slot] = fo;
      A.atom_stress[a] = acc.sx.value();
      if (A.host_f) fo_host_f(A, slot, fo);
    }
  }
}

// ---------------------------------------------------------------------------
// LJ: ljForce.c:151-215 as full pairs; the kinetic stress term is added once
// per (atom, non-empty neighbour box) as at ljForce.c:175
// ---------------------------------------------------------------------------
template <class T>
struct LjPot {
  T s6, s6x12, eps4s6, rc2;  // sigma^6, 12*sigma^6, 4*eps*sigma^6, rc^2
};

template <class T>
__global__ void __launch_bounds__(128) lj_pass_kernel(ForceArgs A, LjPot<T> P) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= A.ntot) return;
  const int slot = A.atom_slot[a];
  const int b = slot >> 6, i = slot & 63;
  T xi, yi, zi;
  PrecT<T>::pos(A.s, slot, xi, yi, zi);
  typename PrecT<T>::Acc fx, fy, fz, ep, sx;
  fx.zero(); fy.zero(); fz.zero(); ep.zero(); sx.zero();
  const T s6 = P.s6, s12 = P.s6x12, c4 = P.eps4s6;
  const T rc2 = P.rc2;
  int cnt = 0;
  auto fn = [&](int js, T dx, T dy, T dz, T r2) {
    if (r2 > rc2) return;
    cnt++;
    T ir2 = T(1.0) / r2;
    T r6 = ir2 * ir2 * ir2;
    ep.add(T(0.5) * r6 * (s6 * r6 - T(1.0)));
    T fr = c4 * r6 * ir2 * (s12 * r6 - T(6.0));
    fx.add(dx * fr);
    fy.add(dy * fr);
    fz.add(dz * fr);
    sx.add(fr * dx * dx);
  };
  for_each_neighbor<T>(A, a, b, i, xi, yi, zi, rc2, fn);
  // kinetic term: -p_x^2/m per non-empty stencil entry
  int ne = A.et.n[b], nonempty = 0;
  for (int e = 0; e < ne; e++) nonempty += A.s.natoms[A.et.box[b * CG_NNBR + e]] > 0;
  d4 p = A.s.p[slot];
  double kin = __ddiv_rn(__dmul_rn(p.x, p.x), A.s.mass[slot]);
  d4 fo;
  fo.x = fx.value();
  fo.y = fy.value();
  fo.z = fz.value();
  fo.w = ep.value();
  A.s.f[slot] = fo;
  A.atom_stress[a] = sx.value() - (double)nonempty * kin;
  A.npair[a] = cnt;
}

// LJ in force order (mixed precision, persistent lists)
// (OBS as in the EAM force pass: energy and stress only where readable)

// The positions that the pass reads.  Inside a step sequence (not OBS) it ends
// with the update, which writes fo.pos while other atoms still gather their
// neighbours, so it reads pf, a copy that fo_lj_settle_kernel makes before it.
// (EAM's force pass reads the copy that its density pass stores.)
template <bool OBS>
__device__ __forceinline__ const float4 *fo_lj_pos(const ForceArgs &A) {
  return OBS ? A.fo.pos : A.fo.pf;
}
static __global__ void __launch_bounds__(PASS_THREADS) fo_lj_settle_kernel(ForceArgs A) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < A.ntot) A.fo.pf[a] = A.fo.pos[a];
}
template <bool MULTI, bool OBS>
__global__ void __launch_bounds__(PASS_THREADS) fo_lj_kernel(ForceArgs A, LjPot<float> P) {
  const float s6 = P.s6, s12 = P.s6x12, c4 = P.eps4s6, rc2 = P.rc2;
  const bool fuse = !OBS && *(volatile const int *)(A.status + ST_FUSE);
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < A.ntot; a += gridDim.x * blockDim.x) {
    const int slot = A.fo.slot[a];
    const int b = slot >> 6;
    KSum fx, fy, fz, ep, sx;
    fx.zero(); fy.zero(); fz.zero(); ep.zero(); sx.zero();
    int cnt = 0;
    auto fn = [&](float, float dx, float dy, float dz, float r2) {
      if (r2 > rc2) return;
      cnt++;
      float ir2 = 1.0f / r2;
      float r6 = ir2 * ir2 * ir2;
      if (OBS) ep.add(0.5f * r6 * (s6 * r6 - 1.0f));
      float fr = c4 * r6 * ir2 * (s12 * r6 - 6.0f);
      fx.add(dx * fr);
      fy.add(dy * fr);
      fz.add(dz * fr);
      if (OBS) sx.add(fr * dx * dx);
    };
    const float4 *pj = fo_lj_pos<OBS>(A);
    fo_for_each<false, MULTI, FO1_UNROLL>(A, a, slot, pj[a], pj, rc2, fn);
    fo_force_end(A, a, slot, fuse, fx.valuef(), fy.valuef(), fz.valuef());
    if (OBS) {
      d4 fo;
      fo.x = fx.value();
      fo.y = fy.value();
      fo.z = fz.value();
      fo.w = ep.value();
      A.s.f[slot] = fo;
      if (A.host_f) fo_host_f(A, slot, fo);
      int ne = A.et.n[b], nonempty = 0;
      for (int e = 0; e < ne; e++) nonempty += A.s.natoms[A.et.box[b * CG_NNBR + e]] > 0;
      d4 p = A.s.p[slot];
      double kin = __ddiv_rn(__dmul_rn(p.x, p.x), A.s.mass[slot]);
      A.atom_stress[a] = sx.value() - (double)nonempty * kin;
    }
    A.npair[a] = cnt;
  }
}

}  // namespace cg
