// force64.cuh -- the FP64 force passes over the per-step list.
//
// What bounds them is the FP64 pipe: about two lanes per SM per clock, so a
// warp's FP64 instruction holds it for 16 clocks while every other pipe (and
// the loads) wait for nothing.  So the passes count FP64 operations:
//   * density first, then forces, as in force order: rho alone in the first
//     pass (7 operations a pair with the Chebyshev polynomials), phi'/r and
//     rho'/r in the second, and phi and the stress only where the caller can
//     read them (OBS);
//   * distances are formed in fixed point (fixed64.cuh), and 1/r and r come
//     from the FP32 reciprocal square root (MUFU) and one cubic step, not from
//     FP64 division;
//   * LANES threads share an atom's list (lane l takes entries l, l + LANES,
//     ...; the sums are combined in a fixed order).  A thread per atom leaves
//     most of the 152 SMs idle on small systems, and on larger ones the last
//     wave of long threads runs nearly empty.
// F'(rho_j) reaches the second pass in the fourth component of the position
// record: one 32-byte gather a pair.
// Measured at 256,000 atoms (no energies), density + forces: table potential
// 3,156 us before (phi, phi' and rho, then rho', a thread per atom, FP64
// division and square root, the skin list walked in FP64), 541 + 682 with the
// list above in FP64 geometry, 354 + 469 in fixed point, 134 + 268 with its
// intervals as polynomials; Chebyshev 1,327, 350 + 560, 160 + 321.  The pipe's
// two lanes a clock would take 135 + 310 for the latter.  LJ: 455.  Relative rms error of
// the forces against extended precision (504 atoms, Cu at 300 K): Chebyshev
// 4.6e-14 before, 2.4e-15 now, table 2.2e-15 and 4.5e-16, LJ 1.4e-15 and
// 0.9e-15; energies and densities are closer as well.
#pragma once

#include "fixed64.cuh"
#include "force_kernels.cuh"

namespace cg {

constexpr int F64_THREADS = 128;

// Threads per atom.  One rule for all FP64 walks; us with 16, 4 and 1 threads,
// density + force pass or the LJ pass without energies, then the other walks:
//             7,488       10,976     12,600     27,436       520,200      1,016,064
//   Chebyshev 33 39 -     42 43 -    45 43 -    83 68 126    - 957 973    - 1,845 1,848
//   table     30 44 -     38 45 -    42 44 -    73 59 131    - 782 850    - 1,500 1,618
//   LJ        23 29 -     30 33 -    36 34 -    64 58 90     - 912 895    - 1,773 1,732
//   virial    28 26 -     38 32 -    41 33 -    81 60 84     - 930 865    - 1,809 1,681
//   adj_w     17 24 -     23 25 -    26 25 -    47 38 81     - 561 543    - 1,083 1,042
//   adj_hvp   39 42 -     53 55 -    59 55 -    115 107 144  - 1,717 1,706  - 3,344 3,322
// (virial: Chebyshev's.)  The lines lie where most of them cross; past the second the
// table potential would be 8% faster with four, the virial before the first
// with four.  Lists of 42 entries leave lanes of 16 short.
inline int lanes64(int ntot) { return ntot < 12000 ? 16 : ntot < (1 << 19) ? 4 : 1; }

// The atom and sub-lane of this thread; false when its whole warp has none.
// Groups past the last atom repeat it (no divergence in the shuffles) and
// store nothing (live).
template <int LANES>
__device__ __forceinline__ bool lane_atom(int ntot, int &a, int &sub, bool &live) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if ((q & ~31L) / LANES >= ntot) return false;
  const long at = q / LANES;
  live = at < ntot;
  a = live ? (int)at : ntot - 1;
  sub = (int)(q % LANES);
  return true;
}

template <int LANES>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// A pair: the differences and r^2 in fixed point, F'(rho_j), j's slot, and
// the entry of i's stencil that it is
struct Pair64 {
  long long x, y, z;
  u64 s;
  double fj;
  int j;
  uint32_t code;
};
// the pair of atom i (its record) and entry code of its box's stencil (off)
__device__ __forceinline__ Pair64 pair64(const ForceArgs &A, const d4 &fi, const d4 *off,
                                         uint32_t code) {
  const d4 o = off[code >> 6];  // the offset, and the neighbour box
  const int j = __double2loint(o.w) * CG_MAXATOMS + (code & 63);
  const d4 q = A.fx[j];
  const long long x =
      __double_as_longlong(fi.x) + __double_as_longlong(o.x) - __double_as_longlong(q.x);
  const long long y =
      __double_as_longlong(fi.y) + __double_as_longlong(o.y) - __double_as_longlong(q.y);
  const long long z =
      __double_as_longlong(fi.z) + __double_as_longlong(o.z) - __double_as_longlong(q.z);
  return Pair64{x, y, z, fx_square(fx_abs(x)) + fx_square(fx_abs(y)) + fx_square(fx_abs(z)),
                q.w, j, code};
}
// s in the range that the integers serve: within the cutoff
__device__ __forceinline__ bool fx_plain(const ForceArgs &A, u64 s) {
  return s - FX_NEAR < A.fx_span;
}

// The same pair in FP64, dr = drbox + r_i - r_j and r^2 operation by operation
// as the reference has them (eam.c:484-521): pairs outside the range of the
// integers.  A coincident pair has r^2 = 0 and so an infinite LJ energy, and
// forces that are not numbers, as with the reference's divisions.
struct Exact64 {
  double x, y, z, r2;
};
__device__ __forceinline__ Exact64 exact64(const EntryTab &et, const d4 *r, int slot,
                                           uint32_t code) {
  const int e = (slot >> 6) * CG_NNBR + (int)(code >> 6);
  const d4 o = et.dr64[e], ri = r[slot];
  const d4 rj = r[et.box[e] * CG_MAXATOMS + (int)(code & 63)];
  Exact64 q;
  q.x = __dsub_rn(__dadd_rn(o.x, ri.x), rj.x);
  q.y = __dsub_rn(__dadd_rn(o.y, ri.y), rj.y);
  q.z = __dsub_rn(__dadd_rn(o.z, ri.z), rj.z);
  q.r2 = __dadd_rn(__dadd_rn(__dmul_rn(q.x, q.x), __dmul_rn(q.y, q.y)), __dmul_rn(q.z, q.z));
  return q;
}
__device__ __forceinline__ Exact64 exact64(const ForceArgs &A, int slot, uint32_t code) {
  return exact64(A.et, A.s.r, slot, code);
}

// This lane's entries of atom a's list: fn(pair), entries past the cutoff
// included; an overflowed list's stencil is scanned by lane 0 (there FP64
// refuses the pairs first: the integers are modulo 2^m).  fi: the atom's
// record.
template <int LANES, class F>
__device__ __forceinline__ void walk64(const ForceArgs &A, int a, int sub, int slot, const d4 &fi,
                                       double rc2, F &&fn) {
  const int n = A.nbr_n[a], b = slot >> 6;
  const d4 *off = A.et.fx + b * CG_NNBR;
  if (n > A.cap) {
    if (sub != 0) return;
    const int ne = A.et.n[b];
    for (int e = 0; e < ne; e++) {
      const int jb = A.et.box[b * CG_NNBR + e], nj = A.s.natoms[jb];
      for (int k = 0; k < nj; k++) {
        if (jb == b && k == (slot & 63)) continue;
        const uint32_t code = (uint32_t)(e << 6 | k);
        const double r2 = exact64(A, slot, code).r2;
        if (r2 > rc2) continue;
        Pair64 q = pair64(A, fi, off, code);
        if (r2 != r2) q.s = 0;  // (not a number: FP64, which keeps it)
        fn(q);
      }
    }
    return;
  }
  const uint16_t *lst = A.nbr + (size_t)a * A.cap;
#pragma unroll 1
  for (int t = sub; t < n; t += LANES) fn(pair64(A, fi, off, __ldg(lst + t)));
}

// rho(r); phi, phi'/r and rho'/r.  false: outside the polynomial tables
static __device__ __forceinline__ bool rho64(const EamPot<double, EVAL_CHEBY> &P, u64 s,
                                             const FxUnit &u, double &rho) {
  int k;
  double x;
  if (!poly_at(P.poly.pair, s, 2 * u.m - 64, k, x)) return false;
  rho = poly_col(P.poly.pair, PF_RHO, k, x);
  return true;
}
template <bool OBS>
static __device__ __forceinline__ bool force64(const EamPot<double, EVAL_CHEBY> &P, u64 s,
                                               const FxUnit &u, double &phi, double &wphi,
                                               double &wrho) {
  int k;
  double x;
  if (!poly_at(P.poly.pair, s, 2 * u.m - 64, k, x)) return false;
  if (OBS) phi = poly_col(P.poly.pair, PF_PHI, k, x);
  wphi = poly_col(P.poly.pair, PF_GPHI, k, x);
  wrho = poly_col(P.poly.pair, PF_GRHO, k, x);
  return true;
}
static __device__ __forceinline__ bool outside64(const EamPot<double, EVAL_CHEBY> &P, u64 s,
                                                 const FxUnit &u) {
  int k;
  double x;
  return !poly_at(P.poly.pair, s, 2 * u.m - 64, k, x);
}
static __device__ __noinline__ double rho64_series(const EamPot<double, EVAL_CHEBY> &P, double r2) {
  double r, inv;
  r_and_inv(r2, r, inv);
  return cheb_series(P, 1, r);
}
static __device__ __noinline__ void force64_series(const EamPot<double, EVAL_CHEBY> &P, double r2,
                                                   double &phi, double &wphi, double &wrho) {
  double r, inv;
  r_and_inv(r2, r, inv);
  phi = cheb_series(P, 0, r);
  wphi = cheb_series(P, 3, r) * inv;
  wrho = cheb_series(P, 4, r) * inv;
}
// The record of s (rec doubles of 32 bytes each) and the argument t = s - S0
// of its polynomials: the interval by an FP32 estimate, good to within one,
// and the ends in the record.
template <int REC>
__device__ __forceinline__ const d4 *tab_record(const TabPoly &T, const d4 *tab, u64 s,
                                                const FxUnit &u, d4 &first, double &t) {
  const float sf = (float)(unsigned)(s >> 32);
  int i = (int)fmaf(sf * rsqrtf(sf), T.ku, T.off);  // (sf = 0: NaN, interval 0)
  i = max(0, min(i, T.n - 1));
  const d4 *rec = tab + REC * i;
  first = rec[0];
  const u64 lo = (u64)__double_as_longlong(first.x), hi = (u64)__double_as_longlong(first.y);
  const int step = s < lo ? (i > 0 ? -1 : 0) : s >= hi ? 1 : 0;
  if (step != 0) {
    rec += REC * step;
    first = rec[0];
  }
  const u64 s0 = (u64)__double_as_longlong(first.x);
  t = fx_area(s > s0 ? s - s0 : 0, u);  // (below the table: its lower end)
  return rec;
}
__device__ __forceinline__ double quartic(double c0, double c1, double c2, double c3, double c4,
                                          double t) {
  return fma(fma(fma(fma(c4, t, c3), t, c2), t, c1), t, c0);
}

static __device__ __forceinline__ bool rho64(const EamPot<double, EVAL_TABLE> &P, u64 s,
                                             const FxUnit &u, double &rho) {
  if (P.tpoly.n > 0) {
    if (s < P.tpoly.s_lo) return false;
    d4 a;
    double t;
    const d4 *rec = tab_record<2>(P.tpoly, P.tpoly.rho, s, u, a, t);
    const d4 b = rec[1];
    rho = quartic(a.z, a.w, b.x, b.y, b.z, t);
    return true;
  }
  double r, inv;
  r_and_inv(fx_area(s, u), r, inv);
  rho = table_value(P.rho, table_at(P.rho, r));
  return true;
}
template <bool OBS>
static __device__ __forceinline__ bool force64(const EamPot<double, EVAL_TABLE> &P, u64 s,
                                               const FxUnit &u, double &phi, double &wphi,
                                               double &wrho) {
  if (P.tpoly.n > 0) {
    if (s < P.tpoly.s_lo) return false;
    d4 a;
    double t;
    const d4 *rec = tab_record<3>(P.tpoly, P.tpoly.force, s, u, a, t);
    const d4 b = rec[1], c = rec[2];
    wphi = quartic(a.z, a.w, b.x, b.y, b.z, t);
    wrho = quartic(b.w, c.x, c.y, c.z, c.w, t);
    if (OBS) {
      const d4 *f = P.tpoly.phi + 2 * ((rec - P.tpoly.force) / 3);
      const d4 e = f[0];
      phi = quartic(e.x, e.y, e.z, e.w, f[1].x, t);
    }
    return true;
  }
  double r, inv;
  r_and_inv(fx_area(s, u), r, inv);
  const TableAt p = table_at(P.phi, r);
  const TableAt q = P.same_grid ? p : table_at(P.rho, r);
  if (OBS) phi = table_value(P.phi, p);
  wphi = __dmul_rn(table_deriv(P.phi, p), inv);
  wrho = __dmul_rn(table_deriv(P.rho, q), inv);
  return true;
}
static __device__ __forceinline__ bool outside64(const EamPot<double, EVAL_TABLE> &P, u64 s,
                                                 const FxUnit &) {
  return P.tpoly.n > 0 && s < P.tpoly.s_lo;
}
static __device__ __noinline__ double rho64_series(const EamPot<double, EVAL_TABLE> &P, double r2) {
  double r, inv;
  r_and_inv(r2, r, inv);
  return table_value(P.rho, table_at(P.rho, r));
}
static __device__ __noinline__ void force64_series(const EamPot<double, EVAL_TABLE> &P, double r2,
                                                   double &phi, double &wphi, double &wrho) {
  double r, inv, dphi, v, drho;
  r_and_inv(r2, r, inv);
  table_eval(P.phi, r, phi, dphi);
  table_eval(P.rho, r, v, drho);
  wphi = dphi * inv;
  wrho = drho * inv;
}

// the pairs of a second sweep: not far beyond the cutoff, and outside the
// range of the integers or of the polynomials
template <int EVAL>
__device__ __forceinline__ bool in_rest64(const ForceArgs &A, const EamPot<double, EVAL> &P,
                                          u64 s) {
  return s <= A.fx_far && (!fx_plain(A, s) || outside64(P, s, A.fxu));
}

// rho_i = sum of rho(r_ij), F'(rho_i) for the force pass; OBS: also rho, F'
// and F(rho_i) (left in f's fourth component) and the pairs counted
template <int EVAL, int LANES, bool OBS>
__global__ void __launch_bounds__(F64_THREADS)
    eam64_density_kernel(ForceArgs A, const __grid_constant__ EamPot<double, EVAL> P) {
  int a, sub;
  bool live;
  if (!lane_atom<LANES>(A.ntot, a, sub, live)) return;
  const int slot = A.atom_slot[a];
  const d4 fi = A.fx[slot];
  double rho = 0.0;
  int cnt = 0;
  bool rest = false;
  walk64<LANES>(A, a, sub, slot, fi, P.rc2, [&](const Pair64 &q) {
    double v;
    if (fx_plain(A, q.s) && rho64(P, q.s, A.fxu, v)) {
      cnt++;
      rho = __dadd_rn(rho, v);
    } else if (q.s <= A.fx_far) {
      rest = true;
    }
  });
  if (rest)  // pairs outside the polynomials or the integers: in FP64, in a second sweep
    walk64<LANES>(A, a, sub, slot, fi, P.rc2, [&](const Pair64 &q) {
      if (!in_rest64(A, P, q.s)) return;
      const double r2 = exact64(A, slot, q.code).r2;
      if (r2 > P.rc2) return;
      cnt++;
      rho = __dadd_rn(rho, rho64_series(P, r2));
    });
  rho = lane_sum<LANES>(rho);
  if (OBS)
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  double F, dF;
  eam_embed<double, EVAL>(P, rho, F, dF);
  if (sub != 0 || !live) return;
  // (atoms still walking gather this record for its position alone, which the
  // store of its last 8 bytes leaves as it is)
  A.fx[slot].w = dF;
  if (OBS) {
    A.s.rho[slot] = rho;
    A.s.fi[slot] = dF;
    A.s.f[slot].w = F;
    A.npair[a] = cnt;
  }
}

// f_i = sum of (phi'(r) + (F'_i + F'_j) rho'(r)) dr/r (eam.c:534-545,
// 595-653); OBS: the per-atom energy and the x-x embedding stress
template <int EVAL, int LANES, bool OBS>
__global__ void __launch_bounds__(F64_THREADS)
    eam64_force_kernel(ForceArgs A, const __grid_constant__ EamPot<double, EVAL> P) {
  int a, sub;
  bool live;
  if (!lane_atom<LANES>(A.ntot, a, sub, live)) return;
  const int slot = A.atom_slot[a];
  const d4 fi = A.fx[slot];
  const double fii = fi.w;
  double fx = 0.0, fy = 0.0, fz = 0.0, ep = 0.0, sx = 0.0;
  bool rest = false;
  auto add = [&](double dx, double dy, double dz, double fs, double phi, double wphi,
                 double wrho) {
    double w;
    if (OBS) {
      const double we = __dmul_rn(fs, wrho);
      w = __dadd_rn(wphi, we);
      ep = __dadd_rn(ep, phi);
      sx = fma(__dmul_rn(we, dx), dx, sx);
    } else {
      w = fma(fs, wrho, wphi);
    }
    fx = fma(w, dx, fx);
    fy = fma(w, dy, fy);
    fz = fma(w, dz, fz);
  };
  walk64<LANES>(A, a, sub, slot, fi, P.rc2, [&](const Pair64 &q) {
    double phi = 0.0, wphi, wrho;
    if (fx_plain(A, q.s) && force64<OBS>(P, q.s, A.fxu, phi, wphi, wrho))
      add(fx_length(q.x, A.fxu), fx_length(q.y, A.fxu), fx_length(q.z, A.fxu),
          __dadd_rn(fii, q.fj), phi, wphi, wrho);
    else if (q.s <= A.fx_far)
      rest = true;
  });
  if (rest)
    walk64<LANES>(A, a, sub, slot, fi, P.rc2, [&](const Pair64 &q) {
      if (!in_rest64(A, P, q.s)) return;
      const Exact64 d = exact64(A, slot, q.code);
      if (d.r2 > P.rc2) return;
      double phi, wphi, wrho;
      force64_series(P, d.r2, phi, wphi, wrho);
      add(d.x, d.y, d.z, d.r2 < P.rc2 ? __dadd_rn(fii, q.fj) : 0.0, phi, wphi, wrho);
    });
  fx = lane_sum<LANES>(fx);
  fy = lane_sum<LANES>(fy);
  fz = lane_sum<LANES>(fz);
  if (OBS) {
    ep = lane_sum<LANES>(ep);
    sx = lane_sum<LANES>(sx);
  }
  if (sub != 0 || !live) return;
  d4 f;
  f.x = fx;
  f.y = fy;
  f.z = fz;
  f.w = 0.0;
  if (OBS) {
    f.w = fma(0.5, ep, A.s.f[slot].w);
    A.atom_stress[a] = sx;
  }
  A.s.f[slot] = f;
}

// the distance of an LJ pair; false: beyond the cutoff
__device__ __forceinline__ bool lj_pair64(const ForceArgs &A, const LjPot<double> &P, int slot,
                                          const Pair64 &q, Exact64 &d) {
  if (fx_plain(A, q.s)) {
    d = Exact64{fx_length(q.x, A.fxu), fx_length(q.y, A.fxu), fx_length(q.z, A.fxu),
                fx_area(q.s, A.fxu)};
    return true;
  }
  if (q.s > A.fx_far) return false;
  d = exact64(A, slot, q.code);
  return !(d.r2 > P.rc2);
}

// LJ: ljForce.c:151-215 as full pairs; the kinetic stress term is added once
// per (atom, non-empty neighbour box) as at ljForce.c:175
template <int LANES, bool OBS>
__global__ void __launch_bounds__(F64_THREADS) lj64_kernel(ForceArgs A, LjPot<double> P) {
  int a, sub;
  bool live;
  if (!lane_atom<LANES>(A.ntot, a, sub, live)) return;
  const int slot = A.atom_slot[a], b = slot >> 6;
  const d4 fi = A.fx[slot];
  const double s6 = P.s6, s12 = P.s6x12, c4 = P.eps4s6;
  double fx = 0.0, fy = 0.0, fz = 0.0, ep = 0.0, sx = 0.0;
  int cnt = 0;
  walk64<LANES>(A, a, sub, slot, fi, P.rc2, [&](const Pair64 &q) {
    Exact64 d;
    if (!lj_pair64(A, P, slot, q, d)) return;
    const double ir2 = reciprocal(d.r2);
    const double r6 = __dmul_rn(__dmul_rn(ir2, ir2), ir2);
    const double fr = __dmul_rn(__dmul_rn(__dmul_rn(c4, r6), ir2), fma(s12, r6, -6.0));
    fx = fma(fr, d.x, fx);
    fy = fma(fr, d.y, fy);
    fz = fma(fr, d.z, fz);
    if (OBS) {
      cnt++;
      ep = fma(r6, fma(s6, r6, -1.0), ep);
      sx = fma(__dmul_rn(fr, d.x), d.x, sx);
    }
  });
  fx = lane_sum<LANES>(fx);
  fy = lane_sum<LANES>(fy);
  fz = lane_sum<LANES>(fz);
  int nonempty = 0;
  if (OBS) {
    ep = lane_sum<LANES>(ep);
    sx = lane_sum<LANES>(sx);
    const int ne = A.et.n[b];
    for (int e = sub; e < ne; e += LANES)
      nonempty += A.s.natoms[A.et.box[b * CG_NNBR + e]] > 0;
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
      cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      nonempty += __shfl_xor_sync(0xffffffffu, nonempty, o);
    }
  }
  if (sub != 0 || !live) return;
  d4 f;
  f.x = fx;
  f.y = fy;
  f.z = fz;
  f.w = 0.0;
  if (OBS) {
    f.w = 0.5 * ep;
    const d4 p = A.s.p[slot];
    const double kin = __ddiv_rn(__dmul_rn(p.x, p.x), A.s.mass[slot]);
    A.atom_stress[a] = sx - (double)nonempty * kin;
    A.npair[a] = cnt;
  }
  A.s.f[slot] = f;
}

}  // namespace cg
