// poly64.cuh -- the FP64 Chebyshev potential as piecewise polynomials.
//
// A 32-term Clenshaw sum costs 93 FP64 operations (and its argument a square
// root and a division), and the FP64 pipe issues about two lanes per SM per
// clock, so summing the series for every pair bounds the FP64 kernels.  The
// pair functions are instead degree-5 polynomials in s = r^2 (no square
// root) on segments that are the 256 equal parts of each binade of s: the
// segment index is the top bits of s and the offset x in it, from -1 to 1, the
// bits below, so an evaluation takes six FP64 operations: one for x, five
// fused multiply-adds.  The embedding function has the same form in rho.  At
// 256,000 atoms the two FP64 passes took 8,342 and 3,267 us with the series and 750
// and 577 us with the polynomials alone changed; force64.cuh has what the passes
// take now.
//
// Accuracy: the coefficients interpolate the series at six Chebyshev nodes
// of each segment, with the series summed in double-double arithmetic, and
// are rounded once.  The fit compares every polynomial with its series and
// the table ends before the first segment that is further off than half an
// FP64 ulp of the sum of the series' coefficients' magnitudes, less than a
// Clenshaw sum in FP64 loses by rounding; arguments outside the table take
// the series.  EAM Cu over 2.1 to 4.96 A, rms error against the series in
// extended precision, Clenshaw in FP64 -> polynomial: phi 4.7e-17 -> 9.5e-19,
// phi'/r 6.6e-17 -> 5.0e-18, rho 3.4e-18 -> 3.5e-19, rho'/r 2.0e-18 ->
// 2.5e-19 (Ha, A).  The Hessian's columns vary faster near the cutoff and
// have twice the segments; the embedding function's table reaches densities
// of 0.46 there, four times the lattice's.
#pragma once

#include <cuda_runtime.h>

#include "fixed64.cuh"

namespace cg {

constexpr int POLY_REC = 3;  // double2 per polynomial: degree 5

// The tables: pair functions (rho, phi, phi'/r, rho'/r), the Hessian's (the
// s-derivatives of phi'/r and rho'/r, doubled: (phi'' - phi'/r) / s and
// (rho'' - rho'/r) / s), and F, F' and F'' of rho; 2^bits segments a binade.
enum { PT_PAIR = 0, PT_HESS, PT_EMBED, PT_COUNT };
enum { PF_RHO = 0, PF_PHI, PF_GPHI, PF_GRHO, PF_COUNT };
enum { HF_PHI = 0, HF_RHO, HF_COUNT };
enum { EF_F = 0, EF_DF, EF_D2F, EF_COUNT };
template <int TABLE>
struct PolyShape;
template <>
struct PolyShape<PT_PAIR> {
  static constexpr int bits = 8, cols = PF_COUNT;
};
template <>
struct PolyShape<PT_HESS> {
  static constexpr int bits = 9, cols = HF_COUNT;
};
template <>
struct PolyShape<PT_EMBED> {
  static constexpr int bits = 8, cols = EF_COUNT;
};

// segment k of the table: arguments whose top bits are base + k; column q of
// it, coefficients in x, at c + (k * cols + q) * POLY_REC.  n = 0: no table.
template <int TABLE>
struct Poly64 {
  const double2 *c;
  int base, n;
};
struct PolyTables {
  Poly64<PT_PAIR> pair;
  Poly64<PT_HESS> hess;
  Poly64<PT_EMBED> embed;
};

// segment k and offset x in it; false outside the table (NaN included)
template <int TABLE>
__device__ __forceinline__ bool poly_at(const Poly64<TABLE> &p, double v, int &k, double &x) {
  constexpr int bits = PolyShape<TABLE>::bits, sh = 20 - bits;
  const int hi = __double2hiint(v), lo = __double2loint(v);
  // 1 + the fraction of the segment
  const double y = __hiloint2double(0x3ff00000 | ((hi << bits) & 0xfffff) |
                                        (int)((unsigned)lo >> (32 - bits)), lo << bits);
  x = __fma_rn(2.0, y, -3.0);
  k = (hi >> sh) - p.base;
  return (unsigned)k < (unsigned)p.n;
}
// the same from a fixed-point argument s * 2^e, s > 0 (fixed64.cuh)
template <int TABLE>
__device__ __forceinline__ bool poly_at(const Poly64<TABLE> &p, unsigned long long s, int e,
                                        int &k, double &x) {
  constexpr int bits = PolyShape<TABLE>::bits;
  const int lz = __clzll((long long)s);
  const unsigned long long m = (s << (lz & 63)) << 1;  // the bits below the leading one
  const unsigned long long f = m << bits;
  const double y = __hiloint2double(0x3ff00000 | (int)(f >> 44), (int)(unsigned)(f >> 12));
  x = __fma_rn(2.0, y, -3.0);
  k = ((1023 + 63 + e - lz) << bits) + (int)(m >> (64 - bits)) - p.base;
  return (unsigned)k < (unsigned)p.n;
}

__device__ __forceinline__ double poly_eval(const double2 *c, double t) {
  const double2 a = __ldg(c), b = __ldg(c + 1), d = __ldg(c + 2);
  return __fma_rn(
      __fma_rn(__fma_rn(__fma_rn(__fma_rn(d.y, t, d.x), t, b.y), t, b.x), t, a.y), t, a.x);
}

// column q at segment k
template <int TABLE>
__device__ __forceinline__ double poly_col(const Poly64<TABLE> &p, int q, int k, double t) {
  return poly_eval(p.c + (size_t)(k * PolyShape<TABLE>::cols + q) * POLY_REC, t);
}

// the series a table is made from: coefficients of phi, rho, F, their first
// and second derivatives (order 0 phi 1 rho 2 F 3 dphi 4 drho 5 dF 6 d2phi
// 7 d2rho 8 d2F) and the intervals
struct PolySeries {
  double c[9][32];
  double a[9], b[9];
};

// First segment and number of segments of a table: pair distances over (lo,
// rc], densities over whole segments of [a, b]; double2 each takes.
void poly_range(int table, double lo, double hi, int *base, int *n);
size_t poly_size(int table, int n);

// Fits n segments of a table into c on the device; *first_bad (device) is
// lowered to the first segment with a polynomial that misses its series.
void launch_poly_fit(int table, const PolySeries *series, int base, int n, double2 *c,
                     int *first_bad, cudaStream_t st);

// The table potential in the same spirit.  eamInterpolateDeriv (eam.c:401-434)
// is a quadratic in r on each of the table's intervals and its derivative
// linear, so phi, rho, phi'/r and rho'/r are smooth functions of s = r^2
// there: degree-4 polynomials in s from the interval's lower end, in place of
// a square root, a division and the index arithmetic (14 FP64 operations a
// pair of the density pass, now five).  The interval has to be the exact one,
// the derivative having a kink at each end: an FP32 estimate of r gives it to
// within one, the record's own ends (integers, fixed64.cuh) decide.
// Fitted and checked as the series' polynomials are: within what half an ulp
// of the value or of r changes.  Pairs below s_lo, inside the first interval
// after the last that misses it (the Cu tables' first, next to their guard
// value, at 1 A), take the formula.
// 256,000 atoms, density + forces: 354 + 469 -> 134 + 268 us.
struct TabPoly {
  const double4_32a *rho;    // [2 n] (S0, S1, c0, c1) (c2, c3, c4, -), S the bits of the ends
  const double4_32a *force;  // [3 n] (S0, S1, a0, a1) (a2, a3, a4, b0) (b1, b2, b3, b4):
                             // a phi'/r, b rho'/r
  const double4_32a *phi;    // [2 n] (c0, c1, c2, c3) (c4, -, -, -)
  float ku, off;             // the interval from sqrt(s >> 32): ku * that + off
  int n;                     // 0: none
  u64 s_lo;
};
constexpr int TABPOLY_MAX = 1 << 16;
constexpr size_t tabpoly_size(int n) { return 7 * (size_t)n; }  // in 32-byte records

// a table as the fit reads it: values v[-1 .. n + 1]
struct TabFit {
  const double *phi, *rho;
  double x0, invDx;
  int n;
};
// into out (the three arrays one after the other); *bad (0 at first) becomes
// one more than the last interval with a polynomial that misses its formula
void launch_tab_fit(const TabFit &t, const FxUnit &u, double4_32a *out, int *bad,
                    cudaStream_t st);

}  // namespace cg
