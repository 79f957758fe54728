// fixed64.cuh -- pair distances of the FP64 passes in 64-bit fixed point.
//
// The FP64 pipe issues two lanes per SM per clock, the integer pipes 128: a
// difference, a square or a comparison of coordinates costs a warp 16 clocks
// of the SM in FP64 and a few in integers.  So the passes form r^2 of a pair
// in integers and turn to FP64 only for the functions of it and the sums.
//
// A coordinate is a 64-bit integer in units of 2^(m-64) A, modulo 2^m, with
// 2^(m-1) larger than any distance in the per-step list: differences wrap, so
// r_i + offset - r_j is exact whatever the box size.  r^2 is the sum of the
// high halves of three squares, in units of 2^(2m-64) A^2.  For EAM Cu (m = 4)
// a unit is 9e-19 A and 1.4e-17 A^2: a position (a double of up to 7 A) is
// held exactly or to 4e-19 A, and r^2 is off by less than 15 units, 2e-16 A^2, where the
// FP64 operations they replace round to 4e-16 A and, at 6 to 25 A^2, 4e-16 to
// 2e-15 A^2.
//
// An error of 15 units is more than those operations' where r^2 is small, and
// r^2 = 0 is no distance at all.  So the integers serve r^2 from FX_NEAR units
// (2^(m-5) A, 0.5 A for EAM Cu: the error is below 1e-15 of r^2) to a hair below
// the cutoff; pairs closer, and those so near to the cutoff that rounding decides on
// which side they lie, take the FP64 operations (exact64 in force64.cuh).
#pragma once

#include <cuda_runtime.h>

namespace cg {

typedef unsigned long long u64;

// the unit: m and 2^-m
struct FxUnit {
  int m;
  double down;
};

// r^2 from which the integers serve, and how near to the squared cutoff: past
// what the rounding of three FP64 differences and squares comes to (2^-50 of
// 2^(2m-2), the largest r^2)
constexpr u64 FX_NEAR = 1ull << 54, FX_TIE = 1ull << 12;

// x in units of 2^(m-64), modulo 2^m
__device__ __forceinline__ long long fx_from(double x, const FxUnit &u) {
  const double y = __dmul_rn(x, u.down);
  return __double2ll_rn(__dmul_rn(__dsub_rn(y, rint(y)), 18446744073709551616.0));
}
__device__ __forceinline__ u64 fx_abs(long long d) { return (u64)(d < 0 ? -d : d); }

// the high half of a^2, at most 3 units short (the square of the low word left
// out)
__device__ __forceinline__ u64 fx_square(u64 a) {
  const unsigned h = (unsigned)(a >> 32), l = (unsigned)a;
  return (u64)h * h + (((u64)h * l) >> 31);
}

// a * 2^e to nearest (ties up) as a double, e + 1086 given: the leading one
// shifted out, the exponent put in front, all in integers
__device__ __forceinline__ double fx_double(u64 a, int e1086) {
  const int lz = __clzll((long long)a);
  const u64 n = a << (lz & 63);
  const unsigned top = lz < 64 ? e1086 - 1 - lz : 0;  // (0 stays 0)
  return __longlong_as_double((long long)(((u64)top << 52) + (n >> 11) + ((n >> 10) & 1)));
}
// a signed difference in A
__device__ __forceinline__ double fx_length(long long d, const FxUnit &u) {
  const double v = fx_double(fx_abs(d), u.m - 64 + 1086);
  return __hiloint2double(__double2hiint(v) | ((int)(d >> 32) & 0x80000000), __double2loint(v));
}
// r^2 in A^2
__device__ __forceinline__ double fx_area(u64 s, const FxUnit &u) {
  return fx_double(s, 2 * u.m - 64 + 1086);
}

}  // namespace cg
