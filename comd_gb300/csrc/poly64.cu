// poly64.cu -- fits the FP64 polynomial tables (poly64.cuh) on the device.
//
// Eight lanes per (segment, column): six sample the series at the segment's
// Chebyshev nodes, two at its ends, in double-double arithmetic (a pair hi +
// lo with about 106 bits; sums by Knuth's two-sum, products by one fused
// multiply-add, Dekker's scheme).  Six lanes then form one monomial
// coefficient each from the samples, by the inverse of the nodes'
// Vandermonde matrix (the same for all segments), and
// round it once; the two others check the ends, where the error of
// interpolation at these nodes peaks.  FP64 operations bound it: 0.37 ms
// for the Cu tables, once per potential (2.75 ms with one thread per
// polynomial).
// Built without FMA contraction: the error terms need the stated roundings.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "poly64.cuh"

namespace cg {
namespace {

constexpr int DEG = 2 * POLY_REC - 1, NP = DEG + 1;
constexpr int FIT_THREADS = 64, FIT_LANES = 8;

struct dd {
  double h, l;
};
__host__ __device__ __forceinline__ dd two_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
__host__ __device__ __forceinline__ dd quick(double a, double b) {
  const double s = a + b;
  return {s, b - (s - a)};
}
__host__ __device__ __forceinline__ dd add(dd a, dd b) {
  const dd s = two_sum(a.h, b.h);
  return quick(s.h, s.l + (a.l + b.l));
}
__host__ __device__ __forceinline__ dd neg(dd a) { return {-a.h, -a.l}; }
__host__ __device__ __forceinline__ dd sub(dd a, dd b) { return add(a, neg(b)); }
__host__ __device__ __forceinline__ dd mul(dd a, dd b) {
  const double p = a.h * b.h;
  const double e = fma(a.h, b.h, -p);
  return quick(p, e + (a.h * b.l + a.l * b.h));
}
__host__ __device__ __forceinline__ dd from(double a) { return {a, 0.0}; }
__host__ __device__ __forceinline__ dd div(dd a, dd b) {
  const double q = a.h / b.h;
  const dd r = sub(a, mul(b, from(q)));
  const double q2 = r.h / b.h;
  const dd r2 = sub(r, mul(b, from(q2)));
  return add(quick(q, q2), from(r2.h / b.h));
}
__device__ __forceinline__ dd root(dd a) {
  const double x = sqrt(a.h);
  const dd r = sub(a, mul(from(x), from(x)));
  return quick(x, r.h / (2.0 * x));
}

// eamCheb (cheby.c:276-310) in double-double
__device__ dd series(const PolySeries &S, int q, dd x) {
  const dd a = from(S.a[q]), b = from(S.b[q]);
  const dd y = div(sub(sub(add(x, x), a), b), sub(b, a)), y2 = add(y, y);
  dd d = from(0.0), e = from(0.0);
#pragma unroll 1
  for (int j = 31; j > 0; j--) {
    const dd t = d;
    d = add(sub(mul(y2, d), e), from(S.c[q][j]));
    e = t;
  }
  return add(sub(mul(y, d), e), from(0.5 * S.c[q][0]));
}

// the series behind column q of a table
template <int TABLE>
__device__ __forceinline__ int series_of(int q) {
  if (TABLE == PT_EMBED) return q == EF_F ? 2 : q == EF_DF ? 5 : 8;
  if (TABLE == PT_HESS) return q == HF_PHI ? 6 : 7;
  return q == PF_RHO ? 1 : q == PF_PHI ? 0 : q == PF_GPHI ? 3 : 4;
}

// column q at argument x (s = r^2 for the pair tables, rho for the embedding)
template <int TABLE>
__device__ dd column(const PolySeries &S, int q, dd x) {
  const int k = series_of<TABLE>(q);
  if (TABLE == PT_EMBED) return series(S, k, x);
  const dd r = root(x), v = series(S, k, r);
  if (TABLE == PT_HESS) return div(sub(v, div(series(S, k - 3, r), r)), x);
  return q == PF_GPHI || q == PF_GRHO ? div(v, r) : v;
}

// what half an ulp of the series' coefficients comes to in column q at x
template <int TABLE>
__device__ double column_bound(const PolySeries &S, int q, double x) {
  double sum = 0.0;
  for (int j = 0; j < 32; j++) sum += fabs(S.c[series_of<TABLE>(q)][j]);
  if (TABLE == PT_PAIR && (q == PF_GPHI || q == PF_GRHO)) sum /= sqrt(x);
  if (TABLE == PT_HESS) sum /= x;
  return 0x1p-53 * sum;
}

// row j: the coefficient of x^j of the polynomial through six values at the
// nodes, x in [-1, 1]
struct NodeMatrix {
  double node[NP];
  dd m[NP][NP];
};

template <int TABLE>
__global__ void __launch_bounds__(FIT_THREADS)
    poly_fit_kernel(const PolySeries *Sp, const __grid_constant__ NodeMatrix N, int base, int n,
                    double2 *c, int *first_bad) {
  __shared__ PolySeries S;
  for (int i = threadIdx.x; i < (int)(sizeof(PolySeries) / sizeof(double)); i += FIT_THREADS)
    reinterpret_cast<double *>(&S)[i] = reinterpret_cast<const double *>(Sp)[i];
  __syncthreads();
  constexpr int cols = PolyShape<TABLE>::cols, sh = 20 - PolyShape<TABLE>::bits;
  const int lane = threadIdx.x % FIT_LANES;
  const int id = (blockIdx.x * FIT_THREADS + threadIdx.x) / FIT_LANES;
  if (id >= n * cols) return;  // (whole groups of lanes)
  const unsigned group = 0xffu << (threadIdx.x & 24);
  const int k = id / cols, q = id - k * cols, i = base + k;
  const double lo = __hiloint2double(i << sh, 0), hi = __hiloint2double((i + 1) << sh, 0);
  const double mid = __hiloint2double((i << sh) | (1 << (sh - 1)), 0);
  const double half = 0.5 * (hi - lo);  // a power of two: the offsets scale exactly
  const double x = lane < NP ? N.node[lane] : lane == NP ? -1.0 : 1.0;
  const dd sample = column<TABLE>(S, q, two_sum(mid, half * x));
  dd p = from(0.0);
#pragma unroll
  for (int j = 0; j < NP; j++) {
    const dd v = {__shfl_sync(group, sample.h, j, FIT_LANES),
                  __shfl_sync(group, sample.l, j, FIT_LANES)};
    p = add(p, mul(v, N.m[lane < NP ? lane : 0][j]));
  }
  dd end = from(0.0);  // at the ends
#pragma unroll
  for (int j = NP - 1; j >= 0; j--) {
    const dd pj = {__shfl_sync(group, p.h, j, FIT_LANES), __shfl_sync(group, p.l, j, FIT_LANES)};
    end = add(mul(end, from(x)), pj);
  }
  if (lane < NP) {
    reinterpret_cast<double *>(c + (size_t)id * POLY_REC)[lane] = p.h + p.l;
  } else if (!(fabs(sub(end, sample).h) <= column_bound<TABLE>(S, q, mid))) {
    atomicMin(first_bad, k);
  }
}

// the unit values' polynomials: Newton's divided differences, expanded
NodeMatrix node_matrix() {
  NodeMatrix N;
  for (int j = 0; j < NP; j++) N.node[j] = std::cos(3.141592653589793 * (j + 0.5) / NP);
  for (int u = 0; u < NP; u++) {
    dd v[NP], p[NP];
    for (int j = 0; j < NP; j++) {
      v[j] = from(j == u ? 1.0 : 0.0);
      p[j] = from(0.0);
    }
    for (int m = 1; m < NP; m++)
      for (int j = NP - 1; j >= m; j--)
        v[j] = div(sub(v[j], v[j - 1]), sub(from(N.node[j]), from(N.node[j - m])));
    for (int m = NP - 1; m >= 0; m--) {
      for (int j = NP - 1; j > 0; j--) p[j] = sub(p[j - 1], mul(p[j], from(N.node[m])));
      p[0] = add(neg(mul(p[0], from(N.node[m]))), v[m]);
    }
    for (int j = 0; j < NP; j++) N.m[j][u] = p[j];
  }
  return N;
}

template <int TABLE>
void fit(const PolySeries *series, int base, int n, double2 *c, int *first_bad, cudaStream_t st) {
  constexpr int per = FIT_THREADS / FIT_LANES;  // polynomials per CTA
  const int work = n * PolyShape<TABLE>::cols;
  if (work > 0)
    poly_fit_kernel<TABLE><<<(work + per - 1) / per, FIT_THREADS, 0, st>>>(
        series, node_matrix(), base, n, c, first_bad);
}

// a double-double number times 2^e as an integer (below 2^63)
__device__ __forceinline__ u64 to_fixed(dd a, int e) {
  return (u64)((long long)ldexp(a.h, e) + __double2ll_rd(ldexp(a.l, e) + (ldexp(a.h, e) - floor(ldexp(a.h, e)))));
}

// One thread per (interval, function): five Chebyshev nodes in s, Newton's
// differences, monomials in s - S0.
__global__ void __launch_bounds__(FIT_THREADS)
    tab_fit_kernel(TabFit T, FxUnit u, double4_32a *out, int *bad) {
  constexpr int M = 5;
  const int id = blockIdx.x * FIT_THREADS + threadIdx.x;
  const int i = id >> 2, q = id & 3;  // rho, phi, phi'/r, rho'/r
  if (i >= T.n) return;
  const int up = 64 - 2 * u.m;
  const double *w = (q == 0 || q == 3) ? T.rho : T.phi;
  const dd inv = from(T.invDx);
  const dd r0 = add(from(T.x0), div(from((double)i), inv));
  const dd r1 = add(from(T.x0), div(from((double)(i + 1)), inv));
  const u64 S0 = to_fixed(mul(r0, r0), up), S1 = to_fixed(mul(r1, r1), up);
  const dd s0 = {ldexp((double)(S0 >> 32), 32 - up), ldexp((double)(unsigned)S0, -up)};
  const double width = ldexp((double)(S1 - S0), -up);
  // the coefficients the formula takes (its table_value and table_deriv)
  const double g0 = w[i + 1] - w[i - 1], g1 = w[i + 2] - w[i];
  const double c0 = w[i], c1 = 0.5 * g0, c2 = 0.5 * (w[i + 1] + w[i - 1] - 2.0 * w[i]);
  const double d0 = i <= 0 ? 0.0 : 0.5 * g0 * T.invDx, d1 = i <= 0 ? 0.0 : 0.5 * (g1 - g0) * T.invDx;
  auto eval = [&](double t) {
    const dd r = root(add(quick(s0.h, s0.l), from(t)));
    const dd v = mul(sub(r, r0), inv);
    if (q < 2) return add(from(c0), mul(v, add(from(c1), mul(v, from(c2)))));
    return div(add(from(d0), mul(v, from(d1))), r);
  };
  double t[M];
  dd v[M], p[M];
#pragma unroll
  for (int j = 0; j < M; j++) {
    t[j] = width * (0.5 + 0.5 * cospi((j + 0.5) / M));
    v[j] = eval(t[j]);
    p[j] = from(0.0);
  }
#pragma unroll
  for (int m = 1; m < M; m++)
#pragma unroll
    for (int j = M - 1; j >= m; j--)
      v[j] = div(sub(v[j], v[j - 1]), sub(from(t[j]), from(t[j - m])));
#pragma unroll
  for (int m = M - 1; m >= 0; m--) {
#pragma unroll
    for (int j = M - 1; j > 0; j--) p[j] = sub(p[j - 1], mul(p[j], from(t[m])));
    p[0] = add(neg(mul(p[0], from(t[m]))), v[m]);
  }
  double c[M];
#pragma unroll
  for (int j = 0; j < M; j++) c[j] = p[j].h + p[j].l;
  for (int e = 0; e < 2; e++) {  // both ends
    const double at = e ? width : 0.0;
    dd s = from(0.0);
#pragma unroll
    for (int j = M - 1; j >= 0; j--) s = add(mul(s, from(at)), p[j]);
    // half an ulp of the value at the lower end, and of r in the rest
    const double steps = r0.h * T.invDx;
    const double size = q < 2 ? fabs(c0) + steps * (fabs(c1) + fabs(c2))
                              : (fabs(d0) + steps * fabs(d1)) / r0.h;
    if (!(fabs(sub(s, eval(at)).h) <= 0x1p-53 * size)) atomicMax(bad, i + 1);
  }
  // the ends of the first and the last interval are open
  const double lo = __longlong_as_double((long long)S0);
  const double hi = __longlong_as_double(i == T.n - 1 ? 0x7fffffffffffffffLL : (long long)S1);
  double *rho = reinterpret_cast<double *>(out) + 8 * (size_t)i;
  double *frc = reinterpret_cast<double *>(out + 2 * (size_t)T.n) + 12 * (size_t)i;
  double *phi = reinterpret_cast<double *>(out + 5 * (size_t)T.n) + 8 * (size_t)i;
  double *to = q == 0 ? rho + 2 : q == 1 ? phi : q == 2 ? frc + 2 : frc + 7;
#pragma unroll
  for (int j = 0; j < M; j++) to[j] = c[j];
  if (q == 0 || q == 2) {
    (q == 0 ? rho : frc)[0] = lo;
    (q == 0 ? rho : frc)[1] = hi;
  }
}

int index_of(double x, int bits) {
  unsigned long long b;
  memcpy(&b, &x, sizeof b);
  return (int)(b >> 32) >> (20 - bits);
}

}  // namespace

// More than eight binades of pair distances are no potential, and densities
// below 2^-6 of the largest are rare: the series serves both.
void poly_range(int table, double lo, double hi, int *base, int *n) {
  *base = 0;
  *n = 0;
  const int bits = table == PT_HESS ? PolyShape<PT_HESS>::bits : PolyShape<PT_PAIR>::bits;
  static_assert((int)PolyShape<PT_PAIR>::bits == (int)PolyShape<PT_EMBED>::bits, "one of two widths");
  if (!(hi > 0.0) || !std::isfinite(hi)) return;
  if (table == PT_EMBED) {
    const double from = std::fmax(lo, hi * 0x1p-6);  // whole segments: below lo F is clamped
    if (!(from < hi)) return;
    *base = index_of(from, bits) + 1;
    *n = std::max(0, index_of(hi, bits) - *base);
    return;
  }
  if (!(lo > 0.0 && lo < hi)) return;
  *base = index_of(lo * lo, bits) + 1;
  const int count = index_of(hi * hi, bits) - *base + 1;
  *n = count > 0 && count <= 8 << bits ? count : 0;
}

size_t poly_size(int table, int n) {
  const int cols = table == PT_PAIR ? (int)PF_COUNT : table == PT_HESS ? (int)HF_COUNT : (int)EF_COUNT;
  return (size_t)n * cols * POLY_REC;
}

void launch_poly_fit(int table, const PolySeries *series, int base, int n, double2 *c,
                     int *first_bad, cudaStream_t st) {
  if (table == PT_PAIR) fit<PT_PAIR>(series, base, n, c, first_bad, st);
  else if (table == PT_HESS) fit<PT_HESS>(series, base, n, c, first_bad, st);
  else fit<PT_EMBED>(series, base, n, c, first_bad, st);
}

void launch_tab_fit(const TabFit &t, const FxUnit &u, double4_32a *out, int *bad,
                    cudaStream_t st) {
  tab_fit_kernel<<<(4 * t.n + FIT_THREADS - 1) / FIT_THREADS, FIT_THREADS, 0, st>>>(t, u, out, bad);
}

}  // namespace cg
