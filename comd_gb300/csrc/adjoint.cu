// adjoint.cu -- gradients of the EAM Chebyshev and LJ potentials with respect
// to their parameters, and the adjoint of the velocity-Verlet loop (FP64).
//
// Parameters: EAM Chebyshev -- the base series c = (phi, rho, F), 3 x 32
// coefficients on their [a, b]; the derivative series follow from them by the
// reference's genDer (cheby.c:219-270), so they are not free parameters.
// LJ -- (epsilon, sigma) at fixed cutoff.  eamCheb (cheby.c:276-310) is
// sum'_k c_k T_k(y), y = (2x - a - b)/(b - a), x clamped below at a, with the
// k = 0 term halved; its derivative in c_k is the basis B_k(y) and d/dx of
// that is B'_k = T'_k(y) * 2/(b - a) (0 below a, where eamCheb is clamped).
//
// With U the total energy, f the reference's forces (EAM f = +grad U,
// eam.c:438-660; LJ f = -grad U, ljForce.c:89-224) and a vector lambda per
// atom, D = sum_i lambda_i . grad_i U.  The force-matching loss
// L = sum_i |f_i - t_i|^2 has dL/dc = +/- dD/dc at lambda = 2 (f - t) (fixed),
// and one reverse velocity-Verlet step needs the same dD/dc at lambda = the
// force adjoint, plus the Hessian-vector product H lambda = grad_r D.
// For EAM, with v_ij = (lambda_i - lambda_j) . (r_i - r_j)/r_ij (symmetric),
// W_i = sum_j v_ij rho'(r_ij) and X_i = F''(rho_i) W_i:
//   D = sum_{i<j} v_ij phi'(r_ij) + sum_i F'(rho_i) W_i
//   dU/dc^phi_k = sum_{i<j} B_k(r_ij)        dD/dc^phi_k = sum_{i<j} v_ij B'_k(r_ij)
//   dU/dc^rho_k = sum_{i<j} (F'_i + F'_j) B_k(r_ij)
//   dD/dc^rho_k = sum_{i<j} [(F'_i + F'_j) v_ij B'_k(r_ij) + (X_i + X_j) B_k(r_ij)]
//   dU/dc^F_k   = sum_i B_k(rho_i)           dD/dc^F_k   = sum_i W_i B'_k(rho_i)
// Unique pairs are the list entries with slot_j > slot_i (duplicate stencil
// entries of small grids are separate terms, as in the reference's sums).
// Sums over atoms and pairs are per CTA in fixed order, then over CTAs in a
// fixed order: results are deterministic.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "force64.cuh"
#include "sim.h"

using namespace cg;
using namespace cgapi;

namespace {

constexpr int NC = CG_NCHEB;
constexpr int BASIS_THREADS = 128;  // CTA of the basis-sum kernels
constexpr int LOG_STEPS = 64;       // backward steps whose sums wait on the device
constexpr int NQ = 4;               // sums per coefficient index at most: three over pairs, one over atoms

// the FP64 series of the simulation and their second derivatives
typedef PolySeries ChebSet;

// eamCheb (cheby.c:276-310), the reference's operation order
__device__ double cheb_val(const ChebSet &S, int q, double x) {
  const double a = S.a[q], b = S.b[q];
  if (x < a) x = a;
  const double y = (2.0 * x - a - b) / (b - a), y2 = 2.0 * y;
  double d = 0.0, dd = 0.0;
  for (int j = NC - 1; j > 0; j--) {
    const double sv = d;
    d = y2 * d - dd + S.c[q][j];
    dd = sv;
  }
  return y * d - dd + 0.5 * S.c[q][0];
}

// x-derivative of a clamped series: 0 below a.  (The reference's forces use
// the derivative series at the clamped argument, eamCheb(dphi, r) -- which
// cheb_val gives -- so D differentiates those values in c, while its
// position derivatives below a are 0.)
__device__ __forceinline__ double cheb_der(const ChebSet &S, int qd, int q, double x) {
  return x < S.a[q] ? 0.0 : cheb_val(S, qd, x);
}

// Pair functions of one distance (r^2 in fixed point) from the polynomial
// table, or from the series outside it (rare: kept out of line).
__device__ __noinline__ double grho_series(const ChebSet &S, double r2) {
  const double r = sqrt(r2);
  return cheb_val(S, 4, r) / r;
}
// rho'(r) / r
__device__ __forceinline__ double pair_grho(const ChebSet &S, const PolyTables &P, u64 s,
                                            const FxUnit &u) {
  int k;
  double t;
  return poly_at(P.pair, s, 2 * u.m - 64, k, t) ? poly_col(P.pair, PF_GRHO, k, t)
                                                : grho_series(S, fx_area(s, u));
}
// the terms of the Hessian: phi'/r and rho'/r, the position derivative of
// the density over r (dr), and (phi'' - phi'/r) / r^2, (rho'' - rho'/r) / r^2
struct HessTerms {
  double gphi, grho, dr, hphi, hrho;
};
__device__ __noinline__ HessTerms hess_series(const ChebSet &S, double r2) {
  const double r = sqrt(r2), ir = 1.0 / r, ir2 = ir * ir;
  HessTerms h;
  h.gphi = cheb_val(S, 3, r) * ir;
  h.grho = cheb_val(S, 4, r) * ir;
  h.dr = cheb_der(S, 4, 1, r) * ir;
  h.hphi = (cheb_der(S, 6, 0, r) - h.gphi) * ir2;
  h.hrho = (cheb_der(S, 7, 1, r) - h.grho) * ir2;
  return h;
}
__device__ __forceinline__ HessTerms hess_terms(const ChebSet &S, const PolyTables &P, u64 s,
                                                const FxUnit &u) {
  int k, kh;
  double t, th;
  if (!poly_at(P.pair, s, 2 * u.m - 64, k, t) || !poly_at(P.hess, s, 2 * u.m - 64, kh, th))
    return hess_series(S, fx_area(s, u));
  HessTerms h;
  h.gphi = poly_col(P.pair, PF_GPHI, k, t);
  h.grho = h.dr = poly_col(P.pair, PF_GRHO, k, t);
  h.hphi = poly_col(P.hess, HF_PHI, kh, th);
  h.hrho = poly_col(P.hess, HF_RHO, kh, th);
  return h;
}
// F''(rho)
__device__ __forceinline__ double embed_d2(const ChebSet &S, const PolyTables &P, double rho) {
  int k;
  double t;
  return poly_at(P.embed, rho, k, t) ? poly_col(P.embed, EF_D2F, k, t) : cheb_der(S, 8, 2, rho);
}

// A pair's distance: from the integers in their range (plain), else in FP64 (for
// the basis sums, which hold every register, out of line).  false: beyond the
// cutoff; strict: within it (the embedding force).  The comparisons in FP64
// stay in the rare branch: for every pair they took 25 us of adj_w_kernel's 304
// at 256,000 atoms and as many of the basis sums'.
__device__ __noinline__ Exact64 exact_distance(EntryTab et, const d4 *r, int slot,
                                               uint32_t code) {
  return exact64(et, r, slot, code);
}
template <bool OUT_OF_LINE = false>
__device__ __forceinline__ bool distance(const ForceArgs &A, int slot, const Pair64 &q, double rc2,
                                         Exact64 &d, bool &plain, bool &strict) {
  plain = strict = fx_plain(A, q.s);
  if (plain) {
    d = Exact64{fx_length(q.x, A.fxu), fx_length(q.y, A.fxu), fx_length(q.z, A.fxu),
                fx_area(q.s, A.fxu)};
    return true;
  }
  if (q.s > A.fx_far) return false;
  d = OUT_OF_LINE ? exact_distance(A.et, A.s.r, slot, q.code) : exact64(A, slot, q.code);
  strict = !(d.r2 >= rc2);
  return !(d.r2 > rc2);
}

struct Lam {
  const d4 *lam;    // [nslots] lambda by slot
  const double *x;  // [nslots] X = F'' W by slot (EAM)
};

// lambda per slot: 2 (f - target[id]) (loss), or u[id] (given vector)
__global__ void adj_lambda_kernel(Slots s, const int *atom_slot, int ntot, const double *target,
                                  const double *u, d4 *lam, double *loss) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= ntot) return;
  const int slot = atom_slot[a];
  const int id = s.id[slot];
  d4 l;
  l.x = l.y = l.z = l.w = 0.0;
  if ((unsigned)id >= (unsigned)ntot) {  // ids must be 0..ntot-1
    lam[slot] = l;
    if (target) loss[a] = 0.0;
    return;
  }
  if (target) {
    const d4 f = s.f[slot];
    const double dx = f.x - target[3 * (size_t)id], dy = f.y - target[3 * (size_t)id + 1],
                 dz = f.z - target[3 * (size_t)id + 2];
    l.x = 2.0 * dx;
    l.y = 2.0 * dy;
    l.z = 2.0 * dz;
    loss[a] = dx * dx + dy * dy + dz * dz;
  } else {
    l.x = u[3 * (size_t)id];
    l.y = u[3 * (size_t)id + 1];
    l.z = u[3 * (size_t)id + 2];
  }
  lam[slot] = l;
}

// W_i = sum_j v_ij rho'(r_ij) over the embedding-force pairs (r2 < rc2,
// eam.c:612) and X_i = F''(rho_i) W_i, per slot.  The walk of the FP64 passes
// (fixed-point distances, LANES threads an atom): a thread per atom in FP64
// geometry took 63 us at 3,960 atoms and 500 us at 256,000, this 12 and 281.
template <int LANES>
__global__ void __launch_bounds__(F64_THREADS)
    adj_w_kernel(ForceArgs A, const __grid_constant__ ChebSet S, PolyTables poly, double rc2,
                 const d4 *lam, double *wout, double *xout) {
  int a, sub;
  bool live;
  if (!lane_atom<LANES>(A.ntot, a, sub, live)) return;
  const int slot = A.atom_slot[a];
  const d4 li = lam[slot];
  double W = 0.0;
  walk64<LANES>(A, a, sub, slot, A.fx[slot], rc2, [&](const Pair64 &q) {
    Exact64 d;
    bool plain, strict;
    if (!distance(A, slot, q, rc2, d, plain, strict) || !strict) return;
    const d4 lj = lam[q.j];
    const double vr = (li.x - lj.x) * d.x + (li.y - lj.y) * d.y + (li.z - lj.z) * d.z;
    W += vr * (plain ? pair_grho(S, poly, q.s, A.fxu) : grho_series(S, d.r2));
  });
  W = lane_sum<LANES>(W);
  if (sub != 0 || !live) return;
  wout[slot] = W;
  xout[slot] = embed_d2(S, poly, A.s.rho[slot]) * W;
}

// y of x on [a, b] after the clamp at a
__device__ __forceinline__ double cheb_y(const ChebSet &S, int q, double x) {
  const double a = S.a[q], b = S.b[q];
  if (x < a) x = a;
  return (2.0 * x - a - b) / (b - a);
}

// Sums over the pairs of w T_k(y), k < 32, for the weights of the gradients:
// without lambda w = 1 (phi) and F'_i + F'_j (rho); with it v (phi) and
// (F'_i + F'_j) v and X_i + X_j (rho).  The sums of the derivative basis
// B'_k = T'_k 2/(b - a) follow on the host, T'_k = k U_{k-1} being twice the
// sum of the T_j of the other parity below k (basis_derivative).
//
// Bound by FP64 operations: one for the recurrence and one per weight and k,
// 124 a pair with lambda.  A thread keeps all its sums in registers (96
// doubles).  Each pair is taken at one of its atoms, the lower slot if the
// slots' sum is even and the higher if it is odd.  So that no lane idles in
// those operations, a warp collects the pairs it takes, over all its atoms, in
// a queue in shared memory and works on 32 at a time; the distances are formed
// in fixed point, r without division.  At 256,000 and 3,960 atoms: 10,450 and
// 750 us with sums in shared memory, 2,158 and 94 us with several threads an
// atom each at its own pairs, 1,406 and 45 us now.
template <int NW>
struct BasisAcc {
  double s[NW][NC];
};
template <int NW, bool SAME>
__device__ __forceinline__ void basis_add(BasisAcc<NW> &A, double yp, double yr, const double *w) {
  double t0 = 1.0, t1 = yp, r0 = 1.0, r1 = yr;
  const double yp2 = 2.0 * yp, yr2 = 2.0 * yr;
#pragma unroll
  for (int k = 0; k < NC; k++) {
    A.s[0][k] = fma(w[0], t0, A.s[0][k]);
#pragma unroll
    for (int q = 1; q < NW; q++) A.s[q][k] = fma(w[q], SAME ? t0 : r0, A.s[q][k]);
    const double t2 = fma(yp2, t1, -t0);
    t0 = t1;
    t1 = t2;
    if (!SAME) {
      const double r2 = fma(yr2, r1, -r0);
      r0 = r1;
      r1 = r2;
    }
  }
}

// A lane hands half of its 2 N rows to its partner O lanes on and adds the
// other half, down to O = 1: a fifth of the additions of a tree per row.
// Returns the lane's first row.
template <int N, int O>
__device__ __forceinline__ int split_rows(double *v, int lane) {
  if constexpr (O == 0) {
    return 0;
  } else {
    const bool upper = lane & O;
#pragma unroll
    for (int r = 0; r < N; r++) {
      const double keep = upper ? v[N + r] : v[r], give = upper ? v[r] : v[N + r];
      v[r] = keep + __shfl_xor_sync(0xffffffffu, give, O);
    }
    return (upper ? N : 0) + split_rows<N / 2, O / 2>(v, lane);
  }
}

// the CTA's sums of NROW per-thread values (a multiple of 32), to
// out[0..NROW): over the lanes of each warp, then the warps in order
template <int NROW, int NT>
__device__ __forceinline__ void block_rows(double *v, double *sh, double *out) {
  static_assert(NROW % 32 == 0, "rows are split over the lanes");
  const int first = split_rows<NROW / 2, 16>(v, threadIdx.x & 31);
#pragma unroll
  for (int r = 0; r < NROW / 32; r++) sh[(threadIdx.x >> 5) * NROW + first + r] = v[r];
  __syncthreads();
  for (int r = threadIdx.x; r < NROW; r += NT) {
    double t = 0.0;
    for (int w = 0; w < NT / 32; w++) t += sh[w * NROW + r];
    out[r] = t;
  }
}

template <int NW, bool SAME>
__global__ void __launch_bounds__(BASIS_THREADS)
    adj_basis_kernel(ForceArgs A, const __grid_constant__ ChebSet S, double rc2, Lam L,
                     double *partial) {
  constexpr int WARPS = BASIS_THREADS / 32;
  __shared__ double sh[WARPS * NW * NC];
  __shared__ uint2 s_queue[WARPS][64];  // (slot i, entry)
  uint2 *queue = s_queue[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const double scale[2] = {1.0 / (S.b[0] - S.a[0]), 1.0 / (S.b[1] - S.a[1])};
  BasisAcc<NW> acc;
#pragma unroll
  for (int q = 0; q < NW; q++)
#pragma unroll
    for (int k = 0; k < NC; k++) acc.s[q][k] = 0.0;
  auto mine = [](int js, int slot) { return ((js > slot) ^ ((js + slot) & 1)) != 0; };
  // cheb_y: 2 (r - a) / (b - a) - 1, the quotient corrected once
  auto y_of = [&](int q, double r) {
    const double d = fmax(r, S.a[q]) - S.a[q], t = d * scale[q];
    return fma(2.0, fma(fma(-t, S.b[q] - S.a[q], d), scale[q], t), -1.0);
  };
  auto pair = [&](int slot, const d4 &fi, const Pair64 &q) {
    Exact64 d;
    bool plain, strict;
    if (!distance<true>(A, slot, q, rc2, d, plain, strict)) return;
    double r, inv;
    r_and_inv(d.r2, r, inv);
    const double fsum = fi.w + q.fj;
    double w[3];
    if (NW == 3) {
      const d4 li = L.lam[slot], lj = L.lam[q.j];
      w[0] = ((li.x - lj.x) * d.x + (li.y - lj.y) * d.y + (li.z - lj.z) * d.z) * inv;
      w[1] = strict ? fsum * w[0] : 0.0;
      w[2] = L.x[slot] + L.x[q.j];
    } else {
      w[0] = 1.0;
      w[1] = fsum;
    }
    const double yp = y_of(0, r);
    basis_add<NW, SAME>(acc, yp, SAME ? yp : y_of(1, r), w);
  };
  int queued = 0;
  auto work = [&](int n) {  // the queue's first n <= 32 pairs
    if (lane < n) {
      const uint2 e = queue[lane];
      const int slot = (int)e.x;
      const d4 fi = A.fx[slot];
      pair(slot, fi, pair64(A, fi, A.et.fx + (slot >> 6) * CG_NNBR, e.y));
    }
    __syncwarp();
  };
  for (int a = blockIdx.x * WARPS + (threadIdx.x >> 5); a < A.ntot; a += gridDim.x * WARPS) {
    const int slot = A.atom_slot[a], n = A.nbr_n[a], ebase = (slot >> 6) * CG_NNBR;
    if (n > A.cap) {  // overflowed list: the stencil, by one lane
      if (lane == 0) {
        const d4 fi = A.fx[slot];
        walk64<1>(A, a, 0, slot, fi, rc2, [&](const Pair64 &q) {
          if (mine(q.j, slot)) pair(slot, fi, q);
        });
      }
      __syncwarp();
      continue;
    }
    const uint16_t *lst = A.nbr + (size_t)a * A.cap;
    for (int t0 = 0; t0 < n; t0 += 32) {
      uint32_t code = 0;
      bool take = false;
      if (t0 + lane < n) {
        code = __ldg(lst + t0 + lane);
        take = mine(__ldg(A.et.box + ebase + (code >> 6)) * CG_MAXATOMS + (int)(code & 63), slot);
      }
      const uint32_t m = __ballot_sync(0xffffffffu, take);
      if (take) queue[queued + __popc(m & ((1u << lane) - 1u))] = make_uint2(slot, code);
      queued += __popc(m);
      __syncwarp();
      if (queued < 32) continue;
      work(32);
      queued -= 32;
      uint2 e;
      if (lane < queued) e = queue[32 + lane];
      __syncwarp();
      if (lane < queued) queue[lane] = e;
      __syncwarp();
    }
  }
  work(queued);
  block_rows<NW * NC, BASIS_THREADS>(&acc.s[0][0], sh, partial + (size_t)blockIdx.x * NW * NC);
}

// sums over the atoms of w T_k(y(rho_i)) for the F series: w = 1, or W_i
__global__ void __launch_bounds__(BASIS_THREADS)
    adj_embed_basis_kernel(ForceArgs A, const __grid_constant__ ChebSet S, const double *wsl,
                           double *partial) {
  __shared__ double sh[BASIS_THREADS / 32 * NC];
  BasisAcc<1> acc;
#pragma unroll
  for (int k = 0; k < NC; k++) acc.s[0][k] = 0.0;
  for (int a = blockIdx.x * BASIS_THREADS + threadIdx.x; a < A.ntot;
       a += gridDim.x * BASIS_THREADS) {
    const int slot = A.atom_slot[a];
    const double y = cheb_y(S, 2, A.s.rho[slot]), w = wsl ? wsl[slot] : 1.0;
    basis_add<1, true>(acc, y, y, &w);
  }
  block_rows<NC, BASIS_THREADS>(&acc.s[0][0], sh, partial + (size_t)blockIdx.x * NC);
}

// out[r] = sum over n partial rows, one CTA per r: thread t takes rows t, t +
// 256, ..., then a tree (a fixed order; one thread over 1,000 rows took 65 us)
__global__ void __launch_bounds__(256)
    adj_sum_kernel(const double *partial, int n, int width, double *out) {
  __shared__ double sh[256];
  double t = 0.0;
  for (int q = threadIdx.x; q < n; q += 256) t += partial[(size_t)q * width + blockIdx.x];
  sh[threadIdx.x] = t;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = sh[0];
}

// LJ (ljForce.c:151-215, U = 4 eps sum_{i<j} (s^12 - s^6), s = sigma/r, no
// shift at the cutoff; f = -grad U): per-CTA sums of dU/deps, dU/dsigma and
// of sum_{i<j} v_ij dV'(r_ij)/d(eps, sigma) (V' = dU_pair/dr), so that
// dL/d(eps, sigma) = -(the last two) for lambda = 2 (f - t)
__global__ void __launch_bounds__(128) adj_lj_kernel(ForceArgs A, double eps, double sigma,
                                                     double rc2, const d4 *lam, double *partial) {
  __shared__ double sh[4][128];
  double ge = 0.0, gs = 0.0, de = 0.0, ds = 0.0;
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < A.ntot; a += gridDim.x * blockDim.x) {
    const int slot = A.atom_slot[a];
    const int b = slot >> 6, i = slot & 63;
    double xi, yi, zi;
    PrecT<double>::pos(A.s, slot, xi, yi, zi);
    d4 li;
    li.x = li.y = li.z = 0.0;
    if (lam) li = lam[slot];
    for_each_neighbor<double, true>(
        A, a, b, i, xi, yi, zi, rc2, [&](int js, double dx, double dy, double dz, double r2) {
          if (js <= slot || r2 > rc2) return;
          const double r = sqrt(r2);
          const double s2 = sigma * sigma / r2, s6 = s2 * s2 * s2, s12 = s6 * s6;
          ge += 4.0 * (s12 - s6);
          gs += 4.0 * eps * (12.0 * s12 - 6.0 * s6) / sigma;
          if (lam) {
            const d4 lj = lam[js];
            const double v = ((li.x - lj.x) * dx + (li.y - lj.y) * dy + (li.z - lj.z) * dz) / r;
            de += v * 4.0 * (-12.0 * s12 + 6.0 * s6) / r;
            ds += v * 4.0 * eps * (-144.0 * s12 + 36.0 * s6) / (sigma * r);
          }
        });
  }
  sh[0][threadIdx.x] = ge;
  sh[1][threadIdx.x] = gs;
  sh[2][threadIdx.x] = de;
  sh[3][threadIdx.x] = ds;
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int c = 0; c < 128; c++) t += sh[threadIdx.x][c];
    partial[blockIdx.x * 4 + threadIdx.x] = t;
  }
}

// EAM Hessian-vector product, (H u)_k = grad_k sum_i u_i . f_i (f the
// reference's forces), per atom over its full list: for each pair (k, j),
// rhat = (r_k - r_j)/r, du = u_k - u_j, v = du . rhat,
//   g  = phi'(r) + (F'_k + F'_j) rho'(r)      (embedding part for r2 < rc2)
//   g' = phi''(r) + (F'_k + F'_j) rho''(r)
//   += g (du - v rhat)/r + v g' rhat + (X_k + X_j) d rho/dr rhat
// with X = F'' W (adj_w_kernel at lambda = u), computed as
//   (g/r) du + [(du . d) (g' - g/r)/r^2 + (X_k + X_j) (d rho/dr)/r] d,
// d = r_k - r_j, whose functions of r^2 are columns of the polynomial table
// (no square root, no division).  Written by atom id.  The walk of adj_w_kernel;
// a thread per atom took 108 us at 3,960 atoms, this 25.
template <int LANES>
__global__ void __launch_bounds__(F64_THREADS)
    adj_hvp_kernel(ForceArgs A, const __grid_constant__ ChebSet S, PolyTables poly, double rc2,
                   const d4 *u, const double *X, double *hv) {
  int a, sub;
  bool live;
  if (!lane_atom<LANES>(A.ntot, a, sub, live)) return;
  const int slot = A.atom_slot[a];
  const d4 fi = A.fx[slot], uk = u[slot];
  const double Xk = X[slot];
  double hx = 0.0, hy = 0.0, hz = 0.0;
  walk64<LANES>(A, a, sub, slot, fi, rc2, [&](const Pair64 &q) {
    Exact64 d;
    bool plain, strict;
    if (!distance(A, slot, q, rc2, d, plain, strict)) return;
    const HessTerms h = plain ? hess_terms(S, poly, q.s, A.fxu) : hess_series(S, d.r2);
    const d4 uj = u[q.j];
    const double ux = uk.x - uj.x, uy = uk.y - uj.y, uz = uk.z - uj.z;
    const double ud = ux * d.x + uy * d.y + uz * d.z;
    const double fs = strict ? fi.w + q.fj : 0.0;
    const double g = h.gphi + fs * h.grho;
    const double c = ud * (h.hphi + fs * h.hrho) + (Xk + X[q.j]) * h.dr;
    hx += g * ux + c * d.x;
    hy += g * uy + c * d.y;
    hz += g * uz + c * d.z;
  });
  hx = lane_sum<LANES>(hx);
  hy = lane_sum<LANES>(hy);
  hz = lane_sum<LANES>(hz);
  if (sub != 0 || !live) return;
  const int id = A.s.id[slot];
  if ((unsigned)id >= (unsigned)A.ntot) return;
  hv[3 * (size_t)id] = hx;
  hv[3 * (size_t)id + 1] = hy;
  hv[3 * (size_t)id + 2] = hz;
}

// per-id vectors, either side of a backward step's Hessian-vector product:
// pb += c rb, u = -dt pb; rb += hv, pb += c rb
__global__ void adj_before_kernel(double c, double dt, const double *rb, double *pb, double *u,
                                  long n) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const double p = c * rb[q] + pb[q];
  pb[q] = p;
  u[q] = -dt * p;
}
__global__ void adj_after_kernel(double c, const double *hv, double *rb, double *pb, long n) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const double r = hv[q] + rb[q];
  rb[q] = r;
  pb[q] = c * r + pb[q];
}
// v[3 id] = f[slot] (the EAM force is grad U)
__global__ void adj_force_by_id_kernel(Slots s, const int *atom_slot, int ntot, double *v) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= ntot) return;
  const int slot = atom_slot[a];
  const int id = s.id[slot];
  if ((unsigned)id >= (unsigned)ntot) return;
  const d4 f = s.f[slot];
  v[3 * (size_t)id] = f.x;
  v[3 * (size_t)id + 1] = f.y;
  v[3 * (size_t)id + 2] = f.z;
}
// per-block sums of x[0..n) (fixed order)
__global__ void adj_block_sum_kernel(const double *x, int n, double *partial) {
  __shared__ double sh[256];
  double t = 0.0;
  for (int q = blockIdx.x * 256 + threadIdx.x; q < n; q += gridDim.x * 256) t += x[q];
  sh[threadIdx.x] = t;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {

ChebSet cheb_set(const comdgb_sim *h) {
  ChebSet S{};
  for (int q = 0; q < 6; q++) {
    memcpy(S.c[q], h->cheb_coef[q], sizeof S.c[q]);
    S.a[q] = h->cheb_a[q];
    S.b[q] = h->cheb_b[q];
  }
  for (int q = 6; q < 9; q++) {
    cheb_derive(S.a[q - 3], S.b[q - 3], S.c[q - 3], S.c[q], NC);
    S.a[q] = S.a[q - 3];
    S.b[q] = S.b[q - 3];
  }
  return S;
}

typedef comdgb_sim::Adj Work;

// the handle's adjoint scratch (allocated once)
int work(comdgb_sim *h, Work *&Wp) {
  Work &W = h->adj;
  Wp = &W;
  if (W.lam) return 0;
  int err = 0;
  size_t ns = (size_t)h->nslots, nv = 3 * (size_t)h->ntot + 3;
  int dev = 0, nsm = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  W.nblk = 2 * nsm;  // resident CTAs of the basis sums
  W.lam = track(h, dalloc<d4>(ns, &err));
  W.w = track(h, dalloc<double>(ns, &err));
  W.x = track(h, dalloc<double>(ns, &err));
  W.loss = track(h, dalloc<double>((size_t)h->ntot + 1, &err));
  W.partial = track(h, dalloc<double>((size_t)W.nblk * NQ * NC + 4096, &err));
  W.out = track(h, dalloc<double>(NQ * NC + 8, &err));
  W.log = track(h, dalloc<double>((size_t)LOG_STEPS * NQ * NC, &err));
  W.target = track(h, dalloc<double>(nv, &err));
  W.rb = track(h, dalloc<double>(nv, &err));
  W.pb = track(h, dalloc<double>(nv, &err));
  W.u = track(h, dalloc<double>(nv, &err));
  W.hv = track(h, dalloc<double>(nv, &err));
  if (err) {
    W.lam = nullptr;
    return set_err(COMDGB_ERR_NOMEM, "cudaMalloc failed for adjoint scratch");
  }
  return 0;
}

// snapshot i of the handle's pool (grown on demand)
int snap(comdgb_sim *h, size_t i, Snapshot *&q) {
  while (h->adj.snaps.size() <= i) {
    Snapshot *n = new Snapshot();
    int rc = snapshot_alloc(h, n);
    if (rc) {
      delete n;
      return rc;
    }
    h->adj.snaps.push_back(n);
  }
  q = (Snapshot *)h->adj.snaps[i];
  return 0;
}

int need_fp64(comdgb_sim *h) {
  if (!h) return set_err(COMDGB_ERR_ARG, "null handle");
  if (h->mixed) return set_err(COMDGB_ERR_UNSUPPORTED, "gradients need an FP64 simulation");
  if (h->opts.potential != COMDGB_POT_EAM_CHEBY && h->opts.potential != COMDGB_POT_LJ)
    return set_err(COMDGB_ERR_UNSUPPORTED, "gradients are for EAM Chebyshev or LJ potentials");
  CK(cudaSetDevice(h->device));
  return 0;
}

unsigned blocks(long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// fn(threads per atom), as the force passes take them
template <class F>
void by_lanes(const comdgb_sim *h, F &&fn) {
  const int lanes = lanes64(h->ntot);
  if (lanes == 16) fn(std::integral_constant<int, 16>());
  else if (lanes == 4) fn(std::integral_constant<int, 4>());
  else fn(std::integral_constant<int, 1>());
}

// sum of W.loss[0..ntot) to the host
int loss_sum(comdgb_sim *h, Work &W, double *loss) {
  const int nb = std::min(1024, (int)blocks(h->ntot));
  adj_block_sum_kernel<<<nb, 256, 0, h->stream>>>(W.loss, h->ntot, W.partial);
  adj_sum_kernel<<<1, 256, 0, h->stream>>>(W.partial, nb, 1, W.out);
  CK(cudaMemcpyAsync(loss, W.out, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return 0;
}

// sums of w T'_k(y) from those of w T_k: T'_k = k U_{k-1}, and U_{k-1} = 2
// (T_{k-1} + T_{k-3} + ...), T_0 counted half
void basis_derivative(const double *t, double *d) {
  for (int k = 0; k < NC; k++) {
    double u = 0.0;
    for (int j = k - 1; j >= 0; j -= 2) u += j == 0 ? 0.5 * t[j] : t[j];
    d[k] = 2.0 * k * u;
  }
}

template <int NW>
void launch_basis(comdgb_sim *h, Work &W, const ChebSet &S, Lam L, double *out) {
  const ForceArgs A = force_args(h);
  const double rc2 = h->eam64c.rc2;
  const bool same = S.a[0] == S.a[1] && S.b[0] == S.b[1];
  const long warps = BASIS_THREADS / 32;
  const int grid = (int)std::max(1L, std::min((long)W.nblk, (h->ntot + warps - 1) / warps));
  auto run = [&](auto kernel) { kernel<<<grid, BASIS_THREADS, 0, h->stream>>>(A, S, rc2, L, W.partial); };
  if (same) run(adj_basis_kernel<NW, true>);
  else run(adj_basis_kernel<NW, false>);
  adj_sum_kernel<<<NW * NC, 256, 0, h->stream>>>(W.partial, grid, NW * NC, out);
}

// The sums of the gradient in the coefficients at the current forces and
// per-step list, to out[0 .. (2 or 3 + 1) NC) on the device.
void enqueue_eam_sums(comdgb_sim *h, Work &W, const ChebSet &S, bool with_lam, double *out) {
  if (with_lam) launch_basis<3>(h, W, S, Lam{W.lam, W.x}, out);
  else launch_basis<2>(h, W, S, Lam{nullptr, nullptr}, out);
  const int nw = with_lam ? 3 : 2;
  const int nb = std::max(1, std::min(W.nblk, (h->ntot + BASIS_THREADS - 1) / BASIS_THREADS));
  adj_embed_basis_kernel<<<nb, BASIS_THREADS, 0, h->stream>>>(force_args(h), S,
                                                              with_lam ? W.w : nullptr, W.partial);
  adj_sum_kernel<<<NC, 256, 0, h->stream>>>(W.partial, nb, NC, out + nw * NC);
}

// the gradient g[3*NC] from those sums: dU/dc, or with lambda set dD/dc
void eam_grad_of(const ChebSet &S, bool with_lam, const double *t, double *g) {
  const int nw = with_lam ? 3 : 2;
  const double *phi = t, *rho = t + NC, *f = t + nw * NC;
  if (!with_lam) {
    for (int k = 0; k < NC; k++) {
      const double c = k == 0 ? 0.5 : 1.0;
      g[k] = c * phi[k];
      g[NC + k] = c * rho[k];
      g[2 * NC + k] = c * f[k];
    }
  } else {
    const double *x = t + 2 * NC;
    double d[3][NC];
    basis_derivative(phi, d[0]);
    basis_derivative(rho, d[1]);
    basis_derivative(f, d[2]);
    for (int k = 0; k < NC; k++)
      for (int q = 0; q < 3; q++) {
        g[q * NC + k] = d[q][k] * (2.0 / (S.b[q] - S.a[q]));
        if (q == 1) g[q * NC + k] += k == 0 ? 0.5 * x[k] : x[k];
      }
  }
}

// both, with the gradient on the host
int eam_grad(comdgb_sim *h, Work &W, const ChebSet &S, bool with_lam, double *g) {
  enqueue_eam_sums(h, W, S, with_lam, W.out);
  double t[NQ * NC];
  CK(cudaMemcpyAsync(t, W.out, sizeof(double) * (with_lam ? 4 : 3) * NC, cudaMemcpyDeviceToHost,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  eam_grad_of(S, with_lam, t, g);
  return check_status(h);
}

// lambda (from target forces by id, or a per-id vector u) and, for EAM, W and X
int set_lambda(comdgb_sim *h, Work &W, const ChebSet &S, const double *d_target,
               const double *d_u) {
  adj_lambda_kernel<<<blocks(h->ntot), 256, 0, h->stream>>>(h->s, h->atom_slot, h->ntot, d_target,
                                                           d_u, W.lam, W.loss);
  if (h->opts.potential == COMDGB_POT_EAM_CHEBY)
    by_lanes(h, [&](auto lanes) {
      constexpr int L = decltype(lanes)::value;
      adj_w_kernel<L><<<blocks((long)h->ntot * L, F64_THREADS), F64_THREADS, 0, h->stream>>>(
          force_args(h), S, h->eam64c.poly, h->eam64c.rc2, W.lam, W.w, W.x);
    });
  CK(cudaGetLastError());
  return 0;
}

// LJ sums: out[0..3] = dU/deps, dU/dsigma, sum v dV'/deps, sum v dV'/dsigma
int lj_sums(comdgb_sim *h, Work &W, bool with_lam, double *out4) {
  const int nb = std::min(W.nblk, 1024);
  adj_lj_kernel<<<nb, 128, 0, h->stream>>>(force_args(h), h->lj_eps, h->lj_sigma, h->lj64.rc2,
                                           with_lam ? W.lam : nullptr, W.partial);
  adj_sum_kernel<<<4, 256, 0, h->stream>>>(W.partial, nb, 4, W.out);
  CK(cudaMemcpyAsync(out4, W.out, sizeof(double) * 4, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return check_status(h);
}

// a force call whose lists are built from the current state (so forces are
// a function of the state alone, whatever the history of list builds)
int force_fresh(comdgb_sim *h, bool wait = true) {
  if (h->pl.slot_of) CK(cudaMemsetAsync(h->status + ST_REBUILD, 0x01, 1, h->stream));
  return wait ? do_force(h) : enqueue_force(h);
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

int comdgb_sim_set_cheby(comdgb_sim *h, const double *coef, const double *x0, const double *xn) {
  if (!h || !coef || !x0 || !xn) return set_err(COMDGB_ERR_ARG, "null argument");
  if (h->opts.potential != COMDGB_POT_EAM_CHEBY)
    return set_err(COMDGB_ERR_UNSUPPORTED, "not an EAM Chebyshev simulation");
  CK(cudaSetDevice(h->device));
  double c6[6][NC], a[6], b[6];
  for (int q = 0; q < 3; q++) {
    if (!(xn[q] > x0[q])) return set_err(COMDGB_ERR_ARG, "series %d: empty interval", q);
    memcpy(c6[q], coef + (size_t)q * NC, sizeof c6[q]);
    a[q] = a[q + 3] = x0[q];
    b[q] = b[q + 3] = xn[q];
    cheb_derive(a[q], b[q], c6[q], c6[q + 3], NC);
  }
  return install_cheby(h, c6, a, b);
}

int comdgb_sim_get_cheby(comdgb_sim *h, double *coef, double *x0, double *xn) {
  if (!h || !coef || !x0 || !xn) return set_err(COMDGB_ERR_ARG, "null argument");
  if (h->opts.potential != COMDGB_POT_EAM_CHEBY)
    return set_err(COMDGB_ERR_UNSUPPORTED, "not an EAM Chebyshev simulation");
  for (int q = 0; q < 3; q++) {
    memcpy(coef + (size_t)q * NC, h->cheb_coef[q], sizeof(double) * NC);
    x0[q] = h->cheb_a[q];
    xn[q] = h->cheb_b[q];
  }
  return 0;
}

int comdgb_sim_set_lj(comdgb_sim *h, double epsilon, double sigma) {
  if (!h) return set_err(COMDGB_ERR_ARG, "null handle");
  if (h->opts.potential != COMDGB_POT_LJ)
    return set_err(COMDGB_ERR_UNSUPPORTED, "not an LJ simulation");
  if (!(sigma > 0.0)) return set_err(COMDGB_ERR_ARG, "sigma must be positive");
  install_lj(h, epsilon, sigma, h->cutoff);
  return 0;
}

int comdgb_sim_energy_grad(comdgb_sim *h, double *energy, double *grad) {
  int rc = need_fp64(h);
  if (rc) return rc;
  if (!grad) return set_err(COMDGB_ERR_ARG, "null argument");
  Work *Wp;
  if ((rc = work(h, Wp)) || (rc = force_fresh(h))) return rc;
  Work &W = *Wp;
  if (energy) *energy = h->e;
  if (h->opts.potential == COMDGB_POT_LJ) {
    double o[4];
    if ((rc = lj_sums(h, W, false, o))) return rc;
    grad[0] = o[0];
    grad[1] = o[1];
    return 0;
  }
  return eam_grad(h, W, cheb_set(h), false, grad);
}

int comdgb_sim_force_loss_grad(comdgb_sim *h, const double *target, double *loss, double *grad) {
  int rc = need_fp64(h);
  if (rc) return rc;
  if (!target || !grad) return set_err(COMDGB_ERR_ARG, "null argument");
  Work *Wp;
  if ((rc = work(h, Wp)) || (rc = force_fresh(h))) return rc;
  Work &W = *Wp;
  double *d_t = W.target;
  CK(cudaMemcpyAsync(d_t, target, sizeof(double) * 3 * h->ntot, cudaMemcpyHostToDevice,
                     h->stream));
  const ChebSet S = h->opts.potential == COMDGB_POT_EAM_CHEBY ? cheb_set(h) : ChebSet{};
  if ((rc = set_lambda(h, W, S, d_t, nullptr))) return rc;
  double l = 0.0;
  if ((rc = loss_sum(h, W, &l))) return rc;
  if (loss) *loss = l;
  if (h->opts.potential == COMDGB_POT_LJ) {
    double o[4];
    if ((rc = lj_sums(h, W, true, o))) return rc;
    grad[0] = -o[2];  // f = -grad U
    grad[1] = -o[3];
    return 0;
  }
  return eam_grad(h, W, S, true, grad);
}

// Reverse velocity Verlet.  Forward: x_{n+1} = Phi(x_n) with r_a = r_n + c p_n,
// p_{n+1} = p_n - dt f(r_a), r_{n+1} = r_a + c p_{n+1}, c = (dt/2)/M.  Given
// the adjoints (rb, pb) of step n+1:  pb += c rb;  u = -dt pb;  rb += H(r_a) u;
// cbar += d(u . f(r_a))/dc;  pb += c rb.  Start: rb = grad U(r_N) (= f for
// EAM), pb = 0, cbar = dU/dc at r_N.  Adjoint vectors are kept by atom id (the
// rebox permutes slots, not atoms).  The host waits once a segment, and for
// the sums of every LOG_STEPS backward steps (a wait after every half step,
// force call and sum took 13.1 ms in 20 steps of 3,960 atoms, this 9.5): errors are
// kept on the device, the first one of a segment is the one reported.
int comdgb_sim_traj_energy_grad(comdgb_sim *h, int n, double dt, int every, double *j,
                                double *grad) {
  int rc = need_fp64(h);
  if (rc) return rc;
  if (h->opts.potential != COMDGB_POT_EAM_CHEBY)
    return set_err(COMDGB_ERR_UNSUPPORTED, "the trajectory adjoint is for EAM Chebyshev");
  if (n < 1 || every < 1 || !grad) return set_err(COMDGB_ERR_ARG, "bad argument");
  const double dt_atu = dt * kBohrPerAtu;
  const double c = (dt_atu / 2.0) / h->rmass;
  const long nv = 3L * h->ntot;
  Work *Wp;
  if ((rc = work(h, Wp))) return rc;
  Work &W = *Wp;
  double *rb = W.rb, *pb = W.pb, *u = W.u, *hv = W.hv;
  const int nseg = (n + every - 1) / every;
  std::vector<Snapshot *> ck((size_t)nseg), mid((size_t)every);
  Snapshot *fin = nullptr;
  size_t si = 0;
  for (auto &q : ck)
    if ((rc = snap(h, si++, q))) return rc;
  for (auto &q : mid)
    if ((rc = snap(h, si++, q))) return rc;
  if ((rc = snap(h, si++, fin))) return rc;
  const ChebSet S = cheb_set(h);
  CK(cudaMemsetAsync(h->status + ST_NONFINITE, 0, sizeof(int), h->stream));
  // forward, keeping the state at the start of every segment
  for (int t = 0; t < n; t++) {
    if (t % every == 0 &&
        ((t && (rc = check_forces(h))) || (rc = snapshot_copy(h, *ck[t / every], true))))
      return rc;
    if ((rc = step_first_half(h, dt_atu)) || (rc = force_fresh(h, false)) ||
        (rc = step_second_half(h, dt_atu)))
      return rc;
  }
  if ((rc = check_forces(h))) return rc;
  if ((rc = force_fresh(h))) return rc;
  if (j) *j = h->e;
  if ((rc = snapshot_copy(h, *fin, true))) return rc;
  double g[3 * NC], cbar[3 * NC];
  if ((rc = eam_grad(h, W, S, false, cbar))) return rc;
  adj_force_by_id_kernel<<<blocks(h->ntot), 256, 0, h->stream>>>(h->s, h->atom_slot, h->ntot, rb);
  CK(cudaMemsetAsync(pb, 0, sizeof(double) * nv, h->stream));
  // the logged sums into cbar, in the order of the steps
  int logged = 0;
  std::vector<double> sums((size_t)LOG_STEPS * NQ * NC);
  auto flush = [&]() -> int {
    if (logged)
      CK(cudaMemcpyAsync(sums.data(), W.log, sizeof(double) * logged * NQ * NC,
                         cudaMemcpyDeviceToHost, h->stream));
    if (int e = check_forces(h)) return e;
    for (int q = 0; q < logged; q++) {
      eam_grad_of(S, true, &sums[(size_t)q * NQ * NC], g);
      for (int k = 0; k < 3 * NC; k++) cbar[k] += g[k];
    }
    logged = 0;
    return 0;
  };
  // backward, segment by segment: recompute the segment's mid-step states
  for (int sgm = nseg - 1; sgm >= 0; sgm--) {
    const int t0 = sgm * every, m = std::min(every, n - t0);
    if ((rc = snapshot_copy(h, *ck[sgm], false))) return rc;
    for (int t = 0; t < m; t++) {
      if ((rc = step_first_half(h, dt_atu)) || (rc = snapshot_copy(h, *mid[t], true)) ||
          (rc = force_fresh(h, false)) || (rc = step_second_half(h, dt_atu)))
        return rc;
    }
    if ((rc = flush())) return rc;
    for (int t = m - 1; t >= 0; t--) {
      if ((rc = snapshot_copy(h, *mid[t], false)) || (rc = force_fresh(h, false))) return rc;
      adj_before_kernel<<<blocks(nv), 256, 0, h->stream>>>(c, dt_atu, rb, pb, u, nv);
      if ((rc = set_lambda(h, W, S, nullptr, u))) return rc;
      by_lanes(h, [&](auto lanes) {
        constexpr int L = decltype(lanes)::value;
        adj_hvp_kernel<L><<<blocks((long)h->ntot * L, F64_THREADS), F64_THREADS, 0, h->stream>>>(
            force_args(h), S, h->eam64c.poly, h->eam64c.rc2, W.lam, W.x, hv);
      });
      enqueue_eam_sums(h, W, S, true, W.log + (size_t)logged * NQ * NC);
      adj_after_kernel<<<blocks(nv), 256, 0, h->stream>>>(c, hv, rb, pb, nv);
      if (++logged == LOG_STEPS && (rc = flush())) return rc;
    }
  }
  if ((rc = flush())) return rc;
  CK(cudaGetLastError());
  for (int q = 0; q < 3 * NC; q++) grad[q] = cbar[q];
  if ((rc = snapshot_copy(h, *fin, false))) return rc;
  return force_fresh(h);
}

}  // extern "C"
