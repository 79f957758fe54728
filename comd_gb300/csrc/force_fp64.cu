// force_fp64.cu -- the FP64 force kernels.  Built with -fmad=false: the sums
// round operation by operation but where a kernel states a fused one.
#include "force64.cuh"
#include "internal.h"

namespace cg {

// Four threads per atom up to 2^20 atoms, then one.  4,000 atoms (LJ): 34 us
// with four, 55 with two, 96 with one.  256,000 (table, density pass): 540 us
// with four, 565 with two, 562 with one, 694 with eight (lists of 42 entries
// leave the eighth lanes short).  1,048,576: 2,137 us with one, 2,235 with two.
static bool four_lanes(int ntot) { return ntot < (1 << 20); }
static unsigned blocks64(int ntot, int lanes) {
  return (unsigned)(((long)ntot * lanes + F64_THREADS - 1) / F64_THREADS);
}

template <int EVAL, bool OBS>
static void launch_eam64_obs(const ForceArgs &A, const EamPot<double, EVAL> &P, int pass,
                             cudaStream_t st) {
  const unsigned n4 = blocks64(A.ntot, 4), n1 = blocks64(A.ntot, 1);
  if (pass == 0) {
    if (four_lanes(A.ntot)) eam64_density_kernel<EVAL, 4, OBS><<<n4, F64_THREADS, 0, st>>>(A, P);
    else eam64_density_kernel<EVAL, 1, OBS><<<n1, F64_THREADS, 0, st>>>(A, P);
  } else {
    if (four_lanes(A.ntot)) eam64_force_kernel<EVAL, 4, OBS><<<n4, F64_THREADS, 0, st>>>(A, P);
    else eam64_force_kernel<EVAL, 1, OBS><<<n1, F64_THREADS, 0, st>>>(A, P);
  }
}

template <int EVAL>
void launch_eam64(const ForceArgs &A, const EamPot<double, EVAL> &P, int pass, cudaStream_t st,
                  bool obs) {
  if (A.ntot <= 0) return;
  if (obs) launch_eam64_obs<EVAL, true>(A, P, pass, st);
  else launch_eam64_obs<EVAL, false>(A, P, pass, st);
}
template void launch_eam64<EVAL_TABLE>(const ForceArgs &, const EamPot<double, EVAL_TABLE> &, int,
                                       cudaStream_t, bool);
template void launch_eam64<EVAL_CHEBY>(const ForceArgs &, const EamPot<double, EVAL_CHEBY> &, int,
                                       cudaStream_t, bool);

template <bool OBS>
static void launch_lj64_obs(const ForceArgs &A, const LjPot<double> &P, cudaStream_t st) {
  if (four_lanes(A.ntot)) lj64_kernel<4, OBS><<<blocks64(A.ntot, 4), F64_THREADS, 0, st>>>(A, P);
  else lj64_kernel<1, OBS><<<blocks64(A.ntot, 1), F64_THREADS, 0, st>>>(A, P);
}
void launch_lj64(const ForceArgs &A, const LjPot<double> &P, cudaStream_t st, bool obs) {
  if (A.ntot <= 0) return;
  if (obs) launch_lj64_obs<true>(A, P, st);
  else launch_lj64_obs<false>(A, P, st);
}

}  // namespace cg
