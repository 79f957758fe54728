// force_fp64.cu -- the FP64 force kernels.  Built with -fmad=false: the sums
// round operation by operation but where a kernel states a fused one.
#include "force64.cuh"
#include "internal.h"

namespace cg {

template <int EVAL, bool OBS, int LANES>
static void launch_eam64_lanes(const ForceArgs &A, const EamPot<double, EVAL> &P, int pass,
                               cudaStream_t st) {
  const unsigned n = (unsigned)(((long)A.ntot * LANES + F64_THREADS - 1) / F64_THREADS);
  if (pass == 0) eam64_density_kernel<EVAL, LANES, OBS><<<n, F64_THREADS, 0, st>>>(A, P);
  else eam64_force_kernel<EVAL, LANES, OBS><<<n, F64_THREADS, 0, st>>>(A, P);
}
template <int EVAL, bool OBS>
static void launch_eam64_obs(const ForceArgs &A, const EamPot<double, EVAL> &P, int pass,
                             cudaStream_t st) {
  const int lanes = lanes64(A.ntot);
  if (lanes == 16) launch_eam64_lanes<EVAL, OBS, 16>(A, P, pass, st);
  else if (lanes == 4) launch_eam64_lanes<EVAL, OBS, 4>(A, P, pass, st);
  else launch_eam64_lanes<EVAL, OBS, 1>(A, P, pass, st);
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

template <bool OBS, int LANES>
static void launch_lj64_lanes(const ForceArgs &A, const LjPot<double> &P, cudaStream_t st) {
  const unsigned n = (unsigned)(((long)A.ntot * LANES + F64_THREADS - 1) / F64_THREADS);
  lj64_kernel<LANES, OBS><<<n, F64_THREADS, 0, st>>>(A, P);
}
template <bool OBS>
static void launch_lj64_obs(const ForceArgs &A, const LjPot<double> &P, cudaStream_t st) {
  const int lanes = lanes64(A.ntot);
  if (lanes == 16) launch_lj64_lanes<OBS, 16>(A, P, st);
  else if (lanes == 4) launch_lj64_lanes<OBS, 4>(A, P, st);
  else launch_lj64_lanes<OBS, 1>(A, P, st);
}
void launch_lj64(const ForceArgs &A, const LjPot<double> &P, cudaStream_t st, bool obs) {
  if (A.ntot <= 0) return;
  if (obs) launch_lj64_obs<true>(A, P, st);
  else launch_lj64_obs<false>(A, P, st);
}

}  // namespace cg
