// force_mixed.cu -- the mixed-precision force kernels (FP32 pair terms on
// box-relative coordinates, Kahan-compensated FP32 per-atom sums) and the list
// builds, which both precisions use.
#include <algorithm>
#include <climits>

#include "comdgb.h"
#include "fo_lanes.cuh"
#include "internal.h"

namespace cg {

// resident CTAs per SM of the EAM pass kernels ([pass][eval]) and the SM
// count, found before any launch or stream capture
static int g_pass_per_sm[2][2];
// force order: [without, with energies][pass 1, pass 2, LJ][eval]
static int g_fo_per_sm[2][3][2];
static int g_num_sms = 1;
// resident CTAs per SM of the FP32 list builds: force order [64, 128, 256
// threads][2, 4, 8 atoms per load], per-step and id-keyed lists
static int g_build_per_sm[3][3], g_build_step_per_sm = 1, g_build_id_per_sm = 1;

template <class K>
static cudaError_t pass_occupancy(K kernel, size_t smem, int *out, int threads = PASS_THREADS) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, kernel, threads, smem);
  if (*out < 1) *out = 1;
  return e;
}

static size_t pass_smem(int pass, int eval) {
  if (eval != EVAL_CHEBY) return 0;
  return sizeof(float4) * (pass == 0 ? 2 : 1) * SEG_N;
}

// force order: what a pass stages (stage_rho, stage_force)
static size_t fo_pass_smem(int pass, int eval, bool obs, int copies, int ntab) {
  if (eval == EVAL_TABLE) return copies > 0 ? sizeof(float4) * (size_t)ntab : 0;
  if (pass == 0) return sizeof(float4) * SEG1_N * copies;
  return sizeof(float4) * (2 * SEG2_N * copies + (obs ? SEG_N : 0));
}

// resident CTAs per SM of the force-order builds with NT threads, for 2, 4
// and 8 atoms per load
template <int NT>
static cudaError_t build_occupancy_nt(int *out) {
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &out[0], nbr_build32_kernel<LIST_FO, NT, 2>, NT, 0);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&out[1], nbr_build32_kernel<LIST_FO, NT, 4>,
                                                      NT, 0);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&out[2], nbr_build32_kernel<LIST_FO, NT, 8>,
                                                      NT, 0);
  for (int i = 0; i < 3; i++) out[i] = out[i] < 1 ? 1 : out[i];
  return e;
}

// resident CTAs per SM of the force-order passes with or without energies
// (g_fo_per_sm[OBS]); every variant's shared-memory limit set
template <bool OBS>
static cudaError_t fo_occupancy() {
  int dummy = 0;
  int(&o)[3][2] = g_fo_per_sm[OBS];
  const size_t s0 = fo_pass_smem(0, EVAL_CHEBY, OBS, RHO_COPIES, 0),
               s1 = fo_pass_smem(1, EVAL_CHEBY, OBS, FORCE_COPIES, 0),
               st = fo_pass_smem(0, EVAL_TABLE, OBS, 1, FOTAB_MAX);
  cudaError_t e = pass_occupancy(fo_eam_pass1_kernel<EVAL_TABLE, false, OBS>, st,
                                 &o[0][EVAL_TABLE], FO1_THREADS);
  if (e == cudaSuccess)
    e = pass_occupancy(fo_eam_pass1_kernel<EVAL_CHEBY, false, OBS>, s0, &o[0][EVAL_CHEBY],
                       FO1_THREADS);
  if (e == cudaSuccess)
    e = pass_occupancy(fo_eam_pass2_kernel<EVAL_TABLE, false, OBS>, st, &o[1][EVAL_TABLE],
                       FO2_MAX_THREADS);
  if (e == cudaSuccess)
    e = pass_occupancy(fo_eam_pass2_kernel<EVAL_CHEBY, false, OBS>, s1, &o[1][EVAL_CHEBY],
                       FO2_MAX_THREADS);
  if (e == cudaSuccess) e = pass_occupancy(fo_lj_kernel<false, OBS>, 0, &o[2][0]);
  if (e == cudaSuccess)
    e = pass_occupancy(fo_eam_pass1_kernel<EVAL_TABLE, true, OBS>, st, &dummy, FO1_THREADS);
  if (e == cudaSuccess)
    e = pass_occupancy(fo_eam_pass1_kernel<EVAL_CHEBY, true, OBS>, s0, &dummy, FO1_THREADS);
  if (e == cudaSuccess)
    e = pass_occupancy(fo_eam_pass2_kernel<EVAL_TABLE, true, OBS>, st, &dummy, FO2_MAX_THREADS);
  if (e == cudaSuccess)
    e = pass_occupancy(fo_eam_pass2_kernel<EVAL_CHEBY, true, OBS>, s1, &dummy, FO2_MAX_THREADS);
  if (e == cudaSuccess) e = pass_occupancy(fo_lj_kernel<true, OBS>, 0, &dummy);
  return e;
}

// grid of a list build: one CTA per box, capped at the resident CTAs
static int build_grid(int nboxes, int per_sm) {
  const long cap = (long)g_num_sms * per_sm;
  return nboxes < cap ? nboxes : (int)cap;
}

// called on the current device before any launch or stream capture
cudaError_t prepare_force_kernels() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = pass_occupancy(eam_pass1_kernel<float, EVAL_TABLE>, pass_smem(0, EVAL_TABLE),
                       &g_pass_per_sm[0][EVAL_TABLE]);
  if (e == cudaSuccess)
    e = pass_occupancy(eam_pass1_kernel<float, EVAL_CHEBY>, pass_smem(0, EVAL_CHEBY),
                       &g_pass_per_sm[0][EVAL_CHEBY]);
  if (e == cudaSuccess)
    e = pass_occupancy(eam_pass2_kernel<float, EVAL_TABLE>, pass_smem(1, EVAL_TABLE),
                       &g_pass_per_sm[1][EVAL_TABLE]);
  if (e == cudaSuccess)
    e = pass_occupancy(eam_pass2_kernel<float, EVAL_CHEBY>, pass_smem(1, EVAL_CHEBY),
                       &g_pass_per_sm[1][EVAL_CHEBY]);
  if (e != cudaSuccess) return e;
  {
    // resident CTAs of the single-replica variants (the batch variants take
    // the same grids; they are grid-stride loops)
    e = fo_occupancy<false>();
    if (e == cudaSuccess) e = fo_occupancy<true>();
    if (e == cudaSuccess) e = build_occupancy_nt<64>(g_build_per_sm[0]);
    if (e == cudaSuccess) e = build_occupancy_nt<128>(g_build_per_sm[1]);
    if (e == cudaSuccess) e = build_occupancy_nt<256>(g_build_per_sm[2]);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &g_build_step_per_sm, nbr_build32_kernel<LIST_STEP>, NB_THREADS, 0);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &g_build_id_per_sm, nbr_build32_kernel<LIST_ID>, NB_THREADS, 0);
    g_build_step_per_sm = g_build_step_per_sm < 1 ? 1 : g_build_step_per_sm;
    g_build_id_per_sm = g_build_id_per_sm < 1 ? 1 : g_build_id_per_sm;
    return e;
  }
}

// grid of a pass: every atom one thread, capped at the resident CTAs
static int pass_grid(int pass, int eval, int ntot, bool fo = false,
                     int threads = PASS_THREADS, bool obs = true) {
  long need = (ntot + threads - 1) / threads;
  long cap = (long)g_num_sms * (fo ? g_fo_per_sm[obs][pass][eval] : g_pass_per_sm[pass][eval]);
  return (int)(need < cap ? need : cap);
}

// the force-order build at the tuned shape (threads per box x atoms per load)
template <int NT>
static void launch_fo_build_nt(const ForceArgs &A, float rc2, int na, cudaStream_t st) {
  const int *per_sm = g_build_per_sm[NT == 64 ? 0 : NT == 128 ? 1 : 2];
  if (na == 2)
    nbr_build32_kernel<LIST_FO, NT, 2><<<build_grid(A.g.nboxes, per_sm[0]), NT, 0, st>>>(A, rc2);
  else if (na == 8)
    nbr_build32_kernel<LIST_FO, NT, 8><<<build_grid(A.g.nboxes, per_sm[2]), NT, 0, st>>>(A, rc2);
  else
    nbr_build32_kernel<LIST_FO, NT, 4><<<build_grid(A.g.nboxes, per_sm[1]), NT, 0, st>>>(A, rc2);
}
static void launch_fo_build(const ForceArgs &A, float rc2, cudaStream_t st, const Tune *t) {
  // The default shape: 64 threads and 2 atoms against 128 and 4 take 200 / 243
  // us at 282,000 atoms (13,000 boxes) and 3.83 / 4.58 ms at 4 M, other shapes
  // between.  With few boxes (the SMs hold eight CTAs of 128 each) a box's own
  // time counts, and 128 threads are the faster ones: 100 steps of 4,000 atoms
  // (216 boxes) 2.39 / 2.36 ms.
  const bool few = A.g.nboxes < 8 * g_num_sms;
  const int nt = t && t->build_threads ? t->build_threads : few ? 128 : 64;
  const int na = t && t->build_atoms ? t->build_atoms : few ? 4 : 2;
  if (nt == 64) launch_fo_build_nt<64>(A, rc2, na, st);
  else if (nt == 256) launch_fo_build_nt<256>(A, rc2, na, st);
  else launch_fo_build_nt<128>(A, rc2, na, st);
}

void launch_nbr_build(const ForceArgs &A, float rc2b, cudaStream_t st, const Tune *tune) {
  if (A.fo.list)
    launch_fo_build(A, rc2b, st, tune);
  else if (A.pl.vlist)
    nbr_build32_kernel<LIST_ID><<<build_grid(A.g.nboxes, g_build_id_per_sm), NB_THREADS, 0, st>>>(
        A, rc2b);
  else
    // (boxes of a per-step list hold 10 to 20 atoms.  32 to 128 threads and 2 to
    // 8 atoms a load: 129 us, this, to 158 us at 256,000 atoms)
    nbr_build32_kernel<LIST_STEP>
        <<<build_grid(A.g.nboxes, g_build_step_per_sm), NB_THREADS, 0, st>>>(A, rc2b);
}

void launch_nbr_cut(const ForceArgs &A, float rc2b, cudaStream_t st) {
  const long threads = 32L * A.ntot;
  if (threads > 0)
    nbr_cut_kernel<<<(unsigned)((threads + NB_THREADS - 1) / NB_THREADS), NB_THREADS, 0, st>>>(
        A, rc2b);
}

// Threads per atom of a force-order pass (1: the thread-per-atom kernels).  The
// lines lie where the sums of both passes cross (us, Cu at 300 K, lattices
// without energies; 8, 4, 2, 1 threads):
//   Chebyshev   4,000 atoms  20.9  23.4  35.0  43.5
//              16,384        27.1  26.3  35.0  43.8
//              32,000          -   31.3  35.0  44.8
//              55,296          -   45.6  43.6  46.0
//             108,000          -   63.4  66.2  62.0
//   table      16,384        25.7  28.7    -   50.5
//              32,000        36.0  32.5    -   51.5
//             108,000          -   63.4  65.4  70.1
//             186,624          -   96.9  94.0 105.3
//             275,684          -  139.9 132.0 130.0
static int fo_lanes(int eval, int ntot) {
  if (eval == EVAL_TABLE)
    return ntot < 24000 ? 8 : ntot < 140000 ? 4 : ntot < 230000 ? 2 : 1;
  return ntot < 12000 ? 8 : ntot < 60000 ? 4 : 1;
}
// and of the LJ pass, whose lists are twice as long (us without / with energies;
// 8, 4, 1 threads):
//      4,000 atoms   9.1 / 11.3  12.5 / 13.9  50.3 / 49.7
//     16,384        11.1 / 14.4  13.1 / 15.4  49.9 / 50.3
//     23,328        15.9 / 20.5  13.5 / 15.6  55.2 / 54.6
//     27,436        16.6 / 22.8  14.1 / 16.6  58.7 / 57.3
//     55,296        25.0 / 34.4  23.3 / 28.9  56.4 / 56.7
//     97,556        40.1 / 54.4  34.2 / 42.9  59.0 / 60.7
//    108,000        43.5 / 59.6  35.7 / 44.1  57.7 / 59.1
//    143,748        55.4 / 76.0  45.4 / 56.8  60.5 / 62.0
// The second line is below where four threads and one cross (past 143,748).
static int fo_lj_lanes(int ntot) { return ntot < 24000 ? 8 : ntot < 100000 ? 4 : 1; }
bool fo_takes_pass2_threads(int potential, long ntot) {
  return potential != COMDGB_POT_LJ &&
         fo_lanes(potential == COMDGB_POT_EAM_TABLE ? EVAL_TABLE : EVAL_CHEBY,
                  (int)std::min(ntot, (long)INT_MAX)) == 1;
}
static unsigned fol_blocks(int ntot, int lanes) {
  return (unsigned)(((long)ntot * lanes + FOL_THREADS - 1) / FOL_THREADS);
}
template <int EVAL, bool OBS, int LANES, int COPIES>
static void launch_fol_eam(const ForceArgs &A, const EamPot<float, EVAL> &P, int pass,
                           cudaStream_t st) {
  const size_t smem = fo_pass_smem(pass, EVAL, OBS, COPIES, P.tab.n);
  const unsigned g = fol_blocks(A.ntot, LANES);
  const bool multi = A.g.nrep > 1;
  if (pass == 0) {
    if (multi) fol_eam_pass1_kernel<EVAL, true, OBS, LANES, COPIES><<<g, FOL_THREADS, smem, st>>>(A, P);
    else fol_eam_pass1_kernel<EVAL, false, OBS, LANES, COPIES><<<g, FOL_THREADS, smem, st>>>(A, P);
  } else {
    if (multi) fol_eam_pass2_kernel<EVAL, true, OBS, LANES, COPIES><<<g, FOL_THREADS, smem, st>>>(A, P);
    else fol_eam_pass2_kernel<EVAL, false, OBS, LANES, COPIES><<<g, FOL_THREADS, smem, st>>>(A, P);
  }
}
template <bool OBS, int LANES>
static void launch_fol_lj(const ForceArgs &A, const LjPot<float> &P, cudaStream_t st) {
  const unsigned g = fol_blocks(A.ntot, LANES);
  if (A.g.nrep > 1) fol_lj_kernel<true, OBS, LANES><<<g, FOL_THREADS, 0, st>>>(A, P);
  else fol_lj_kernel<false, OBS, LANES><<<g, FOL_THREADS, 0, st>>>(A, P);
}

template <int EVAL, bool OBS>
static void launch_fo_eam_obs(const ForceArgs &A, const EamPot<float, EVAL> &P, int pass,
                              cudaStream_t st, const Tune *tune) {
  // the tables once a CTA, or (table potential) from global memory
  constexpr int copies = EVAL == EVAL_TABLE ? 0 : 1;
  switch (fo_lanes(EVAL, A.ntot)) {
    case 8: return launch_fol_eam<EVAL, OBS, 8, copies>(A, P, pass, st);
    case 4: return launch_fol_eam<EVAL, OBS, 4, copies>(A, P, pass, st);
    case 2: return launch_fol_eam<EVAL, OBS, 2, copies>(A, P, pass, st);
  }
  const size_t smem = fo_pass_smem(pass, EVAL, OBS, pass == 0 ? RHO_COPIES : FORCE_COPIES, P.tab.n);
  const bool multi = A.g.nrep > 1;
  if (pass == 0) {
    const int g0 = pass_grid(0, EVAL, A.ntot, true, FO1_THREADS, OBS);
    if (multi) fo_eam_pass1_kernel<EVAL, true, OBS><<<g0, FO1_THREADS, smem, st>>>(A, P);
    else fo_eam_pass1_kernel<EVAL, false, OBS><<<g0, FO1_THREADS, smem, st>>>(A, P);
  } else {
    const int threads = tune ? tune->pass2_threads : FO2_MAX_THREADS;
    const int tuned = tune ? (OBS ? tune->pass2_blocks : tune->pass2_blocks_fast) : 0;
    int g1;
    if (tuned > 0) {
      const long need = ((long)A.ntot + threads - 1) / threads;
      g1 = (int)(need < tuned ? need : tuned);
    } else {
      g1 = pass_grid(1, EVAL, A.ntot, true, threads, OBS);
    }
    if (multi) fo_eam_pass2_kernel<EVAL, true, OBS><<<g1, threads, smem, st>>>(A, P);
    else fo_eam_pass2_kernel<EVAL, false, OBS><<<g1, threads, smem, st>>>(A, P);
  }
}

template <int EVAL>
void launch_fo_eam(const ForceArgs &A, const EamPot<float, EVAL> &P, int pass, cudaStream_t st,
                   const Tune *tune, bool obs) {
  if (A.ntot <= 0) return;
  if (obs) launch_fo_eam_obs<EVAL, true>(A, P, pass, st, tune);
  else launch_fo_eam_obs<EVAL, false>(A, P, pass, st, tune);
}
template void launch_fo_eam<EVAL_TABLE>(const ForceArgs &, const EamPot<float, EVAL_TABLE> &,
                                        int, cudaStream_t, const Tune *, bool);
template void launch_fo_eam<EVAL_CHEBY>(const ForceArgs &, const EamPot<float, EVAL_CHEBY> &,
                                        int, cudaStream_t, const Tune *, bool);

template <int EVAL, bool OBS>
static int fo_pass2_per_sm(bool multi, int threads) {
  int per_sm = 0;
  const size_t smem = fo_pass_smem(1, EVAL, OBS, FORCE_COPIES, FOTAB_MAX);
  const cudaError_t e =
      multi ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                  &per_sm, fo_eam_pass2_kernel<EVAL, true, OBS>, threads, smem)
            : cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                  &per_sm, fo_eam_pass2_kernel<EVAL, false, OBS>, threads, smem);
  return e != cudaSuccess || per_sm < 1 ? 1 : per_sm;
}

int fo_pass2_blocks(int eval, bool multi, int threads, bool obs) {
  int per_sm;
  if (eval == EVAL_CHEBY)
    per_sm = obs ? fo_pass2_per_sm<EVAL_CHEBY, true>(multi, threads)
                 : fo_pass2_per_sm<EVAL_CHEBY, false>(multi, threads);
  else
    per_sm = obs ? fo_pass2_per_sm<EVAL_TABLE, true>(multi, threads)
                 : fo_pass2_per_sm<EVAL_TABLE, false>(multi, threads);
  return per_sm * g_num_sms;
}

void launch_fo_lj(const ForceArgs &A, const LjPot<float> &P, cudaStream_t st, bool obs) {
  if (A.ntot <= 0) return;
  if (!obs)
    fo_lj_settle_kernel<<<(A.ntot + PASS_THREADS - 1) / PASS_THREADS, PASS_THREADS, 0, st>>>(A);
  const int lanes = fo_lj_lanes(A.ntot);
  if (lanes > 1) {
    if (lanes == 8) obs ? launch_fol_lj<true, 8>(A, P, st) : launch_fol_lj<false, 8>(A, P, st);
    else obs ? launch_fol_lj<true, 4>(A, P, st) : launch_fol_lj<false, 4>(A, P, st);
    return;
  }
  const int grid = pass_grid(2, 0, A.ntot, true, PASS_THREADS, obs);
  const bool multi = A.g.nrep > 1;
  if (obs) {
    if (multi) fo_lj_kernel<true, true><<<grid, PASS_THREADS, 0, st>>>(A, P);
    else fo_lj_kernel<false, true><<<grid, PASS_THREADS, 0, st>>>(A, P);
  } else {
    if (multi) fo_lj_kernel<true, false><<<grid, PASS_THREADS, 0, st>>>(A, P);
    else fo_lj_kernel<false, false><<<grid, PASS_THREADS, 0, st>>>(A, P);
  }
}

template <>
void launch_eam_pass1<float, EVAL_TABLE>(const ForceArgs &A, const EamPot<float, EVAL_TABLE> &P,
                                      cudaStream_t st) {
  if (A.ntot <= 0) return;
  const size_t smem = P.seg.n > 0 ? pass_smem(0, EVAL_TABLE) : 0;
  eam_pass1_kernel<float, EVAL_TABLE><<<pass_grid(0, EVAL_TABLE, A.ntot), PASS_THREADS, smem, st>>>(A, P);
}
template <>
void launch_eam_pass1<float, EVAL_CHEBY>(const ForceArgs &A, const EamPot<float, EVAL_CHEBY> &P,
                                      cudaStream_t st) {
  if (A.ntot <= 0) return;
  const size_t smem = P.seg.n > 0 ? pass_smem(0, EVAL_CHEBY) : 0;
  eam_pass1_kernel<float, EVAL_CHEBY><<<pass_grid(0, EVAL_CHEBY, A.ntot), PASS_THREADS, smem, st>>>(A, P);
}
template <>
void launch_eam_pass2<float, EVAL_TABLE>(const ForceArgs &A, const EamPot<float, EVAL_TABLE> &P,
                                      cudaStream_t st) {
  if (A.ntot <= 0) return;
  const size_t smem = P.seg.n > 0 ? pass_smem(1, EVAL_TABLE) : 0;
  eam_pass2_kernel<float, EVAL_TABLE><<<pass_grid(1, EVAL_TABLE, A.ntot), PASS_THREADS, smem, st>>>(A, P);
}
template <>
void launch_eam_pass2<float, EVAL_CHEBY>(const ForceArgs &A, const EamPot<float, EVAL_CHEBY> &P,
                                      cudaStream_t st) {
  if (A.ntot <= 0) return;
  const size_t smem = P.seg.n > 0 ? pass_smem(1, EVAL_CHEBY) : 0;
  eam_pass2_kernel<float, EVAL_CHEBY><<<pass_grid(1, EVAL_CHEBY, A.ntot), PASS_THREADS, smem, st>>>(A, P);
}
template <>
void launch_lj<float>(const ForceArgs &A, const LjPot<float> &P, cudaStream_t st) {
  if (A.ntot > 0) lj_pass_kernel<float><<<(A.ntot + 127) / 128, 128, 0, st>>>(A, P);
}

}  // namespace cg
