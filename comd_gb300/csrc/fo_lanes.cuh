// fo_lanes.cuh -- the force-order passes with LANES threads per atom.
//
// One thread per atom (force_kernels.cuh) fills the 152 SMs from about
// 155,000 atoms on; below, a pass takes as long as one thread's walk over its
// list, 20 us whatever the size.  Here LANES neighbouring threads share a
// list (lane l takes entries l, l + LANES, ..., FOL_BATCH gathers in flight),
// their compensated sums are added in a fixed order, and lane k < 3 makes
// component k of the step update.  The Chebyshev tables are staged once
// instead of in 8 interleaved copies (8 KB a CTA instead of 64 KB: less to
// load than the bank conflicts cost at these sizes) and the table potential's
// are read from global memory.  At 4,000 atoms both Chebyshev passes took 46.3
// us with one thread an atom and take 20.9, the table potential's 78.7 and
// 20.9; fo_lanes in force_mixed.cu has the other sizes.
#pragma once

#include "force_kernels.cuh"

namespace cg {

constexpr int FOL_THREADS = 128;
constexpr int FOL_BATCH = 3;  // entries per lane loaded before the first is used

// the sum of the lanes' compensated sums, lane by lane (all lanes get it)
template <int LANES>
__device__ __forceinline__ KSum ksum_lanes(const KSum &k) {
  KSum t;
  t.zero();
#pragma unroll
  for (int l = 0; l < LANES; l++) {
    t.add(__shfl_sync(0xffffffffu, k.s, l, LANES));
    t.add(-__shfl_sync(0xffffffffu, k.c, l, LANES));
  }
  return t;
}

// fn(a, live) for the atom of this thread's group.  The groups of a warp stay
// together: past the last atom they repeat it and store nothing (live).
template <int LANES, class F>
__device__ __forceinline__ void fol_atom(int ntot, F &&fn) {
  const long q = (long)blockIdx.x * FOL_THREADS + threadIdx.x, at = q / LANES;
  if ((q & ~31L) / LANES < ntot) fn(at < ntot ? (int)at : ntot - 1, at < ntot);
}

// this lane's entries of a force-order list (skin or cut) of n entries:
// fn(q, dx, dy, dz, r2), q the neighbour's record of pj (pos or pf)
template <bool MULTI, int LANES, class F>
__device__ __forceinline__ void fol_walk(const ForceArgs &A, const uint32_t *list, int n, int a,
                                         int slot, int sub, float4 pi, const float4 *pj, F &&fn) {
  const FoFrame fr = fo_frame<MULTI>(A, slot);
  const uint32_t *lst = list + fo_row(a, A.fo.vcap);
  for (int t0 = sub; t0 < n; t0 += LANES * FOL_BATCH) {
    uint32_t p[FOL_BATCH];
    float4 q[FOL_BATCH];
#pragma unroll
    for (int u = 0; u < FOL_BATCH; u++) p[u] = __ldg(lst + (size_t)min(t0 + u * LANES, n - 1) * 32);
#pragma unroll
    for (int u = 0; u < FOL_BATCH; u++) q[u] = __ldg(pj + (p[u] >> 6));
#pragma unroll
    for (int u = 0; u < FOL_BATCH; u++) {
      float dx, dy, dz;
      const float r2 = fo_dr(fr, p[u], pi, q[u], dx, dy, dz);
      if (t0 + u * LANES < n) fn(q[u], dx, dy, dz, r2);
    }
  }
}

// an overflowed skin list: the stencil, by lane 0
template <bool NEED_FI, class F>
__device__ __forceinline__ void fol_scan(const ForceArgs &A, int slot, int sub, float rc2, F &&fn) {
  if (sub != 0) return;
  const float4 p = __ldg(A.s.pos32 + slot);
  scan_stencil<float>(A, slot >> 6, slot & 63, p.x, p.y, p.z, rc2,
                      [&](int js, float dx, float dy, float dz, float r2) {
                        fn(NEED_FI ? __ldg(A.s.fi32 + js) : 0.f, dx, dy, dz, r2);
                      });
}

// fo_eam_pass1_kernel with LANES threads per atom: the same cut list, in the
// same order (each round's hits packed by a ballot of the group)
template <int EVAL, bool MULTI, bool OBS, int LANES, int COPIES>
__device__ __forceinline__ void fol_density(const ForceArgs &A, const EamPot<float, EVAL> &P,
                                            const float4 *seg_sm, int a, int sub, bool live) {
  const float rc2 = P.rc2;
  const int slot = A.fo.slot[a];
  const float4 pi = A.fo.pos[a];
  const int n = A.fo.n[a];
  KSum rh;
  rh.zero();
  int cnt = 0, ncut;
  if (n > A.fo.vcap) {
    fol_scan<false>(A, slot, sub, rc2, [&](float, float, float, float, float r2) {
      if (r2 > rc2) return;
      cnt++;
      float rho;
      if (!fo_rho<COPIES>(P, seg_sm, r2, rho)) rho = fo_rho_series(P, r2);
      rh.add(rho);
    });
    ncut = A.fo.vcap + 1;
  }
  // (groups of one warp may differ in n and in overflow: every group takes
  // the rounds of the longest list, the ballots being the warp's)
  const int m = n > A.fo.vcap ? 0 : n;
  int most = m;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  const FoFrame fr = fo_frame<MULTI>(A, slot);
  const size_t row = fo_row(a, A.fo.vcap);
  const uint32_t *lst = A.fo.list + row;
  uint32_t *cut = A.fo.cut + row;
  const unsigned group = (threadIdx.x & 31) / LANES * LANES;
  bool low = false;
  for (int t0 = 0; t0 < most; t0 += LANES * FOL_BATCH) {
    uint32_t p[FOL_BATCH];
    float4 q[FOL_BATCH];
#pragma unroll
    for (int u = 0; u < FOL_BATCH; u++) {
      const int t = t0 + u * LANES + sub;
      p[u] = t < m ? __ldg(lst + (size_t)t * 32) : 0u;
    }
#pragma unroll
    for (int u = 0; u < FOL_BATCH; u++) q[u] = __ldg(A.fo.pos + (p[u] >> 6));
#pragma unroll
    for (int u = 0; u < FOL_BATCH; u++) {
      float dx, dy, dz;
      const float r2 = fo_dr(fr, p[u], pi, q[u], dx, dy, dz);
      const bool hit = t0 + u * LANES + sub < m && !(r2 > rc2);
      const uint32_t hits = (__ballot_sync(0xffffffffu, hit) >> group) & ((1u << LANES) - 1u);
      if (hit) {
        if (live) cut[(size_t)(cnt + __popc(hits & ((1u << sub) - 1u))) * 32] = p[u];
        float rho;
        if (fo_rho<COPIES>(P, seg_sm, r2, rho)) rh.add(rho);
        else low = true;
      }
      cnt += __popc(hits);
    }
  }
  if (low)  // pairs below the table: the series, in a second sweep
    fol_walk<MULTI, LANES>(A, A.fo.list, m, a, slot, sub, pi, A.fo.pos,
                           [&](float4, float, float, float, float r2) {
                             if (!(r2 > rc2) && below_seg(P, r2)) rh.add(fo_rho_series(P, r2));
                           });
  if (n <= A.fo.vcap) ncut = cnt;
  __syncwarp();
  rh = ksum_lanes<LANES>(rh);
  if (sub == 0 && live) fo_density_store<EVAL, OBS>(A, P, rh, a, slot, pi, cnt, ncut);
}
template <int EVAL, bool MULTI, bool OBS, int LANES, int COPIES>
__global__ void __launch_bounds__(FOL_THREADS)
    fol_eam_pass1_kernel(ForceArgs A, const __grid_constant__ EamPot<float, EVAL> P) {
  extern __shared__ float4 seg_sm[];
  stage_rho<COPIES>(seg_sm, P);
  const float4 *sm = fo_copy<EVAL, COPIES>(seg_sm);
  fol_atom<LANES>(A.ntot, [&](int a, bool live) {
    fol_density<EVAL, MULTI, OBS, LANES, COPIES>(A, P, sm, a, threadIdx.x % LANES, live);
  });
}

// fo_force_end with lane k < 3 of the group making component k (all lanes of
// the warp call it; fx, fy, fz are the group's sums)
template <int LANES>
__device__ __forceinline__ void fol_force_end(const ForceArgs &A, int a, int slot, int sub,
                                              bool live, bool fuse, float fx, float fy, float fz) {
  if (!fuse) {
    if (sub == 0 && live) A.fo.force[a] = make_float4(fx, fy, fz, 0.f);
    return;
  }
  if (LANES < 4) {
    if (sub == 0 && live) fo_force_end(A, a, slot, true, fx, fy, fz);
    return;
  }
  const int k = min(sub, 2), b = slot >> 6;
  const bool mine = sub < 3 && live;
  const float f = k == 0 ? fx : k == 1 ? fy : fz;
  double *pk = reinterpret_cast<double *>(A.s.p + slot) + k;
  double *rk = reinterpret_cast<double *>(A.s.r + slot) + k;
  const double p = fma(-A.vv_dt, (double)f, *pk);
  const double r = fma(p, A.vv_c, *rk);
  const RepGeo &R = rep_of(A.g, b);
  const float4 q = A.fo.ref[a];
  const float qk = k == 0 ? q.x : k == 1 ? q.y : q.z;
  const int sh = 10 * k;
  int db = ((__ldg(A.g.boxc + b) >> sh) & 1023) -
           ((__ldg(A.g.boxc + __float_as_int(q.w)) >> sh) & 1023);
  if (A.g.periodic) {
    if (db > 1) db -= R.nbx[k];
    else if (db < -1) db += R.nbx[k];
  }
  float v = d2f_rn(r - R.half[k]);
  const bool far = db > 1 || db < -1 || !(fabsf(v) <= 1.5f * R.hi[k]);
  if (db != 0) v = d2f_rn(fma((double)db, R.boxsize[k], r - R.half[k]));
  const float d = v - qk;
  if (mine) {
    *pk = p;
    *rk = r;
    reinterpret_cast<float *>(A.fo.pos + a)[k] = v;
  }
  // |d|^2 in the order of fo_track_at, the skin test on the first lane
  const float d0 = __shfl_sync(0xffffffffu, d, 0, LANES), d1 = __shfl_sync(0xffffffffu, d, 1, LANES),
              d2 = __shfl_sync(0xffffffffu, d, 2, LANES);
  const unsigned away = __ballot_sync(0xffffffffu, far && mine);
  const unsigned group = (threadIdx.x & 31) / LANES * LANES;
  if (sub != 0 || !live) return;
  const float s = fmaf(d2, d2, fmaf(d1, d1, fmaf(d0, d0, 0.f)));
  if (a == 0) cond_pending(A.cond, A.status);
  if ((((away >> group) & 7u) != 0 || !(s <= A.fo.half_skin2)) &&
      atomicExch(A.status + ST_REBUILD, 1) == 0 && A.cond)
    set_condition(A.cond);
}

// fo_eam_pass2_kernel with LANES threads per atom
template <int EVAL, bool MULTI, bool OBS, int LANES, int COPIES>
__device__ __forceinline__ void fol_force(const ForceArgs &A, const EamPot<float, EVAL> &P,
                                          const float4 *sm, const float4 *phi_sm, int a, int sub,
                                          bool live, bool fuse) {
  const float rc2 = P.rc2;
  const int slot = A.fo.slot[a];
  const float4 pi = A.fo.pf[a];
  const float fii = pi.w;
  const int n = A.fo.ncut[a];
  ForceSums<OBS> acc;
  acc.zero();
  bool low = false;
  auto add = [&](float fj, float dx, float dy, float dz, float r2) {
    if (r2 > rc2) return;
    float phi = 0.f, wphi, wrho;
    if (!fo_pair<OBS, COPIES>(P, sm, phi_sm, r2, phi, wphi, wrho)) {
      low = true;
      return;
    }
    const float we = r2 < rc2 ? (fii + fj) * wrho : 0.f;
    acc.add(phi, wphi, we, dx, dy, dz);
  };
  auto add_low = [&](float fj, float dx, float dy, float dz, float r2) {
    if (r2 > rc2 || !below_seg(P, r2)) return;
    float phi, wphi, wrho;
    fo_pair_series(P, r2, phi, wphi, wrho);
    const float we = r2 < rc2 ? (fii + fj) * wrho : 0.f;
    acc.add(phi, wphi, we, dx, dy, dz);
  };
  auto entry = [](auto &&fn) {
    return [&fn](float4 q, float dx, float dy, float dz, float r2) { fn(q.w, dx, dy, dz, r2); };
  };
  if (n > A.fo.vcap) {
    fol_scan<true>(A, slot, sub, rc2, add);
    if (low) fol_scan<true>(A, slot, sub, rc2, add_low);
  } else {
    fol_walk<MULTI, LANES>(A, A.fo.cut, n, a, slot, sub, pi, A.fo.pf, entry(add));
    if (low) fol_walk<MULTI, LANES>(A, A.fo.cut, n, a, slot, sub, pi, A.fo.pf, entry(add_low));
  }
  __syncwarp();
  acc.fx = ksum_lanes<LANES>(acc.fx);
  acc.fy = ksum_lanes<LANES>(acc.fy);
  acc.fz = ksum_lanes<LANES>(acc.fz);
  const float fx = acc.fx.valuef(), fy = acc.fy.valuef(), fz = acc.fz.valuef();
  fol_force_end<LANES>(A, a, slot, sub, live, fuse, fx, fy, fz);
  if (OBS) {
    acc.ep = ksum_lanes<LANES>(acc.ep);
    acc.sx = ksum_lanes<LANES>(acc.sx);
    if (sub != 0 || !live) return;
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
template <int EVAL, bool MULTI, bool OBS, int LANES, int COPIES>
__global__ void __launch_bounds__(FOL_THREADS)
    fol_eam_pass2_kernel(ForceArgs A, const __grid_constant__ EamPot<float, EVAL> P) {
  extern __shared__ float4 seg_sm[];
  stage_force<COPIES, OBS>(seg_sm, P);
  const float4 *sm = fo_copy<EVAL, COPIES>(seg_sm), *phi_sm = seg_sm + 2 * SEG2_N * COPIES;
  const bool fuse = !OBS && *(volatile const int *)(A.status + ST_FUSE);
  fol_atom<LANES>(A.ntot, [&](int a, bool live) {
    fol_force<EVAL, MULTI, OBS, LANES, COPIES>(A, P, sm, phi_sm, a, threadIdx.x % LANES, live,
                                               fuse);
  });
}

// fo_lj_kernel with LANES threads per atom
template <bool MULTI, bool OBS, int LANES>
__device__ __forceinline__ void fol_lj(const ForceArgs &A, const LjPot<float> &P, int a, int sub,
                                       bool live, bool fuse) {
  const float s6 = P.s6, s12 = P.s6x12, c4 = P.eps4s6, rc2 = P.rc2;
  const int slot = A.fo.slot[a], n = A.fo.n[a];
  KSum fx, fy, fz, ep, sx;
  fx.zero(); fy.zero(); fz.zero(); ep.zero(); sx.zero();
  int cnt = 0;
  auto add = [&](float, float dx, float dy, float dz, float r2) {
    if (r2 > rc2) return;
    cnt++;
    const float ir2 = 1.0f / r2;
    const float r6 = ir2 * ir2 * ir2;
    if (OBS) ep.add(0.5f * r6 * (s6 * r6 - 1.0f));
    const float fr = c4 * r6 * ir2 * (s12 * r6 - 6.0f);
    fx.add(dx * fr);
    fy.add(dy * fr);
    fz.add(dz * fr);
    if (OBS) sx.add(fr * dx * dx);
  };
  const float4 *pj = fo_lj_pos<OBS>(A);
  if (n > A.fo.vcap)
    fol_scan<false>(A, slot, sub, rc2, add);
  else
    fol_walk<MULTI, LANES>(A, A.fo.list, n, a, slot, sub, pj[a], pj,
                           [&](float4, float dx, float dy, float dz, float r2) {
                             add(0.f, dx, dy, dz, r2);
                           });
  __syncwarp();
  fx = ksum_lanes<LANES>(fx);
  fy = ksum_lanes<LANES>(fy);
  fz = ksum_lanes<LANES>(fz);
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  fol_force_end<LANES>(A, a, slot, sub, live, fuse, fx.valuef(), fy.valuef(), fz.valuef());
  if (OBS) {
    ep = ksum_lanes<LANES>(ep);
    sx = ksum_lanes<LANES>(sx);
  }
  if (sub != 0 || !live) return;
  if (OBS) {
    const int b = slot >> 6;
    d4 fo;
    fo.x = fx.value();
    fo.y = fy.value();
    fo.z = fz.value();
    fo.w = ep.value();
    A.s.f[slot] = fo;
    if (A.host_f) fo_host_f(A, slot, fo);
    int ne = A.et.n[b], nonempty = 0;
    for (int e = 0; e < ne; e++) nonempty += A.s.natoms[A.et.box[b * CG_NNBR + e]] > 0;
    const d4 p = A.s.p[slot];
    const double kin = __ddiv_rn(__dmul_rn(p.x, p.x), A.s.mass[slot]);
    A.atom_stress[a] = sx.value() - (double)nonempty * kin;
  }
  A.npair[a] = cnt;
}
template <bool MULTI, bool OBS, int LANES>
__global__ void __launch_bounds__(FOL_THREADS)
    fol_lj_kernel(ForceArgs A, LjPot<float> P) {
  const bool fuse = !OBS && *(volatile const int *)(A.status + ST_FUSE);
  fol_atom<LANES>(A.ntot, [&](int a, bool live) {
    fol_lj<MULTI, OBS, LANES>(A, P, a, threadIdx.x % LANES, live, fuse);
  });
}

}  // namespace cg
