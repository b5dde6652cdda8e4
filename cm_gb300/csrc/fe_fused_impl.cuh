// libcm_fe: the staged assembly in one launch, device code and launcher shared
// by the mixed-precision (fe_mixed.cu) and FP64 (fe_fp64.cu) translation units.
#pragma once
#include "fe_mixed_impl.cuh"
#include "fe_surface_impl.cuh"

#include <atomic>

namespace {

// Staged assembly in one launch: CTAs take element groups in element order
// from a global counter, store each group's records (and the surface-pressure
// faces of its boundary elements), then count, for every row node of the
// group, how many of the elements around the node are done.  The CTA whose
// count completes a node gathers that node's rows right away, while the
// records of the elements around it are still in L2 -- no CTA ever waits for
// another.  Sh: elements per group EG, threads NT and CTAs per SM MINB.
//
// Bound by the FP64 pipe and by the barriers between a group's phases: the
// 32^3 box's mixed assembly takes 1.78 ms (2.72 with the contraction on the
// tensor cores and records laid out by element), without the gathers 1.26.  By
// the counters of the 16^3 box it issues 600 FP64 warp instructions an element
// (480 of them element work), which keep that pipe 55 % busy.  The 16^3 box's
// FP64 Jacobian takes 1.10 ms (6.5 with one launch per colour contracting over
// all Gauss points), without the gathers 0.91: 3,715 an element, 77 % busy.
template <int N1, int PM, class T, class H, class Sh>
__global__ void __launch_bounds__(Sh::NT, Sh::MINB) fe_fused_kernel(KParams P, cmfe::StageOut so, cmfe::FusedArgs F) {
  using C = MixCfg<N1, PM, Sh::EG, T, Sh::NT>;
  constexpr int NPE = C::NPE, NPP = C::NPP, EG = C::EG;
  static_assert(C::THREADS / 32 * (int)sizeof(SurfWarpSmem) <= C::O_NODE1 - C::O_Z, "surface scratch");
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_grp, s_nready, s_next;
  mix_tables<N1, PM, EG, T, H, Sh::NT>(P, sm);
  const int ngroups = min((P.count + EG - 1) / EG, F.g1);
  const bool p4_first = (blockIdx.x / P.wave) & 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* s_node = reinterpret_cast<const int*>(sm + C::O_NODE1);
  unsigned char* scratch = sm + C::O_Z;
  for (;;) {
    if (tid == 0) s_grp = F.g0 + atomicAdd(F.work, 1);
    __syncthreads();
    const int grp = s_grp;
    if (grp >= ngroups) break;
    mix_group<N1, PM, EG, T, H, 1, Sh::NT>(P, nullptr, P.count, grp, p4_first, sm, &so);
    const int nvalid = min(EG, P.count - grp * EG);
    __syncthreads();  // the group's records are complete within the CTA; the scratch is free
    if (F.bmask) {
      SurfWarpSmem* ws = reinterpret_cast<SurfWarpSmem*>(scratch);
      for (int el = warp; el < nvalid; el += C::THREADS / 32) {
        const int e = grp * EG + el;
        if (F.bmask[e]) surface_element<N1, NPP, T>(P, e, F.bmask, 2, 1, ws[warp], lane, &so);
      }
      __syncthreads();
    }
    GroupGather<NPE, NPP, EG, Sh::NT, T>::run(P, so, F, s_node, nvalid, scratch, &s_nready, &s_next);
  }
}

// Resident blocks per SM of the fused kernel (its shared-memory attribute set
// once per device first); 0 on error, with the error in *err.
template <int N1, int PM, class T, class H, class Sh>
int fused_per_sm(cudaError_t* err) {
  using C = MixCfg<N1, PM, Sh::EG, T, Sh::NT>;
  static std::atomic<bool> attr[64];
  auto kern = fe_fused_kernel<N1, PM, T, H, Sh>;
  int dev = 0;
  *err = cudaGetDevice(&dev);
  if (*err != cudaSuccess) return 0;
  if (dev < 0 || dev >= 64 || !attr[dev].load()) {
    *err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM1);
    if (*err != cudaSuccess) return 0;
    if (dev >= 0 && dev < 64) attr[dev].store(true);
  }
  int per_sm = 0;
  *err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::THREADS, C::SMEM1);
  if (*err != cudaSuccess) return 0;
  return per_sm < 1 ? 1 : per_sm;
}

// Groups [fa.g0, fa.g1) in one launch.  Launches of one assembly share nothing
// but the node counts, which are atomic, so they may run at the same time.
template <int N1, int PM, class T, class H, class Sh>
int launch_fused_t(const KParams& kp, const cmfe::StageOut& so, cmfe::FusedArgs fa, int num_sms, cudaStream_t st) {
  using C = MixCfg<N1, PM, Sh::EG, T, Sh::NT>;
  auto kern = fe_fused_kernel<N1, PM, T, H, Sh>;
  cudaError_t e;
  const int per_sm = fused_per_sm<N1, PM, T, H, Sh>(&e);
  if (!per_sm) return (int)e;
  const int all = (kp.count + C::EG - 1) / C::EG;
  if (fa.g1 > all) fa.g1 = all;
  if (fa.g0 < 0 || fa.g0 >= fa.g1) return (int)cudaSuccess;  // no groups in this launch
  const int groups = fa.g1 - fa.g0;
  int grid = per_sm * num_sms;
  grid = grid < groups ? grid : groups;
  grid = grid < 1 ? 1 : grid;
  KParams k = kp;
  k.wave = num_sms > 0 ? num_sms : 1;
  kern<<<grid, C::THREADS, C::SMEM1, st>>>(k, so, fa);
  return (int)cudaGetLastError();
}

}  // namespace
