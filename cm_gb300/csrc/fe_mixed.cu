// libcm_fe: mixed-precision element assembly (sm_103a), one launch per
// element colour of one equations set.  The device code is in
// fe_mixed_impl.cuh.
#include "fe_mixed_impl.cuh"
#include "fe_surface_impl.cuh"

#include <atomic>


namespace {

template <int N1, int PM, class H>
__global__ void __launch_bounds__(256, MixCfg<N1, PM>::MINB) fe_mixed_kernel(KParams P) {
  using C = MixCfg<N1, PM>;
  extern __shared__ __align__(16) unsigned char sm[];
  mix_tables<N1, PM, C::EG, float, H>(P, sm);
  const int ngroups = (P.count + C::EG - 1) / C::EG;
  const bool p4_first = (blockIdx.x / P.wave) & 1;
  for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) mix_group<N1, PM, C::EG, float, H>(P, P.elems, P.count, grp, p4_first, sm);
}

// Elements per group, threads per CTA and CTAs per SM of the fused kernel.
template <int N1, int PM>
struct FusedShape {
  static constexpr int EG = N1 == 3 ? 3 : 4;
  static constexpr int NT = 256;
  static constexpr int MINB = N1 == 3 ? 3 : 2;
};

// Staged assembly in one launch: CTAs take element groups in element order
// from a global counter, store each group's records (and the surface-pressure
// faces of its boundary elements), then count, for every row node of the
// group, how many of the elements around the node are done.  The CTA whose
// count completes a node gathers that node's rows right away, while the
// records of the elements around it are still in L2 -- no CTA ever waits for
// another.
template <int N1, int PM, class H>
__global__ void __launch_bounds__(FusedShape<N1, PM>::NT, FusedShape<N1, PM>::MINB)
    fe_mixed_fused_kernel(KParams P, cmfe::StageOut so, cmfe::FusedArgs F) {
  using Sh = FusedShape<N1, PM>;
  using C = MixCfg<N1, PM, Sh::EG, float, Sh::NT>;
  constexpr int NPE = C::NPE, NPP = C::NPP, EG = C::EG;
  static_assert(C::THREADS / 32 * (int)sizeof(SurfWarpSmem) <= C::O_NODE1 - C::O_Z, "surface scratch");
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_grp, s_nready, s_next;
  mix_tables<N1, PM, EG, float, H, Sh::NT>(P, sm);
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
    mix_group<N1, PM, EG, float, H, 1, Sh::NT>(P, nullptr, P.count, grp, p4_first, sm, &so);
    const int nvalid = min(EG, P.count - grp * EG);
    __syncthreads();  // the group's records are complete within the CTA; the scratch is free
    if (F.bmask) {
      SurfWarpSmem* ws = reinterpret_cast<SurfWarpSmem*>(scratch);
      for (int el = warp; el < nvalid; el += C::THREADS / 32) {
        const int e = grp * EG + el;
        if (F.bmask[e]) surface_element<N1, NPP, float>(P, e, F.bmask, 2, 1, ws[warp], lane, &so);
      }
      __syncthreads();
    }
    GroupGather<NPE, NPP, EG, Sh::NT, float>::run(P, so, F, s_node, nvalid, scratch, &s_nready, &s_next);
  }
}

// Resident blocks per SM of the fused kernel (its shared-memory attribute set
// once per device first); 0 on error, with the error in *err.
template <int N1, int PM, class H>
int fused_per_sm(cudaError_t* err) {
  using C = MixCfg<N1, PM, FusedShape<N1, PM>::EG, float, FusedShape<N1, PM>::NT>;
  constexpr int SMEM = C::SMEM1;
  static std::atomic<bool> attr[64];
  auto kern = fe_mixed_fused_kernel<N1, PM, H>;
  int dev = 0;
  *err = cudaGetDevice(&dev);
  if (*err != cudaSuccess) return 0;
  if (dev < 0 || dev >= 64 || !attr[dev].load()) {
    *err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (*err != cudaSuccess) return 0;
    if (dev >= 0 && dev < 64) attr[dev].store(true);
  }
  int per_sm = 0;
  *err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::THREADS, SMEM);
  if (*err != cudaSuccess) return 0;
  return per_sm < 1 ? 1 : per_sm;
}

template <int N1, int PM, class H>
int launch_fused_t(const KParams& kp, const cmfe::StageOut& so, cmfe::FusedArgs fa, int num_sms,
                   cudaStream_t st) {
  using C = MixCfg<N1, PM, FusedShape<N1, PM>::EG, float, FusedShape<N1, PM>::NT>;
  auto kern = fe_mixed_fused_kernel<N1, PM, H>;
  cudaError_t e;
  const int per_sm = fused_per_sm<N1, PM, H>(&e);
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

template <class H>
int launch_fused_h(const HostSetup& s, const KParams& kp, const cmfe::StageOut& so, const cmfe::FusedArgs& fa,
                   int num_sms, cudaStream_t st) {
  if (s.n1 == 2 && s.pmode == 0) return launch_fused_t<2, 0, H>(kp, so, fa, num_sms, st);
  if (s.n1 == 2 && s.pmode == 1) return launch_fused_t<2, 1, H>(kp, so, fa, num_sms, st);
  if (s.n1 == 3 && s.pmode == 0) return launch_fused_t<3, 0, H>(kp, so, fa, num_sms, st);
  return launch_fused_t<3, 1, H>(kp, so, fa, num_sms, st);
}

template <int N1, int PM, class H>
int launch_t(const KParams& kp, int num_sms, cudaStream_t st) {
  using C = MixCfg<N1, PM>;
  constexpr int SMEM = C::SMEM0;
  // the attribute belongs to the device that is current: set once per device
  static std::atomic<bool> attr[64];
  auto kern = fe_mixed_kernel<N1, PM, H>;
  int dev = 0;
  cudaError_t e0 = cudaGetDevice(&dev);
  if (e0 != cudaSuccess) return (int)e0;
  if (dev < 0 || dev >= 64 || !attr[dev].load()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) attr[dev].store(true);
  }
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::THREADS, SMEM);
  if (e != cudaSuccess) return (int)e;
  per_sm = per_sm < 1 ? 1 : per_sm;
  const int groups = (kp.count + C::EG - 1) / C::EG;
  int grid = per_sm * num_sms;
  grid = grid < groups ? grid : groups;
  grid = grid < 1 ? 1 : grid;
  KParams k = kp;
  k.wave = num_sms > 0 ? num_sms : 1;
  kern<<<grid, C::THREADS, SMEM, st>>>(k);
  return (int)cudaGetLastError();
}

template <class H>
int launch_h(const HostSetup& s, const KParams& kp, int num_sms, cudaStream_t st) {
  if (s.n1 == 2 && s.pmode == 0) return launch_t<2, 0, H>(kp, num_sms, st);
  if (s.n1 == 2 && s.pmode == 1) return launch_t<2, 1, H>(kp, num_sms, st);
  if (s.n1 == 3 && s.pmode == 0) return launch_t<3, 0, H>(kp, num_sms, st);
  return launch_t<3, 1, H>(kp, num_sms, st);
}

}  // namespace

namespace cmfe {

int launch_mixed(const HostSetup& s, const KParams& kp, int num_sms, void* stream, bool double_float) {
  cudaStream_t st = (cudaStream_t)stream;
  if (kp.count <= 0) return 0;
  return double_float ? launch_h<dd>(s, kp, num_sms, st) : launch_h<double>(s, kp, num_sms, st);
}

int fused_wave(const HostSetup& s, int num_sms, bool double_float) {
  cudaError_t e;
  int per_sm;
  if (double_float)
    per_sm = s.n1 == 2 ? (s.pmode ? fused_per_sm<2, 1, dd>(&e) : fused_per_sm<2, 0, dd>(&e))
                       : (s.pmode ? fused_per_sm<3, 1, dd>(&e) : fused_per_sm<3, 0, dd>(&e));
  else
    per_sm = s.n1 == 2 ? (s.pmode ? fused_per_sm<2, 1, double>(&e) : fused_per_sm<2, 0, double>(&e))
                       : (s.pmode ? fused_per_sm<3, 1, double>(&e) : fused_per_sm<3, 0, double>(&e));
  if (!per_sm) return -(int)e;
  return per_sm * (num_sms > 0 ? num_sms : 1);
}

int fused_group_size(const HostSetup& s) {
  if (s.n1 == 2) return s.pmode ? FusedShape<2, 1>::EG : FusedShape<2, 0>::EG;
  return s.pmode ? FusedShape<3, 1>::EG : FusedShape<3, 0>::EG;
}

int launch_mixed_fused(const HostSetup& s, const KParams& kp, const StageOut& so, const FusedArgs& fa, int num_sms,
                       void* stream, bool double_float) {
  cudaStream_t st = (cudaStream_t)stream;
  if (kp.count <= 0) return 0;
  return double_float ? launch_fused_h<dd>(s, kp, so, fa, num_sms, st)
                      : launch_fused_h<double>(s, kp, so, fa, num_sms, st);
}

}  // namespace cmfe
