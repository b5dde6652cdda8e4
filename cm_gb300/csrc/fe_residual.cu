// libcm_fe: the residual in one launch (sm_103a): the element code of the fused
// assembly without the displacement block and the coupling, a residual record
// per element, and a node's rows summed by the CTA that finishes its last
// element, in element colour order: the order, and with the same element code
// the bits, of the colour-by-colour assembly.  With a surface load the two agree
// to rounding: here an element's faces are added to its record, there to the row
// after the volume terms of the element's colour.
//
// The FP64 pipe binds a large mesh: about 270 warp instructions per
// triquadratic element (267 counted), 19 cycles each, are 0.53 ms on the 32^3 box, which
// takes 0.64 (0.86 in eight launches, one per element colour, with a third
// more of them).  A small mesh is bound by the latency of one group, which the
// eight launches paid eight times (9x7x8: 197 -> 23 us).
#include "fe_mixed_impl.cuh"
#include "fe_surface_impl.cuh"

#include <atomic>

namespace {

// Elements per group, threads and CTAs per SM.  Large meshes: groups whose
// Gauss points fill the warps (7 x 27 points on six warps, 8 x 27 on seven) and
// two CTAs an SM (16^3 box: 85 us against 101 with groups of four).  Up to four
// elements per SM: one or two elements per CTA (9x7x8: 23 against 30 us).
template <int N1, bool SMALL>
struct ShapeR {
  static constexpr int EG = SMALL ? (N1 == 3 ? 1 : 2) : (N1 == 3 ? 7 : 8);
  static constexpr int NT = SMALL ? (N1 == 3 ? 128 : 64) : (N1 == 3 ? 224 : 256);
  static constexpr int MINB = SMALL ? (N1 == 3 ? 4 : 8) : 2;
};

template <int N1, int PM, class H, class Sh>
__global__ void __launch_bounds__(Sh::NT, Sh::MINB) fe_residual_kernel(KParams P, cmfe::StageOut so, cmfe::FusedArgs F) {
  constexpr int EG = Sh::EG, NT = Sh::NT;
  using C = MixCfg<N1, PM, EG, float, NT, true>;
  constexpr int NPE = C::NPE, NPP = C::NPP, NR = C::NR;
  using RR = cmfe::RecR<NPE, NPP>;
  static_assert(NT / 32 * (int)sizeof(SurfWarpSmem) <= C::O_NODE2 - C::O_Z, "surface scratch");
  static_assert(EG * NR * 16 <= C::O_NODE2 - C::O_Z, "ready list");
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_count;
  mix_tables<N1, PM, EG, float, H, NT>(P, sm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* s_node = reinterpret_cast<const int*>(sm + C::O_NODE2);
  ReadyNode* ready = reinterpret_cast<ReadyNode*>(sm + C::O_Z);
  const int ngroups = (P.count + EG - 1) / EG;
  for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    mix_group<N1, PM, EG, float, H, 2, NT>(P, nullptr, P.count, grp, false, sm, &so);
    const int nvalid = min(EG, P.count - grp * EG);
    if (tid == 0) s_count = 0;
    __syncthreads();  // the group's records are complete within the CTA; the scratch is free
    if (F.bmask) {
      SurfWarpSmem* ws = reinterpret_cast<SurfWarpSmem*>(sm + C::O_Z);
      for (int el = warp; el < nvalid; el += NT / 32) {
        const int e = grp * EG + el;
        if (F.bmask[e]) surface_element<N1, NPP>(P, e, F.bmask, 3, 0, ws[warp], lane, &so);
      }
      __syncthreads();
    }
    // count the finished elements around the group's row nodes (publication as
    // in GroupGather::run); a complete count goes back to zero
    __threadfence();
    __syncthreads();
    for (int i = tid; i < nvalid * NR; i += NT) {
      __threadfence();
      const int el = i / NR, r = i % NR;
      const int node = s_node[el * (NR + 1) + r];
      const bool un = r < NPE;
      const int id = un ? node : P.nu + node;
      const int32_t* ptr = un ? F.u_inc_ptr + node : F.p_inc_ptr + node;
      const int k0 = ptr[0], cnt = ptr[1] - k0;
      if (atomicAdd(F.node_done + id, 1) + 1 == cnt) {
        __threadfence();
        F.node_done[id] = 0;
        ready[atomicAdd(&s_count, 1)] = {id, k0, cnt, 0};
      }
    }
    __syncthreads();
    const int nready = s_count;
    for (int i = tid; i < 3 * nready; i += NT) {  // (row node, component)
      const ReadyNode rn = ready[i / 3];
      const int m = i % 3;
      const bool un = rn.id < P.nu;
      if (!un && m) continue;
      double acc = 0.0;
      for (int kb = 0; kb < rn.cnt; kb += 8) {  // eight elements' loads in flight
        double v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = 0.0;
          if (kb + j < rn.cnt) {
            const int pk = (un ? F.u_inc : F.p_inc)[rn.k0 + kb + j];
            const double* r = un ? RR::of(so, pk >> 5) + 3 * (pk & 31) + m : RR::of(so, pk >> 3) + 3 * NPE + (pk & 7);
            v[j] = __ldcg(r);
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (kb + j < rn.cnt) acc += v[j];
      }
      P.r[un ? (size_t)m * P.nu + rn.id : (size_t)2 * P.nu + rn.id] = acc;
    }
    // mix_group begins with a barrier before it reuses the scratch
  }
}

template <int N1, int PM, class H, class Sh>
int launch_t(const KParams& kp, const cmfe::StageOut& so, const cmfe::FusedArgs& fa, int num_sms, cudaStream_t st) {
  using C = MixCfg<N1, PM, Sh::EG, float, Sh::NT, true>;
  auto kern = fe_residual_kernel<N1, PM, H, Sh>;
  static std::atomic<bool> attr[64];
  static std::atomic<int> resident[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  if (dev < 0 || dev >= 64 || !attr[dev].load()) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM2);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, Sh::NT, C::SMEM2);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) {
      resident[dev].store(per_sm);
      attr[dev].store(true);
    }
  } else {
    per_sm = resident[dev].load();
  }
  const int groups = (kp.count + Sh::EG - 1) / Sh::EG;
  int grid = (per_sm < 1 ? 1 : per_sm) * num_sms;
  grid = grid < groups ? grid : groups;
  KParams k = kp;
  k.wave = num_sms > 0 ? num_sms : 1;
  kern<<<grid < 1 ? 1 : grid, Sh::NT, C::SMEM2, st>>>(k, so, fa);
  return (int)cudaGetLastError();
}

template <int N1, int PM>
int launch_h(const KParams& kp, const cmfe::StageOut& so, const cmfe::FusedArgs& fa, int num_sms, cudaStream_t st,
             bool double_float) {
  if (double_float) return launch_t<N1, PM, dd, ShapeR<N1, false>>(kp, so, fa, num_sms, st);
  if (kp.count <= 4 * num_sms) return launch_t<N1, PM, double, ShapeR<N1, true>>(kp, so, fa, num_sms, st);
  return launch_t<N1, PM, double, ShapeR<N1, false>>(kp, so, fa, num_sms, st);
}

}  // namespace

namespace cmfe {

size_t record_bytes_residual(const HostSetup& s) {
  if (s.n1 == 2) return 8 * (s.pmode ? RecR<8, 8>::N : RecR<8, 1>::N);
  return 8 * (s.pmode ? RecR<27, 8>::N : RecR<27, 1>::N);
}

int launch_residual_fused(const HostSetup& s, const KParams& kp, const StageOut& so, const FusedArgs& fa, int num_sms,
                          void* stream, bool double_float) {
  cudaStream_t st = (cudaStream_t)stream;
  if (s.n1 == 2 && s.pmode == 0) return launch_h<2, 0>(kp, so, fa, num_sms, st, double_float);
  if (s.n1 == 2 && s.pmode == 1) return launch_h<2, 1>(kp, so, fa, num_sms, st, double_float);
  if (s.n1 == 3 && s.pmode == 0) return launch_h<3, 0>(kp, so, fa, num_sms, st, double_float);
  return launch_h<3, 1>(kp, so, fa, num_sms, st, double_float);
}

}  // namespace cmfe
