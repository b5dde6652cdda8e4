// libcm_fe: FP64 assembly of the Jacobian and the residual in one launch
// (sm_103a): the fused staged assembly (fe_fused_impl.cuh) with the
// displacement block in FP64 as well.
//
// The FP64 pipe binds it: GB300 issues one FP64 warp instruction per 19
// cycles and SM.  The sum-factorised contraction (fe_uu.cuh) and the tangent
// as outer products take about 3,000 such instructions per triquadratic
// element; contracting every entry over every Gauss point in the reference's
// order (fe_element_kernel in fe_kernels.cu, which stays for the
// element-level calls) takes about 12,000.  With the row gathers a 16^3 box's
// launch issues 3,715 an element and keeps that pipe 77 % busy (counters).
#include "fe_fused_impl.cuh"

namespace {

// Elements per group, threads per CTA and CTAs per SM.  The contraction is
// nine warp tasks for two triquadratic elements; 255 registers hold its
// accumulators without spills, so two CTAs of four warps (one to an SM
// sub-partition) beat three of three (16^3 box: 1100 against 1282 us).  Meshes
// that leave SMs without a group take one element per CTA and a warp for
// every contraction task (6x5x4: 96 us in one launch, 102 in eight, against 156;
// 9x7x7: 204 and 221 against 211, the lines cross near three elements per SM;
// trilinear 4x4x4: 59 and 68 against 108).
template <int N1, bool SMALL>
struct Shape64 {
  static constexpr int EG = SMALL ? 1 : (N1 == 3 ? 2 : 4);
  static constexpr int NT = SMALL && N1 == 3 ? 160 : 128;
  static constexpr int MINB = 2;
};

template <int N1>
bool small_mesh(const HostSetup& s, int num_sms) {
  return s.ne <= (N1 == 3 ? 3 : 2) * num_sms;
}

template <int N1, int PM>
int launch_shape(const HostSetup& s, const KParams& kp, const cmfe::StageOut& so, const cmfe::FusedArgs& fa,
                 int num_sms, cudaStream_t st) {
  return small_mesh<N1>(s, num_sms)
             ? launch_fused_t<N1, PM, double, double, Shape64<N1, true>>(kp, so, fa, num_sms, st)
             : launch_fused_t<N1, PM, double, double, Shape64<N1, false>>(kp, so, fa, num_sms, st);
}

}  // namespace

namespace cmfe {

size_t record_bytes_fp64(const HostSetup& s) {
  if (s.n1 == 2) return s.pmode ? Rec<8, 8, double>::BYTES : Rec<8, 1, double>::BYTES;
  return s.pmode ? Rec<27, 8, double>::BYTES : Rec<27, 1, double>::BYTES;
}

int fp64_groups(const HostSetup& s, int num_sms, bool* small) {
  *small = s.n1 == 2 ? small_mesh<2>(s, num_sms) : small_mesh<3>(s, num_sms);
  const int eg = s.n1 == 2 ? (*small ? Shape64<2, true>::EG : Shape64<2, false>::EG)
                           : (*small ? Shape64<3, true>::EG : Shape64<3, false>::EG);
  return (s.ne + eg - 1) / eg;
}

int launch_fp64_fused(const HostSetup& s, const KParams& kp, const StageOut& so, const FusedArgs& fa, int num_sms,
                      void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (s.n1 == 2 && s.pmode == 0) return launch_shape<2, 0>(s, kp, so, fa, num_sms, st);
  if (s.n1 == 2 && s.pmode == 1) return launch_shape<2, 1>(s, kp, so, fa, num_sms, st);
  if (s.n1 == 3 && s.pmode == 0) return launch_shape<3, 0>(s, kp, so, fa, num_sms, st);
  return launch_shape<3, 1>(s, kp, so, fa, num_sms, st);
}

}  // namespace cmfe
