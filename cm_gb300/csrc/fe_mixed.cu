// libcm_fe: mixed-precision assembly of the Jacobian (and the residual) in one
// launch (sm_103a): the fused staged assembly of fe_fused_impl.cuh with the
// displacement block in FP32.  fe_mixed_coloured.cu has the launches per
// element colour.
#include "fe_fused_impl.cuh"

#include <type_traits>

namespace {

// Elements per group, threads per CTA and CTAs per SM.  The FP64 pipe binds
// the large shapes: three elements per group fill their warps' lanes (81 Gauss
// points on 96 lanes), and three CTAs of 192 threads beat three of 256 and two
// of 224 with four elements (32^3 triquadratic, us: 1800, 1895, 1995; trilinear
// 24x23x22 with four elements: 305 against 331 for two CTAs of 256).  A mesh
// whose groups are all resident at once is bound by the latency of one group
// and its gather, so it takes small groups with the same warps (triquadratic
// 9x7x8: 68 against 89 us, 6x5x4: 50 against 76; at 16^3, seven times as many
// elements as are resident, 339 against 292; trilinear 12x11x10: 55 against
// 62, 24x23x22: 320 against 305).
template <int N1, bool SMALL>
struct FusedShape {
  static constexpr int EG = SMALL ? (N1 == 3 ? 1 : 2) : (N1 == 3 ? 3 : 4);
  static constexpr int NT = SMALL && N1 == 2 ? 128 : 192;
  static constexpr int MINB = SMALL ? (N1 == 3 ? 4 : 5) : 3;
};

// Meshes whose groups are resident at once in the small shape take it
// (double-float phases keep the large one).
template <int N1>
bool small_mesh(const HostSetup& s, int num_sms, bool double_float) {
  using S = FusedShape<N1, true>;
  return !double_float && s.ne <= S::EG * S::MINB * num_sms;
}

// fn.template run<N1, PM, H, Shape>() for the mesh's element type and size.
template <class F>
auto with_shape(const HostSetup& s, int num_sms, bool double_float, F fn) {
  auto typed = [&](auto n1, auto pm) {
    constexpr int N1 = decltype(n1)::value, PM = decltype(pm)::value;
    if (double_float) return fn.template run<N1, PM, dd, FusedShape<N1, false>>();
    return small_mesh<N1>(s, num_sms, false) ? fn.template run<N1, PM, double, FusedShape<N1, true>>()
                                             : fn.template run<N1, PM, double, FusedShape<N1, false>>();
  };
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  using I2 = std::integral_constant<int, 2>;
  using I3 = std::integral_constant<int, 3>;
  if (s.n1 == 2) return s.pmode ? typed(I2{}, I1{}) : typed(I2{}, I0{});
  return s.pmode ? typed(I3{}, I1{}) : typed(I3{}, I0{});
}

struct PerSm {
  template <int N1, int PM, class H, class Sh>
  int run() const {
    cudaError_t e;
    const int per_sm = fused_per_sm<N1, PM, float, H, Sh>(&e);
    return per_sm ? per_sm : -(int)e;
  }
};

struct GroupSize {
  template <int N1, int PM, class H, class Sh>
  int run() const { return Sh::EG; }
};

struct Launch {
  const KParams& kp;
  const cmfe::StageOut& so;
  const cmfe::FusedArgs& fa;
  int num_sms;
  cudaStream_t st;
  template <int N1, int PM, class H, class Sh>
  int run() const { return launch_fused_t<N1, PM, float, H, Sh>(kp, so, fa, num_sms, st); }
};

}  // namespace

namespace cmfe {

int fused_wave(const HostSetup& s, int num_sms, bool double_float) {
  const int per_sm = with_shape(s, num_sms, double_float, PerSm{});
  return per_sm <= 0 ? per_sm : per_sm * (num_sms > 0 ? num_sms : 1);
}

int fused_group_size(const HostSetup& s, int num_sms, bool double_float) {
  return with_shape(s, num_sms, double_float, GroupSize{});
}

int launch_mixed_fused(const HostSetup& s, const KParams& kp, const StageOut& so, const FusedArgs& fa, int num_sms,
                       void* stream, bool double_float) {
  if (kp.count <= 0) return 0;
  return with_shape(s, num_sms, double_float, Launch{kp, so, fa, num_sms, (cudaStream_t)stream});
}

}  // namespace cmfe
