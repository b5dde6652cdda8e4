// libcm_fe: the displacement block of the element Jacobian, device code
// templated on its arithmetic type T (float: mixed-precision assembly;
// double: FP64 assembly).
//
//   K^{mn}(a, b) = sum_g sum_kl dN_a/dxi_k(g) D^{mn}_{kl}(g) dN_b/dxi_l(g),
//   D^{mn}_{kl} = J_z w sum_ij dxi_k/dz_i (c_imjn + delta_mn sigma_ij) dxi_l/dz_j
//
// (FiniteElasticity_FiniteElementJacobianEvaluate, finite_elasticity_routines.f90:
// 842-1175, pulled back to xi space).  Basis and quadrature are tensor
// products, so the sum over the 27 Gauss points is done one direction at a
// time: with B / D the 1-D basis values / derivatives and
// MM_t(a, b; g) the four products BB, BD, DB, DD,
//   stage 1  S1[kl][a1 b1][g2 g3] = sum_g1 MM_{t1(kl)}(a1, b1; g1) D_kl(g1, g2, g3)
//   stage 2  w[t3][g3] = sum_{kl with type t3 along xi3} sum_g2 MM_{t2(kl)}(a2, b2; g2) S1[kl][a1 b1][g2, g3]
//   stage 3  K(a, b) = sum_t3 sum_g3 MM_{t3}(a3, b3; g3) w[t3][g3].
// A triquadratic element takes about 70 k multiply-adds this way instead of the
// 354 k of the 81 x 81 x 81 product over (Gauss point, derivative) pairs, in
// full T precision.
#pragma once

#include <cuda_runtime.h>

#include "../../include/cm_fe.h"
#include "fe_dd.cuh"

namespace {

// 1-D Lagrange basis function a of n nodes on [0, 1] (derivative when d) at
// Gauss point g of the 3-point rule, as a compile-time constant.
__host__ __device__ constexpr double uu_lag(int n, int a, int d, int g) {
  const double t = g == 0 ? 0.11270166537925831 : (g == 1 ? 0.5 : 0.88729833462074169);
  if (n == 2) return d ? (a == 0 ? -1.0 : 1.0) : (a == 0 ? 1.0 - t : t);
  if (d) return a == 0 ? 4.0 * t - 3.0 : (a == 1 ? 4.0 - 8.0 * t : 4.0 * t - 1.0);
  return a == 0 ? 1.0 - 3.0 * t + 2.0 * t * t : (a == 1 ? 4.0 * t * (1.0 - t) : t * (t + t - 1.0));
}
// MM_t(a, b; g): bit 1 of t takes the derivative on a, bit 0 on b.
__host__ __device__ constexpr double uu_mm(int n, int t, int a, int b, int g) {
  return uu_lag(n, a, t >> 1, g) * uu_lag(n, b, t & 1, g);
}

// Slots of the D^{blk}_{kl} records of one Gauss point: the diagonal blocks
// are symmetric in (k, l) and keep k <= l (6 slots each), the lower blocks 9.
constexpr int UU_REC = 45;
__host__ __device__ constexpr int uu_sym(int k, int l) {
  const int i = k < l ? k : l, j = k < l ? l : k;
  return i == 0 ? j : (i == 1 ? 2 + j : 5);
}
__host__ __device__ constexpr int uu_slot(int blk, int k, int l) {
  return blk < 3 ? 6 * blk + uu_sym(k, l) : 18 + 9 * (blk - 3) + 3 * k + l;
}

template <class T>
__device__ __forceinline__ T uu_rcbrt(T x);
template <>
__device__ __forceinline__ float uu_rcbrt<float>(float x) { return rcbrtf(x); }
template <>
__device__ __forceinline__ double uu_rcbrt<double>(double x) { return hrcbrt(x); }
__device__ __forceinline__ bool uu_finite(float v) { return isfinite(v); }
__device__ __forceinline__ bool uu_finite(double v) { return hfinite(v); }
template <class T>
__device__ __forceinline__ T uu_exp(T x);
template <>
__device__ __forceinline__ float uu_exp<float>(float x) { return expf(x); }
template <>
__device__ __forceinline__ double uu_exp<double>(double x) { return exp(x); }

// The 45 values D^{blk}_{kl} of one Gauss point.  M = dz/dxi, dn = dxi/dnu,
// rjx = 1 / J_x, w = quadrature weight, p = pressure.  The tangent is the
// reference's (FINITE_ELASTICITY_GAUSS_ELASTICITY_TENSOR, :609-835) in index
// form: with P the deviatoric projection, tau = sigma_bar, s = dev tau,
//   c = P : c_bar : P + 2/3 tr(tau) P - 2/3 (I x s + s x I) + p (I x I - 2 1),
// and c_bar pushed forward analytically, so that every term of D is an outer
// product of vectors contracted with dxi_k/dz once (no 6 x 6 matrices:
// F_bar^T dxi_k/dz = J^(-1/3) dxi_k/dnu).  Returns whether it is finite.
template <class T>
__device__ __forceinline__ bool uu_tangent(int law, const T* c, const T M[3][3], const T* dn, T rjx, T w, T p, T* rec) {
  const T third = T(1.0 / 3.0), half = T(0.5), two = T(2.0);
  T G[3][3], F[3][3];
  G[0][0] = M[1][1] * M[2][2] - M[1][2] * M[2][1];
  G[0][1] = M[0][2] * M[2][1] - M[0][1] * M[2][2];
  G[0][2] = M[0][1] * M[1][2] - M[0][2] * M[1][1];
  G[1][0] = M[1][2] * M[2][0] - M[1][0] * M[2][2];
  G[1][1] = M[0][0] * M[2][2] - M[0][2] * M[2][0];
  G[1][2] = M[0][2] * M[1][0] - M[0][0] * M[1][2];
  G[2][0] = M[1][0] * M[2][1] - M[1][1] * M[2][0];
  G[2][1] = M[0][1] * M[2][0] - M[0][0] * M[2][1];
  G[2][2] = M[0][0] * M[1][1] - M[0][1] * M[1][0];
  const T det = M[0][0] * G[0][0] + M[0][1] * G[1][0] + M[0][2] * G[2][0];
  const T rdet = T(1) / det;
  const T jz = det < T(0) ? -det : det;
  const T J = jz * rjx;
  const T s = uu_rcbrt<T>(J), rJ = s * s * s, jw = jz * w;
  T f[3][3];  // F_bar^T dxi_k/dz
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      G[i][j] = G[i][j] * rdet;
      f[i][j] = s * dn[3 * i + j];
      F[i][j] = s * (M[i][0] * dn[j] + M[i][1] * dn[3 + j] + M[i][2] * dn[6 + j]);
    }
  // symmetric 3 x 3 tensors in the order 00 11 22 01 02 12
  constexpr int V0[6] = {0, 1, 2, 0, 0, 1}, V1[6] = {0, 1, 2, 1, 2, 2};
  T sb[6], q[6];  // sigma_bar; q = -1/3 c_bar : I - 2/3 s
  T t;            // I : c_bar : I
  T Bv[6];        // MR: left Cauchy-Green tensor B_bar; Guccione: F_bar DQ F_bar^T
  T e0, eb[6];    // scale of the rank-one part; Guccione: scales of the six basis tensors
  if (law == FE_LAW_MOONEY_RIVLIN) {
#pragma unroll
    for (int v = 0; v < 6; ++v)
      Bv[v] = F[V0[v]][0] * F[V1[v]][0] + F[V0[v]][1] * F[V1[v]][1] + F[V0[v]][2] * F[V1[v]][2];
    const T I1 = Bv[0] + Bv[1] + Bv[2];
    const T al = two * rJ * (c[0] + I1 * c[1]), be = -two * rJ * c[1];
    e0 = T(4) * rJ * c[1];
    T trb2 = T(0);
#pragma unroll
    for (int v = 0; v < 6; ++v) {
      const int i = V0[v], j = V1[v];
      T b2 = T(0);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int ik = i == k ? i : (i + k == 1 ? 3 : (i + k == 2 ? 4 : 5));
        const int kj = k == j ? j : (k + j == 1 ? 3 : (k + j == 2 ? 4 : 5));
        b2 += Bv[ik] * Bv[kj];
      }
      if (v < 3) trb2 += b2;
      sb[v] = al * Bv[v] + be * b2;
      q[v] = e0 * (I1 * Bv[v] - b2);
    }
    t = e0 * (I1 * I1 - trb2);
#pragma unroll
    for (int v = 0; v < 6; ++v) eb[v] = T(0);
  } else {
    T C[6];
#pragma unroll
    for (int v = 0; v < 6; ++v)
      C[v] = F[0][V0[v]] * F[0][V1[v]] + F[1][V0[v]] * F[1][V1[v]] + F[2][V0[v]] * F[2][V1[v]];
    const T b[6] = {two * c[1], two * c[2], two * c[2], c[3], c[3], c[2]};
    T DQ[6], dot = T(0);
#pragma unroll
    for (int v = 0; v < 6; ++v) {
      const T E = v < 3 ? half * (C[v] - T(1)) : C[v];
      DQ[v] = b[v] * E;
      dot += E * DQ[v];
    }
    e0 = half * c[0] * uu_exp<T>(half * dot) * rJ;
    t = T(0);
    T trs = T(0);
#pragma unroll
    for (int v = 0; v < 6; ++v) {
      const int i = V0[v], j = V1[v];
      T sum = T(0);
#pragma unroll
      for (int I = 0; I < 3; ++I) {
        const T Si0 = DQ[I == 0 ? 0 : (I == 1 ? 3 : 4)], Si1 = DQ[I == 0 ? 3 : (I == 1 ? 1 : 5)],
                Si2 = DQ[I == 0 ? 4 : (I == 1 ? 5 : 2)];
        sum += F[i][I] * (Si0 * F[j][0] + Si1 * F[j][1] + Si2 * F[j][2]);
      }
      Bv[v] = sum;
      if (v < 3) trs += sum;
    }
#pragma unroll
    for (int v = 0; v < 6; ++v) eb[v] = e0 * b[v];
#pragma unroll
    for (int v = 0; v < 6; ++v) {
      sb[v] = e0 * Bv[v];
      T h = e0 * Bv[v] * trs;
#pragma unroll
      for (int u = 0; u < 6; ++u) {  // basis tensor u: F_U0 F_U1^T, symmetrised for the shears; its trace
        const T tr = u < 3 ? C[u] : two * C[u];
        T b2 = F[V0[v]][V0[u]] * F[V1[v]][V1[u]];
        if (u >= 3) b2 += F[V0[v]][V1[u]] * F[V1[v]][V0[u]];
        h += eb[u] * tr * b2;
      }
      q[v] = h;
      if (v < 3) t += h;
    }
  }
  // every term of D is linear in what follows: J_z w goes in here
  const T tr = sb[0] + sb[1] + sb[2];
  const T jw3 = third * jw;
  T sg[6];  // J_z w (sigma + mu/2 1), mu/2 = tr / 3 - p: the delta_mn part
  const T mu2 = jw * (third * tr - p);
#pragma unroll
  for (int v = 0; v < 6; ++v) {
    const T sd = v < 3 ? sb[v] - third * tr : sb[v];
    q[v] = -jw3 * (q[v] + two * sd);
    sg[v] = v < 3 ? jw * (sd + p) + mu2 : jw * sd;
  }
  const T kap = jw * (t * T(1.0 / 9.0) - T(2.0 / 9.0) * tr + p);
  e0 = jw * e0;
#pragma unroll
  for (int v = 0; v < 6; ++v) eb[v] = jw * eb[v];
  T r[3][3], rho[3][3], b[3][3], sG[3][3], mG[3][3], ob[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r[k][0] = q[0] * G[k][0] + q[3] * G[k][1] + q[4] * G[k][2];
    r[k][1] = q[3] * G[k][0] + q[1] * G[k][1] + q[5] * G[k][2];
    r[k][2] = q[4] * G[k][0] + q[5] * G[k][1] + q[2] * G[k][2];
    sG[k][0] = sg[0] * G[k][0] + sg[3] * G[k][1] + sg[4] * G[k][2];
    sG[k][1] = sg[3] * G[k][0] + sg[1] * G[k][1] + sg[5] * G[k][2];
    sG[k][2] = sg[4] * G[k][0] + sg[5] * G[k][1] + sg[2] * G[k][2];
    if (law == FE_LAW_MOONEY_RIVLIN) {
#pragma unroll
      for (int m = 0; m < 3; ++m) b[k][m] = F[m][0] * f[k][0] + F[m][1] * f[k][1] + F[m][2] * f[k][2];
    } else {
      b[k][0] = Bv[0] * G[k][0] + Bv[3] * G[k][1] + Bv[4] * G[k][2];
      b[k][1] = Bv[3] * G[k][0] + Bv[1] * G[k][1] + Bv[5] * G[k][2];
      b[k][2] = Bv[4] * G[k][0] + Bv[5] * G[k][1] + Bv[2] * G[k][2];
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      mG[k][m] = mu2 * G[k][m];
      rho[k][m] = r[k][m] + kap * G[k][m];
      ob[k][m] = e0 * b[k][m];
    }
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      // delta_mn part, and MR's -e0/2 (dxi_k/dz . B_bar . dxi_l/dz) B_bar
      const T iso = G[l][0] * sG[k][0] + G[l][1] * sG[k][1] + G[l][2] * sG[k][2];
      T bkl = T(0);
      if (law == FE_LAW_MOONEY_RIVLIN) bkl = -half * (G[l][0] * ob[k][0] + G[l][1] * ob[k][1] + G[l][2] * ob[k][2]);
#pragma unroll
      for (int blk = 0; blk < 6; ++blk) {
        if (blk < 3 && k > l) continue;
        const int m = blk < 3 ? blk : (blk == 3 ? 1 : 2), n = blk < 3 ? blk : (blk == 5 ? 1 : 0);
        T v = G[k][m] * rho[l][n] + r[k][m] * G[l][n] + mG[k][n] * G[l][m];
        if (law == FE_LAW_MOONEY_RIVLIN) {
          const int vm = m == n ? m : (m + n == 1 ? 3 : (m + n == 2 ? 4 : 5));
          v += bkl * Bv[vm];
          if (m == n)
            v += (half * ob[k][m]) * b[l][m];
          else
            v += ob[k][m] * b[l][n] - (half * ob[k][n]) * b[l][m];
        } else {
          v += ob[k][m] * b[l][n];
#pragma unroll
          for (int u = 0; u < 6; ++u) {
            const int I = V0[u], J2 = V1[u];
            T x = f[k][I] * F[m][J2], y = f[l][I] * F[n][J2];
            if (u >= 3) {
              x += f[k][J2] * F[m][I];
              y += f[l][J2] * F[n][I];
            }
            v += eb[u] * x * y;
          }
        }
        if (m == n) v += iso;
        if (blk == 0 && k == l) ok = ok && uu_finite(v);
        rec[uu_slot(blk, k, l)] = v;
      }
    }
  return ok;
}

// Work split of the contraction: warp tasks over (element, block) units.
// Triquadratic: a lower block takes 27 lanes, lane = (a1 b1, a2), three b2
// each; of a diagonal block only the entries up to the mirror (a <-> b) are
// formed, 15 lanes with three (a2, b2) pairs each, two such blocks to a
// warp.  Trilinear: 8 lanes to a block, lane = (a1 b1, a2), two b2 each,
// four blocks to a warp.
template <int N1>
struct UUCfg {
  static constexpr int NP = N1 * N1;
  static constexpr int JP = N1;                                 // (a2, b2) pairs per lane
  static constexpr int S1 = N1 == 3 ? 2 * 6 * 81 : 4 * 9 * 36;  // stage-1 values of one warp task
  static_assert(S1 >= (N1 == 3 ? 9 : 4 * 9) * NP * 9 && S1 >= (N1 == 3 ? 2 * 6 * NP * 9 : 0), "units of a warp task");
  static constexpr int MM = 4 * NP * 4;                         // table [t][a b][g], g padded to 4
  __host__ __device__ static constexpr int tasks(int nvalid) {
    return N1 == 3 ? 3 * nvalid + (3 * nvalid + 1) / 2 : (6 * nvalid + 3) / 4;
  }
};

template <int N1, class T>
__device__ __forceinline__ void uu_table(T* s_mm, int tid, int threads) {
  constexpr int NP = N1 * N1;
  for (int i = tid; i < 4 * NP * 4; i += threads) {
    const int g = i % 4, ab = (i / 4) % NP, t = i / (4 * NP);
    const int gg = g < 3 ? g : 0;
    const T v = T(uu_lag(N1, ab / N1, t >> 1, gg) * uu_lag(N1, ab % N1, t & 1, gg));
    s_mm[i] = g < 3 ? v : T(0);
  }
}

template <class T>
__device__ __forceinline__ void uu_load3(const T* p, T (&v)[3]) {
  if constexpr (sizeof(T) == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z;
  } else {
    const double2 x = *reinterpret_cast<const double2*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = p[2];
  }
}

// One warp task: stages 1 to 3 of its units.  s_D: [el][g][UU_REC]; s1: this
// warp's scratch (UUCfg::S1 values).  out(el, blk, a12, b12, K) receives, for
// one pair of partial node indices a12 = a1 + N1 a2 and b12, the N1 x N1 values
// K[a3][b3].
template <int N1, class T, class Out>
__device__ __forceinline__ void uu_warp_task(const T* s_D, const T* s_mm, T* s1, int task, int nvalid, int lane, Out out) {
  using C = UUCfg<N1>;
  constexpr int NP = C::NP, JP = C::JP;
  constexpr bool SYM = N1 == 3;
  const bool off = SYM && task < 3 * nvalid;  // a lower block of a triquadratic element
  // ---- units of this task
  int units, per_unit, first;  // units, stage-1 slots per unit, first unit number
  if (SYM) {
    units = off ? 1 : min(2, 3 * nvalid - 2 * (task - 3 * nvalid));
    per_unit = off ? 9 : 6;
    first = off ? task : 2 * (task - 3 * nvalid);
  } else {
    units = min(4, 6 * nvalid - 4 * task);
    per_unit = 9;
    first = 4 * task;
  }
  auto unit_of = [&](int u, int& el, int& blk) {
    const int d = first + u;
    el = SYM ? d / 3 : d / 6;
    blk = SYM ? (off ? 3 : 0) + d % 3 : d % 6;
  };
  __syncwarp();
  // ---- stage 1
  for (int i = lane; i < units * per_unit * 9; i += 32) {
    const int j = i % 9, s = (i / 9) % per_unit, u = i / (9 * per_unit);
    int el, blk, k, l;
    unit_of(u, el, blk);
    if (SYM && !off) {
      k = s < 3 ? 0 : (s < 5 ? 1 : 2);
      l = s < 3 ? s : (s < 5 ? s - 2 : 2);
    } else {
      k = s / 3;
      l = s % 3;
    }
    const int t1 = (k == 0 ? 2 : 0) + (l == 0 ? 1 : 0);
    const T* d = s_D + (size_t)(el * 27 + 3 * j) * UU_REC + uu_slot(blk, k, l);
    const T d0 = d[0], d1 = d[UU_REC], d2 = d[2 * UU_REC];
    T* o = s1 + (u * per_unit + s) * NP * 9 + j;
    const T* mm = s_mm + t1 * NP * 4;
#pragma unroll
    for (int ab = 0; ab < NP; ++ab) {
      T m[3];
      uu_load3(mm + 4 * ab, m);
      o[ab * 9] = m[0] * d0 + m[1] * d1 + m[2] * d2;
    }
  }
  __syncwarp();
  // ---- stages 2 and 3
  int u, a1, b1, a2[JP], b2[JP];
  bool work;
  if (SYM && off) {
    u = 0;
    work = lane < 27;
    const int r = work ? lane : 26;
    a1 = r / 3 % 3;
    b1 = r % 3;
#pragma unroll
    for (int j = 0; j < JP; ++j) {
      a2[j] = r / 9;
      b2[j] = j;
    }
  } else if (SYM) {
    u = lane >= 15 ? 1 : 0;
    const int r = lane - 15 * u;
    work = lane < 30 && u < units;
    if (!work) u = 0;
    if (r < 9) {  // a1 < b1: all nine (a2, b2)
      const int pr = r / 3;
      a1 = pr == 2 ? 1 : 0;
      b1 = pr == 0 ? 1 : 2;
#pragma unroll
      for (int j = 0; j < JP; ++j) {
        a2[j] = r % 3;
        b2[j] = j;
      }
    } else {  // a1 = b1: a2 <= b2
      const int h = (r - 9) % 2;
      a1 = b1 = min((r - 9) / 2, 2);
#pragma unroll
      for (int j = 0; j < JP; ++j) {
        a2[j] = h ? (j == 2 ? 2 : 1) : 0;
        b2[j] = h ? (j == 0 ? 1 : 2) : j;
      }
    }
  } else {
    u = lane / 8;
    work = u < units;
    if (!work) u = 0;
    a1 = lane % 8 / 4;
    b1 = lane % 2;
#pragma unroll
    for (int j = 0; j < JP; ++j) {
      a2[j] = lane % 4 / 2;
      b2[j] = j;
    }
  }
  int el, blk;
  unit_of(u, el, blk);
  const T* su = s1 + u * per_unit * NP * 9;
  const bool sym = SYM && !off;
  const T* row = su + (a1 * N1 + b1) * 9;   // S1[.][a1 b1]
  const T* rowt = su + (b1 * N1 + a1) * 9;  // S1[.][b1 a1]: the (l, k) entries of a symmetric block
  constexpr int JW = sizeof(T) == 4 ? JP : 1;  // pairs formed together (registers)
#pragma unroll
  for (int j0 = 0; j0 < JP; j0 += JW) {
    T w[JW][4][3];
#pragma unroll
    for (int j = 0; j < JW; ++j)
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int g = 0; g < 3; ++g) w[j][t][g] = T(0);
#pragma unroll
    for (int t2 = 0; t2 < 4; ++t2) {
      T m[JW][3];
#pragma unroll
      for (int j = 0; j < JW; ++j) uu_load3(s_mm + (t2 * NP + a2[j0 + j] * N1 + b2[j0 + j]) * 4, m[j]);
#pragma unroll
      for (int kl = 0; kl < 9; ++kl) {
        const int k = kl / 3, l = kl % 3;
        if ((k == 1 ? 2 : 0) + (l == 1 ? 1 : 0) != t2) continue;
        const int t3 = (k == 2 ? 2 : 0) + (l == 2 ? 1 : 0);
        const T* s = (sym ? (k > l ? rowt : row) + uu_sym(k, l) * (NP * 9) : row + kl * (NP * 9));
#pragma unroll
        for (int g3 = 0; g3 < 3; ++g3)
#pragma unroll
          for (int g2 = 0; g2 < 3; ++g2) {
            const T v = s[3 * g3 + g2];
#pragma unroll
            for (int j = 0; j < JW; ++j) w[j][t3][g3] += m[j][g2] * v;
          }
      }
    }
#pragma unroll
    for (int j = 0; j < JW; ++j) {
      // stage 3 in even and odd combinations: the reflection of xi3 takes
      // (a3, b3) to (N1 - 1 - a3, N1 - 1 - b3) and changes the sign of the
      // types with one derivative, so the entries come in pairs P + Q, P - Q
      T K[N1][N1], e[4], o[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        e[t] = w[j][t][0] + w[j][t][2];
        o[t] = w[j][t][0] - w[j][t][2];
      }
#pragma unroll
      for (int a3 = 0; a3 < N1; ++a3)
#pragma unroll
        for (int b3 = 0; b3 < N1; ++b3) {
          const int ma = N1 - 1 - a3, mb = N1 - 1 - b3;
          if (ma * N1 + mb < a3 * N1 + b3) continue;
          T P = T(0), Q = T(0);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const double m0 = uu_mm(N1, t, a3, b3, 0), m1 = uu_mm(N1, t, a3, b3, 1), m2 = uu_mm(N1, t, a3, b3, 2);
            const double me = 0.5 * (m0 + m2), mo = 0.5 * (m0 - m2);
            T& E = t == 0 || t == 3 ? P : Q;
            T& O = t == 0 || t == 3 ? Q : P;
            const bool self = ma == a3 && mb == b3;
            if (!(self && (t == 1 || t == 2))) {
              E += T(me) * e[t];
              if (m1 != 0.0) E += T(m1) * w[j][t][1];
            }
            if (!(self && (t == 0 || t == 3))) O += T(mo) * o[t];
          }
          K[a3][b3] = P + Q;
          if (ma != a3 || mb != b3) K[ma][mb] = P - Q;
        }
      if (work) out(el, blk, a1 + N1 * a2[j0 + j], b1 + N1 * b2[j0 + j], K);
    }
  }
}

}  // namespace
