// libcm_fe: element assembly, device code shared by the fused kernels
// (fe_mixed.cu, fe_fp64.cu), the residual (fe_residual.cu), the launches per
// colour (fe_mixed_coloured.cu) and the batched kernel (fe_batch.cu).
//
// Same arithmetic content as the reference's element residual and Jacobian
// (FiniteElasticity_FiniteElement{Residual,Jacobian}Evaluate,
// finite_elasticity_routines.f90:1260-1639 and :842-1175), reorganised for
// the GB300:
//
//  * FP64 only where the residual and the pressure coupling need it.  Per
//    Gauss point the kinematics use the adjugate of dz/dxi (J_z dxi/dz =
//    adj(dz/dxi), so no 3x3 division), the Cauchy stress is formed as
//    F_bar S_bar F_bar^T / J (the push-forward of :1221-1253 written as a
//    matrix product), and the residual is contracted against the fixed table
//    of reference-element gradients: r(m,a) = sum_g sum_k dN_a/dxi_k (g) *
//    P_g(k,m) with P_g = J_z w_g dxi/dz sigma.  The pressure-coupling block
//    K(p_q, u_nb) = sum_g psi_q(g) J_z w_g dN_b/dz_n is contracted with the
//    tensor-product (sum-factorised) form of the trilinear pressure basis.
//  * The displacement block is FP32: the reference's tangent (:1003-1034) is
//    pulled back to xi space per Gauss point and contracted over the Gauss
//    points by sum factorisation on the FP32 pipes (fe_uu.cuh).  Warps do it
//    on their own, one block of an element (or two symmetric ones) at a time.
//  * Elements of one colour share no node; a CTA processes EG elements at a
//    time for the per-Gauss-point work (so 100+ threads do the FP64
//    kinematics at once) and then contracts them one by one.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fe_dd.cuh"
#include "fe_internal.h"
#include "fe_math.cuh"
#include "fe_line.cuh"
#include "fe_uu.cuh"
#include "fe_gather_impl.cuh"

using cmfe::HostSetup;
using cmfe::KParams;
using cmfe::NG;

namespace {

constexpr int align16(int x) { return (x + 15) & ~15; }

// Elements per group of the launches per colour: 3 for triquadratic with nodal pressure
// (about 72 KB of shared memory, so three 256-thread CTAs fit on an SM, which
// measured 17 % faster than two CTAs of 4 elements despite the register
// spills the 80-register budget causes), 4 for element-based pressure, 8 for
// trilinear elements.
// RES: the residual alone (no displacement block, no coupling).
template <int N1, int PM, int EG_ = (N1 == 3 ? (PM ? 3 : 4) : 8), class T = float, int NT = 256, bool RES = false>
struct MixCfg {
  static constexpr int MINB = (N1 == 3 && PM) ? 3 : 2;  // CTAs per SM the launch bounds ask for
  static constexpr int NPE = N1 * N1 * N1;
  static constexpr int NPP = PM ? 8 : 1;
  static constexpr int NR = NPE + NPP;
  static constexpr int NU3 = 3 * NPE;
  static constexpr int NROW = NU3 + NPP;
  static constexpr int THREADS = NT;
  static constexpr int EG = EG_;                // elements per group
  static constexpr int REC64 = RES ? 11 : 20;  // P(9), A(9), t1, pad; RES: P(9), t1, pad
  static constexpr int T1 = RES ? 9 : 18;      // place of t1
  static constexpr int O_PSI64 = 0;
  static constexpr int O_W = align16(O_PSI64 + NG * 8 * 8);
  // constant tables first, then the per-group scratch from O_Z on (the fused
  // kernel reuses the scratch between groups for its row gathers)
  static constexpr int O_MM = align16(O_W + NG * 8);
  static constexpr int O_Z = align16(O_MM + UUCfg<N1>::MM * (int)sizeof(T));
  static constexpr int O_P = align16(O_Z + EG * 3 * NPE * 8);
  static constexpr int O_PG = align16(O_P + EG * 8 * 8);
  static constexpr int O_R64 = align16(O_PG + EG * NG * 8);
  static constexpr int P1S = EG * (18 * N1 * N1 + 81 * N1) * 8;  // scratch of the gradients' first two stages
  static constexpr int L2 = 2 * N1;                               // linear x 1-D basis products of a line
  static constexpr int T1S = EG * 3 * L2 * 9 * 8;                 // coupling, per component: stage 1
  static constexpr int W2S = EG * L2 * L2 * 3 * 8;                //   and each of the two stage-2 arrays
  static constexpr int P3S = PM && !RES ? 3 * T1S + 6 * W2S : 0;
  static constexpr int RECS = RES ? 0 : EG * NG * UU_REC * (int)sizeof(T);
  static constexpr int O_R32 = align16(O_R64 + EG * NG * REC64 * 8);
  // the gradients and the FP64 stages' scratch share their space with the
  // warps' stage-1 values of the displacement block
  static constexpr int O_DZ = align16(O_R32 + (RECS > P1S ? RECS : P1S));
  static constexpr int P3R = EG * (9 * N1 * 9 + 6 * N1 * N1 * 3 + 64) * 8;  // scratch of the residual stages
  static constexpr int O_U1 = O_DZ, O_U2 = O_U1 + EG * 9 * N1 * 9 * 8, O_U3 = O_U2 + EG * 6 * N1 * N1 * 3 * 8;
  static constexpr int WS1 = RES ? 0 : THREADS / 32 * UUCfg<N1>::S1 * (int)sizeof(T);
  static constexpr int big(int x, int y) { return x > y ? x : y; }
  static constexpr int O_BASE = align16(O_DZ + big(big(EG * NG * 9 * 8, WS1), big(P3R, P3S)));
  // coloured order only: scatter addresses and rank tables of the group
  static constexpr int O_TAB = align16(O_BASE + EG * 9 * NPE * 4);
  static constexpr int O_NODE0 = align16(O_TAB + EG * NPE * NPE * 2);
  static constexpr int SMEM0 = align16(O_NODE0 + EG * (NR + 1) * 4);
  // staged order: the node numbers follow the scratch, which the row gathers
  // reuse from O_Z on
  static constexpr int GATHER_END = align16(O_Z + GroupGather<NPE, NPP, EG, THREADS, T>::SCRATCH);
  static constexpr int O_NODE1 = O_BASE > GATHER_END ? O_BASE : GATHER_END;
  static constexpr int SMEM1 = align16(O_NODE1 + EG * (NR + 1) * 4);
  // residual alone: no row gathers in the scratch
  static constexpr int O_NODE2 = O_BASE;
  static constexpr int SMEM2 = align16(O_NODE2 + EG * (NR + 1) * 4);
};

// Block (m, n) of the lower-triangle displacement blocks: 0..2 diagonal,
// 3 = (1,0), 4 = (2,0), 5 = (2,1).
__device__ __forceinline__ void blk_mn(int blk, int& m, int& n) {
  m = blk < 3 ? blk : (blk == 3 ? 1 : 2);
  n = blk < 3 ? blk : (blk == 5 ? 1 : 0);
}

// Cauchy stress of the MR or Guccione law in the high-precision type H from
// F (material frame) and J = Jznu: sigma = dev(F_bar S_bar F_bar^T / J) + p I.
template <class H>
__device__ void mix_stress(int law, const H* c, const H F[3][3], H J, H p, H sig[3][3]) {
  const H s = hrcbrt(J), s2 = s * s, rJ = s * s2;
  const H zero = hval<H>(0.0), one = hval<H>(1.0), two = hval<H>(2.0), half = hval<H>(0.5);
  if (law == FE_LAW_MOONEY_RIVLIN) {
    // S_bar = al I + be C_bar, so F_bar S_bar F_bar^T = al B_bar + be B_bar^2
    // with B_bar = J^(-2/3) F F^T (and tr C_bar = tr B_bar); the powers of J
    // and 1/J go into the two coefficients
    H B[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) {
        B[i][j] = hfma(F[i][2], F[j][2], hfma(F[i][1], F[j][1], F[i][0] * F[j][0]));
        B[j][i] = B[i][j];
      }
    const H I1 = s2 * (B[0][0] + B[1][1] + B[2][2]);
    const H q = two * rJ * s2;
    const H al = q * hfma(I1, c[1], c[0]);
    const H be = -(q * s2 * c[1]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) {
        const H b2 = hfma(B[i][2], B[2][j], hfma(B[i][1], B[1][j], B[i][0] * B[0][j]));
        sig[i][j] = hfma(be, b2, al * B[i][j]);
        sig[j][i] = sig[i][j];
      }
    const H sh = hfma(hval<H>(-1.0 / 3.0), sig[0][0] + sig[1][1] + sig[2][2], p);
#pragma unroll
    for (int i = 0; i < 3; ++i) sig[i][i] = sig[i][i] + sh;
    return;
  }
  H Fb[3][3], Cb[3][3], S[3][3], T[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Fb[i][j] = F[i][j] * s;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j) {
      Cb[i][j] = hfma(Fb[2][i], Fb[2][j], hfma(Fb[1][i], Fb[1][j], Fb[0][i] * Fb[0][j]));
      Cb[j][i] = Cb[i][j];
    }
  const H B[6] = {two * c[1], two * c[2], two * c[2], c[3], c[3], c[2]};
  const H E[6] = {half * (Cb[0][0] - one), half * (Cb[1][1] - one), half * (Cb[2][2] - one), Cb[1][0], Cb[2][0],
                  Cb[2][1]};
  H DQ[6], dot = zero;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    DQ[i] = B[i] * E[i];
    dot = hfma(E[i], DQ[i], dot);
  }
  const H t1 = half * c[0] * hexp(half * dot) * rJ;
  S[0][0] = t1 * DQ[0];
  S[1][1] = t1 * DQ[1];
  S[2][2] = t1 * DQ[2];
  S[0][1] = S[1][0] = t1 * DQ[3];
  S[0][2] = S[2][0] = t1 * DQ[4];
  S[1][2] = S[2][1] = t1 * DQ[5];
  // sigma_bar = F_bar (S / J) F_bar^T
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) T[i][j] = hfma(Fb[i][2], S[2][j], hfma(Fb[i][1], S[1][j], Fb[i][0] * S[0][j]));
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j) {
      sig[i][j] = hfma(T[i][2], Fb[j][2], hfma(T[i][1], Fb[j][1], T[i][0] * Fb[j][0]));
      sig[j][i] = sig[i][j];
    }
  const H sh = hfma(hval<H>(-1.0 / 3.0), sig[0][0] + sig[1][1] + sig[2][2], p);
#pragma unroll
  for (int i = 0; i < 3; ++i) sig[i][i] = sig[i][i] + sh;
}

// Geometric Gauss-point data (dXi/dNu row-major, J_x, 1 / J_x) in H.
__device__ __forceinline__ void load_geo(const KParams& P, int e, int g, double dn[9], double& jx, double& rjx) {
  const double* geo = &P.geo[((size_t)e * NG + g) * 10];
#pragma unroll
  for (int i = 0; i < 9; ++i) dn[i] = geo[i];
  jx = geo[9];
  rjx = P.geo_rj[(size_t)e * NG + g];
}
__device__ __forceinline__ void load_geo(const KParams& P, int e, int g, dd dn[9], dd& jx, dd& rjx) {
  const float2* geo = reinterpret_cast<const float2*>(P.geo_dd) + ((size_t)e * NG + g) * 10;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const float2 v = geo[i];
    dn[i] = {v.x, v.y};
  }
  const float2 v = geo[9];
  jx = {v.x, v.y};
  rjx = to_dd(P.geo_rj[(size_t)e * NG + g]);
}
// The same data in the displacement block's type T; FP32 takes the leading
// parts of the double-float copy, which are the values rounded to FP32 (a
// conversion takes the FP64 pipe as long as an FP64 operation).
__device__ __forceinline__ void load_geo_t(const KParams& P, int e, int g, double dn[9], double& rjx) {
  double jx;
  load_geo(P, e, g, dn, jx, rjx);
}
__device__ __forceinline__ void load_geo_t(const KParams& P, int e, int g, float dn[9], float& rjx) {
  const float2* geo = reinterpret_cast<const float2*>(P.geo_dd) + ((size_t)e * NG + g) * 10;
#pragma unroll
  for (int i = 0; i < 9; ++i) dn[i] = geo[i].x;
  rjx = 1.0f / geo[9].x;
}

template <class T, class H>
__device__ __forceinline__ T to_t(H v) {
  if constexpr (sizeof(T) == 4)
    return hf(v);
  else
    return hd(v);
}

// Constant tables (pressure basis and weights at the Gauss points, products of
// the 1-D basis functions) into shared memory.
template <int N1, int PM, int EG_, class T, class H, int NT = 256>
__device__ __forceinline__ void mix_tables(const KParams& P, unsigned char* sm) {
  using C = MixCfg<N1, PM, EG_, T, NT>;
  H* s_psi = reinterpret_cast<H*>(sm + C::O_PSI64);  // [g][q]
  H* s_w = reinterpret_cast<H*>(sm + C::O_W);        // [g]
  const int tid = threadIdx.x;
  // ---- constant tables
  for (int i = tid; i < NG * 8; i += C::THREADS) s_psi[i] = hval<H>(P.gbf_p[i]);
  for (int i = tid; i < NG; i += C::THREADS) s_w[i] = hval<H>(P.gw[i]);
  uu_table<N1, T>(reinterpret_cast<T*>(sm + C::O_MM), tid, C::THREADS);
}

// Element number of entry i of an element list (NULL: P.first_elem + i).
__device__ __forceinline__ int elem_at(const KParams& P, const int32_t* elems, int i) {
  return elems ? elems[i] : P.first_elem + i;
}

// One group of up to EG elements, elems[grp*EG ...] of the count elements
// of the current colour.  p4_first swaps the order of the independent stages
// P3 (residual and coupling) and P4 (displacement block).  OUT = 0 adds the
// element's entries into the CSR values and the residual (first contributor
// in colour order stores, later ones add); OUT = 1 stores them into the
// element's staging records (*SO), which the row gather sums afterwards;
// OUT = 2 forms the residual alone and stores it into the element's residual
// record (cmfe::RecR).
template <int N1, int PM, int EG_, class T, class H, int OUT = 0, int NT = 256>
__device__ __forceinline__ void mix_group(const KParams& P, const int32_t* elems, int count, int grp, bool p4_first,
                                          unsigned char* sm, const cmfe::StageOut* SO = nullptr) {
  constexpr bool RES = OUT == 2;
  using C = MixCfg<N1, PM, EG_, T, NT, RES>;
  constexpr int NPE = C::NPE, NPP = C::NPP, NR = C::NR, NU3 = C::NU3, EG = C::EG;
  using R = cmfe::Rec<NPE, NPP, T>;
  using RR = cmfe::RecR<NPE, NPP>;
  H* s_psi = reinterpret_cast<H*>(sm + C::O_PSI64);  // [g][q]
  H* s_w = reinterpret_cast<H*>(sm + C::O_W);        // [g]
  H* s_z = reinterpret_cast<H*>(sm + C::O_Z);        // [el][c][a]
  H* s_p = reinterpret_cast<H*>(sm + C::O_P);        // [el][q]
  H* s_dz = reinterpret_cast<H*>(sm + C::O_DZ);      // [el][g][c*3+k]
  H* s_pg = reinterpret_cast<H*>(sm + C::O_PG);      // [el][g]
  H* s_r64 = reinterpret_cast<H*>(sm + C::O_R64);    // [el][g][REC64]
  T* s_D = reinterpret_cast<T*>(sm + C::O_R32);                // [el][g][UU_REC]
  T* s_mm = reinterpret_cast<T*>(sm + C::O_MM);
  int* s_node = reinterpret_cast<int*>(sm + (OUT == 2 ? C::O_NODE2 : OUT == 1 ? C::O_NODE1 : C::O_NODE0));  // [el][NR+1]
  // Every scratch array ends inside its region (a region begins where the one
  // before it ends, and what shares one is separated by barriers: the stages
  // below; run thread by thread on the CPU, none leaves its array or races).
  static_assert(sizeof(H) == 8 && EG * 3 * NPE * 8 <= C::O_P - C::O_Z && EG * 8 * 8 <= C::O_PG - C::O_P &&
                    EG * NG * 8 <= C::O_R64 - C::O_PG && EG * NG * C::REC64 * 8 <= C::O_R32 - C::O_R64 &&
                    EG * NG * 9 * 8 <= C::O_BASE - C::O_DZ,
                "positions, pressures, Gauss-point records, gradients");
  static_assert(OUT != 0 || (EG * 9 * NPE * 4 <= C::O_TAB - C::O_BASE && EG * NPE * NPE * 2 <= C::O_NODE0 - C::O_TAB),
                "scatter addresses and rank tables");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // FP64 items are dealt to the warps from a different first warp in each
  // CTA of an SM: an SM sub-partition takes 64 cycles per FP64 warp
  // instruction, and most stages have fewer items than threads
  const int vt = ((warp + blockIdx.x / P.wave) % (C::THREADS / 32)) * 32 + lane;
  const int nu = P.nu;
  const int nvalid = min(EG, count - grp * EG);
  __syncthreads();
  // ---- P0: element nodes and table ids
  for (int i = tid; i < EG * (NR + 1); i += C::THREADS) {
    const int el = i / (NR + 1), r = i % (NR + 1);
    int v = 0;
    if (el < nvalid) {
      const int e = elem_at(P, elems, grp * EG + el);
      if (r < NPE)
        v = P.elem_u[(size_t)e * NPE + r];
      else if (r < NR)
        v = PM ? P.elem_p[(size_t)e * 8 + (r - NPE)] : e;
      else
        v = P.elem_table[e];
    }
    s_node[i] = v;
  }
  __syncthreads();
  // positions from a node of the element: only their derivatives are wanted,
  // and the lines below then round values of the element's size, not the
  // mesh's.  Against 113-bit arithmetic the FP64 Jacobian of nine meshes is 0.73
  // to 0.94 times, the residual 0.69 to 0.79 times as far off as contracting
  // over all Gauss points in the reference's order (16^3 box: 2.6e-15 against
  // 3.5e-15, 5.8e-14 against 7.6e-14); residual of the 32^3 box 635 -> 638 us.
  for (int i = tid; i < EG * 3 * NPE; i += C::THREADS) {
    const int el = i / (3 * NPE), c = (i / NPE) % 3, a = i % NPE;
    const int* nd = s_node + el * (NR + 1);
    const double* x = P.x + (size_t)c * nu;
    s_z[i] = hval<H>(el < nvalid ? x[nd[a]] - x[nd[NPE / 2]] : 0.0);
  }
  for (int i = tid; i < EG * NPP; i += C::THREADS) {
    const int el = i / NPP, q = i % NPP;
    s_p[el * 8 + q] = hval<H>(el < nvalid ? P.x[(size_t)3 * nu + s_node[el * (NR + 1) + NPE + q]] : 0.0);
  }
  __syncthreads();
  // ---- P1: dz/dxi at the Gauss points by sum factorisation over the
  // tensor-product basis: xi1, then xi2, then xi3, one line of nodes or points
  // per item (fe_line.cuh; B = values, D = derivatives).
  {
    constexpr int N2 = N1 * N1;
    H* S1 = reinterpret_cast<H*>(sm + C::O_R32);  // [B|D][ec][g1][a2a3]
    H* S2 = S1 + EG * 3 * 2 * 3 * N2;             // [BB|BD|DB][ec][g1][g2][a3]
    constexpr int S1T = EG * 3 * 3 * N2, S2T = EG * 3 * 9 * N1;
    static_assert((2 * S1T + 3 * S2T) * 8 <= C::O_DZ - C::O_R32, "scratch of the gradients");
    for (int i = vt; i < EG * 3 * N2; i += C::THREADS) {
      const int j = i % N2, ec = i / N2;
      H z[N1], B[3], D[3];
#pragma unroll
      for (int a1 = 0; a1 < N1; ++a1) z[a1] = s_z[ec * NPE + N1 * j + a1];
      line_BD<N1, H>(z, B, D);
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        S1[(ec * 3 + g) * N2 + j] = B[g];
        S1[S1T + (ec * 3 + g) * N2 + j] = D[g];
      }
    }
    __syncthreads();
    constexpr int L2I = EG * 3 * 3 * N1;  // (ec, g1, a3)
    for (int i = vt; i < 2 * L2I; i += C::THREADS) {
      const bool d1 = i >= L2I;
      const int r = d1 ? i - L2I : i;
      const int a3 = r % N1, eg = r / N1;  // eg = ec * 3 + g1
      const H* s = S1 + (d1 ? S1T : 0) + eg * N2 + N1 * a3;
      H z[N1], B[3];
#pragma unroll
      for (int a2 = 0; a2 < N1; ++a2) z[a2] = s[a2];
      if (d1) {
        line_B<N1, H>(z, B);
#pragma unroll
        for (int g = 0; g < 3; ++g) S2[2 * S2T + (eg * 3 + g) * N1 + a3] = B[g];
      } else {
        H D[3];
        line_BD<N1, H>(z, B, D);
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          S2[(eg * 3 + g) * N1 + a3] = B[g];
          S2[S2T + (eg * 3 + g) * N1 + a3] = D[g];
        }
      }
    }
    __syncthreads();
    constexpr int L3I = EG * 3 * 9;  // (ec, g1, g2)
    for (int i = vt; i < 3 * L3I; i += C::THREADS) {
      const int k = i / L3I, r = i % L3I;  // d/dxi1: DB, d/dxi2: BD, d/dxi3: BB
      const int g2 = r % 3, g1 = (r / 3) % 3, ec = r / 9, el = ec / 3, c = ec % 3;
      const H* s = S2 + (2 - k) * S2T + r * N1;
      H z[N1], o[3];
#pragma unroll
      for (int a3 = 0; a3 < N1; ++a3) z[a3] = s[a3];
      if (k == 2)
        line_D<N1, H>(z, o);
      else
        line_B<N1, H>(z, o);
#pragma unroll
      for (int g3 = 0; g3 < 3; ++g3) s_dz[(el * NG + g1 + 3 * g2 + 9 * g3) * 9 + c * 3 + k] = o[g3];
    }
  }
  for (int i = vt; i < EG * NG; i += C::THREADS) {
    const int el = i / NG, g = i % NG;
    H pg;
    if (PM) {
      pg = hval<H>(0.0);
#pragma unroll
      for (int q = 0; q < 8; ++q) pg = hfma(s_psi[g * 8 + q], s_p[el * 8 + q], pg);
    } else {
      pg = s_p[el * 8];
    }
    s_pg[i] = pg;
  }
  __syncthreads();
  // ---- P2 (H: kinematics, stress and the residual / coupling records per
  // Gauss point) and P2b (T: the spatial tangent pulled back to xi space)
  // run at the same time on the two halves of the CTA, so that the FP64 and
  // the FP32 pipes overlap; P2b forms the kinematics it needs itself from
  // the same gradients.
  // (The residual alone: P2 on all warps.)
  constexpr int HALF = RES ? C::THREADS : C::THREADS / 2;
  if (vt < HALF) {
    for (int t = vt; t < EG * NG; t += HALF) {
      const int el = t / NG, g = t % NG;
      if (el >= nvalid) continue;
      const int e = elem_at(P, elems, grp * EG + el);
      H M[3][3], adj[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k) M[c][k] = s_dz[t * 9 + c * 3 + k];
      adj[0][0] = M[1][1] * M[2][2] - M[1][2] * M[2][1];
      adj[0][1] = M[0][2] * M[2][1] - M[0][1] * M[2][2];
      adj[0][2] = M[0][1] * M[1][2] - M[0][2] * M[1][1];
      adj[1][0] = M[1][2] * M[2][0] - M[1][0] * M[2][2];
      adj[1][1] = M[0][0] * M[2][2] - M[0][2] * M[2][0];
      adj[1][2] = M[0][2] * M[1][0] - M[0][0] * M[1][2];
      adj[2][0] = M[1][0] * M[2][1] - M[1][1] * M[2][0];
      adj[2][1] = M[0][1] * M[2][0] - M[0][0] * M[2][1];
      adj[2][2] = M[0][0] * M[1][1] - M[0][1] * M[1][0];
      const H det = M[0][0] * adj[0][0] + M[0][1] * adj[1][0] + M[0][2] * adj[2][0];
      H dn[9], jx, rjx;
      load_geo(P, e, g, dn, jx, rjx);
      const H jz = habs(det);
      const H w = s_w[g];
      const bool dpos = hpos(det);
      const H sw = dpos ? w : -w;  // J_z w dxi/dz = sign(det) w adj
      const H pgv = s_pg[t];
      H* rec = &s_r64[t * C::REC64];
      bool ok = dpos;
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          adj[k][n] = sw * adj[k][n];
          if (!RES) rec[9 + k * 3 + n] = adj[k][n];
        }
      if (P.r != nullptr) {
        H F[3][3], sig[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) F[i][j] = hfma(M[i][2], dn[6 + j], hfma(M[i][1], dn[3 + j], M[i][0] * dn[j]));
        const double* cm = P.mat + (P.matpe ? (size_t)e * P.nmat : 0);
        const H cc[4] = {hval<H>(cm[0]), hval<H>(cm[1]), hval<H>(P.nmat > 2 ? cm[2] : 0.0),
                         hval<H>(P.nmat > 3 ? cm[3] : 0.0)};
        mix_stress<H>(P.law, cc, F, jz * rjx, pgv, sig);
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const H v = hfma(adj[k][2], sig[2][m], hfma(adj[k][1], sig[1][m], adj[k][0] * sig[0][m]));
            rec[k * 3 + m] = v;
            ok = ok && hfinite(v);
          }
        rec[C::T1] = w * (jz - jx);  // J_x w (J - 1)
      }
      if (!ok) atomicOr(P.status, 1u);
    }
  } else if constexpr (!RES) {
    for (int t = vt - HALF; t < (P.res_only ? 0 : EG * NG); t += HALF) {
      const int el = t / NG, g = t % NG;
      if (el >= nvalid) continue;
      const int e = elem_at(P, elems, grp * EG + el);
      T Mt[3][3], dn[9], rjx, ct[4];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k) Mt[c][k] = to_t<T>(s_dz[t * 9 + c * 3 + k]);
      load_geo_t(P, e, g, dn, rjx);
      const double* cm = P.mat + (P.matpe ? (size_t)e * P.nmat : 0);
#pragma unroll
      for (int i = 0; i < 4; ++i) ct[i] = i < P.nmat ? (T)cm[i] : T(0);
      if (!uu_tangent<T>(P.law, ct, Mt, dn, rjx, to_t<T>(s_w[g]), to_t<T>(s_pg[t]), &s_D[t * UU_REC]))
        atomicOr(P.status, 1u);
    }
  }
  __syncthreads();
  // P3 (FP64 pipe) and P4 (displacement block) are independent; the
  // second wave of CTAs runs them in the opposite order so that the two
  // CTAs sharing an SM work on different pipes.
  for (int ph = 0; ph < (RES ? 1 : 2); ++ph) {
    if (RES || (ph == 0) != p4_first) {
      // ---- P3: residual rows and pressure-coupling columns (high precision H)
      __syncthreads();
      constexpr int N2 = N1 * N1;
      // Sum factorisation over the tensor-product basis, line by line: for
      // V = rec[roff + 3 k + m],
      //   R(m, a) = sum_g sum_k M_k(g; a) V_g(k, m),
      // M_k the product of the 1-D derivatives along xi_k and the 1-D values
      // along the other two.  xi1 is contracted for each k, xi2 with the k = 0
      // and k = 1 terms merged (both take values along xi3), xi3 with all
      // merged.  roff = 0: V = P, the residual rows; roff = 9: V = A = J_z w
      // dxi/dz, the element-based pressure coupling column.
      H* U1 = reinterpret_cast<H*>(sm + C::O_U1);  // [el][m][k][a1][g2 + 3 g3]
      H* U2 = reinterpret_cast<H*>(sm + C::O_U2);  // [W|U][el][m][a1 + N1 a2][g3]
      H* Lq = reinterpret_cast<H*>(sm + C::O_U3);  // residual pressure rows: [el][q1][j], then [el][q1 q2][g3]
      static_assert(EG * 9 * N1 * 9 * 8 <= C::O_U2 - C::O_U1 && 2 * EG * 3 * N2 * 3 * 8 <= C::O_U3 - C::O_U2 &&
                        (EG * 2 * 9 + EG * 4 * 3) * 8 <= C::O_BASE - C::O_U3,
                    "scratch of the residual");
      auto sumfact = [&](int roff, bool prows, auto emit, auto emit_p) {
        for (int i = vt; i < EG * 81; i += C::THREADS) {
          const int j = i % 9, k = (i / 9) % 3, m = (i / 27) % 3, el = i / 81;
          const H* rec = &s_r64[(el * NG + 3 * j) * C::REC64 + roff + k * 3 + m];
          const H v[3] = {rec[0], rec[C::REC64], rec[2 * C::REC64]};
          H o[N1];
          if (k == 0)
            line_Dt<N1, H>(v, o);
          else
            line_Bt<N1, H>(v, o);
#pragma unroll
          for (int a = 0; a < N1; ++a) U1[((i / 9) * N1 + a) * 9 + j] = o[a];
        }
        if (PM && prows) {  // the pressure rows, on the warps the lines leave over
          for (int i = C::THREADS - 1 - vt; i < EG * 9; i += C::THREADS) {
            const H* rec = &s_r64[(i / 9 * NG + 3 * (i % 9)) * C::REC64 + C::T1];
            const H v[3] = {rec[0], rec[C::REC64], rec[2 * C::REC64]};
            H o[2];
            line_Lt<H>(v, o);
            Lq[(i / 9 * 2) * 9 + i % 9] = o[0];
            Lq[(i / 9 * 2 + 1) * 9 + i % 9] = o[1];
          }
        }
        __syncthreads();
        constexpr int I2 = EG * 9 * N1;  // (el, m, a1, g3)
        for (int i = vt; i < 2 * I2; i += C::THREADS) {
          const bool third = i >= I2;
          const int r = third ? i - I2 : i;
          const int g3 = r % 3, a1 = (r / 3) % N1, em = r / (3 * N1);
          const H* u = U1 + (em * 3 * N1 + a1) * 9 + 3 * g3;
          H o[N1];
          if (third)
            line_Bt<N1, H>(u + 2 * N1 * 9, o);
          else
            line_BtDt<N1, H>(u, u + N1 * 9, o);
#pragma unroll
          for (int a = 0; a < N1; ++a) U2[((third ? EG * 3 : 0) + em) * N2 * 3 + (a1 + N1 * a) * 3 + g3] = o[a];
        }
        if (PM && prows) {
          H* Lq2 = Lq + EG * 18;
          for (int i = C::THREADS - 1 - vt; i < EG * 6; i += C::THREADS) {  // (el, q1, g3)
            H o[2];
            line_Lt<H>(Lq + (i / 3) * 9 + 3 * (i % 3), o);
            const int q1 = (i / 3) % 2, el = i / 6;
            Lq2[(el * 4 + q1) * 3 + i % 3] = o[0];
            Lq2[(el * 4 + q1 + 2) * 3 + i % 3] = o[1];
          }
        }
        __syncthreads();
        for (int i = vt; i < EG * 3 * N2; i += C::THREADS) {
          const int a12 = i % N2, m = (i / N2) % 3, el = i / (3 * N2);
          H o[N1];
          line_BtDt<N1, H>(U2 + i * 3, U2 + (EG * 3 * N2 + i) * 3, o);
          if (el < nvalid) emit(el, m, a12, o);
        }
        if (prows) {
          if (PM) {
            const H* Lq2 = Lq + EG * 18;
            for (int i = C::THREADS - 1 - vt; i < EG * 4; i += C::THREADS) {  // (el, q1 q2)
              H o[2];
              line_Lt<H>(Lq2 + i * 3, o);
              if (i / 4 < nvalid) {
                emit_p(i / 4, i % 4, o[0]);
                emit_p(i / 4, i % 4 + 4, o[1]);
              }
            }
          } else {
            for (int el = C::THREADS - 1 - vt; el < nvalid; el += C::THREADS) {
              H acc = hval<H>(0.0);
              for (int g = 0; g < NG; ++g) acc = acc + s_r64[(el * NG + g) * C::REC64 + C::T1];
              emit_p(el, 0, acc);
            }
          }
        }
        __syncthreads();
      };
      if (P.r != nullptr) {
        auto add_r = [&](int el, int ln, size_t gr, double v) {
          const int* nd = &s_node[el * (NR + 1)];
          const uint16_t* tab = P.tables + (size_t)nd[NR] * NR * NR;
          if (tab[ln * NR + ln] & 0x8000)
            P.r[gr] = v;
          else
            atomicAdd(&P.r[gr], v);
        };
        sumfact(
            0, true,
            [&](int el, int m, int a12, const H (&o)[N1]) {
#pragma unroll
              for (int a3 = 0; a3 < N1; ++a3) {
                const int a = a12 + N2 * a3;
                if constexpr (OUT == 1) {
                  unsigned char* er = SO->rec + (size_t)elem_at(P, elems, grp * EG + el) * R::BYTES;
                  reinterpret_cast<double*>(er + a * R::ROW + R::OR)[m] = hd(o[a3]);
                } else if constexpr (OUT == 2) {
                  RR::of(*SO, elem_at(P, elems, grp * EG + el))[3 * a + m] = hd(o[a3]);
                } else {
                  add_r(el, a, (size_t)m * nu + s_node[el * (NR + 1) + a], hd(o[a3]));
                }
              }
            },
            [&](int el, int q, H v) {
              if constexpr (OUT == 1) {
                unsigned char* er = SO->rec + (size_t)elem_at(P, elems, grp * EG + el) * R::BYTES;
                reinterpret_cast<double*>(er + R::P0 + q * R::PROW)[NU3] = hd(v);
              } else if constexpr (OUT == 2) {
                RR::of(*SO, elem_at(P, elems, grp * EG + el))[NU3 + q] = hd(v);
              } else {
                add_r(el, NPE + q, (size_t)3 * nu + s_node[el * (NR + 1) + NPE + q], hd(v));
              }
            });
      }
      // one pressure-coupling entry K(q, (n, b)) and its mirror
      if constexpr (!RES) {
      auto emit_c = [&](int el, int q, int n, int b, double kv) {
        if constexpr (OUT == 1) {
          unsigned char* er = SO->rec + (size_t)elem_at(P, elems, grp * EG + el) * R::BYTES;
          reinterpret_cast<double*>(er + R::P0 + q * R::PROW)[n * NPE + b] = kv;
          reinterpret_cast<double*>(er + b * R::ROW + R::OC)[n * NPP + q] = kv;
        } else {
          const int* nd = &s_node[el * (NR + 1)];
          const uint16_t* tab = P.tables + (size_t)nd[NR] * NR * NR;
          const int lq = NPE + q, pq = nd[lq], nb = nd[b];
          const uint16_t tqb = tab[lq * NR + b], tbq = tab[b * NR + lq];
          const size_t p1 = (size_t)P.cp_row_ptr[(size_t)3 * nu + pq] + (size_t)n * P.wp[pq] + (tqb & 0x7fff);
          if (tqb & 0x8000)
            P.vals[p1] = kv;
          else
            atomicAdd(&P.vals[p1], kv);
          const size_t p2 = (size_t)P.cp_row_ptr[(size_t)n * nu + nb] + (tbq & 0x7fff);
          if (tbq & 0x8000)
            P.vals[p2] = kv;
          else
            atomicAdd(&P.vals[p2], kv);
        }
      };
      if (!PM && !P.res_only)
        sumfact(
            9, false,
            [&](int el, int n, int b12, const H (&o)[N1]) {
#pragma unroll
              for (int b3 = 0; b3 < N1; ++b3) emit_c(el, 0, n, b12 + N2 * b3, hd(o[b3]));
            },
            [](int, int, H) {});
      // Pressure-coupling block for nodal (trilinear) pressure,
      //   K(q, n, b) = sum_k sum_g psi_q(g) A_g(k, n) dN_b/dxi_k(g),  A_g = J_z w dxi/dz,
      // psi_q = L(q1) L(q2) L(q3), dN_b/dxi_k = M1k(b1) M2k(b2) M3k(b3), line by
      // line with the products of the linear and the 1-D basis functions
      // (line_L): xi1 for every k, xi2 with k = 0 and 1 merged, xi3 with all.
      if (PM && !P.res_only) {
        constexpr int L2 = C::L2;
        H* T1 = reinterpret_cast<H*>(sm + C::O_DZ);  // [n][el][k][q1 b1][g2 + 3 g3]
        H* W2 = T1 + EG * 9 * L2 * 9;                // [n][el][q1 b1][q2 b2][g3]
        H* V2 = W2 + EG * 3 * L2 * L2 * 3;           // the k = 2 terms
        static_assert(!PM || (EG * 9 * L2 * 9 + 2 * EG * 3 * L2 * L2 * 3) * 8 <= C::O_BASE - C::O_DZ,
                      "scratch of the coupling");
        for (int i = vt; i < EG * 81; i += C::THREADS) {
          const int j = i % 9, k = (i / 9) % 3, el = (i / 27) % EG, n = i / (27 * EG);
          const H* a = &s_r64[(el * NG + 3 * j) * C::REC64 + 9 + 3 * k + n];
          const H v[3] = {a[0], a[C::REC64], a[2 * C::REC64]};
          H o[L2];
          if (k == 0)
            line_L<N1, 0, 1, H>(v, v, o);
          else
            line_L<N1, 1, 0, H>(v, v, o);
#pragma unroll
          for (int b = 0; b < L2; ++b) T1[((i / 9) * L2 + b) * 9 + j] = o[b];
        }
        __syncthreads();
        constexpr int I2 = EG * 3 * L2 * 3;  // (n, el, q1 b1, g3)
        for (int i = vt; i < 2 * I2; i += C::THREADS) {
          const bool third = i >= I2;
          const int r = third ? i - I2 : i;
          const int g3 = r % 3, b1 = (r / 3) % L2, ne = r / (3 * L2);
          const H* t = T1 + (ne * 3 * L2 + b1) * 9 + 3 * g3;
          H o[L2];
          if (third)
            line_L<N1, 1, 0, H>(t + 2 * L2 * 9, t, o);
          else
            line_L<N1, 1, 1, H>(t, t + L2 * 9, o);
          H* out = (third ? V2 : W2) + (ne * L2 + b1) * L2 * 3 + g3;
#pragma unroll
          for (int b = 0; b < L2; ++b) out[b * 3] = o[b];
        }
        __syncthreads();
        for (int i = vt; i < EG * 3 * L2 * L2; i += C::THREADS) {
          const int qb2 = i % L2, qb1 = (i / L2) % L2, el = (i / (L2 * L2)) % EG, n = i / (L2 * L2 * EG);
          H o[L2];
          line_L<N1, 1, 1, H>(W2 + i * 3, V2 + i * 3, o);
          if (el >= nvalid) continue;
          const int q12 = qb1 / N1 + 2 * (qb2 / N1), b12 = qb1 % N1 + N1 * (qb2 % N1);
#pragma unroll
          for (int qb3 = 0; qb3 < L2; ++qb3)
            emit_c(el, q12 + 4 * (qb3 / N1), n, b12 + N2 * (qb3 % N1), hd(o[qb3]));
        }
      }
      // structurally zero pressure-pressure entries, stored by their first contributor
      for (int i = tid; i < (P.res_only || OUT == 1 ? 0 : EG * NPP * NPP); i += C::THREADS) {
        const int el = i / (NPP * NPP), q = (i / NPP) % NPP, q2 = i % NPP;
        if (el >= nvalid) continue;
        const int* nd = &s_node[el * (NR + 1)];
        const uint16_t t = P.tables[(size_t)nd[NR] * NR * NR + (NPE + q) * NR + NPE + q2];
        if (t & 0x8000) {
          const int pq = nd[NPE + q];
          P.vals[(size_t)P.cp_row_ptr[(size_t)3 * nu + pq] + 3 * (size_t)P.wp[pq] + (t & 0x7fff)] = 0.0;
        }
      }
      }
    } else if constexpr (!RES) {
      // ---- P4: displacement blocks by sum factorisation, warp by warp
      if (!P.res_only) {
        // Coloured order: scatter addresses staged in shared memory:
        // base[el][3m+n][a] = start of the n-block of row (m, node a), and the
        // element's rank table over its u nodes.
        int* s_base = reinterpret_cast<int*>(sm + C::O_BASE);
        uint16_t* s_tab = reinterpret_cast<uint16_t*>(sm + C::O_TAB);
        T* s1 = reinterpret_cast<T*>(sm + C::O_DZ) + (size_t)warp * UUCfg<N1>::S1;
        static_assert(C::THREADS / 32 * UUCfg<N1>::S1 * (int)sizeof(T) <= C::O_BASE - C::O_DZ &&
                          EG * NG * UU_REC * (int)sizeof(T) <= C::O_DZ - C::O_R32,
                      "scratch of the displacement block");
        if constexpr (OUT == 0) {
          for (int i = tid; i < EG * 9 * NPE; i += C::THREADS) {
            const int a = i % NPE, mn = (i / NPE) % 9, el = i / (9 * NPE);
            const int na = s_node[el * (NR + 1) + a];
            s_base[i] = el < nvalid ? P.uu_row_ptr[(size_t)(mn / 3) * nu + na] + (mn % 3) * P.wu[na] : 0;
          }
          for (int i = tid; i < EG * NPE * NPE; i += C::THREADS) {
            const int ab = i % (NPE * NPE), el = i / (NPE * NPE);
            const int a = ab / NPE, b = ab % NPE;
            s_tab[i] = el < nvalid ? P.tables[(size_t)s_node[el * (NR + 1) + NR] * NR * NR + a * NR + b] : 0;
          }
        }
        __syncthreads();  // the scratch below is free (P3 done or not begun)
        for (int task = warp; task < UUCfg<N1>::tasks(nvalid); task += C::THREADS / 32) {
          uu_warp_task<N1, T>(s_D, s_mm, s1, task, nvalid, lane,
                              [&](int el, int blk, int a12, int b12, const T (&K)[N1][N1]) {
            int m, n;
            blk_mn(blk, m, n);
            // a diagonal block's entries beyond its diagonal are mirrors
            const bool diag = blk < 3 && a12 == b12;
            constexpr int NP = N1 * N1;
            if constexpr (OUT == 1) {
              unsigned char* er = SO->rec + (size_t)elem_at(P, elems, grp * EG + el) * R::BYTES;
              T* s0 = reinterpret_cast<T*>(er + a12 * R::ROW) + (3 * m + n) * NPE + b12;
              T* s1m = reinterpret_cast<T*>(er + b12 * R::ROW) + (3 * n + m) * NPE + a12;
              constexpr int A3 = NP * (R::ROW / (int)sizeof(T));  // next a3: NP node rows on
#pragma unroll
              for (int a3 = 0; a3 < N1; ++a3)
#pragma unroll
                for (int b3 = 0; b3 < N1; ++b3) {
                  if (diag && a3 > b3) continue;
                  if (N1 == 2 && blk < 3 && a12 + NP * a3 > b12 + NP * b3) continue;
                  s0[a3 * A3 + b3 * NP] = K[a3][b3];
                  if (!(diag && a3 == b3)) s1m[b3 * A3 + a3 * NP] = K[a3][b3];
                }
            } else {
              const int* bs = &s_base[el * 9 * NPE];
              const uint16_t* tb = &s_tab[el * NPE * NPE];
#pragma unroll
              for (int a3 = 0; a3 < N1; ++a3)
#pragma unroll
                for (int b3 = 0; b3 < N1; ++b3) {
                  if (diag && a3 > b3) continue;
                  const int a = a12 + NP * a3, b = b12 + NP * b3;
                  if (N1 == 2 && blk < 3 && a > b) continue;
                  const float v = (float)K[a3][b3];
                  const uint16_t tab_ab = tb[a * NPE + b];
                  const int p1 = bs[(m * 3 + n) * NPE + a] + (tab_ab & 0x7fff);
                  if (tab_ab & 0x8000)
                    P.vals_uu[p1] = v;
                  else
                    atomicAdd(&P.vals_uu[p1], v);
                  if (diag && a3 == b3) continue;
                  const uint16_t tab_ba = tb[b * NPE + a];
                  const int p2 = bs[(n * 3 + m) * NPE + b] + (tab_ba & 0x7fff);
                  if (tab_ba & 0x8000)
                    P.vals_uu[p2] = v;
                  else
                    atomicAdd(&P.vals_uu[p2], v);
                }
            }
          });
        }
        __syncthreads();  // P3 may run next and reuse the scratch
      }
    }
  }
}

}  // namespace
