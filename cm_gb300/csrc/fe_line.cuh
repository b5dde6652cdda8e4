// libcm_fe: one-dimensional transforms of the sum-factorised FP64 stages.
//
// A triquadratic (trilinear) element is a tensor product of lines of N1 = 3
// (2) equally spaced nodes, integrated with the symmetric 3-point
// Gauss-Legendre rule at s = -sqrt(0.6), 0, sqrt(0.6) on [-1, 1].  Written in
// the even and odd combinations of a line's values, a transform takes about
// half the operations of its 3 x N1 matrix: for a quadratic,
//   z(s) = z1 - s/2 o + s^2/2 t,  dz/dxi(s) = -o + 2 s t,  o = z0 - z2, t = z0 - 2 z1 + z2,
// and the transposes (Gauss points to nodes) follow.  What counts is the
// number of warp instructions on the FP64 pipe: one takes 19 cycles of an SM
// (measured, DFMA and DADD alike, whatever lanes are active).
#pragma once

#include "fe_dd.cuh"

namespace {

constexpr double LN_S = 0.77459666924148340;  // sqrt(0.6)

template <class H>
__device__ __forceinline__ H hc(double x) { return hval<H>(x); }

// Values at the Gauss points from nodal values.
template <int N1, class H>
__device__ __forceinline__ void line_B(const H* z, H* B) {
  if constexpr (N1 == 2) {
    const H s = hc<H>(0.5) * (z[0] + z[1]), o = z[0] - z[1];
    B[0] = hfma(hc<H>(0.5 * LN_S), o, s);
    B[1] = s;
    B[2] = hfma(hc<H>(-0.5 * LN_S), o, s);
  } else {
    const H o = z[0] - z[2], t = hfma(hc<H>(-2.0), z[1], z[0] + z[2]);
    const H e = hfma(hc<H>(0.3), t, z[1]);
    B[0] = hfma(hc<H>(0.5 * LN_S), o, e);
    B[1] = z[1];
    B[2] = hfma(hc<H>(-0.5 * LN_S), o, e);
  }
}
// Derivatives at the Gauss points.
template <int N1, class H>
__device__ __forceinline__ void line_D(const H* z, H* D) {
  if constexpr (N1 == 2) {
    D[0] = D[1] = D[2] = z[1] - z[0];
  } else {
    const H o = z[2] - z[0], t = hfma(hc<H>(-2.0), z[1], z[0] + z[2]);
    D[0] = hfma(hc<H>(-2.0 * LN_S), t, o);
    D[1] = o;
    D[2] = hfma(hc<H>(2.0 * LN_S), t, o);
  }
}
// Both.
template <int N1, class H>
__device__ __forceinline__ void line_BD(const H* z, H* B, H* D) {
  if constexpr (N1 == 2) {
    line_B<N1, H>(z, B);
    line_D<N1, H>(z, D);
  } else {
    const H o = z[2] - z[0], t = hfma(hc<H>(-2.0), z[1], z[0] + z[2]);
    const H e = hfma(hc<H>(0.3), t, z[1]);
    B[0] = hfma(hc<H>(-0.5 * LN_S), o, e);
    B[1] = z[1];
    B[2] = hfma(hc<H>(0.5 * LN_S), o, e);
    D[0] = hfma(hc<H>(-2.0 * LN_S), t, o);
    D[1] = o;
    D[2] = hfma(hc<H>(2.0 * LN_S), t, o);
  }
}
// Transposes: out[a] = sum_g B_a(g) v[g], sum_g D_a(g) v[g], and their sum.
template <int N1, class H>
__device__ __forceinline__ void line_Bt(const H* v, H* out) {
  const H p = v[0] + v[2], m = v[0] - v[2];
  if constexpr (N1 == 2) {
    const H h = hc<H>(0.5) * (p + v[1]);
    out[0] = hfma(hc<H>(0.5 * LN_S), m, h);
    out[1] = hfma(hc<H>(-0.5 * LN_S), m, h);
  } else {
    const H q = hc<H>(0.3) * p;
    out[0] = hfma(hc<H>(0.5 * LN_S), m, q);
    out[1] = hfma(hc<H>(0.4), p, v[1]);
    out[2] = hfma(hc<H>(-0.5 * LN_S), m, q);
  }
}
template <int N1, class H>
__device__ __forceinline__ void line_Dt(const H* v, H* out) {
  const H S = v[0] + v[2] + v[1];
  if constexpr (N1 == 2) {
    out[0] = -S;
    out[1] = S;
  } else {
    const H m = v[2] - v[0];
    out[0] = hfma(hc<H>(2.0 * LN_S), m, -S);
    out[1] = hc<H>(-4.0 * LN_S) * m;
    out[2] = hfma(hc<H>(2.0 * LN_S), m, S);
  }
}
template <int N1, class H>
__device__ __forceinline__ void line_BtDt(const H* vb, const H* vd, H* out) {
  const H p = vb[0] + vb[2], m = vb[0] - vb[2], S = vd[0] + vd[2] + vd[1];
  const H odd = hfma(hc<H>(0.5 * LN_S), m, -S);
  if constexpr (N1 == 2) {
    const H h = hc<H>(0.5) * (p + vb[1]);
    out[0] = h + odd;
    out[1] = h - odd;
  } else {
    const H md = vd[2] - vd[0];
    const H even = hfma(hc<H>(2.0 * LN_S), md, hc<H>(0.3) * p);
    out[0] = even + odd;
    out[1] = hfma(hc<H>(-4.0 * LN_S), md, hfma(hc<H>(0.4), p, vb[1]));
    out[2] = even - odd;
  }
}
// out[q] = sum_g L_q(g) v[g] for the two linear functions L.
template <class H>
__device__ __forceinline__ void line_Lt(const H* v, H* out) { line_Bt<2, H>(v, out); }

// Products with the linear functions: out[q N1 + a] = sum_g L_q(g) M_a(g) v[g]
// (+ the same with the derivatives of vd).  The reflection s -> -s takes
// (q, a) to (1 - q, N1 - 1 - a) and the derivative to its negative, so the
// outputs come in pairs P + Q, P - Q.
__host__ __device__ constexpr double ln_val(int n, int a, int d, double s) {
  const double t = 0.5 * (1.0 + s);
  if (n == 2) return d ? (a == 0 ? -1.0 : 1.0) : (a == 0 ? 1.0 - t : t);
  if (d) return a == 0 ? 4.0 * t - 3.0 : (a == 1 ? 4.0 - 8.0 * t : 4.0 * t - 1.0);
  return a == 0 ? 1.0 - 3.0 * t + 2.0 * t * t : (a == 1 ? 4.0 * t * (1.0 - t) : t * (t + t - 1.0));
}
__host__ __device__ constexpr double ln_prod(int n, int q, int a, int d, double s) {
  return (q == 0 ? 0.5 * (1.0 - s) : 0.5 * (1.0 + s)) * ln_val(n, a, d, s);
}
// coefficients of the even and odd combinations and of the middle point
__host__ __device__ constexpr double ln_e(int n, int q, int a, int d) {
  return 0.5 * (ln_prod(n, q, a, d, -LN_S) + ln_prod(n, q, a, d, LN_S));
}
__host__ __device__ constexpr double ln_o(int n, int q, int a, int d) {
  return 0.5 * (ln_prod(n, q, a, d, -LN_S) - ln_prod(n, q, a, d, LN_S));
}
__host__ __device__ constexpr double ln_m(int n, int q, int a, int d) { return ln_prod(n, q, a, d, 0.0); }

template <int N1, int B, int D, class H>
__device__ __forceinline__ void line_L(const H* vb, const H* vd, H* out) {
  H be, bo, de, dd_o;
  if (B) {
    be = vb[0] + vb[2];
    bo = vb[0] - vb[2];
  }
  if (D) {
    de = vd[0] + vd[2];
    dd_o = vd[0] - vd[2];
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int a = 0; a < N1; ++a) {
      const int mate = (1 - q) * N1 + (N1 - 1 - a);
      if (mate < q * N1 + a) continue;
      H P, Q;  // even under the reflection, odd under it
      if constexpr (B && D) {
        P = hfma(hc<H>(ln_e(N1, q, a, 0)), be, hc<H>(ln_o(N1, q, a, 1)) * dd_o);
        Q = hfma(hc<H>(ln_o(N1, q, a, 0)), bo, hc<H>(ln_e(N1, q, a, 1)) * de);
        if (ln_m(N1, q, a, 0) != 0.0) P = hfma(hc<H>(ln_m(N1, q, a, 0)), vb[1], P);
        if (ln_m(N1, q, a, 1) != 0.0) Q = hfma(hc<H>(ln_m(N1, q, a, 1)), vd[1], Q);
        out[q * N1 + a] = P + Q;
        out[mate] = P - Q;
      } else if constexpr (B) {
        P = hc<H>(ln_e(N1, q, a, 0)) * be;
        if (ln_m(N1, q, a, 0) != 0.0) P = hfma(hc<H>(ln_m(N1, q, a, 0)), vb[1], P);
        out[q * N1 + a] = hfma(hc<H>(ln_o(N1, q, a, 0)), bo, P);
        out[mate] = hfma(hc<H>(-ln_o(N1, q, a, 0)), bo, P);
      } else {
        Q = hc<H>(ln_e(N1, q, a, 1)) * de;
        if (ln_m(N1, q, a, 1) != 0.0) Q = hfma(hc<H>(ln_m(N1, q, a, 1)), vd[1], Q);
        out[q * N1 + a] = hfma(hc<H>(ln_o(N1, q, a, 1)), dd_o, Q);
        out[mate] = hfma(hc<H>(ln_o(N1, q, a, 1)), dd_o, -Q);
      }
    }
}

}  // namespace
