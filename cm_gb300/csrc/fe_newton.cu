// libcm_fe: Newton load step on the device (sm_103a).
//
// The solve the reference runs around the assembly for one load increment
// (SOLVER_NEWTON_LINESEARCH, solver_routines.f90:17803-17812 and
// 18772-18775): Newton from the given state, the FP64 Jacobian and residual
// of this library, Dirichlet rows and columns dropped from the linear system
// (solver_mapping_routines.f90:1420,1592), each Newton system solved by
// restarted GMRES (the reference's KSP default, solver_routines.f90:
// 10979-10987) with a block-diagonal preconditioner, then a cubic
// backtracking line search (the published Dennis-Schnabel algorithm that
// PETSc's "bt" line search implements) on f = 1/2 ||r_free||^2.
//
// The free-dof system is never extracted: vectors keep the full dof
// numbering with zeros on the fixed dofs, and the matrix-vector product masks
// rows and columns of fixed dofs.  Every reduction is a fixed-order two-pass
// sum, so a solve is bit-identical from run to run.
//
// On the meshes this solver suits (its preconditioner is diagonal) a GMRES
// iteration is a handful of vectors of a few thousand entries, bound by
// launches and by the latency of FP64 reductions.  While the rows fit the SMs'
// shared memory, a whole cycle is one cooperative launch (k_cycle).  Else an
// iteration is four launches: dots, update with the second pass's dots, update
// with the norm, the preconditioning and the Hessenberg column, matrix-vector
// product with the scaling; a block owns a chunk of rows and its warps take
// different basis vectors, so no dot waits on a block-wide reduction, the sums
// over the chunks (row_chunks) are formed by the kernel that uses them, the host
// rotates the columns, and the next iteration is queued before it waits for one.
#include "fe_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

namespace {

constexpr int NT = 256;
constexpr int NWARP = NT / 32;
constexpr int MAX_CHUNKS = 608;  // row chunks of a reduction: one block each

// y = P A x on the free rows (P: the free-dof mask), 0 on the fixed ones, for
// x zero on the fixed dofs; with scale: y and v scaled by *scale.  One warp
// takes two rows, lanes over the entries, and reduces both with five
// additions instead of ten: the FP64 pipe (19 cycles of an SM per warp
// instruction) and two waits for memory bind it.  U entries a lane are loaded
// at once: eight for the rows of a triquadratic mesh (100 to 400 entries), four
// for the shorter ones of a trilinear one, whose multiply-adds past the end of
// the row would hold the pipe as long as real ones (a GMRES iteration on
// 270,763 rows of about 80 entries: 243 against 315 us with eight).
template <int U>
__global__ void __launch_bounds__(NT) k_spmv(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                                             const double* __restrict__ val, const uint8_t* __restrict__ free_dof,
                                             const double* __restrict__ x, double* __restrict__ y,
                                             const double* __restrict__ scale, double* __restrict__ v) {
  const int lane = threadIdx.x & 31;
  const double sc = scale ? *scale : 1.0;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = 2 * ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); i < n; i += 2 * nw) {
    double s[2] = {0.0, 0.0};
    int at[2], end[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const bool in = i + r < n && free_dof[i + r];
      at[r] = in ? rp[i + r] + lane : 0;
      end[r] = in ? rp[i + r + 1] : 0;
    }
    while (__any_sync(0xffffffffu, at[0] < end[0] || at[1] < end[1])) {
      double a[2][U];
      int c[2][U];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool in = at[r] + 32 * u < end[r];
          a[r][u] = in ? val[at[r] + 32 * u] : 0.0;
          c[r][u] = in ? col[at[r] + 32 * u] : 0;
        }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (at[r] + 32 * u < end[r]) s[r] = fma(a[r][u], x[c[r][u]], s[r]);
        at[r] += 32 * U;
      }
    }
    // lanes 0..15 go on with the first row, 16..31 with the second
    const bool hi = lane & 16;
    double t = (hi ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, hi ? s[0] : s[1], 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    const int64_t row = i + (hi ? 1 : 0);
    if ((lane & 15) == 0 && row < n) {
      y[row] = scale ? sc * t : t;
      if (scale) v[row] *= sc;
    }
  }
}

// Diagonal of A (0 where a row has no diagonal entry).
__global__ void k_diag(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                       const double* __restrict__ val, double* __restrict__ d) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += nw) {
    double v = 0.0;
    for (int64_t j = rp[i] + lane; j < rp[i + 1]; j += 32)
      if (col[j] == i) v = val[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) d[i] = v;
  }
}

// Preconditioner: 1/A_ii on free displacement rows; on free pressure rows
// -1/s_i with s_i = sum over free displacement columns j of B_ij^2 / A_jj
// (the diagonal of the Schur complement B diag(A)^-1 B^T), 1 if s_i = 0;
// 0 on fixed dofs.
__global__ void k_precond(int64_t n, int64_t nu3, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                          const double* __restrict__ val, const uint8_t* __restrict__ free_dof,
                          const double* __restrict__ d, double* __restrict__ minv) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += nw) {
    if (!free_dof[i]) {
      if (lane == 0) minv[i] = 0.0;
      continue;
    }
    if (i < nu3) {
      if (lane == 0) minv[i] = 1.0 / d[i];
      continue;
    }
    double s = 0.0;
    for (int64_t j = rp[i] + lane; j < rp[i + 1]; j += 32) {
      const int c = col[j];
      if (c < nu3 && free_dof[c]) s += val[j] * val[j] / d[c];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) minv[i] = -1.0 / (s != 0.0 ? s : 1.0);
  }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;  // valid in lane 0
}

// Chunk blockIdx.x of gridDim.x of the rows: [r0, r1).
__device__ __forceinline__ void chunk_rows(int64_t n, int64_t& r0, int64_t& r1) {
  const int64_t len = (n + gridDim.x - 1) / gridDim.x;
  r0 = blockIdx.x * len;
  r1 = r0 + len < n ? r0 + len : n;
}

// part[j * gridDim.x + chunk] = the chunk's share of V_j . w, j < m (V
// row-major, leading dimension ld), each by one warp.
__device__ __forceinline__ void chunk_dots(int64_t r0, int64_t r1, const double* __restrict__ V, int64_t ld, int m,
                                           const double* w, double* __restrict__ part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j = warp; j < m; j += NWARP) {
    double s = 0.0;
    const double* v = V + j * ld;
#pragma unroll 4
    for (int64_t i = r0 + lane; i < r1; i += 32) s = fma(v[i], w[i], s);
    s = warp_sum(s);
    if (lane == 0) part[j * (int)gridDim.x + blockIdx.x] = s;
  }
}

// Sum of v over each group of G neighbouring lanes (G a power of two), in
// every lane of the group, by a fixed tree.
template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// h[j] = sum of the chunks' shares for j < m (shared memory): eight lanes to a
// j, as a chain of FP64 additions waits 64 cycles for each.
__device__ __forceinline__ void sum_parts(const double* __restrict__ part, int m, double* h) {
  const int q = threadIdx.x & 7;
  for (int j0 = 0; j0 < m; j0 += NT / 8) {
    const int j = j0 + (threadIdx.x >> 3);
    double s = 0.0;
    if (j < m)
      for (int c = q; c < (int)gridDim.x; c += 8) s += part[j * (int)gridDim.x + c];
    s = group_sum<8>(s);
    if (j < m && q == 0) h[j] = s;
  }
}

constexpr int MAX_BASIS = 208;  // restart limit 200 and a few

// Dots of m vectors with w; V = w and m = 1 give the squared norm.
__global__ void __launch_bounds__(NT) k_dots(int64_t n, const double* __restrict__ V, int64_t ld, int m,
                                             const double* __restrict__ w, double* __restrict__ part) {
  int64_t r0, r1;
  chunk_rows(n, r0, r1);
  chunk_dots(r0, r1, V, ld, m, w, part);
}

// *out = sum over the chunks (one block of one warp).
__global__ void k_sum(const double* __restrict__ part, int chunks, double* __restrict__ out) {
  double s = 0.0;
  for (int c = threadIdx.x; c < chunks; c += 32) s += part[c];
  s = warp_sum(s);
  if (threadIdx.x == 0) *out = s;
}

// w -= sum_j h[j] V_j on the block's chunk (and z = minv .* w): four lanes to a
// row.  Returns this thread's share of the new w's squared norm.
__device__ __forceinline__ double chunk_update(int64_t r0, int64_t r1, const double* __restrict__ V, int64_t ld, int m,
                                               const double* h, double* w, const double* __restrict__ minv = nullptr,
                                               double* __restrict__ z = nullptr) {
  const int q = threadIdx.x & 3;
  double nrm = 0.0;
  for (int64_t b = r0; b < r1; b += NT / 4) {
    const int64_t i = b + (threadIdx.x >> 2);
    double s = 0.0;
    if (i < r1) {
#pragma unroll 8
      for (int j = q; j < m; j += 4) s = fma(h[j], V[j * ld + i], s);
    }
    s = group_sum<4>(s);
    if (i < r1 && q == 0) {
      const double t = w[i] - s;
      w[i] = t;
      if (z) z[i] = minv[i] * t;
      nrm = fma(t, t, nrm);
    }
  }
  return nrm;
}

// First Gram-Schmidt update and the second pass's dots.  col[j] = h[j].
__global__ void __launch_bounds__(NT) k_update_dots(int64_t n, const double* __restrict__ V, int64_t ld, int m,
                                                    const double* __restrict__ part, double* w, double* __restrict__ col,
                                                    double* __restrict__ part2) {
  __shared__ double h[MAX_BASIS];
  int64_t r0, r1;
  chunk_rows(n, r0, r1);
  sum_parts(part, m, h);
  __syncthreads();
  chunk_update(r0, r1, V, ld, m, h, w);
  if (blockIdx.x == 0)
    for (int j = threadIdx.x; j < m; j += NT) col[j] = h[j];
  __syncthreads();
  chunk_dots(r0, r1, V, ld, m, w, part2);
}

// Second Gram-Schmidt update, the result preconditioned (z = minv .* w), and
// its squared norm.  The last block to finish writes the Hessenberg column to
// the host (page-locked memory): col[j] + h[j], and the squared norm; col[m] =
// 1 / norm (0 when it is 0: an Arnoldi breakdown, after which the vector is
// not used).
__global__ void __launch_bounds__(NT) k_update_norm(int64_t n, const double* __restrict__ V, int64_t ld, int m,
                                                    const double* __restrict__ part2, double* w, double* __restrict__ col,
                                                    double* __restrict__ npart, int* __restrict__ done,
                                                    const double* __restrict__ minv, double* __restrict__ z, double* host) {
  __shared__ double h[MAX_BASIS];
  __shared__ double sh[NWARP];
  __shared__ bool last;
  int64_t r0, r1;
  chunk_rows(n, r0, r1);
  sum_parts(part2, m, h);
  __syncthreads();
  const double s = warp_sum(chunk_update(r0, r1, V, ld, m, h, w, minv, z));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 8) {
    double t = sh[threadIdx.x];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffu, t, o);
    if (threadIdx.x == 0) {
      npart[blockIdx.x] = t;
      __threadfence();
      last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int j = threadIdx.x; j < m; j += NT) host[j] = col[j] + h[j];
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int c = threadIdx.x; c < (int)gridDim.x; c += 32) t += __ldcg(npart + c);
    t = warp_sum(t);
    if (threadIdx.x == 0) {
      host[m] = t;
      col[m] = t > 0.0 ? 1.0 / sqrt(t) : 0.0;
      *done = 0;
    }
  }
}

// One GMRES cycle in one cooperative launch, for systems whose rows fit the
// SMs' shared memory: block b holds the matrix entries of rows [bound[b],
// bound[b + 1]) (as many as fit; the rest is read from L2), the basis vectors'
// and w's entries of these rows, and one more block turns the Hessenberg
// columns into the triangular system while the others form the next product.
// What crosses SMs is the preconditioned vector z and the blocks' shares of
// the dots and the norm: three grid barriers an iteration (blocks that poll
// the shares themselves until all have come take twice the time).
//
// Bound by the barriers (1.9 us each) and FP64 latency (an instruction holds a
// quarter SM's pipe for 64 cycles).  Load steps of triquadratic boxes, with the
// cycle and with four launches an iteration, ms: 1,093 rows 9.0 and 13.7, 4,071
// rows and 700,000 entries 22.1 and 32.9 (20.7 and 30.8 us an iteration, the
// assemblies included), 9,223 rows 54.1 and 75.6; trilinear, 8,970 rows 51.9 and
// 86.4.
struct CycleArgs {
  int n, nb, restart, kmax, cap;
  int* bound;  // [nb + 1]
  double beta, tol, breakdown;
  const int32_t *rp, *col;
  const double *vals, *minv, *b;
  const uint8_t* free_dof;
  double *res, *dx, *z, *part, *part2, *npart, *y;
  double* scale;  // 1 / norm of the newest basis vector, -1: converged
  int* ctl;       // barrier arrivals; zeroed before the launch
  unsigned polls;  // of a barrier, before it gives up
  int extra_from;  // barriers from this one on wait for one arrival more than there are
  double* host;  // page-locked: squared norm of the true residual, iterations, converged
};

constexpr int CT = 512;                  // threads
constexpr int CYCLE_ROWS = 64;           // rows of a block at most
constexpr int LD = CYCLE_ROWS + 1;       // between basis vectors in shared memory
constexpr int MAX_SHARES = 160;          // blocks at most
constexpr unsigned CYCLE_POLLS = 1u << 21;  // a wait gives up after about a second

// Row bounds of k_cycle's blocks: equal shares of entries + 24 x rows (a row's
// reduction takes as long as 24 entries), no block above CYCLE_ROWS rows.
__global__ void __launch_bounds__(MAX_SHARES + 32) k_cycle_bounds(int n, int nb, const int32_t* __restrict__ rp,
                                                                  int* __restrict__ bound) {
  __shared__ int at[MAX_SHARES + 1];
  const int b = threadIdx.x;
  if (b <= nb) {
    const int64_t target = ((int64_t)rp[n] + 24 * (int64_t)n) * b / nb;
    int lo = 0, hi = n;  // first row whose share starts at or after the target
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (rp[mid] + 24 * (int64_t)mid < target) lo = mid + 1;
      else hi = mid;
    }
    at[b] = lo;
  }
  __syncthreads();
  if (b == 0) {
    int prev = 0;
    bound[0] = 0;
    for (int i = 1; i <= nb; ++i) {
      const int least = max(prev, n - (nb - i) * CYCLE_ROWS);
      bound[i] = prev = min(max(at[i], least), min(prev + CYCLE_ROWS, n));
    }
  }
}

// Grid barrier number k = 1, 2, ... of the launch; false when it gave up.
__device__ __forceinline__ bool cycle_barrier(const CycleArgs& A, int k) {
  __shared__ bool ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    const int target = k * (int)gridDim.x + (k >= A.extra_from);
    unsigned polls = A.polls;
    int v;
    __threadfence();
    atomicAdd(A.ctl, 1);
    do {
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(A.ctl) : "memory");
    } while (v < target && --polls);
    ok = v >= target;
    __threadfence();
  }
  __syncthreads();
  return ok;
}

// Squared norm of the vector whose blocks' shares npart holds (one warp).
__device__ __forceinline__ double cycle_norm(const double* __restrict__ npart, int nb) {
  double v[MAX_SHARES / 32], t = 0.0;
#pragma unroll
  for (int u = 0; u < MAX_SHARES / 32; ++u) {
    const int c = (threadIdx.x & 31) + 32 * u;
    v[u] = c < nb ? __ldcg(npart + c) : 0.0;
  }
#pragma unroll
  for (int u = 0; u < MAX_SHARES / 32; ++u) t += v[u];
  return group_sum<32>(t);
}

// Sums over the blocks of part[j nb + block], j < m, eight lanes to a j:
// done(j, sum) on one of them.
template <class F>
__device__ __forceinline__ void cycle_sums(const double* part, int nb, int m, F done) {
  const int q = threadIdx.x & 7;
  for (int j0 = 0; j0 < m; j0 += CT / 8) {
    const int j = j0 + (threadIdx.x >> 3);
    if ((threadIdx.x >> 5) * 4 + j0 >= m) break;  // whole warps
    double v[MAX_SHARES / 8], s = 0.0;
#pragma unroll
    for (int u = 0; u < MAX_SHARES / 8; ++u) v[u] = j < m && q + 8 * u < nb ? __ldcg(part + j * nb + q + 8 * u) : 0.0;
#pragma unroll
    for (int u = 0; u < MAX_SHARES / 8; ++u) s += v[u];
    s = group_sum<8>(s);
    if (j < m && q == 0) done(j, s);
  }
}

__global__ void __launch_bounds__(CT, 1) k_cycle(const __grid_constant__ CycleArgs A) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[CYCLE_ROWS / 8];
  __shared__ int groups;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = tid & 3, grp = tid >> 2;
  const bool givens = (int)blockIdx.x == A.nb;
  const int r0 = givens ? A.n : A.bound[blockIdx.x];
  const int rows = givens ? 0 : A.bound[blockIdx.x + 1] - r0;
  const bool row_warp = warp * 8 < rows;  // warps with a row in combine()
  int bar = 0;
  bool near = false;           // the matrix entries are in shared memory
  double* h = sm;              // [MAX_BASIS]
  double* c = h + MAX_BASIS;   // [MAX_BASIS]: the Hessenberg column (the last block)
  double* V = c + MAX_BASIS;   // [restart + 1][LD]; the last vector found is not scaled yet
  double* wn = V + (size_t)(A.restart + 1) * LD;  // the product
  double* mi = wn + LD;
  double* sval = mi + LD + (~A.restart & 1);  // [cap], 16-byte aligned
  int32_t* rps = reinterpret_cast<int32_t*>(sval + A.cap);  // [CYCLE_ROWS]: a row's first entry there
  int32_t* rpe = rps + CYCLE_ROWS;  // and its groups of 32
  uint16_t* scol = reinterpret_cast<uint16_t*>(rpe + CYCLE_ROWS);
  // the last block's arrays take the place of the matrix
  double *cs = V, *sn = cs + A.restart, *g = sn + A.restart, *xs = g + A.restart + 1, *pr = xs + A.restart + 1,
         *U = pr + A.restart;  // U: packed columns of the triangular matrix

  if (!givens) {
    // groups of 32 entries of every free row, the last one filled up with
    // zeros; a lane's four are neighbours and eight apart in the row
    if (warp == 0) {
      int first = 1;
      for (int r = lane; r < CYCLE_ROWS; r += 32) {
        const int ng = r < rows && A.free_dof[r0 + r] ? (A.rp[r0 + r + 1] - A.rp[r0 + r] + 31) / 32 : 0;
        int sum = ng;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += t;
        }
        rps[r] = 32 * (first + sum - ng);
        rpe[r] = ng;
        first += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) groups = first;
    }
    __syncthreads();
    near = 32 * groups <= A.cap;
    if (near) {
      if (tid < 32) {
        sval[tid] = 0.0;
        scol[tid] = 0;
      }
      for (int r = warp; r < rows; r += CT / 32) {
        const int e0 = A.rp[r0 + r], len = A.rp[r0 + r + 1] - e0;
        for (int g = 0; g < rpe[r]; ++g) {
          const int e = 32 * g + lane, to = rps[r] + 32 * g + 4 * (lane & 7) + (lane >> 3);
          sval[to] = e < len ? A.vals[e0 + e] : 0.0;
          scol[to] = e < len ? (uint16_t)A.col[e0 + e] : (uint16_t)0;
        }
      }
    }
    for (int r = tid; r < rows; r += CT) {
      const double m = A.minv[r0 + r], v = A.res[r0 + r] * (1.0 / A.beta);
      mi[r] = m;
      V[r] = v;
      A.z[r0 + r] = m * v;
    }
  } else if (tid == 0) {
    g[0] = A.beta;
  }

  // wn = P A x on the block's rows: eight lanes to a row, 32 entries at a time.
  // x goes through L1 (the barrier before makes the other blocks' part
  // visible), as a block's rows share most of their columns.
  static_assert(CYCLE_ROWS * 8 == CT, "one row per eight threads");
  auto product = [&](const double* x) {
    const int r = tid >> 3, l = tid & 7;
    if (warp * 4 < rows) {
      double s0 = 0.0, s1 = 0.0;
      const int start = r < rows ? rps[r] : 0, ng = r < rows ? rpe[r] : 0;
      if (near) {
        const int most = __reduce_max_sync(0xffffffffu, ng);
        for (int g0 = 0; g0 < most; g0 += 4) {
          int at[4];
          double xv[4][4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            at[g] = (g0 + g < ng ? start + 32 * (g0 + g) : 0) + 4 * l;  // the first group holds zeros
            const ushort4 cc = *reinterpret_cast<const ushort4*>(scol + at[g]);
            xv[g][0] = x[cc.x];
            xv[g][1] = x[cc.y];
            xv[g][2] = x[cc.z];
            xv[g][3] = x[cc.w];
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (g0 + g >= most) break;
            const double2 a = *reinterpret_cast<const double2*>(sval + at[g]);
            const double2 b = *reinterpret_cast<const double2*>(sval + at[g] + 2);
            s0 = fma(a.x, xv[g][0], s0);
            s1 = fma(a.y, xv[g][1], s1);
            s0 = fma(b.x, xv[g][2], s0);
            s1 = fma(b.y, xv[g][3], s1);
          }
        }
      } else if (ng) {
        for (int e = A.rp[r0 + r] + l; e < A.rp[r0 + r + 1]; e += 8) s0 = fma(A.vals[e], x[A.col[e]], s0);
      }
      __syncwarp();
      const double s = group_sum<8>(s0 + s1);
      if (l == 0 && r < rows) wn[r] = s;
    }
    __syncthreads();
  };
  // the block's shares of V_j . w, j < m
  auto dots = [&](int m, const double* w, double* part) {
    for (int j0 = 0; j0 < m; j0 += CT / 4) {
      const int j = j0 + grp;
      if (warp * 8 + j0 >= m) continue;
      double s = 0.0;
      if (j < m) {
#pragma unroll 8
        for (int r = q; r < rows; r += 4) s = fma(V[j * LD + r], w[r], s);
      }
      s = group_sum<4>(s);
      if (j < m && q == 0) part[j * A.nb + blockIdx.x] = s;
    }
  };
  // sum_j h[j] V_j on row grp (the row's four lanes; whole warps)
  auto combine = [&](int m) {
    double s = 0.0;
    if (grp < rows) {
#pragma unroll 8
      for (int j = q; j < m; j += 4) s = fma(h[j], V[j * LD + grp], s);
    }
    return group_sum<4>(s);
  };
  // the block's share of a squared norm, v on the threads with q == 0
  auto norm_share = [&](double v) {
    if (row_warp) {
      double t = (q == 0 && grp < rows) ? v * v : 0.0;
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) red[warp] = t;
    }
    __syncthreads();
    if (warp == 0) {
      const double t = group_sum<8>(lane < 8 && lane * 8 < rows ? red[lane] : 0.0);
      if (lane == 0) A.npart[blockIdx.x] = t;
    }
  };
  // column k of the Hessenberg matrix: the previous rotations, then the one
  // that zeroes its last entry (the last block, all threads); true when the
  // cycle has converged or broken down
  auto rotate = [&](int k) -> bool {
    __syncthreads();
    for (int i = tid; i < k; i += CT) pr[i] = cs[i] * c[i + 1];
    __syncthreads();
    double* Uk = U + k * (k + 1) / 2;
    if (tid == 0) {
      double x = c[0];
      xs[0] = x;
      for (int i = 0; i < k; ++i) xs[i + 1] = x = fma(-sn[i], x, pr[i]);
      const double bb = c[k + 1], den = hypot(x, bb);
      const double ck = den > 0.0 ? x / den : 1.0, sk = den > 0.0 ? bb / den : 0.0;
      Uk[k] = den;
      cs[k] = ck;
      sn[k] = sk;
      g[k + 1] = -sk * g[k];
      g[k] = ck * g[k];
    }
    __syncthreads();
    for (int i = tid; i < k; i += CT) Uk[i] = fma(cs[i], xs[i], sn[i] * c[i + 1]);
    return fabs(g[k + 1]) <= A.tol || c[k + 1] <= A.breakdown;
  };

  if (!cycle_barrier(A, ++bar)) return;
  int K = 0;
  bool converged = false;
  for (int k = 0;; ++k) {
    const int m = k + 1;
    double* w = V + m * LD;
    if (!givens) {
      product(A.z);
      dots(m, wn, A.part);
    } else if (k) {
      if (warp == 0) {
        const double t = cycle_norm(A.npart, A.nb);
        if (lane == 0) {
          c[k] = sqrt(t);
          red[0] = t > 0.0 ? rsqrt(t) : 0.0;
        }
      }
      converged = rotate(k - 1);
      if (tid == 0) *A.scale = converged ? -1.0 : red[0];
    }
    if (!cycle_barrier(A, ++bar)) return;
    // V_k, the product and its dots still lack the scale of V_k
    const double a = k ? __ldcg(A.scale) : 1.0;
    cycle_sums(A.part, A.nb, m, [&](int j, double s) { h[j] = j == k ? s * a * a : s * a; });
    for (int r = tid; r < rows; r += CT) {
      V[k * LD + r] *= a;
      w[r] = a * wn[r];
    }
    if (a < 0.0) {  // column k - 1 was the last one
      K = k;
      break;
    }
    __syncthreads();
    if (!givens) {
      if (row_warp) {
        const double s = combine(m);
        if (grp < rows && q == 0) w[grp] -= s;
      }
      __syncthreads();
      dots(m, w, A.part2);
    } else {
      for (int j = tid; j < m; j += CT) c[j] = h[j];
    }
    if (!cycle_barrier(A, ++bar)) return;
    cycle_sums(A.part2, A.nb, m, [&](int j, double s) { h[j] = s; });
    __syncthreads();
    if (!givens) {
      double t = 0.0;
      if (row_warp) {
        const double s = combine(m);
        if (grp < rows && q == 0) {
          t = w[grp] - s;
          w[grp] = t;
          A.z[r0 + grp] = mi[grp] * t;
        }
      }
      norm_share(t);
    } else {
      for (int j = tid; j < m; j += CT) c[j] += h[j];
    }
    if (!cycle_barrier(A, ++bar)) return;
    if (m == A.kmax) {
      if (givens) {
        if (warp == 0) {
          const double t = cycle_norm(A.npart, A.nb);
          if (lane == 0) c[m] = sqrt(t);
        }
        converged = rotate(k);
      }
      K = m;
      break;
    }
  }
  // the cycle's correction: U y = g, dx += M^-1 V y
  if (givens) {
    __syncthreads();
    for (int i = K - 1; i >= 0; --i) {
      const double* Ui = U + i * (i + 1) / 2;
      const double yi = Ui[i] != 0.0 ? g[i] / Ui[i] : 0.0;
      __syncthreads();
      if (tid == 0) A.y[i] = yi;
      for (int j = tid; j < i; j += CT) g[j] = fma(-Ui[j], yi, g[j]);
      __syncthreads();
    }
  }
  if (!cycle_barrier(A, ++bar)) return;
  if (!givens) {
    for (int j = tid; j < K; j += CT) h[j] = __ldcg(A.y + j);
    __syncthreads();
    const double s = row_warp ? combine(K) : 0.0;
    if (grp < rows && q == 0) A.dx[r0 + grp] = fma(mi[grp], s, A.dx[r0 + grp]);
  }
  if (!cycle_barrier(A, ++bar)) return;
  // the true residual and its norm
  if (!givens) {
    product(A.dx);
    double t = 0.0;
    if (grp < rows && q == 0) A.res[r0 + grp] = t = A.b[r0 + grp] - wn[grp];
    norm_share(t);
  }
  if (!cycle_barrier(A, ++bar)) return;
  if (givens && warp == 0) {
    const double r2 = cycle_norm(A.npart, A.nb);
    if (lane == 0) {
      A.host[0] = r2;
      A.host[1] = K;
      A.host[2] = converged ? 1.0 : 0.0;
    }
  }
}

// v = a * x, z = minv .* v
__global__ void __launch_bounds__(NT) k_scale_precond(int64_t n, double a, const double* __restrict__ minv,
                                                      const double* __restrict__ x, double* __restrict__ v,
                                                      double* __restrict__ z) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double t = a * x[i];
    v[i] = t;
    z[i] = minv[i] * t;
  }
}

// y = a * x
__global__ void k_scale(int64_t n, double a, const double* x, double* y) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = a * x[i];
}

// y = a * x + b * y
__global__ void k_axpby(int64_t n, double a, const double* __restrict__ x, double b, double* __restrict__ y) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = a * x[i] + b * y[i];
}

// x += sum_{j < m} y[j] (minv .* V_j)
__global__ void __launch_bounds__(NT) k_combine(int64_t n, const double* __restrict__ V, int64_t ld, int m,
                                                const double* __restrict__ minv, const double* __restrict__ y,
                                                double* __restrict__ x) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double s = x[i];
    const double mi = minv[i];
#pragma unroll 8
    for (int j = 0; j < m; ++j) s = fma(y[j], mi * V[j * ld + i], s);
    x[i] = s;
  }
}

// r <- -r on free dofs, 0 on fixed ones (in place when out == r)
__global__ void k_mask(int64_t n, const uint8_t* __restrict__ free_dof, double sign, const double* r, double* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = free_dof[i] ? sign * r[i] : 0.0;
}

// x[dofs[k]] = values[k]; free[dofs[k]] = 0
__global__ void k_fix(int64_t m, const int32_t* __restrict__ dofs, const double* __restrict__ values,
                      double* __restrict__ x, uint8_t* __restrict__ free_dof) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
    x[dofs[k]] = values[k];
    free_dof[dofs[k]] = 0;
  }
}

// Row chunks of a reduction: one, two or four to an SM of the 152.  Every block
// adds up all chunks' shares (eight lanes to a sum), so more of them help only
// where the rows are what takes the time.  A GMRES iteration with 64, 152, 304
// and 608 chunks, us: 13,653 rows 51, 45, 47, 47; 49,072 rows 147, 108, 100,
// 116; 216,024 rows 509, 351, 294, 295; 859,812 rows 2,510, 1,485, 1,136, 998.
int row_chunks(int64_t n) {
  const int64_t most = MAX_CHUNKS / 4 * (n < 24000 ? 1 : n < 200000 ? 2 : 4);
  return (int)std::min<int64_t>((n + 63) / 64, most);
}

int blocks_for(int64_t n) {
  const int64_t b = (n + NT - 1) / NT;
  return (int)(b < 4096 ? (b < 1 ? 1 : b) : 4096);
}

// Blocks for one row per warp, and for k_spmv's two.
int warp_blocks_for(int64_t n) {
  const int64_t b = (n + (NT / 32) - 1) / (NT / 32);
  return (int)(b < 8192 ? (b < 1 ? 1 : b) : 8192);
}

#define NT_TRY(expr)                                                                                 \
  do {                                                                                              \
    cudaError_t e_ = (expr);                                                                        \
    if (e_ != cudaSuccess) return cmfe::record_error(FE_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Device work space of one call in one allocation, freed on scope exit: the
// arrays are announced with add() and placed by alloc().
struct Work {
  struct Slot {
    void** p;
    size_t at;
  };
  std::vector<Slot> slots;
  size_t bytes = 0;
  void* base = nullptr;
  double* pinned = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  ~Work() {
    if (base) cudaFree(base);
    if (pinned) cudaFreeHost(pinned);
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
  }
  template <class T>
  void add(T** p, size_t count) {
    slots.push_back({reinterpret_cast<void**>(p), bytes});
    bytes += (count * sizeof(T) + 255) / 256 * 256;
  }
  int alloc(size_t host_doubles) {
    cudaError_t e = cudaMalloc(&base, bytes);
    if (e == cudaSuccess) e = cudaMallocHost(&pinned, host_doubles * sizeof(double));
    for (cudaEvent_t& v : ev)
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return cmfe::record_error(FE_ERR_OUT_OF_MEMORY, std::string("Newton work space: ") + cudaGetErrorString(e));
    }
    for (const Slot& s : slots) *s.p = static_cast<char*>(base) + s.at;
    return FE_NO_ERROR;
  }
};

struct Solver {
  fe_handle h;
  cudaStream_t st;
  int64_t n, nnz, nu3;
  const int32_t *rp, *col;
  double *vals, *r, *rn, *d, *xs, *w, *minv, *diag, *V, *z, *col_d, *part, *part2, *npart, *scal;
  int* done;
  uint8_t* free_dof;
  double* pinned;   // page-locked: the Hessenberg column, and single sums
  const cudaEvent_t* ev;  // two: the columns' copies
  int restart, chunks;
  std::vector<cudaGraphExec_t> graphs;  // iteration k of a cycle
  cudaStream_t capture = nullptr;
  int64_t cycles = 0;
  bool no_graphs = false;
  CycleArgs cyc{};     // of k_cycle, when the system takes it
  size_t cyc_smem = 0;  // 0: it does not

  Solver() = default;
  Solver(const Solver&) = delete;
  ~Solver() {
    for (cudaGraphExec_t g : graphs)
      if (g) cudaGraphExecDestroy(g);
    if (capture) cudaStreamDestroy(capture);
  }

  int spmv(const double* x, double* y) {
    return spmv(x, y, nullptr, nullptr, st);
  }

  // y = P A x; with scale, y and v scaled by it.
  int spmv(const double* x, double* y, const double* scale, double* v, cudaStream_t t) {
    auto kern = nnz <= 128 * n ? k_spmv<4> : k_spmv<8>;
    kern<<<warp_blocks_for((n + 1) / 2), NT, 0, t>>>(n, rp, col, vals, free_dof, x, y, scale, v);
    NT_TRY(cudaGetLastError());
    return FE_NO_ERROR;
  }

  int dot_host(const double* a, const double* b, double* out) {
    k_dots<<<chunks, NT, 0, st>>>(n, a, n, 1, b, npart);
    k_sum<<<1, 32, 0, st>>>(npart, chunks, scal);
    NT_TRY(cudaGetLastError());
    NT_TRY(cudaMemcpyAsync(pinned, scal, sizeof(double), cudaMemcpyDeviceToHost, st));
    NT_TRY(cudaStreamSynchronize(st));
    *out = *pinned;
    return FE_NO_ERROR;
  }

  // r_out = -(residual at x) on free dofs; *inverted when an element of x
  // has det F <= 0 or a non-finite stress (the kernels' status word).
  int residual(double* x, double* r_out, bool* inverted) {
    *inverted = false;
    int rc = fe_residual_evaluate(h, x, r_out, st);
    if (rc) return rc;
    rc = fe_check(h, st);
    if (rc == FE_ERR_NUMERICAL) {
      *inverted = true;
      return FE_NO_ERROR;
    }
    if (rc) return rc;
    k_mask<<<blocks_for(n), NT, 0, st>>>(n, free_dof, 1.0, r_out, r_out);
    NT_TRY(cudaGetLastError());
    return FE_NO_ERROR;
  }

  // GMRES iteration k on the stream t: orthogonalise V_{k+1} (holding
  // A M^-1 v_k), its Hessenberg column to the host, then scale it and form the
  // next product.
  int iteration_kernels(int k, cudaStream_t t) {
    const int m = k + 1;
    double* wv = V + (size_t)m * n;
    double* cd = col_d + (size_t)(k & 1) * (restart + 2);
    // classical Gram-Schmidt, twice
    k_dots<<<chunks, NT, 0, t>>>(n, V, n, m, wv, part);
    k_update_dots<<<chunks, NT, 0, t>>>(n, V, n, m, part, wv, cd, part2);
    k_update_norm<<<chunks, NT, 0, t>>>(n, V, n, m, part2, wv, cd, npart, done, minv, z,
                                        pinned + (size_t)(k & 1) * (restart + 2));
    NT_TRY(cudaGetLastError());
    return m < restart ? spmv(z, V + (size_t)(m + 1) * n, cd + m, wv, t) : FE_NO_ERROR;
  }

  // The same, from the second cycle on as one graph launch: single launches
  // from the host take longer than the work of a few thousand rows.
  // The buffers stay the same over the whole load step; a graph is recorded
  // when its iteration comes up again.
  int queue_iteration(int k) {
    if (cycles > 0 && !graphs[k] && !no_graphs) {
      cudaGraph_t g = nullptr;
      bool ok = cudaStreamBeginCapture(capture, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
      if (ok) {
        const int rc = iteration_kernels(k, capture);
        ok = cudaStreamEndCapture(capture, &g) == cudaSuccess && rc == FE_NO_ERROR;
      }
      ok = ok && cudaGraphInstantiate(&graphs[k], g, 0) == cudaSuccess;
      if (g) cudaGraphDestroy(g);
      if (!ok) {
        cudaGetLastError();
        graphs[k] = nullptr;
        no_graphs = true;
      }
    }
    if (graphs[k]) {
      NT_TRY(cudaGraphLaunch(graphs[k], st));
    } else {
      const int rc = iteration_kernels(k, st);
      if (rc) return rc;
    }
    NT_TRY(cudaEventRecord(ev[k & 1], st));
    return FE_NO_ERROR;
  }

  // Rows and shared memory of k_cycle for this system; cyc_smem stays 0 when
  // it has more rows than the blocks take: 64 each, a row per eight threads,
  // with which the basis of the longest restart still fits.  Up to that line
  // k_cycle is the faster one at every size (see there).
  void plan_cycle(int* ctl, int* bound) {
    int dev = 0, sms = 0, smem = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop || sms < 2)
      return;
    // a block has 16 rows or more while that many blocks are not all in use
    const int nb = (int)std::min<int64_t>(std::min(sms - 1, MAX_SHARES), (n + 15) / 16);
    if (n > (int64_t)nb * CYCLE_ROWS || n > 65535 || nnz > INT32_MAX) return;
    const int64_t fixed = 8 * (2 * MAX_BASIS + (restart + 3) * LD + 1) + 8 * CYCLE_ROWS;
    const int64_t last = 8 * (2 * (int64_t)MAX_BASIS + 5 * (restart + 1) + (int64_t)restart * (restart + 1) / 2);
    const int64_t room = smem - 1024;  // the kernel's static arrays
    const int64_t cap = (room - fixed) / 10 & ~(int64_t)31;
    if (cap < 0 || last > room) return;
    if (cudaFuncSetAttribute(k_cycle, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    CycleArgs& a = cyc;
    a.n = (int)n;
    a.nb = nb;
    a.restart = restart;
    a.cap = (int)cap;
    a.rp = rp;
    a.col = col;
    a.vals = vals;
    a.minv = minv;
    a.free_dof = free_dof;
    a.z = z;
    a.npart = npart;
    a.part = part;
    a.part2 = part2;
    a.scale = scal;
    a.y = col_d;
    a.ctl = ctl;
    unsigned polls = 0;
    cmfe::newton_barrier_limits(h, &polls, &a.extra_from);
    a.polls = polls ? polls : CYCLE_POLLS;
    if (!a.extra_from) a.extra_from = INT32_MAX;
    a.bound = bound;
    a.host = pinned;
    k_cycle_bounds<<<1, MAX_SHARES + 32, 0, st>>>((int)n, nb, rp, bound);
    if (cudaGetLastError() == cudaSuccess) cyc_smem = (size_t)room;
  }

  // One cycle of at most kmax iterations by k_cycle; *ran false when the GPU
  // cannot hold its blocks at once or one of its barriers gave up, after which
  // res and dx hold nothing of use.
  int cycle(const double* b, double* res, double* dx, double beta, double tol, int kmax, bool* ran, int* K,
            bool* converged, double* r2) {
    CycleArgs a = cyc;
    a.b = b;
    a.res = res;
    a.dx = dx;
    a.beta = beta;
    a.tol = tol;
    a.breakdown = 1e-14 * beta;
    a.kmax = kmax;
    NT_TRY(cudaMemsetAsync(a.ctl, 0, sizeof(int), st));
    pinned[1] = -1.0;
    void* args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_cycle, dim3(a.nb + 1), dim3(CT), args, cyc_smem, st);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
      cudaGetLastError();
      *ran = false;
      return FE_NO_ERROR;
    }
    NT_TRY(e);
    NT_TRY(cudaStreamSynchronize(st));
    *ran = pinned[1] >= 0.0;
    if (!*ran) return FE_NO_ERROR;
    *r2 = pinned[0];
    *K = (int)pinned[1];
    *converged = pinned[2] != 0.0;
    return FE_NO_ERROR;
  }

  // Right-preconditioned GMRES(restart) for A dx = b (b on free dofs, dx
  // zero on fixed ones); returns the iterations in *its.
  int gmres(const double* b, double* dx, double rtol, int max_it, int64_t* its) {
    *its = 0;
    NT_TRY(cudaMemsetAsync(dx, 0, sizeof(double) * n, st));
    double bnorm2 = 0.0;
    int rc = dot_host(b, b, &bnorm2);
    if (rc) return rc;
    const double bnorm = std::sqrt(bnorm2);
    if (bnorm == 0.0) return FE_NO_ERROR;
    double* res = w;  // current residual b - A dx before each cycle
    NT_TRY(cudaMemcpyAsync(res, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    double beta = bnorm;
    std::vector<double> H((size_t)(restart + 1) * restart), cs(restart), sn(restart), g(restart + 1), y(restart);
    std::vector<double> col_h(restart + 2);
    while (*its < max_it) {
      if (beta <= rtol * bnorm) break;
      if (cyc_smem) {
        bool ran = false, conv = false;
        int K = 0;
        double r2 = 0.0;
        const int kmax = (int)std::min<int64_t>(restart, max_it - *its);
        if ((rc = cycle(b, res, dx, beta, rtol * bnorm, kmax, &ran, &K, &conv, &r2))) return rc;
        if (ran) {
          *its += K;
          beta = std::sqrt(r2);
          if (conv && beta <= rtol * bnorm) break;
          continue;
        }
        // the four kernels, from the start of this solve
        cyc_smem = 0;
        *its = 0;
        beta = bnorm;
        NT_TRY(cudaMemsetAsync(dx, 0, sizeof(double) * n, st));
        NT_TRY(cudaMemcpyAsync(res, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
      }
      std::fill(g.begin(), g.end(), 0.0);
      g[0] = beta;
      int k = 0;
      bool done_it = false;
      k_scale_precond<<<blocks_for(n), NT, 0, st>>>(n, 1.0 / beta, minv, res, V, z);
      if ((rc = spmv(z, V + n))) return rc;
      int queued = 0;  // iterations queued: one ahead of the column the host waits for
      while (k < restart && *its < max_it) {
        for (; queued < restart && queued <= k + 1 && *its + (queued - k) < max_it; ++queued) {
          if ((rc = queue_iteration(queued))) return rc;
        }
        NT_TRY(cudaEventSynchronize(ev[k & 1]));
        const double* hc = pinned + (size_t)(k & 1) * (restart + 2);
        std::copy(hc, hc + k + 2, col_h.begin());
        col_h[k + 1] = std::sqrt(col_h[k + 1]);
        // apply the previous rotations, then a new one that zeroes H[k+1][k]
        for (int i = 0; i < k; ++i) {
          const double t = cs[i] * col_h[i] + sn[i] * col_h[i + 1];
          col_h[i + 1] = -sn[i] * col_h[i] + cs[i] * col_h[i + 1];
          col_h[i] = t;
        }
        const double a = col_h[k], bb = col_h[k + 1];
        const double den = std::hypot(a, bb);
        cs[k] = den > 0.0 ? a / den : 1.0;
        sn[k] = den > 0.0 ? bb / den : 0.0;
        for (int i = 0; i <= k; ++i) H[(size_t)i * restart + k] = col_h[i];
        H[(size_t)k * restart + k] = den;
        g[k + 1] = -sn[k] * g[k];
        g[k] = cs[k] * g[k];
        ++k;
        ++*its;
        if (std::fabs(g[k]) <= rtol * bnorm || bb <= 1e-14 * beta) {
          done_it = true;
          break;
        }
      }
      // back substitution for the rotated upper-triangular system
      for (int i = k - 1; i >= 0; --i) {
        double s = g[i];
        for (int j = i + 1; j < k; ++j) s -= H[(size_t)i * restart + j] * y[j];
        const double hii = H[(size_t)i * restart + i];
        y[i] = hii != 0.0 ? s / hii : 0.0;
      }
      NT_TRY(cudaMemcpyAsync(col_d, y.data(), sizeof(double) * k, cudaMemcpyHostToDevice, st));
      k_combine<<<blocks_for(n), NT, 0, st>>>(n, V, n, k, minv, col_d, dx);
      // true residual of the cycle
      if ((rc = spmv(dx, res))) return rc;
      k_axpby<<<blocks_for(n), NT, 0, st>>>(n, 1.0, b, -1.0, res);
      double r2 = 0.0;
      if ((rc = dot_host(res, res, &r2))) return rc;
      beta = std::sqrt(r2);
      ++cycles;
      if (done_it && beta <= rtol * bnorm) break;
    }
    return FE_NO_ERROR;
  }
};

}  // namespace

extern "C" {

void fe_newton_options_default(fe_newton_options* o) {
  if (!o) return;
  o->max_iterations = 50;
  o->atol = 1e-10;
  o->alpha = 1e-4;
  o->max_step = 1e8;
  o->min_lambda = 1e-10;
  o->ksp_rtol = 1e-5;
  o->ksp_restart = 30;
  o->ksp_max_iterations = 600;
  o->forcing = 0;
}

int fe_newton_load_step(fe_handle h, const int32_t* fixed_dofs, const double* fixed_values, int64_t num_fixed,
                        double* x, const fe_newton_options* options, fe_newton_report* report, void* stream) {
  if (!h || !x || !report) return cmfe::record_error(FE_ERR_INVALID_ARGUMENT, "NULL handle, x or report");
  if (num_fixed < 0 || (num_fixed > 0 && (!fixed_dofs || !fixed_values)))
    return cmfe::record_error(FE_ERR_INVALID_ARGUMENT, "fixed dofs and values must be given together");
  fe_newton_options o;
  fe_newton_options_default(&o);
  if (options) o = *options;
  if (o.ksp_restart < 1 || o.ksp_restart > 200 || o.max_iterations < 0 || !(o.atol >= 0.0))
    return cmfe::record_error(FE_ERR_INVALID_ARGUMENT, "invalid Newton options");
  std::memset(report, 0, sizeof(*report));
  Solver S;
  S.h = h;
  S.st = (cudaStream_t)stream;
  S.restart = o.ksp_restart;
  int rc = cmfe::device_pattern(h, &S.rp, &S.col, &S.n, &S.nnz, &S.nu3);
  if (rc) return rc;
  const int64_t n = S.n;
  for (int64_t k = 0; k < num_fixed; ++k)
    if (fixed_dofs[k] < 0 || fixed_dofs[k] >= n) return cmfe::record_error(FE_ERR_INVALID_ARGUMENT, "fixed dof out of range");
  Work W;
  double *dx_state, *fvals;
  int32_t* fdofs;
  int* bound;
  const size_t rs = (size_t)S.restart;
  const size_t basis = rs + 1;
  S.chunks = row_chunks(n);
  W.add(&S.vals, (size_t)S.nnz);
  for (double** p : {&S.r, &S.rn, &S.d, &S.xs, &S.w, &S.minv, &S.diag, &S.z, &dx_state}) W.add(p, (size_t)n);
  W.add(&S.V, (basis + 1) * n);
  W.add(&S.col_d, 2 * (rs + 2));
  const size_t shares = std::max(MAX_CHUNKS, MAX_SHARES);
  W.add(&S.part, (basis + 1) * shares);
  W.add(&S.part2, (basis + 1) * shares);
  W.add(&S.npart, shares);
  W.add(&S.scal, 4);
  W.add(&S.done, 4);
  W.add(&bound, MAX_SHARES + 1);
  W.add(&S.free_dof, (size_t)n);
  W.add(&fvals, num_fixed > 0 ? num_fixed : 1);
  W.add(&fdofs, num_fixed > 0 ? num_fixed : 1);
  if ((rc = W.alloc(2 * (rs + 2) + 4))) return rc;
  S.graphs.assign(rs, nullptr);
  S.no_graphs = cudaStreamCreateWithFlags(&S.capture, cudaStreamNonBlocking) != cudaSuccess;
  S.pinned = W.pinned;
  S.ev = W.ev;
  S.plan_cycle(S.done + 1, bound);
  cudaStream_t st = S.st;
  // the state on the device (x may be host memory)
  cudaPointerAttributes pa;
  bool host_x = true;
  if (cudaPointerGetAttributes(&pa, x) == cudaSuccess)
    host_x = !(pa.type == cudaMemoryTypeDevice || pa.type == cudaMemoryTypeManaged);
  else
    cudaGetLastError();
  double* xd = host_x ? dx_state : x;
  if (host_x) NT_TRY(cudaMemcpyAsync(xd, x, sizeof(double) * n, cudaMemcpyHostToDevice, st));
  NT_TRY(cudaMemsetAsync(S.free_dof, 1, n, st));
  NT_TRY(cudaMemsetAsync(S.done, 0, sizeof(int), st));
  if (num_fixed > 0) {
    NT_TRY(cudaMemcpyAsync(fdofs, fixed_dofs, sizeof(int32_t) * num_fixed, cudaMemcpyHostToDevice, st));
    NT_TRY(cudaMemcpyAsync(fvals, fixed_values, sizeof(double) * num_fixed, cudaMemcpyHostToDevice, st));
    k_fix<<<blocks_for(num_fixed), NT, 0, st>>>(num_fixed, fdofs, fvals, xd, S.free_dof);
    NT_TRY(cudaGetLastError());
  }
  auto finish = [&](int code) -> int {
    if (host_x) {
      const cudaError_t e = cudaMemcpyAsync(x, xd, sizeof(double) * n, cudaMemcpyDeviceToHost, st);
      const cudaError_t e2 = cudaStreamSynchronize(st);
      if (!code && (e != cudaSuccess || e2 != cudaSuccess))
        return cmfe::record_error(FE_ERR_CUDA, "copying the state back failed");
    } else {
      cudaStreamSynchronize(st);
    }
    return code;
  };
  bool inverted = false;
  if ((rc = S.residual(xd, S.r, &inverted))) return finish(rc);
  if (inverted) return finish(cmfe::record_error(FE_ERR_NUMERICAL, "the initial state has an element with det F <= 0"));
  double r2 = 0.0;
  if ((rc = S.dot_host(S.r, S.r, &r2))) return finish(rc);
  double fnorm = std::sqrt(r2), fnorm_prev = -1.0, prev_eta = -1.0;
  report->residual_norm_initial = fnorm;
  report->residual_norm = fnorm;
  report->last_lambda = 0.0;
  int it = 0;
  while (fnorm > o.atol && it < o.max_iterations) {
    if ((rc = fe_jacobian_evaluate(h, xd, S.vals, nullptr, st))) return finish(rc);
    k_diag<<<warp_blocks_for(n), NT, 0, st>>>(n, S.rp, S.col, S.vals, S.diag);
    k_precond<<<warp_blocks_for(n), NT, 0, st>>>(n, S.nu3, S.rp, S.col, S.vals, S.free_dof, S.diag, S.minv);
    NT_TRY(cudaGetLastError());
    double eta = o.ksp_rtol;
    if (o.forcing == 1) {
      // Eisenstat & Walker (1996), choice 2 (gamma 0.9, alpha 2) with their safeguard
      eta = fnorm_prev < 0.0 ? 0.5 : 0.9 * (fnorm / fnorm_prev) * (fnorm / fnorm_prev);
      if (prev_eta >= 0.0 && 0.9 * prev_eta * prev_eta > 0.1) eta = std::fmax(eta, 0.9 * prev_eta * prev_eta);
      eta = std::fmin(std::fmax(eta, o.ksp_rtol), 0.5);
      prev_eta = eta;
    }
    // Newton system A d = -r on the free dofs
    k_mask<<<blocks_for(n), NT, 0, st>>>(n, S.free_dof, -1.0, S.r, S.rn);
    int64_t lits = 0;
    if ((rc = S.gmres(S.rn, S.d, eta, o.ksp_max_iterations, &lits))) return finish(rc);
    report->linear_iterations += lits;
    double dn2 = 0.0;
    if ((rc = S.dot_host(S.d, S.d, &dn2))) return finish(rc);
    if (std::sqrt(dn2) > o.max_step) k_scale<<<blocks_for(n), NT, 0, st>>>(n, o.max_step / std::sqrt(dn2), S.d, S.d);
    // slope of f = 1/2 ||r||^2 along d: r . (A d)
    if ((rc = S.spmv(S.d, S.w))) return finish(rc);
    double slope = 0.0;
    if ((rc = S.dot_host(S.r, S.w, &slope))) return finish(rc);
    if (slope > 0.0) slope = -slope;
    const double f0 = 0.5 * fnorm * fnorm;
    double lam = 1.0, lam_prev = -1.0, f_prev = 0.0, f1 = 0.0;
    bool accepted = false;
    NT_TRY(cudaMemcpyAsync(S.xs, xd, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    while (true) {
      NT_TRY(cudaMemcpyAsync(xd, S.xs, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
      k_axpby<<<blocks_for(n), NT, 0, st>>>(n, lam, S.d, 1.0, xd);  // d is zero on fixed dofs
      if ((rc = S.residual(xd, S.rn, &inverted))) return finish(rc);
      if (inverted) {
        f1 = INFINITY;
      } else {
        double q = 0.0;
        if ((rc = S.dot_host(S.rn, S.rn, &q))) return finish(rc);
        f1 = 0.5 * q;
      }
      if (std::isfinite(f1) && f1 <= f0 + o.alpha * lam * slope) {
        accepted = true;
        break;
      }
      if (lam < o.min_lambda) break;
      double lt;
      if (lam_prev < 0.0 || !std::isfinite(f1)) {
        lt = std::isfinite(f1) ? -slope / (2.0 * (f1 - f0 - slope)) : 0.1 * lam;
      } else {
        const double a1 = f1 - f0 - lam * slope, a2 = f_prev - f0 - lam_prev * slope, den = lam - lam_prev;
        const double a = (a1 / (lam * lam) - a2 / (lam_prev * lam_prev)) / den;
        const double b = (-lam_prev * a1 / (lam * lam) + lam * a2 / (lam_prev * lam_prev)) / den;
        if (a == 0.0) {
          lt = -slope / (2.0 * b);
        } else {
          const double disc = std::fmax(b * b - 3.0 * a * slope, 0.0);
          lt = (-b + std::sqrt(disc)) / (3.0 * a);
        }
      }
      lam_prev = lam;
      f_prev = f1;
      lam = std::fmin(std::fmax(lt, 0.1 * lam), 0.5 * lam);
    }
    report->last_lambda = lam;
    ++it;
    if (!accepted) {
      // No trial step gave sufficient decrease: keep the state, residual and
      // norm from before the step (as PETSc's bt line search leaves X on a
      // failed reduction) and stop.
      NT_TRY(cudaMemcpyAsync(xd, S.xs, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
      report->line_search_failed = 1;
      break;
    }
    std::swap(S.r, S.rn);
    fnorm_prev = fnorm;
    fnorm = std::sqrt(2.0 * f1);
  }
  report->iterations = it;
  report->residual_norm = fnorm;
  report->converged = fnorm <= o.atol;
  return finish(FE_NO_ERROR);
}

}  // extern "C"
