// libcm_fe: kernels of the learned Newton warm start (include/cm_warmstart.h).
//
// Training runs in FP32 on the CUDA cores (the network is 4-256-256-256-64,
// so one training step is a few tens of MFLOP), one launch per layer and
// direction; inference runs the whole
// network in one launch with BF16 weights on the tensor cores
// (mma.sync m16n8k16, FP32 accumulation), one cluster of eight CTAs per 16 input
// rows with the activations held in shared memory between layers.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <string>

#include "cm_fe.h"
#include "cm_warmstart.h"
#include "fe_internal.h"

namespace {

int cuda_status(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cmfe::record_error(FE_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return FE_NO_ERROR;
}

int bad(const char* what) { return cmfe::record_error(FE_ERR_INVALID_ARGUMENT, what); }

// ---------------------------------------------------------------- FP32 GEMM
constexpr int TM = 64, TN = 64, TK = 16;

__global__ void __launch_bounds__(256) gemm_kernel(int M, int N, int K, const float* __restrict__ A, int64_t a_sm,
                                                   int64_t a_sk, const float* __restrict__ B, int64_t b_sk,
                                                   int64_t b_sn, float* __restrict__ C, int64_t ldc, float beta) {
  __shared__ float As[TK][TM + 4];
  __shared__ float Bs[TK][TN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  const int tr = tid / 16, tc = tid % 16;  // 16 x 16 threads, 4 x 4 outputs each
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += TK) {
    for (int i = tid; i < TM * TK; i += 256) {
      const int mm = i / TK, kk = i % TK;
      const int gm = m0 + mm, gk = k0 + kk;
      As[kk][mm] = (gm < M && gk < K) ? A[(int64_t)gm * a_sm + (int64_t)gk * a_sk] : 0.0f;
    }
    for (int i = tid; i < TN * TK; i += 256) {
      const int kk = i / TN, nn = i % TN;
      const int gn = n0 + nn, gk = k0 + kk;
      Bs[kk][nn] = (gn < N && gk < K) ? B[(int64_t)gk * b_sk + (int64_t)gn * b_sn] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][tr + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tc + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gm = m0 + tr + 16 * i, gn = n0 + tc + 16 * j;
      if (gm < M && gn < N) {
        float* c = &C[(int64_t)gm * ldc + gn];
        *c = beta == 0.0f ? acc[i][j] : acc[i][j] + beta * *c;
      }
    }
}

// ------------------------------------------------- FP32 network training
// One tile of C = A B^T over the whole contraction length: TBM x TBN outputs by
// eight warps, each over an eighth of every 256-long chunk of the contraction,
// their sums added in warp order (deterministic).  On the networks trained
// here (256 x 256 layers, minibatches of 256) a product is a few hundred
// thousand multiply-adds per SM and its time is latency: one wait for the
// operands of a chunk and one reduction, where 64 x 64 tiles walking the
// contraction 16 at a time left 16 CTAs 33 us.
constexpr int TBM = 32, TBN = 16, TBK = 256, TWARPS = 8;
constexpr int TLDA = TBM + 1, TLDB = TBN + 4;
constexpr int TSMEM = ((TBK + 4) * (TLDA + TLDB)) * 4;  // operands; the warps' sums reuse it
static_assert(TWARPS * TBM * (TBN + 1) * 4 <= TSMEM, "reduction scratch");

// Rows r0 .. r0 + ROWS of an operand (R rows in all), chunk [k0, k0 + TBK) of the
// contraction (K long): all loads first (fetch), then into s[k][row] (put).  KC:
// stored [row][K] (contraction contiguous), else [K][row].  Four values at a
// time where the alignment and the sizes allow (vec).  PAR: a parameter, else
// written by a kernel before this one, maybe after this one started: read from
// L2.
template <bool KC, int ROWS, int LD, bool PAR>
struct TileOperand {
  static constexpr int Q = ROWS * TBK / 4 / (32 * TWARPS);
  float4 v[Q];
  static __device__ __forceinline__ bool vec(const float* src, int64_t ld, int R, int K) {
    return (reinterpret_cast<uintptr_t>(src) & 15) == 0 && ld % 4 == 0 && (KC ? K : R) % 4 == 0;
  }
  template <class V>
  static __device__ __forceinline__ V get(const V* p) {
    return PAR ? *p : __ldcg(p);
  }
  static __device__ __forceinline__ void at(int u, int& r, int& k) {
    const int i = u * 32 * TWARPS + threadIdx.x;
    r = KC ? i / (TBK / 4) : i % (ROWS / 4) * 4;
    k = KC ? i % (TBK / 4) * 4 : i / (ROWS / 4);
  }
  __device__ __forceinline__ void fetch(const float* __restrict__ src, int64_t ld, int r0, int R, int k0, int K, bool vec) {
#pragma unroll
    for (int u = 0; u < Q; ++u) {
      int r, k;
      at(u, r, k);
      const float* p = KC ? src + (int64_t)(r0 + r) * ld + k0 + k : src + (int64_t)(k0 + k) * ld + r0 + r;
      v[u] = float4{0.f, 0.f, 0.f, 0.f};
      if (r0 + r < R && k0 + k < K) {
        if (vec) {
          v[u] = get(reinterpret_cast<const float4*>(p));
        } else {
          const int left = KC ? K - k0 - k : R - r0 - r;
          v[u].x = get(p);
          if (left > 1) v[u].y = get(p + 1);
          if (left > 2) v[u].z = get(p + 2);
          if (left > 3) v[u].w = get(p + 3);
        }
      }
    }
  }
  __device__ __forceinline__ void put(float* __restrict__ s, int kn) const {
#pragma unroll
    for (int u = 0; u < Q; ++u) {
      int r, k;
      at(u, r, k);
      if (k >= kn) continue;
      float* d = s + k * LD + r;
      constexpr int st = KC ? LD : 1;
      d[0] = v[u].x;
      d[st] = v[u].y;
      d[2 * st] = v[u].z;
      d[3 * st] = v[u].w;
    }
  }
};

// Programmatic dependent launch along a training step: a kernel lets the next
// one start at once, and the next one waits for the whole of it before it
// touches anything that a kernel of the step writes.  Only the parameters (the
// step's first kernel starts after all earlier work of the stream) are read
// before the wait.  Without the launch attribute both do nothing.  The nine
// launches of a step are bound by their latencies and the gaps between them:
// 64 -> 46 us for the 4-256-256-256-64 network on 256 rows.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The tile at (m0, n0).  Outputs go to out(m, n, value) for m < M, n < N; with
// colsum, sum over the contraction of A's rows to csum(m, value).  BPAR: B is a
// parameter, loaded before the wait for the previous kernel; else the wait is
// the first thing.
template <bool AKC, bool BKC, bool BPAR, class Out, class Sum>
__device__ __forceinline__ void tile_product(int M, int N, int K, const float* A, int64_t lda, const float* B,
                                             int64_t ldb, int m0, int n0, bool colsum, Out out, Sum csum) {
  extern __shared__ __align__(16) float tsm[];
  float* As = tsm;
  float* Bs = tsm + (TBK + 4) * TLDA;  // a chunk's last quadruple may pass its end
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tr = lane >> 2, tc = lane & 3;  // rows tr + 8 i, columns 4 tc + j
  float acc[4][4] = {}, asum = 0.0f;
  TileOperand<AKC, TBM, TLDA, false> ta;
  TileOperand<BKC, TBN, TLDB, BPAR> tb;
  const bool va = ta.vec(A, lda, M, K), vb = tb.vec(B, ldb, N, K);
  for (int k0 = 0; k0 < K; k0 += TBK) {
    const int kn = min(TBK, K - k0);
    if (!BPAR && !k0) wait_for_previous();
    tb.fetch(B, ldb, n0, N, k0, K, vb);
    if (BPAR && !k0) wait_for_previous();
    ta.fetch(A, lda, m0, M, k0, K, va);
    if (k0) __syncthreads();
    ta.put(As, kn);
    tb.put(Bs, kn);
    __syncthreads();
    const int kw = warp * (TBK / TWARPS);
    const int ke = min(TBK / TWARPS, K - k0 - kw);
#pragma unroll 8
    for (int kk = 0; kk < ke; ++kk) {
      const float* a = As + (kw + kk) * TLDA + tr;
      const float4 b = *reinterpret_cast<const float4*>(Bs + (kw + kk) * TLDB + 4 * tc);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float v = a[8 * i];
        acc[i][0] = fmaf(v, b.x, acc[i][0]);
        acc[i][1] = fmaf(v, b.y, acc[i][1]);
        acc[i][2] = fmaf(v, b.z, acc[i][2]);
        acc[i][3] = fmaf(v, b.w, acc[i][3]);
      }
    }
    if (colsum)
      for (int kk = 0; kk < ke; ++kk) asum += As[(kw + kk) * TLDA + lane];
  }
  __syncthreads();
  constexpr int LDR = TBN + 1;
  float* red = tsm + warp * TBM * LDR;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) red[(tr + 8 * i) * LDR + 4 * tc + j] = acc[i][j];
  red[lane * LDR + TBN] = asum;
  __syncthreads();
  for (int i = threadIdx.x; i < TBM * TBN; i += 32 * TWARPS) {
    const int m = i / TBN, n = i % TBN;
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < TWARPS; ++w) v += tsm[w * TBM * LDR + m * LDR + n];
    if (m0 + m < M && n0 + n < N) out(m0 + m, n0 + n, v);
  }
  if (colsum && threadIdx.x < TBM && m0 + (int)threadIdx.x < M) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < TWARPS; ++w) v += tsm[w * TBM * LDR + threadIdx.x * LDR + TBN];
    csum(m0 + threadIdx.x, v);
  }
}

__device__ __forceinline__ float act_fwd(float x, int act);

// y = act(x W^T + b), x: [n][in], W: [out][in].  With target (the last layer of
// a training step): dz = 2 (y - target) / (n out) and this CTA's share of
// sum (y - target)^2 in part.
__global__ void __launch_bounds__(32 * TWARPS) linear_kernel(int n, int in, int out, const float* __restrict__ x,
                                                             const float* __restrict__ W, const float* __restrict__ b,
                                                             int act, float* __restrict__ y,
                                                             const float* __restrict__ target, float* __restrict__ dz,
                                                             float* __restrict__ part) {
  __shared__ float sq[TWARPS];
  let_next_start();
  const int tn = (out + TBN - 1) / TBN;
  const float inv2 = target ? 2.0f / ((float)n * (float)out) : 0.0f;
  float s = 0.0f;
  tile_product<true, true, true>(
      n, out, in, x, in, W, in, blockIdx.x / tn * TBM, blockIdx.x % tn * TBN, false,
      [&](int m, int c, float v) {
        v = act_fwd(v + (b ? b[c] : 0.0f), act);
        const int64_t at = (int64_t)m * out + c;
        if (y) y[at] = v;
        if (target) {
          const float d = v - target[at];
          s = fmaf(d, d, s);
          dz[at] = d * inv2;
        }
      },
      [](int, float) {});
  if (target) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sq[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.0f;
      for (int w = 0; w < TWARPS; ++w) t += sq[w];
      part[blockIdx.x] = t;
    }
  }
}

// Backward of one layer from dz: [n][out]: dW = dz^T h, db = column sums of dz
// (first tw CTAs), and with dprev the previous layer's dz = (dz W) act'(h) (the
// others).  With part: the loss from the last layer's shares, in order.
__global__ void __launch_bounds__(32 * TWARPS) backward_kernel(int n, int in, int out, const float* __restrict__ dz,
                                                               const float* __restrict__ h, const float* __restrict__ W,
                                                               int act, float* __restrict__ dW, float* __restrict__ db,
                                                               float* __restrict__ dprev, int tw,
                                                               const float* __restrict__ part, int parts,
                                                               float* __restrict__ loss) {
  let_next_start();
  if ((int)blockIdx.x < tw) {
    const int tn = (in + TBN - 1) / TBN;
    const int tm = blockIdx.x / tn, tc = blockIdx.x % tn;
    tile_product<false, false, false>(
        out, in, n, dz, out, h, in, tm * TBM, tc * TBN, tc == 0,
        [&](int o, int i, float v) { dW[(int64_t)o * in + i] = v; }, [&](int o, float v) { db[o] = v; });
    if (part && blockIdx.x == 0 && threadIdx.x < 32) {
      float s = 0.0f;
      for (int c = threadIdx.x; c < parts; c += 32) s += __ldcg(part + c);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (threadIdx.x == 0) *loss = s / ((float)n * (float)out);
    }
    return;
  }
  const int t = blockIdx.x - tw, tn = (in + TBN - 1) / TBN;
  tile_product<true, false, true>(
      n, in, out, dz, out, W, in, t / tn * TBM, t % tn * TBN, false,
      [&](int m, int i, float v) {
        const int64_t at = (int64_t)m * in + i;
        const float a = __ldcg(h + at);
        dprev[at] = act == WS_ACT_TANH ? v * (1.0f - a * a) : v;
      },
      [](int, float) {});
}

// Launch that may start before the previous kernel of the stream has ended
// (early) and then waits for it in the kernel.
template <class... P, class... A>
cudaError_t launch_next(void (*kern)(P...), int grid, int threads, size_t smem, cudaStream_t st, bool early, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

int tiles(int m, int n) { return ((m + TBM - 1) / TBM) * ((n + TBN - 1) / TBN); }

// The kernels' shared memory, set once per device.
int tile_attributes() {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && (dev < 0 || dev >= 64 || !done[dev].load())) {
    e = cudaFuncSetAttribute(linear_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TSMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TSMEM);
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev].store(true);
  }
  return e == cudaSuccess ? FE_NO_ERROR
                          : cmfe::record_error(FE_ERR_CUDA, std::string("training kernels: ") + cudaGetErrorString(e));
}

__device__ __forceinline__ float act_fwd(float x, int act) { return act == WS_ACT_TANH ? tanhf(x) : x; }

__global__ void bias_act_kernel(float* y, const float* bias, int rows, int cols, int act) {
  const int64_t n = (int64_t)rows * cols;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(i % cols);
    y[i] = act_fwd(y[i] + (bias ? bias[j] : 0.0f), act);
  }
}

__global__ void act_backward_kernel(const float* y, const float* dy, float* dz, int64_t n, int act) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float g = dy[i];
    dz[i] = act == WS_ACT_TANH ? g * (1.0f - y[i] * y[i]) : g;
  }
}

__global__ void column_sum_kernel(const float* dz, float* db, int rows, int cols) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= cols) return;
  float s = 0.0f;
  for (int i = 0; i < rows; ++i) s += dz[(int64_t)i * cols + j];
  db[j] = s;
}

// One CTA: fixed thread-to-element assignment and a fixed-order tree, so the
// loss does not depend on scheduling.
__global__ void __launch_bounds__(1024) mse_kernel(const float* p, const float* t, float* dp, float* loss, int64_t n) {
  __shared__ float part[1024];
  const float inv = 1.0f / (float)n;
  float s = 0.0f;
  for (int64_t i = threadIdx.x; i < n; i += 1024) {
    const float d = p[i] - t[i];
    s = fmaf(d, d, s);
    if (dp) dp[i] = 2.0f * d * inv;
  }
  part[threadIdx.x] = s;
  __syncthreads();
  for (int w = 512; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = part[0] * inv;
}

__global__ void adam_kernel(float* p, const float* g, float* m, float* v, int64_t n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  wait_for_previous();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = __ldcg(g + i);
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

__global__ void to_bf16_kernel(const float* s, uint16_t* d, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const __nv_bfloat16 h = __float2bfloat16_rn(s[i]);
    d[i] = *reinterpret_cast<const uint16_t*>(&h);
  }
}

// ------------------------------------------------------ BF16 inference
constexpr int MAXW = 256;
constexpr int ICLUSTER = 8;                  // CTAs that share 16 input rows
constexpr int IW = MAXW / 8 / ICLUSTER;      // warps per CTA: one per tile of 8 features
constexpr int ILD = MAXW / 2 + 4;  // activation row in 32-bit words (BF16 pairs), padded off the banks

struct MlpArgs {
  int layers;
  int widths[WS_MAX_LAYERS + 1];
  const uint32_t* w[WS_MAX_LAYERS];  // BF16 pairs, [out][in/2]
  const float* b[WS_MAX_LAYERS];
};

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// The whole network for 16 input rows by a cluster of eight CTAs.  A few rows
// are a latency problem: one CTA walking 256 x 256 layers waits for its weights
// at every step (26 us for the 4-256-256-256-64 network on 256 rows).  Here each
// warp has at most one tile of 8 features of a layer; its weights are at most
// 32 registers and are loaded one layer ahead, and the activations, rounded to
// BF16 as the products take them, go to all eight CTAs' shared memory.  Every
// output is summed over the contraction in order by one warp.
__global__ void __cluster_dims__(ICLUSTER, 1, 1) __launch_bounds__(32 * IW)
    mlp_bf16_kernel(MlpArgs a, int n, const float* __restrict__ x, int xcols, float* __restrict__ y, int act) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ uint32_t buf[2][16][ILD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int tile = cluster.block_rank() * IW + warp;  // of every layer that has as many
  const int row0 = blockIdx.x / ICLUSTER * 16;
  constexpr int MAXS = MAXW / 16;  // k16 steps
  uint32_t w[2][2 * MAXS];
  auto load = [&](int l, uint32_t (&f)[2 * MAXS]) {
    const int steps = 8 * tile < a.widths[l + 1] ? a.widths[l] / 16 : 0;
    const uint32_t* wr = a.w[l] + (int64_t)(8 * tile + gq) * a.widths[l] / 2;
#pragma unroll
    for (int k = 0; k < MAXS; ++k)
      if (k < steps) {
        f[2 * k] = wr[8 * k + tq];
        f[2 * k + 1] = wr[8 * k + tq + 4];
      }
  };
  load(0, w[0]);
  for (int i = threadIdx.x; i < 16 * a.widths[0] / 2; i += blockDim.x) {
    const int r = i / (a.widths[0] / 2), c = 2 * (i % (a.widths[0] / 2));
    const float* xr = x + (int64_t)(row0 + r) * xcols;
    const bool in = row0 + r < n;
    buf[0][r][c / 2] = pack2(in && c < xcols ? xr[c] : 0.0f, in && c + 1 < xcols ? xr[c + 1] : 0.0f);
  }
  cluster.sync();  // every CTA of the cluster has started: its shared memory may be written
  auto layer = [&](int l, uint32_t (&f)[2 * MAXS], uint32_t (&next)[2 * MAXS]) {
    const bool last = l + 1 == a.layers;
    if (!last) load(l + 1, next);
    const int out = a.widths[l + 1], steps = a.widths[l] / 16;
    if (8 * tile < out) {
      const uint32_t(*in)[ILD] = buf[l & 1];
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < MAXS; ++k)
        if (k < steps) {
          const int c = 8 * k + tq;
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
              "{%0,%1,%2,%3};\n"
              : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
              : "r"(in[gq][c]), "r"(in[gq + 8][c]), "r"(in[gq][c + 4]), "r"(in[gq + 8][c + 4]), "r"(f[2 * k]),
                "r"(f[2 * k + 1]));
        }
      const int c = 8 * tile + 2 * tq;
      const float b0 = a.b[l][c], b1 = a.b[l][c + 1];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = gq + 8 * h;
        const float v0 = d[2 * h] + b0, v1 = d[2 * h + 1] + b1;
        if (last) {
          if (row0 + r < n) {
            y[(int64_t)(row0 + r) * out + c] = v0;
            y[(int64_t)(row0 + r) * out + c + 1] = v1;
          }
        } else {
          const uint32_t v = pack2(act_fwd(v0, act), act_fwd(v1, act));
          uint32_t* dst = &buf[(l + 1) & 1][r][c / 2];
#pragma unroll
          for (int q = 0; q < ICLUSTER; ++q) *cluster.map_shared_rank(dst, q) = v;
        }
      }
    }
    // the activations are everywhere; and nobody writes a CTA that has ended
    if (!last) cluster.sync();
  };
  for (int l = 0; l < a.layers; l += 2) {
    layer(l, w[0], w[1]);
    if (l + 1 < a.layers) layer(l + 1, w[1], w[0]);
  }
}

// The same by one CTA of eight warps per 16 rows, which walks the layers' tiles
// of 8 features and waits for their weights from L2: with enough rows to fill
// the SMs that wait is hidden and there are no exchanges between CTAs.  The sums
// and roundings are those of mlp_bf16_kernel.
__global__ void __launch_bounds__(256) mlp_bf16_rows_kernel(MlpArgs a, int n, const float* __restrict__ x, int xcols,
                                                            float* __restrict__ y, int act) {
  __shared__ float buf[2][16][MAXW + 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int row0 = blockIdx.x * 16;
  const int w0 = a.widths[0];
  for (int i = threadIdx.x; i < 16 * w0; i += blockDim.x) {
    const int r = i / w0, c = i % w0;
    buf[0][r][c] = row0 + r < n && c < xcols ? x[(int64_t)(row0 + r) * xcols + c] : 0.0f;
  }
  __syncthreads();
  for (int l = 0; l < a.layers; ++l) {
    const int in = a.widths[l], out = a.widths[l + 1], cur = l & 1;
    const bool last = l + 1 == a.layers;
    for (int nt = warp; nt < out / 8; nt += 8) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      const uint32_t* wr = a.w[l] + (int64_t)(8 * nt + gq) * in / 2;
      for (int k0 = 0; k0 < in; k0 += 16) {
        const float* A0 = &buf[cur][gq][k0 + 2 * tq];
        const float* A1 = &buf[cur][gq + 8][k0 + 2 * tq];
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};\n"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(pack2(A0[0], A0[1])), "r"(pack2(A1[0], A1[1])), "r"(pack2(A0[8], A0[9])), "r"(pack2(A1[8], A1[9])),
              "r"(wr[k0 / 2 + tq]), "r"(wr[k0 / 2 + tq + 4]));
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int r = gq + (h >= 2 ? 8 : 0), c = 8 * nt + 2 * tq + (h & 1);
        const float v = d[h] + a.b[l][c];
        if (!last)
          buf[cur ^ 1][r][c] = act_fwd(v, act);
        else if (row0 + r < n)
          y[(int64_t)(row0 + r) * out + c] = v;
      }
    }
    __syncthreads();
  }
}

int grid_for(int64_t n) {
  int64_t g = (n + 255) / 256;
  return (int)(g < 4096 ? (g < 1 ? 1 : g) : 4096);
}

}  // namespace

extern "C" {

int ws_gemm_f32(int32_t m, int32_t n, int32_t k, const float* a, int64_t a_sm, int64_t a_sk, const float* b,
                int64_t b_sk, int64_t b_sn, float* c, int64_t ldc, float beta, void* stream) {
  if (m < 0 || n < 0 || k < 0 || !a || !b || !c || ldc < n) return bad("ws_gemm_f32: bad sizes or NULL pointer");
  if (m == 0 || n == 0) return FE_NO_ERROR;
  const dim3 grid((n + TN - 1) / TN, (m + TM - 1) / TM);
  gemm_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(m, n, k, a, a_sm, a_sk, b, b_sk, b_sn, c, ldc, beta);
  return cuda_status("ws_gemm_f32");
}

// Many rows: the 64 x 64 tiles of gemm_kernel use their operands four times as
// often as linear_kernel's 32 x 16 ones, whose split contraction and epilogue
// are for the latency of few; the shorter the contraction, the sooner that
// tells.  us, linear_kernel against gemm_kernel and bias_act_kernel, [in x out]:
// 4 x 256 1,024 rows 12.4, 15.7, 2,048 rows 17.0, 16.1, 131,072 rows 509, 163;
// 64 x 64 8,192 rows 20.9, 23.3, 16,384 rows 31.5, 29.2; 256 x 256 8,192 rows
// 95, 100, 16,384 rows 181, 173, 131,072 rows 1,399, 1,096.
static bool many_rows(int n, int in, int out) {
  return tiles(n, out) >= 768 + 18 * (in < 256 ? in : 256) && (n + TM - 1) / TM <= 65535;
}

int ws_linear_f32(int32_t n, int32_t in, int32_t out, const float* x, const float* w, const float* bias, int32_t act,
                  float* y, void* stream) {
  if (n < 0 || in <= 0 || out <= 0 || !x || !w || !y || (act != WS_ACT_IDENTITY && act != WS_ACT_TANH))
    return bad("ws_linear_f32: bad arguments");
  if (n == 0) return FE_NO_ERROR;
  if (many_rows(n, in, out)) {
    gemm_kernel<<<dim3((out + TN - 1) / TN, (n + TM - 1) / TM), 256, 0, (cudaStream_t)stream>>>(n, out, in, x, in, 1, w,
                                                                                                1, in, y, out, 0.0f);
    bias_act_kernel<<<grid_for((int64_t)n * out), 256, 0, (cudaStream_t)stream>>>(y, bias, n, out, act);
    return cuda_status("ws_linear_f32");
  }
  const int rc = tile_attributes();
  if (rc) return rc;
  linear_kernel<<<tiles(n, out), 32 * TWARPS, TSMEM, (cudaStream_t)stream>>>(n, in, out, x, w, bias, act, y, nullptr,
                                                                             nullptr, nullptr);
  return cuda_status("ws_linear_f32");
}

int64_t ws_mlp_workspace(int32_t n, int32_t layers, const int32_t* widths) {
  if (n <= 0 || layers < 1 || layers > WS_MAX_LAYERS || !widths) return 0;
  int64_t floats = tiles(n, widths[layers]);
  for (int l = 1; l <= layers; ++l) floats += 2 * (int64_t)n * widths[l];
  return floats;
}

int ws_mlp_loss_grad(int32_t n, int32_t layers, const int32_t* widths, const float* params, float* grad, const float* x,
                     const float* target, float* loss, float* workspace, void* stream) {
  if (n <= 0 || layers < 1 || layers > WS_MAX_LAYERS || !widths || !params || !grad || !x || !target || !loss || !workspace)
    return bad("ws_mlp_loss_grad: bad arguments");
  for (int l = 0; l <= layers; ++l)
    if (widths[l] <= 0) return bad("ws_mlp_loss_grad: widths must be positive");
  int rc = tile_attributes();
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const float* h[WS_MAX_LAYERS + 1];   // layer outputs
  float* dz[WS_MAX_LAYERS + 1];        // gradients before the activations
  int64_t off[WS_MAX_LAYERS + 1];      // W_l, b_l in params and grad
  float* ws = workspace;
  h[0] = x;
  off[0] = 0;
  for (int l = 0; l < layers; ++l) {
    off[l + 1] = off[l] + (int64_t)widths[l + 1] * (widths[l] + 1);
    h[l + 1] = ws;
    ws += (int64_t)n * widths[l + 1];
    dz[l + 1] = ws;
    ws += (int64_t)n * widths[l + 1];
  }
  float* part = ws;
  for (int l = 0; l < layers; ++l) {
    const int in = widths[l], out = widths[l + 1];
    const float* W = params + off[l];
    const bool last = l + 1 == layers;
    const cudaError_t e =
        launch_next(linear_kernel, tiles(n, out), 32 * TWARPS, TSMEM, st, l > 0, n, in, out, h[l], W,
                    W + (int64_t)out * in, (int)(last ? WS_ACT_IDENTITY : WS_ACT_TANH),
                    last ? nullptr : const_cast<float*>(h[l + 1]), last ? target : nullptr, dz[l + 1], part);
    if (e != cudaSuccess) return cuda_status("ws_mlp_loss_grad");
  }
  for (int l = layers - 1; l >= 0; --l) {
    const int in = widths[l], out = widths[l + 1], tw = tiles(out, in);
    float* dW = grad + off[l];
    const bool last = l + 1 == layers;
    const cudaError_t e =
        launch_next(backward_kernel, tw + (l > 0 ? tiles(n, in) : 0), 32 * TWARPS, TSMEM, st, true, n, in, out, dz[l + 1],
                    h[l], params + off[l], (int)WS_ACT_TANH, dW, dW + (int64_t)out * in, l > 0 ? dz[l] : nullptr, tw,
                    last ? part : nullptr, tiles(n, widths[layers]), loss);
    if (e != cudaSuccess) return cuda_status("ws_mlp_loss_grad");
  }
  return cuda_status("ws_mlp_loss_grad");
}

int ws_bias_act(float* y, const float* bias, int32_t rows, int32_t cols, int32_t act, void* stream) {
  if (!y || rows < 0 || cols <= 0 || (act != WS_ACT_IDENTITY && act != WS_ACT_TANH)) return bad("ws_bias_act: bad arguments");
  bias_act_kernel<<<grid_for((int64_t)rows * cols), 256, 0, (cudaStream_t)stream>>>(y, bias, rows, cols, act);
  return cuda_status("ws_bias_act");
}

int ws_act_backward(const float* y, const float* dy, float* dz, int64_t count, int32_t act, void* stream) {
  if (!y || !dy || !dz || count < 0 || (act != WS_ACT_IDENTITY && act != WS_ACT_TANH)) return bad("ws_act_backward: bad arguments");
  if (count == 0) return FE_NO_ERROR;
  act_backward_kernel<<<grid_for(count), 256, 0, (cudaStream_t)stream>>>(y, dy, dz, count, act);
  return cuda_status("ws_act_backward");
}

int ws_column_sum(const float* dz, float* db, int32_t rows, int32_t cols, void* stream) {
  if (!dz || !db || rows < 0 || cols <= 0) return bad("ws_column_sum: bad arguments");
  column_sum_kernel<<<(cols + 127) / 128, 128, 0, (cudaStream_t)stream>>>(dz, db, rows, cols);
  return cuda_status("ws_column_sum");
}

int ws_mse(const float* pred, const float* target, float* dpred, float* loss, int64_t count, void* stream) {
  if (!pred || !target || !loss || count <= 0) return bad("ws_mse: bad arguments");
  mse_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(pred, target, dpred, loss, count);
  return cuda_status("ws_mse");
}

int ws_adam(float* param, const float* grad, float* m, float* v, int64_t count, float lr, float beta1, float beta2,
            float eps, int32_t step, void* stream) {
  if (!param || !grad || !m || !v || count < 0 || step < 1) return bad("ws_adam: bad arguments");
  if (count == 0) return FE_NO_ERROR;
  const float c1 = 1.0f - std::pow(beta1, (float)step), c2 = 1.0f - std::pow(beta2, (float)step);
  launch_next(adam_kernel, grid_for(count), 256, 0, (cudaStream_t)stream, true, param, grad, m, v, count, lr, beta1, beta2,
              eps, c1, c2);
  return cuda_status("ws_adam");
}

int ws_to_bf16(const float* src, uint16_t* dst, int64_t count, void* stream) {
  if (!src || !dst || count < 0) return bad("ws_to_bf16: bad arguments");
  if (count == 0) return FE_NO_ERROR;
  to_bf16_kernel<<<grid_for(count), 256, 0, (cudaStream_t)stream>>>(src, dst, count);
  return cuda_status("ws_to_bf16");
}

int ws_mlp_forward_bf16(int32_t n, int32_t layers, const int32_t* widths, const uint16_t* const* weights,
                        const float* const* bias, const float* x, float* y, int32_t act, void* stream) {
  return ws_mlp_forward_bf16_cols(n, layers, widths, weights, bias, x, widths ? widths[0] : 0, y, act, stream);
}

int ws_mlp_forward_bf16_cols(int32_t n, int32_t layers, const int32_t* widths, const uint16_t* const* weights,
                             const float* const* bias, const float* x, int32_t x_cols, float* y, int32_t act,
                             void* stream) {
  if (n < 0 || layers < 1 || layers > WS_MAX_LAYERS || !widths || !weights || !bias || !x || !y)
    return bad("ws_mlp_forward_bf16: bad arguments");
  MlpArgs a;
  a.layers = layers;
  for (int l = 0; l <= layers; ++l) {
    if (widths[l] <= 0 || widths[l] % 16 != 0 || widths[l] > MAXW)
      return bad("ws_mlp_forward_bf16: every width must be a positive multiple of 16, at most 256");
    a.widths[l] = widths[l];
  }
  for (int l = 0; l < layers; ++l) {
    if (!weights[l] || !bias[l]) return bad("ws_mlp_forward_bf16: NULL weight or bias");
    if (reinterpret_cast<uintptr_t>(weights[l]) % 4 != 0) return bad("ws_mlp_forward_bf16: weights must be 4-byte aligned");
    a.w[l] = reinterpret_cast<const uint32_t*>(weights[l]);
    a.b[l] = bias[l];
  }
  if (x_cols <= 0 || x_cols > widths[0]) return bad("ws_mlp_forward_bf16: x has 1 to widths[0] columns");
  if (n == 0) return FE_NO_ERROR;
  // A cluster per 16 rows or a CTA, us a call of the 4-256-256-256-64 network: 16
  // rows 30 and 46, 256 rows 33 and 47, 1,024 rows 46 and 47, 2,048 rows 60 and
  // 48, 16,384 rows 276 and 166, 131,072 rows 1,977 and 1,128; of 4-64-64-32:
  // 1,024 rows 32 and 34, 2,048 rows 37 and 33, 131,072 rows 874 and 86.
  if (n <= 1024)
    mlp_bf16_kernel<<<(n + 15) / 16 * ICLUSTER, 32 * IW, 0, (cudaStream_t)stream>>>(a, n, x, x_cols, y, act);
  else
    mlp_bf16_rows_kernel<<<(n + 15) / 16, 256, 0, (cudaStream_t)stream>>>(a, n, x, x_cols, y, act);
  return cuda_status("ws_mlp_forward_bf16");
}

}  // extern "C"
