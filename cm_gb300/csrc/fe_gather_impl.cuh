// libcm_fe: the row gather of the staged assembly, device code of the fused
// assembly kernels, which gather a node's rows as soon as the last element
// around the node has stored its record.
//
// One warp forms the rows of one row node from the per-element records
// (cmfe::Rec) of the elements around it, adding them in increasing element
// number -- a fixed order, so the result is deterministic -- and writes each
// row once, contiguously.  This is the addition of
// EQUATIONS_MATRICES_JACOBIAN_ELEMENT_ADD / MATRIX_VALUES_ADD_DP2
// (equations_matrices_routines.f90:3174-3225, matrix_vector.f90:2756-2880) and
// of the residual vector add (distributed_matrix_vector.f90:8853-8927),
// organised by rows instead of by elements: every matrix sector is written
// once, in full, and never read.
//
// What bounds it is latency (a corner node of a triquadratic box sums eight
// elements), so nothing waits in a chain: what a row node needs of an element
// is one contiguous piece of the element's record, the pieces of four
// elements are copied to shared memory at once (cp.async), and every lane
// keeps its columns of the rows in registers.  Which of an element's nodes
// belongs to a column is read from the node's pattern (HostSetup::pat), which
// nodes with equal surroundings share, while the copies are in flight.
//
// Row layout of the mixed split: a displacement row (m, a) holds
// [u_x | u_y | u_z] blocks of wu[a] columns in the FP32 array at
// uu_row_ptr[m nu + a] and its pressure columns in the FP64 array at
// cp_row_ptr[m nu + a]; a pressure row q holds [u_x | u_y | u_z] blocks of
// wp[q] columns and then its pressure-pressure columns (structural zeros) at
// cp_row_ptr[3 nu + q].  With FP64 blocks (T = double) all of a row is in one
// array at row_ptr: [u_x | u_y | u_z | p].  The column of a neighbour inside a
// block is its rank in the row node's neighbour list.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fe_internal.h"

namespace {

constexpr int GR = 4;           // elements whose pieces are in flight together
constexpr int GPOS = 128;       // columns of a u block in registers at a time (4 per lane)
constexpr int GPP = 32;         // pressure columns at a time (1 per lane)
constexpr int GNONE = 255;      // no local node at this column
constexpr int GLIST = 8;        // incidences of a ready node read ahead by the whole CTA

// A row node whose elements are all assembled: u node id < nu, else pressure
// row node id - nu; its incidences [k0, k0 + cnt).
struct ReadyNode {
  int id, k0, cnt, pad;
};

// Shared scratch of one gathering warp: the pieces in flight; u nodes: the
// sums of the pressure columns and the residual; pressure nodes: the sums of
// the row.
template <int NPE, int NPP, class T>
struct GatherCfg {
  using R = cmfe::Rec<NPE, NPP, T>;
  static constexpr int O_ACC = GR * R::ROW;                 // u: [3][GPP], residual [3], then FP64 blocks [9][GPOS]
  static constexpr int O_ACCP = GR * R::PROW;               // p: [3][GPOS], residual
  static constexpr int UB = O_ACC + (3 * GPP + 4 + (sizeof(T) == 8 ? 9 * GPOS : 0)) * 8, PB = O_ACCP + (3 * GPOS + 2) * 8;
  static constexpr int BYTES = UB > PB ? UB : PB;           // multiples of 16
};

// Copies n bytes (a multiple of 16) from global memory to the warp's shared
// memory, through L2 only: other CTAs of the same launch wrote them.
__device__ __forceinline__ void copy_piece(unsigned char* dst, const unsigned char* src, int n, int lane) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  for (int i = 16 * lane; i < n; i += 512)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + i), "l"(src + i) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// One 32-bit word holds the local nodes of the four elements of a round at
// one column.
static_assert(GR == 4, "one byte per element of a round");
__device__ __forceinline__ int inv_at(uint32_t w, int j) { return (w >> (8 * j)) & 255; }

// The three displacement rows of a u node, by one warp.  list: its first
// GLIST incidences (element and local node, rank-table row).
template <int NPE, int NPP, class T, bool ROWS>
__device__ __forceinline__ void gather_unode(const cmfe::KParams& P, const cmfe::StageOut& S, const cmfe::FusedArgs& F,
                                             const ReadyNode& rn, const int2* list, unsigned char* mine, int lane) {
  using R = cmfe::Rec<NPE, NPP, T>;
  constexpr int NR = NPE + NPP;
  constexpr bool FULL = sizeof(T) == 8;
  const int nu = P.nu, a = rn.id;
  const int wu = P.wu[a];
  T* du[3];
  double* dc[3];
  int wc;
  if constexpr (FULL) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      du[m] = P.vals + P.row_ptr[(size_t)m * nu + a];
      dc[m] = du[m] + 3 * wu;
    }
    wc = P.row_ptr[(size_t)a + 1] - P.row_ptr[(size_t)a] - 3 * wu;
  } else {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      du[m] = P.vals_uu + P.uu_row_ptr[(size_t)m * nu + a];
      dc[m] = P.vals + P.cp_row_ptr[(size_t)m * nu + a];
    }
    wc = P.cp_row_ptr[(size_t)a + 1] - P.cp_row_ptr[(size_t)a];  // the same for m = 0..2
  }
  using G = GatherCfg<NPE, NPP, T>;
  double* cacc = reinterpret_cast<double*>(mine + G::O_ACC);
  const uint32_t* pat = F.pat + F.u_pat[a];
  const int passes = max((wu + GPOS - 1) / GPOS, (wc + GPP - 1) / GPP);
  for (int pass = 0; pass < passes; ++pass) {  // one pass unless the neighbourhood is very large
    const int p0 = pass * GPOS, q0 = pass * GPP;
    T acc[FULL ? 1 : GPOS / 32][9];
    double* uacc = cacc + 3 * GPP + 4;
    for (int i = lane; i < 3 * GPP + 3; i += 32) cacc[i] = 0.0;
    if constexpr (FULL) {
      for (int i = lane; i < 9 * GPOS; i += 32) uacc[i] = 0.0;
    } else {
#pragma unroll
      for (int i = 0; i < GPOS / 32; ++i)
#pragma unroll
        for (int mn = 0; mn < 9; ++mn) acc[i][mn] = T(0);
    }
    for (int kb = 0; kb < rn.cnt; kb += GR) {
      const int cnt = min(GR, rn.cnt - kb);
      int2 in = {0, 0};
      if (lane < cnt) in = kb + lane < GLIST ? list[kb + lane] : int2{F.u_inc[rn.k0 + kb + lane], F.u_inc_row[rn.k0 + kb + lane]};
      __syncwarp();
#pragma unroll
      for (int j = 0; j < GR; ++j) {
        const int packed = __shfl_sync(0xffffffffu, in.x, j);
        if (j < cnt)
          copy_piece(mine + j * R::ROW, S.rec + (size_t)(packed >> 5) * R::BYTES + (packed & 31) * R::ROW, R::ROW, lane);
      }
      // the columns' local nodes (FP64: the local nodes' columns) and the
      // pressure parameters' ranks
      const uint32_t* pr = pat + (size_t)(kb / GR) * (wu + 2 * NPP);
      int rq = -1;
      if (lane < 4 * NPP) rq = (int)reinterpret_cast<const uint16_t*>(pr + wu)[lane] - q0;
      if constexpr (FULL) {
        int rk[GR];
#pragma unroll
        for (int j = 0; j < GR; ++j) {
          const int row = __shfl_sync(0xffffffffu, in.y, j);
          rk[j] = j < cnt && lane < NPE ? (P.tables[(size_t)row * NR + lane] & 0x7fff) - p0 : -1;
        }
        copies_done();
        __syncwarp();
        // value i of a piece, [m][n][b], to its column: added in shared
        // memory, where every lane holds a value (the columns of one element
        // are a quarter of a corner node's, so sums per column would issue
        // three times the FP64 instructions)
#pragma unroll
        for (int j = 0; j < GR; ++j) {
          if (j >= cnt) break;
          const double* v = reinterpret_cast<const double*>(mine + j * R::ROW);
#pragma unroll
          for (int s = 0; s < (9 * NPE + 31) / 32; ++s) {
            const int i = 32 * s + lane;
            const int tk = __shfl_sync(0xffffffffu, rk[j], i % NPE);
            if (i < 9 * NPE && tk >= 0 && tk < GPOS) uacc[i / NPE * GPOS + tk] += v[i];
          }
          __syncwarp();
        }
      } else {
        uint32_t w[GPOS / 32];
#pragma unroll
        for (int i = 0; i < GPOS / 32; ++i) w[i] = p0 + 32 * i + lane < wu ? pr[p0 + 32 * i + lane] : 0xffffffffu;
        copies_done();
        __syncwarp();
#pragma unroll
        for (int i = 0; i < GPOS / 32; ++i) {
          if (p0 + 32 * i >= wu) break;
#pragma unroll
          for (int j = 0; j < GR; ++j) {
            const int b = inv_at(w[i], j);
            if (b != GNONE) {
              const T* v = reinterpret_cast<const T*>(mine + j * R::ROW) + b;
#pragma unroll
              for (int mn = 0; mn < 9; ++mn) acc[i][mn] += v[mn * NPE];
            }
          }
        }
      }
      // the piece's FP64 values, [m][q] coupling and [m] residual, one per
      // lane: an FP64 warp instruction costs the same for 3 lanes as for 32
#pragma unroll
      for (int j = 0; j < GR; ++j) {
        if (j >= cnt) break;
        const int tq = __shfl_sync(0xffffffffu, rq, j * NPP + lane % NPP);
        const int at = lane < 3 * NPP ? (tq >= 0 && tq < GPP ? lane / NPP * GPP + tq : -1) : 3 * GPP + lane - 3 * NPP;
        if (lane < 3 * NPP + 3 && at >= 0) cacc[at] += reinterpret_cast<const double*>(mine + j * R::ROW + R::OC)[lane];
        __syncwarp();
      }
    }
    // Row after row (ROWS), so that the sectors a store begins or ends in are
    // completed by the next one: over the host link (outputs in page-locked
    // memory) every part of a sector is a write of its own (32^3 box 7.10 ms with
    // the columns as the outer loop, 6.00 so; device outputs 1.80 and 1.78).  On
    // meshes that are resident at once the columns go first (9x7x8 69.2 us, rows
    // first 69.7).
    constexpr int NC = GPOS / 32;
#pragma unroll
    for (int k = 0; k < 9 * NC; ++k) {
      const int mn = ROWS ? k / NC : k % 9, i = ROWS ? k % NC : k / 9;
      const int pos = p0 + 32 * i + lane;
      if (pos < wu) du[mn / 3][mn % 3 * wu + pos] = FULL ? (T)uacc[mn * GPOS + 32 * i + lane] : acc[FULL ? 0 : i][mn];
    }
    if (q0 + lane < wc) {
#pragma unroll
      for (int m = 0; m < 3; ++m) dc[m][q0 + lane] = cacc[m * GPP + lane];
    }
    if (pass == 0 && lane < 3 && P.r) P.r[(size_t)lane * nu + a] = cacc[3 * GPP + lane];
    __syncwarp();
  }
}

// The row of pressure row node q, by one warp.
template <int NPE, int NPP, class T>
__device__ __forceinline__ void gather_pnode(const cmfe::KParams& P, const cmfe::StageOut& S, const cmfe::FusedArgs& F,
                                             const ReadyNode& rn, const int2* list, unsigned char* mine, int lane) {
  using R = cmfe::Rec<NPE, NPP, T>;
  constexpr int NR = NPE + NPP;
  const int q = rn.id - P.nu;
  const size_t row = (size_t)3 * P.nu + q;
  const int32_t* rp = sizeof(T) == 8 ? P.row_ptr : P.cp_row_ptr;
  const int wp = P.wp[q];
  const int len = rp[row + 1] - rp[row];
  double* out = P.vals + rp[row];
  double* acc = reinterpret_cast<double*>(mine + GatherCfg<NPE, NPP, T>::O_ACCP);
  constexpr int NV = 3 * NPE + 1;  // values of a piece: [n][b] coupling, residual
  for (int p0 = 0; p0 < wp || p0 == 0; p0 += GPOS) {
    for (int i = lane; i < 3 * GPOS + 1; i += 32) acc[i] = 0.0;
    for (int kb = 0; kb < rn.cnt; kb += GR) {
      const int cnt = min(GR, rn.cnt - kb);
      int2 in = {0, 0};
      if (lane < cnt) in = kb + lane < GLIST ? list[kb + lane] : int2{F.p_inc[rn.k0 + kb + lane], F.p_inc_row[rn.k0 + kb + lane]};
      __syncwarp();
      int rk[GR];
#pragma unroll
      for (int j = 0; j < GR; ++j) {
        const int packed = __shfl_sync(0xffffffffu, in.x, j);
        const uint16_t* tab = P.tables + (size_t)__shfl_sync(0xffffffffu, in.y, j) * NR;
        rk[j] = -1;
        if (j < cnt) {
          if (lane < NPE) rk[j] = (tab[lane] & 0x7fff) - p0;
          copy_piece(mine + j * R::PROW, S.rec + (size_t)(packed >> 3) * R::BYTES + R::P0 + (packed & 7) * R::PROW,
                     R::PROW, lane);
        }
      }
      copies_done();
      __syncwarp();
#pragma unroll
      for (int j = 0; j < GR; ++j) {
        if (j >= cnt) break;
        const double* v = reinterpret_cast<const double*>(mine + j * R::PROW);
#pragma unroll
        for (int s = 0; s < (NV + 31) / 32; ++s) {
          const int i = 32 * s + lane;
          const int tk = __shfl_sync(0xffffffffu, rk[j], i % NPE);
          const int at = i < 3 * NPE ? (tk >= 0 && tk < GPOS ? i / NPE * GPOS + tk : -1) : 3 * GPOS;
          if (i < NV && at >= 0) acc[at] += v[i];
        }
        __syncwarp();
      }
    }
    for (int i = lane; i < min(GPOS, wp - p0); i += 32) {
#pragma unroll
      for (int n = 0; n < 3; ++n) out[n * wp + p0 + i] = acc[n * GPOS + i];
    }
    if (p0 == 0) {
      for (int i = 3 * wp + lane; i < len; i += 32) out[i] = 0.0;  // pressure-pressure entries
      if (lane == 0 && P.r) P.r[row] = acc[3 * GPOS];
    }
    __syncwarp();
  }
}

// Counts the finished elements around the row nodes of one element group
// (nvalid elements, local node numbers s_node[el][NR + 1]) and gathers the
// rows of the nodes this completes, by all threads of a CTA.  The records of
// the group are stored; the caller's threads are past a barrier after that.
// Publication follows the release/acquire pattern: every thread fences its
// record stores before the counting, and a completing count is followed by a
// fence before the records are read.  scratch: gather_scratch bytes.
template <int NPE, int NPP, int EG, int THREADS, class T>
struct GroupGather {
  using G = GatherCfg<NPE, NPP, T>;
  static constexpr int NR = NPE + NPP;
  static constexpr int O_READY = THREADS / 32 * G::BYTES;
  static constexpr int O_LIST = O_READY + EG * NR * (int)sizeof(ReadyNode);
  static constexpr int SCRATCH = O_LIST + EG * NR * GLIST * (int)sizeof(int2);

  static __device__ __forceinline__ void run(const cmfe::KParams& P, const cmfe::StageOut& S, const cmfe::FusedArgs& F,
                                             const int* s_node, int nvalid, unsigned char* scratch, int* s_count,
                                             int* s_next) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    ReadyNode* ready = reinterpret_cast<ReadyNode*>(scratch + O_READY);
    int2* list = reinterpret_cast<int2*>(scratch + O_LIST);
    __threadfence();  // release: this thread's record stores before the counts below
    if (tid == 0) *s_count = *s_next = 0;
    __syncthreads();
    for (int i = tid; i < nvalid * NR; i += THREADS) {
      __threadfence();  // cumulative release, after the barrier, for the stores of the whole CTA
      const int el = i / NR, r = i % NR;
      const int node = s_node[el * (NR + 1) + r];
      const bool un = r < NPE;
      const int id = un ? node : P.nu + node;
      const int32_t* ptr = un ? F.u_inc_ptr + node : F.p_inc_ptr + node;
      const int k0 = ptr[0], cnt = ptr[1] - k0;
      if (atomicAdd(F.node_done + id, 1) + 1 == cnt) {
        __threadfence();  // acquire: the records of every element around the node
        ready[atomicAdd(s_count, 1)] = {id, k0, cnt, 0};
      }
    }
    __syncthreads();
    const int nready = *s_count;
    // the incidences of all ready nodes in one go
    for (int i = tid; i < nready * GLIST; i += THREADS) {
      const ReadyNode rn = ready[i / GLIST];
      const int j = i % GLIST;
      if (j < rn.cnt) {
        const bool un = rn.id < P.nu;
        list[i] = int2{(un ? F.u_inc : F.p_inc)[rn.k0 + j], (un ? F.u_inc_row : F.p_inc_row)[rn.k0 + j]};
      }
    }
    __syncthreads();
    unsigned char* mine = scratch + (size_t)warp * G::BYTES;
    for (;;) {  // nodes differ in cost: each warp takes the next one
      int j = 0;
      if (lane == 0) j = atomicAdd(s_next, 1);
      j = __shfl_sync(0xffffffffu, j, 0);
      if (j >= nready) break;
      const ReadyNode rn = ready[j];
      if (rn.id < P.nu)
        gather_unode<NPE, NPP, T, (EG > 2)>(P, S, F, rn, list + j * GLIST, mine, lane);
      else
        gather_pnode<NPE, NPP, T>(P, S, F, rn, list + j * GLIST, mine, lane);
    }
    __syncthreads();  // the next group reuses the scratch
  }
};

}  // namespace
