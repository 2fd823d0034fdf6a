// Sinkhorn-balanced routing in one kernel.
//
// Replaces SinkhornRouter.forward (models/decoder_moe.py:92-123: 2 + 4*iters elementwise and
// reduction launches over a [T,E] fp32 matrix) and the unbuilt kernels of
// kernels/fused_sinkhorn.cu:56-209 (6 launches per iteration, global float atomics).
//
// The reference iterates on the matrix q itself:
//     q = exp(s - rowmax);  iters x { q /= rowsum(q) + eps ;  q = q / (colsum(q) + eps) * T/E };
//     q /= rowsum(q) + eps ;  top-k of q ;  w = vals / (sum(vals) + eps)
// Every step scales whole rows or whole columns, so q_ij = a_i * K_ij * b_j with K = exp(s - rowmax)
// fixed: only the vectors a (rows) and b (columns) change.  K stays on chip for the whole
// run (each CTA owns a block of rows), a row step is local to a CTA, and a column step needs one
// sum over all CTAs: per-CTA partial sums go to a double-buffered global scratch, a grid barrier
// follows, and every CTA adds the partials in the same fixed order (bit-identical b everywhere,
// run-to-run deterministic).  One grid barrier per iteration; the grid is launched cooperatively so
// that all CTAs are co-resident, and the barrier spin is bounded in time.
#include <atomic>
#include <cfloat>
#include <cstdlib>

#include "sm100.cuh"

namespace moe {
namespace {

constexpr int kThreads = 256;

struct SParams {
  const void* logits;
  int logits_dtype;
  int vec_rows;  // rows are a multiple of 16 bytes and 16-byte aligned
  int tokens, experts, top_k, iters;
  float eps, temperature;
  int rows_per_cta;
  void* idx;         // int32, or int64 with idx64
  void* gates;       // fp32, or the logits' type with gate_dtype
  int idx64, gate_dtype;
  float* scratch;    // [2][gridDim.x][experts]
  int32_t* control;  // [0] arrival count, [1] generation
  int32_t* status;
};

// CLUSTER = false: any number of co-resident CTAs (cooperative launch), column partials through a
// global scratch and a grid barrier.  CLUSTER = true: the whole matrix fits the shared memory of
// ONE thread-block cluster (16 or 8 CTAs x 1024 threads); column partials are pushed into every CTA's
// shared memory (st.shared::cluster) and a hardware cluster barrier replaces the grid barrier, which
// takes the global-memory round trips out of every iteration.
__device__ __forceinline__ void store_pick(const SParams& p, size_t at, int pick, float gate) {
  if (p.idx64) static_cast<int64_t*>(p.idx)[at] = pick;
  else static_cast<int32_t*>(p.idx)[at] = pick;
  if (p.gate_dtype == MOE_F32) static_cast<float*>(p.gates)[at] = gate;
  else if (p.gate_dtype == MOE_F16) static_cast<__half*>(p.gates)[at] = __float2half_rn(gate);
  else static_cast<__nv_bfloat16*>(p.gates)[at] = __float2bfloat16_rn(gate);
}

// The column step: b_j <- b_j * (T/E) / (b_j * sum_i a_i K_ij + eps).  Where a column is empty (an expert whose
// logits are all -inf or far below the others) b_j grows by T/E / eps in every iteration; it is kept finite, so
// that q = a * 0 * b stays 0, as it does where q itself is iterated.  (NaN passes.)
__device__ __forceinline__ float next_column_scale(float b, float sum, float eps, float ct) {
  const float next = b / (b * sum + eps) * ct;
  return next > FLT_MAX ? FLT_MAX : next;
}

// One thread per row: scan q_ij = a_i K_ij b_j over the columns keeping the best KMAX entries under
// "larger value, then lower index" (the first slot a candidate beats takes it, the rest shifts down).
template <int KMAX>
__device__ __forceinline__ void topk_rows(const SParams& p, const float* s_k, const float* s_a, const float* s_b,
                                          int SK, int row0, int nrows) {
  for (int r = threadIdx.x; r < nrows; r += (int)blockDim.x) {
    const float* kr = s_k + r * SK;
    const float a = s_a[r];
    float tv[KMAX];
    int ti[KMAX];
#pragma unroll
    for (int j = 0; j < KMAX; ++j) { tv[j] = -INFINITY; ti[j] = 0x7fffffff; }
    for (int c = 0; c < p.experts; ++c) {
      float cv = a * kr[c] * s_b[c];
      int ci = c;
      bool placed = false;
#pragma unroll
      for (int j = 0; j < KMAX; ++j) {
        if (placed || better(cv, ci, tv[j], ti[j])) {
          const float fv = tv[j];
          const int fi = ti[j];
          tv[j] = cv; ti[j] = ci;
          cv = fv; ci = fi;
          placed = true;
        }
      }
    }
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
      if (j < p.top_k) sum += tv[j];
    const float inv = 1.f / (sum + p.eps);
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
      if (j < p.top_k)
        store_pick(p, (size_t)(row0 + r) * p.top_k + j, ti[j] == 0x7fffffff ? 0 : ti[j], tv[j] * inv);
  }
}

template <typename T, bool CLUSTER>
__global__ void __launch_bounds__(CLUSTER ? 1024 : kThreads)
sinkhorn_kernel(const SParams p) {
  extern __shared__ __align__(16) float s_f[];
  const int E = p.experts;
  const int R = p.rows_per_cta;
  const int nthreads = (int)blockDim.x;
  const int nblk = (int)gridDim.x;
  const int cw = min(E, nthreads);       // columns handled side by side
  const int groups = nthreads / cw;      // row groups working on the same column
  const int SK = E + 1;                  // row stride of K in shared memory
  float* s_k = s_f;                      // [R][SK]  K = exp(s - rowmax)
  float* s_a = s_k + (size_t)R * SK;     // [R]      row scale
  float* s_b = s_a + R;                  // [E]      column scale
  float* s_part = s_b + E;               // [groups][E] partial column sums of this CTA
  float* s_all = s_part + (size_t)groups * E;  // [2][nblk][E] partials of all CTAs (CLUSTER only)
  __shared__ int s_flag;

  const int row0 = blockIdx.x * R;
  const int nrows = max(0, min(R, p.tokens - row0));
  const T* logits = static_cast<const T*>(p.logits);
  const float ct = (float)p.tokens / (float)max(E, 1);
  // Remote shared-memory stores below need every CTA of the cluster to be running: arrive now, wait
  // just before the first store (by then the others have long started, so the wait costs nothing).
  if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

  // ---- K = exp(s - rowmax), s = (logits / temperature) rounded to the logits dtype ----
  // coalesced load of the CTA's rows, then one thread per row (rows are SK = E+1 floats apart, so
  // threads of a warp working on consecutive rows hit different banks)
  for (int i = threadIdx.x; i < nrows * E; i += nthreads) {
    const int r = i / E, j = i - r * E;
    float v = to_float(logits[(size_t)row0 * E + i]);
    if (p.temperature != 1.0f) v = to_float(from_float<T>(v / p.temperature));
    s_k[r * SK + j] = v;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < nrows; r += nthreads) {
    float* kr = s_k + r * SK;
    float m = -INFINITY;
    for (int j = 0; j < E; ++j) m = fmaxf(m, kr[j]);
    for (int j = 0; j < E; ++j) kr[j] = expf(kr[j] - m);
    s_a[r] = 1.f;
  }
  for (int j = threadIdx.x; j < E; j += nthreads) s_b[j] = 1.f;
  __syncthreads();

  const int g = threadIdx.x / cw;
  const int jc = threadIdx.x % cw;

  bool ok = true;
  for (int it = 0; it <= p.iters && ok; ++it) {
    // ---- row step: a_i <- a_i / (a_i * sum_j K_ij b_j + eps), one thread per row ----
    for (int r = threadIdx.x; r < nrows; r += nthreads) {
      const float* kr = s_k + r * SK;
      float s0 = 0.f, s1 = 0.f;
      int j = 0;
      for (; j + 1 < E; j += 2) {
        s0 = fmaf(kr[j], s_b[j], s0);
        s1 = fmaf(kr[j + 1], s_b[j + 1], s1);
      }
      if (j < E) s0 = fmaf(kr[j], s_b[j], s0);
      const float a = s_a[r];
      s_a[r] = a / (a * (s0 + s1) + p.eps);
    }
    __syncthreads();
    if (it == p.iters) break;  // the last pass is the final row normalisation only

    // ---- column step: b_j <- b_j * (T/E) / (b_j * sum_i a_i K_ij + eps) ----
    if (g < groups) {
      for (int j = jc; j < E; j += cw) {
        float s = 0.f;
        for (int r = g; r < nrows; r += groups) s = fmaf(s_a[r], s_k[r * SK + j], s);
        s_part[(size_t)g * E + j] = s;
      }
    }
    __syncthreads();
    if constexpr (CLUSTER) {
      // this CTA's column sums go into slot [it & 1][my rank] of every CTA of the cluster
      const uint32_t me = sm100::cluster_ctarank();
      if (it == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      float* slot = s_all + ((size_t)(it & 1) * nblk + me) * E;
      for (int j = threadIdx.x; j < E; j += nthreads) {
        float s = 0.f;
        for (int gg = 0; gg < groups; ++gg) s += s_part[(size_t)gg * E + j];
        const uint32_t local = sm100::smem_u32(slot + j);
        for (int c = 0; c < nblk; ++c) sm100::st_cluster_f32(sm100::map_to_cta(local, (uint32_t)c), s);
      }
      sm100::cluster_sync_all();
      const float* all = s_all + (size_t)(it & 1) * nblk * E;
      for (int j = threadIdx.x; j < E; j += nthreads) {
        float s = 0.f;
        for (int c = 0; c < nblk; ++c) s += all[(size_t)c * E + j];  // same order in every CTA
        const float b = s_b[j];
        s_b[j] = next_column_scale(b, s, p.eps, ct);
      }
      __syncthreads();
    } else {
      float* mine = p.scratch + ((size_t)(it & 1) * nblk + blockIdx.x) * E;
      for (int j = threadIdx.x; j < E; j += nthreads) {
        float s = 0.f;
        for (int gg = 0; gg < groups; ++gg) s += s_part[(size_t)gg * E + j];
        mine[j] = s;
      }
      ok = grid_barrier(p.control, nblk, p.status, &s_flag);
      if (!ok) break;
      // every CTA adds the partials of all CTAs in the same fixed order: `groups` threads per column
      // each take a contiguous range of CTAs (loads in flight together), then the ranges are added
      // in order
      const float* all = p.scratch + (size_t)(it & 1) * nblk * E;
      const int per = (nblk + groups - 1) / groups;
      if (g < groups) {
        for (int j = jc; j < E; j += cw) {
          const int c0 = g * per, c1 = min(nblk, c0 + per);
          float s = 0.f;
          int c = c0;
          for (; c + 7 < c1; c += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = __ldcg(all + (size_t)(c + u) * E + j);
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
          }
          for (; c < c1; ++c) s += __ldcg(all + (size_t)c * E + j);
          s_part[(size_t)g * E + j] = s;
        }
      }
      __syncthreads();
      for (int j = threadIdx.x; j < E; j += nthreads) {
        float s = 0.f;
        for (int gg = 0; gg < groups; ++gg) s += s_part[(size_t)gg * E + j];
        const float b = s_b[j];
        s_b[j] = next_column_scale(b, s, p.eps, ct);
      }
      __syncthreads();
    }
  }
  if (!ok) return;

  // ---- top-k of q_ij = a_i K_ij b_j (lowest index wins ties), w = vals / (sum(vals) + eps) ----
  if (p.top_k <= 1) topk_rows<1>(p, s_k, s_a, s_b, SK, row0, nrows);
  else if (p.top_k <= 2) topk_rows<2>(p, s_k, s_a, s_b, SK, row0, nrows);
  else if (p.top_k <= 4) topk_rows<4>(p, s_k, s_a, s_b, SK, row0, nrows);
  else topk_rows<8>(p, s_k, s_a, s_b, SK, row0, nrows);
}

// ---------------------------------------------------------------------------------------------------
// The matrix in registers.  One cluster of up to 16 CTAs x 512 threads; a lane holds RPL rows x 8 columns
// of K, LPR lanes share a row (8 * LPR >= E), so a warp holds 32 / LPR * RPL rows.  An iteration is a chain
// of short dependent steps, and its latency is all that counts (the arithmetic, 2 * T * E FMA, takes 16 SMs
// 0.13 us at T = 4096, E = 64):
//   row step      b of the lane's columns from shared memory, dot products in registers, sums over the row's
//                 LPR lanes by exchanges that halve the number of rows per lane, so that a row's division is
//                 done once and not by every lane
//   column step   sums over the lane's rows in registers, over the warp by halving exchanges, over the 16
//                 warps and then over the CTAs by half a warp per four columns: CTA partials travel as one
//                 16-byte remote store per CTA and column quad that counts its bytes on the receiver's
//                 mbarrier, so that no CTA waits for a cluster-wide barrier
// with two block-wide barriers and one mbarrier wait.  Every sum is added in an order that depends on the
// shape alone and is the same in every CTA.
// T = 4096, E = 64, 10 iterations: 44.0 -> 21.3 us on the device (the shared-memory form below: K in shared
// memory, one thread per row, partials exchanged behind a cluster barrier), of which 1.3 per iteration, 1.0 per
// pick and the rest launch, loads and exponentials; 256 x 64: 12.7 us, 8192 x 32: 19.1, 8192 x 64: 36.9.  Larger
// matrices keep the forms below (16384 x 64: 76 us).
constexpr int kRegThreads = 512;
constexpr int kRegWarps = kRegThreads / 32;
constexpr int kRegCols = 8;    // columns per lane
constexpr int kRegMaxCtas = 16;
static_assert(kRegWarps == 16 && kRegMaxCtas == 16, "half a warp adds the partials of all warps / all CTAs");

// Sums over the lanes that differ in the bits [LO, HI) of the lane id of N values per lane: each exchange
// halves the values a lane is responsible for until one is left.  Leaves value `owned<N, LO, HI>(lane)`
// (and, while N is larger than the number of lanes, the ones behind it) in v[0..].
template <int N, int LO, int HI>
__device__ __forceinline__ void reduce_lanes(float* v, int lane) {
  if constexpr (LO < HI) {
    if constexpr (N > 1) {
      const bool up = (lane & LO) != 0;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        const float give = up ? v[i] : v[i + N / 2], keep = up ? v[i + N / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, LO);
      }
      reduce_lanes<N / 2, LO * 2, HI>(v, lane);
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], LO);
      reduce_lanes<1, LO * 2, HI>(v, lane);
    }
  }
}
// First of the values that reduce_lanes leaves with this lane.
template <int N, int LO, int HI>
__device__ __forceinline__ int owned(int lane) {
  if constexpr (LO < HI && N > 1) return ((lane & LO) ? N / 2 : 0) + owned<N / 2, LO * 2, HI>(lane);
  else return 0;
}
constexpr int owned_count(int n, int lanes) { return n > lanes ? n / lanes : 1; }
// The way back: every lane gets all N values.
template <int N, int LO, int HI>
__device__ __forceinline__ void spread_lanes(float* v, int lane) {
  if constexpr (LO < HI && N > 1) {
    spread_lanes<N / 2, LO * 2, HI>(v, lane);
    const bool up = (lane & LO) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const float mine = v[i], other = __shfl_xor_sync(0xffffffffu, mine, LO);
      v[i] = up ? other : mine;
      v[i + N / 2] = up ? mine : other;
    }
  }
}

__device__ __forceinline__ void st_async_v4(uint32_t dst_cluster, const float (&v)[4], uint32_t bar_cluster) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   dst_cluster),
               "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar_cluster)
               : "memory");
}

// 8 consecutive logits of RPL rows (RG rows apart) as fp32; rows and columns past the end: -inf.  All loads are
// under way before the first is used: one round trip to memory, not one per row.
template <typename T, int RPL, int RG>
__device__ __forceinline__ void load_logits(const SParams& p, int row0, int c0, float (&k)[RPL][kRegCols]) {
  const T* src = static_cast<const T*>(p.logits) + (size_t)row0 * p.experts + c0;
  const size_t step = (size_t)RG * p.experts;
  if (p.vec_rows && c0 + kRegCols <= p.experts) {
    constexpr int W = 16 / sizeof(T), Q = kRegCols / W;
    union Piece { uint4 q[Q]; T e[kRegCols]; } u[RPL];
#pragma unroll
    for (int r = 0; r < RPL; ++r)
#pragma unroll
      for (int i = 0; i < Q; ++i)
        if (row0 + r * RG < p.tokens) u[r].q[i] = __ldg(reinterpret_cast<const uint4*>(src + r * step) + i);
#pragma unroll
    for (int r = 0; r < RPL; ++r)
#pragma unroll
      for (int j = 0; j < kRegCols; ++j) k[r][j] = row0 + r * RG < p.tokens ? to_float(u[r].e[j]) : -INFINITY;
  } else {
#pragma unroll
    for (int r = 0; r < RPL; ++r)
#pragma unroll
      for (int j = 0; j < kRegCols; ++j)
        k[r][j] = row0 + r * RG < p.tokens && c0 + j < p.experts ? to_float(src[r * step + j]) : -INFINITY;
  }
  if (p.temperature != 1.0f) {
#pragma unroll
    for (int r = 0; r < RPL; ++r)
#pragma unroll
      for (int j = 0; j < kRegCols; ++j) k[r][j] = to_float(from_float<T>(k[r][j] / p.temperature));
  }
}

template <int LPR, int RPL>
__global__ void __launch_bounds__(kRegThreads, 1) sinkhorn_regs_kernel(const SParams p) {
  constexpr int RG = 32 / LPR;          // rows side by side in a warp
  constexpr int EP = LPR * kRegCols;    // columns with padding
  constexpr int SP = EP + 4;            // row of a partial table: conflict-free 16-byte accesses
  constexpr int QUADS = EP / 4;
  constexpr int QPH = (QUADS + 2 * kRegWarps - 1) / (2 * kRegWarps);  // column quads per half warp
  extern __shared__ __align__(16) float s_f[];
  float* s_part = s_f;                       // [warps][SP]        column sums of every warp
  float* s_all = s_part + kRegWarps * SP;    // [2][16][SP]        column sums of every CTA
  float* s_b = s_all + 2 * kRegMaxCtas * SP; // [EP]               column scale
  __shared__ __align__(8) uint64_t s_bar[2];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int E = p.experts, nblk = (int)gridDim.x;
  const uint32_t me = sm100::cluster_ctarank();
  const uint32_t bar0 = sm100::smem_u32(s_bar);
  const uint32_t tx_bytes = (uint32_t)(nblk * EP * sizeof(float));
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) sm100::mbar_init(bar0 + 8 * i, 1);
    sm100::fence_barrier_init();
    for (int i = 0; i < 2; ++i) sm100::mbar_expect_tx(bar0 + 8 * i, tx_bytes);
  }
  for (int j = threadIdx.x; j < EP; j += kRegThreads) s_b[j] = j < E ? 1.f : 0.f;
  __syncthreads();
  // remote stores need every CTA of the cluster running with its barriers initialised: arrive now, wait
  // before the first store
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  // Launched with programmatic stream serialisation: placing a cluster and everything above go on while the kernel in
  // front (a router GEMM, another call's Sinkhorn on 16 of the other SMs) is running; nothing in global memory is
  // touched before the wait.  Calls one behind the other, 4096 x 64: 22.55 -> 20.75 us.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // ---- K = exp(s - rowmax), s = (logits / temperature) rounded to the logits dtype ----
  const int rg = lane / LPR, c0 = (lane % LPR) * kRegCols;
  const int row0 = (int)blockIdx.x * p.rows_per_cta + warp * (RG * RPL) + rg;  // + r * RG
  float k[RPL][kRegCols];
  if (p.logits_dtype == MOE_F16) load_logits<__half, RPL, RG>(p, row0, c0, k);
  else if (p.logits_dtype == MOE_BF16) load_logits<__nv_bfloat16, RPL, RG>(p, row0, c0, k);
  else load_logits<float, RPL, RG>(p, row0, c0, k);
#pragma unroll
  for (int r = 0; r < RPL; ++r) {
    float m = k[r][0];
#pragma unroll
    for (int j = 1; j < kRegCols; ++j) m = fmaxf(m, k[r][j]);
#pragma unroll
    for (int ofs = 1; ofs < LPR; ofs <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, ofs));
    if (row0 + r * RG >= p.tokens) m = 0.f;
#pragma unroll
    for (int j = 0; j < kRegCols; ++j) k[r][j] = expf(k[r][j] - m);  // past the matrix: -inf -> 0
  }

  // the row scales this lane is responsible for (1 inside the matrix, 0 past its end)
  constexpr int AN = owned_count(RPL, LPR);
  const int a_first = owned<RPL, 1, LPR>(lane);
  float a_own[AN];
#pragma unroll
  for (int i = 0; i < AN; ++i) a_own[i] = row0 + (a_first + i) * RG < p.tokens ? 1.f : 0.f;
  float a[RPL];

  // quads: the half warp h of warp w adds the partials of column quads h + 2 w, + 32, ..
  const int half = lane >> 4, src = lane & 15;
  const int col_in_quad = owned<4, 1, 16>(src);
  float b_own[QPH];
#pragma unroll
  for (int i = 0; i < QPH; ++i) b_own[i] = 0.f;
#pragma unroll
  for (int i = 0; i < QPH; ++i)
    if ((i * 2 * kRegWarps + 2 * warp + half) * 4 + col_in_quad < E) b_own[i] = 1.f;
  const float ct = (float)p.tokens / (float)max(E, 1);

  // The exchange that this thread has given up because its wait ran into the limit.  It then takes no further part
  // in any: it stores nothing, so that the CTAs that count on its sums give up in their turn, and arms nothing (a
  // phase that has not completed must not be armed again).  The kernel runs to its end; the status block says why.
  int given_up = p.iters;
  for (int it = 0;; ++it) {
    // ---- row step: a_i <- a_i / (a_i * sum_j K_ij b_j + eps) ----
    float b[kRegCols];
#pragma unroll
    for (int j = 0; j < kRegCols; j += 4) {
      const float4 t = *reinterpret_cast<const float4*>(s_b + c0 + j);
      b[j] = t.x; b[j + 1] = t.y; b[j + 2] = t.z; b[j + 3] = t.w;
    }
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int j = 0; j < kRegCols; j += 2) {
        s0 = fmaf(k[r][j], b[j], s0);
        s1 = fmaf(k[r][j + 1], b[j + 1], s1);
      }
      a[r] = s0 + s1;
    }
    reduce_lanes<RPL, 1, LPR>(a, lane);
#pragma unroll
    for (int i = 0; i < AN; ++i) a[i] = a_own[i] = a_own[i] / (a_own[i] * a[i] + p.eps);
    spread_lanes<RPL, 1, LPR>(a, lane);
    if (it == p.iters) break;  // the last pass is the final row normalisation only

    // ---- column step: b_j <- b_j * (T/E) / (b_j * sum_i a_i K_ij + eps) ----
    float s[kRegCols];
#pragma unroll
    for (int j = 0; j < kRegCols; ++j) {
      s[j] = a[0] * k[0][j];
#pragma unroll
      for (int r = 1; r < RPL; ++r) s[j] = fmaf(a[r], k[r][j], s[j]);
    }
    reduce_lanes<kRegCols, LPR, 32>(s, lane);
    constexpr int SN = owned_count(kRegCols, RG);
    float* part = s_part + warp * SP + c0 + owned<kRegCols, LPR, 32>(lane);
#pragma unroll
    for (int j = 0; j < SN; ++j) part[j] = s[j];  // (lanes with the same columns hold the same sums)
    __syncthreads();
    if (it == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t bar = bar0 + 8u * (uint32_t)(it & 1);
    float* all = s_all + (it & 1) * kRegMaxCtas * SP;
#pragma unroll
    for (int i = 0; i < QPH; ++i) {
      const int quad = i * 2 * kRegWarps + 2 * warp + half;
      if (i * 2 * kRegWarps + 2 * warp < QUADS) {  // uniform over the warp (QUADS is even)
        const float4 t = *reinterpret_cast<const float4*>(s_part + src * SP + quad * 4);
        float v[4] = {t.x, t.y, t.z, t.w};
        reduce_lanes<4, 1, 16>(v, src);
        spread_lanes<4, 1, 16>(v, src);
        if (src < nblk && given_up == p.iters)
          st_async_v4(sm100::map_to_cta(sm100::smem_u32(all + me * SP + quad * 4), (uint32_t)src), v,
                      sm100::map_to_cta(bar, (uint32_t)src));
      }
    }
    if (given_up == p.iters) {
      if (!sm100::mbar_wait_cluster(bar, (uint32_t)(it >> 1) & 1u, p.status, 9)) given_up = it;
      else if (threadIdx.x == 0) sm100::mbar_expect_tx(bar, tx_bytes);  // the buffer's next use, two iterations on
    }
#pragma unroll
    for (int i = 0; i < QPH; ++i) {
      const int quad = i * 2 * kRegWarps + 2 * warp + half;
      if (i * 2 * kRegWarps + 2 * warp < QUADS) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (src < nblk) t = *reinterpret_cast<const float4*>(all + src * SP + quad * 4);
        float v[4] = {t.x, t.y, t.z, t.w};
        reduce_lanes<4, 1, 16>(v, src);
        b_own[i] = next_column_scale(b_own[i], v[0], p.eps, ct);
        if (src < 4) s_b[quad * 4 + col_in_quad] = b_own[i];
      }
    }
    __syncthreads();
  }

  // ---- top-k of q_ij = a_i K_ij b_j (lowest index wins ties), w = vals / (sum(vals) + eps) ----
  float b[kRegCols];
#pragma unroll
  for (int j = 0; j < kRegCols; ++j) b[j] = s_b[c0 + j];
#pragma unroll
  for (int r = 0; r < RPL; ++r) {
    const int row = row0 + r * RG;
#pragma unroll
    for (int j = 0; j < kRegCols; ++j) k[r][j] = c0 + j < E ? a[r] * k[r][j] * b[j] : -INFINITY;
    float sum = 0.f;
    float pv[8];
    int pi[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      if (t < p.top_k) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < kRegCols; ++j)  // ascending columns: the first of equal values stays
          if (k[r][j] > bv) { bv = k[r][j]; bi = c0 + j; }
#pragma unroll
        for (int ofs = 1; ofs < LPR; ofs <<= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, bv, ofs);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, ofs);
          if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
#pragma unroll
        for (int j = 0; j < kRegCols; ++j)
          if (bi == c0 + j) k[r][j] = -INFINITY;  // taken (q itself is never negative)
        pv[t] = bv;
        pi[t] = bi;
        sum += bv;
      }
    }
    const float inv = 1.f / (sum + p.eps);
    if (row < p.tokens && lane % LPR == 0) {
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (t < p.top_k) store_pick(p, (size_t)row * p.top_k + t, pi[t] == 0x7fffffff ? 0 : pi[t], pv[t] * inv);
    }
  }
  // no CTA leaves while another may still store into its shared memory
  sm100::cluster_sync_all();
  // Nobody stores any more, but what was stored for an exchange that was given up, and for the one behind it (no
  // CTA gets past that), may still be under way to this CTA: one more limited wait for each.
  for (int late = given_up; late < min(given_up + 2, p.iters); ++late)
    (void)sm100::mbar_wait_cluster(bar0 + 8u * (uint32_t)(late & 1), (uint32_t)(late >> 1) & 1u, p.status, 9);
}

using RegKernel = void (*)(const SParams);
template <int LPR>
RegKernel reg_kernel_rows(int rpl) {
  return rpl == 1 ? sinkhorn_regs_kernel<LPR, 1> : rpl == 2 ? sinkhorn_regs_kernel<LPR, 2>
         : rpl == 4 ? sinkhorn_regs_kernel<LPR, 4> : sinkhorn_regs_kernel<LPR, 8>;
}
RegKernel reg_kernel(int lpr, int rpl) {
  switch (lpr) {
    case 1: return reg_kernel_rows<1>(rpl);
    case 2: return reg_kernel_rows<2>(rpl);
    case 4: return reg_kernel_rows<4>(rpl);
    case 8: return reg_kernel_rows<8>(rpl);
    case 16: return reg_kernel_rows<16>(rpl);
    default: return reg_kernel_rows<32>(rpl);
  }
}

// Whether the current device can place a cluster of 16 such CTAs: a property of the device (one CTA per SM,
// 16 SMs in one GPC), asked once.
bool places_wide_cluster(RegKernel kernel, const cudaLaunchConfig_t& cfg) {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> known[kMaxDevices];  // 0: not asked yet, 1: no, 2: yes
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
  int v = known[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    int clusters = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess) (void)cudaGetLastError();
    v = e == cudaSuccess && clusters > 0 ? 2 : 1;
    known[dev].store(v, std::memory_order_relaxed);
  }
  return v == 2;
}

// MOE_B200_SINKHORN_CLUSTER=8 in the environment keeps every cluster at the portable size.
bool wide_clusters_allowed() {
  static const bool allowed = [] { const char* v = getenv("MOE_B200_SINKHORN_CLUSTER"); return !(v && atoi(v) == 8); }();
  return allowed;
}

// Launches the register kernel where the matrix fits one cluster's registers: at most 64 elements a thread,
// 16 CTAs (8 where the device cannot place 16 or the environment keeps the portable size), E <= 256:
// T * E <= 524288 (262144) with E rounded up to 8 * 2^n.
// MOE_ERR_UNSUPPORTED, with nothing launched, where it does not.
int launch_sinkhorn_regs(SParams p, cudaStream_t s) {
  int lpr = 1;
  while (lpr * kRegCols < p.experts) lpr *= 2;
  if (lpr > 32) return MOE_ERR_UNSUPPORTED;
  const int rows_per_set = kRegWarps * (32 / lpr);  // rows per CTA and row slot of a lane
  for (int max_ctas = wide_clusters_allowed() ? kRegMaxCtas : kRegMaxCtas / 2; max_ctas >= kRegMaxCtas / 2; max_ctas /= 2) {
    int rpl = 1;
    while (rpl <= 8 && (long long)rows_per_set * rpl * max_ctas < p.tokens) rpl *= 2;
    if (rpl > 8) return MOE_ERR_UNSUPPORTED;
    int ctas = 1;
    while ((long long)rows_per_set * rpl * ctas < p.tokens) ctas *= 2;
    p.rows_per_cta = rows_per_set * rpl;
    RegKernel kernel = reg_kernel(lpr, rpl);
    const int sp = lpr * kRegCols + 4;
    const size_t smem = ((size_t)(kRegWarps + 2 * kRegMaxCtas) * sp + lpr * kRegCols) * sizeof(float);
    cudaError_t e = cudaSuccess;
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && ctas > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return fail(MOE_ERR_LAUNCH, "moe_sinkhorn: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(kRegThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (ctas > 8 && !places_wide_cluster(kernel, cfg)) continue;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kernel, static_cast<const SParams>(p));
    if (e != cudaSuccess) return fail(MOE_ERR_LAUNCH, "sinkhorn_regs_kernel: %s", cudaGetErrorString(e));
    note_launch();
    return MOE_OK;
  }
  return MOE_ERR_UNSUPPORTED;
}

constexpr int kClusterCtas = 8;        // portable cluster size
constexpr int kClusterCtasWide = 16;   // needs cudaFuncAttributeNonPortableClusterSizeAllowed
constexpr int kClusterThreads = 1024;

// Shared memory (bytes) of a launch with `rows` rows per CTA.
size_t sinkhorn_smem(int rows, int experts, int threads, int nblk, bool cluster) {
  const int cw = experts < threads ? experts : threads;
  const int groups = threads / cw;
  size_t floats = (size_t)rows * (experts + 1) + rows + experts + (size_t)groups * experts;
  if (cluster) floats += (size_t)2 * nblk * experts;
  return floats * sizeof(float);
}

// Launch as ONE cluster of `ctas` CTAs.  Returns MOE_ERR_UNSUPPORTED (nothing launched, no error text
// kept) when `probe` is set and the device cannot place such a cluster, so that the caller can fall
// back to the portable size.
template <typename T>
int launch_sinkhorn_cluster(SParams& p, int ctas, size_t smem, cudaStream_t s, bool probe) {
  cudaError_t e = cudaFuncSetAttribute(sinkhorn_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(MOE_ERR_LAUNCH, "moe_sinkhorn: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  if (ctas > kClusterCtas) {
    e = cudaFuncSetAttribute(sinkhorn_kernel<T, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return MOE_ERR_UNSUPPORTED;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, 1, 1);
  cfg.blockDim = dim3(kClusterThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (probe) {
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, sinkhorn_kernel<T, true>, &cfg);
    if (e != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      return MOE_ERR_UNSUPPORTED;
    }
  }
  e = cudaLaunchKernelEx(&cfg, sinkhorn_kernel<T, true>, p);
  if (e != cudaSuccess) return fail(MOE_ERR_LAUNCH, "sinkhorn_kernel (cluster): %s", cudaGetErrorString(e));
  note_launch();
  return MOE_OK;
}

template <typename T>
int launch_sinkhorn(SParams& p, int grid, size_t smem, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(sinkhorn_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(MOE_ERR_LAUNCH, "moe_sinkhorn: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sinkhorn_kernel<T, false>, kThreads, smem);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess || per_sm * sms < grid)
    return fail(MOE_ERR_UNSUPPORTED, "moe_sinkhorn: a grid of %d CTAs cannot be co-resident on this device", grid);
  void* args[] = {&p};
  e = cudaLaunchCooperativeKernel(reinterpret_cast<void*>(sinkhorn_kernel<T, false>), dim3(grid), dim3(kThreads), args, smem, s);
  if (e != cudaSuccess) return fail(MOE_ERR_LAUNCH, "sinkhorn_kernel: %s", cudaGetErrorString(e));
  note_launch();
  return MOE_OK;
}

}  // namespace
}  // namespace moe

namespace moe {
namespace {

int sinkhorn_route(const void* logits, int logits_dtype, int tokens, int experts, int top_k, int iters, float epsilon,
                   float temperature, void* idx, int idx64, void* gates, int gate_dtype, void* workspace,
                   size_t workspace_bytes, void* stream) {
  if (tokens < 0 || experts <= 0) return fail(MOE_ERR_ARG, "moe_sinkhorn: bad shape");
  if (iters <= 0) return fail(MOE_ERR_ARG, "SinkhornRouter.iters must be > 0");
  if (!(epsilon > 0.f)) return fail(MOE_ERR_ARG, "SinkhornRouter.epsilon must be > 0");
  if (!(temperature > 0.f)) return fail(MOE_ERR_ARG, "SinkhornRouter.temperature must be > 0");
  if (top_k <= 0) return fail(MOE_ERR_ARG, "top_k must be > 0");
  if (top_k > experts) return fail(MOE_ERR_ARG, "top_k must be <= n_experts");
  if (top_k > 8) return fail(MOE_ERR_UNSUPPORTED, "moe_sinkhorn: top_k must be <= 8, got %d", top_k);
  if (experts > 1024) return fail(MOE_ERR_UNSUPPORTED, "moe_sinkhorn: experts must be <= 1024");
  if (tokens == 0) return MOE_OK;
  if (!logits || !idx || !gates) return fail(MOE_ERR_ARG, "moe_sinkhorn: null pointer");
  if (!workspace || workspace_bytes < workspace_bytes_for(tokens, experts, top_k))
    return fail(MOE_ERR_WORKSPACE, "moe_sinkhorn: workspace too small (need %zu bytes)",
                workspace_bytes_for(tokens, experts, top_k));
  Workspace ws = carve(workspace, tokens, experts);

  SParams p;
  p.logits = logits; p.logits_dtype = logits_dtype; p.tokens = tokens; p.experts = experts; p.top_k = top_k; p.iters = iters;
  p.eps = epsilon; p.temperature = temperature;
  p.idx = idx; p.idx64 = idx64; p.gates = gates; p.gate_dtype = gate_dtype; p.scratch = ws.fscratch; p.control = ws.control; p.status = ws.status;
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  if (logits_dtype != MOE_F16 && logits_dtype != MOE_BF16 && logits_dtype != MOE_F32)
    return fail(MOE_ERR_ARG, "moe_sinkhorn: logits must be fp16/bf16/fp32");
  p.vec_rows = (((size_t)experts * (logits_dtype == MOE_F32 ? 4 : 2)) | reinterpret_cast<uintptr_t>(logits)) % 16 == 0;
  const int rc_regs = launch_sinkhorn_regs(p, s);
  if (rc_regs != MOE_ERR_UNSUPPORTED) return rc_regs;

  // One cluster when the matrix fits its shared memory (T=4096, E=64 does): no global round trips
  // inside the iterations.  16 CTAs where the device can place such a cluster (half the rows per CTA:
  // every pass of the iteration is shorter), else the portable 8.
  for (int ctas : {kClusterCtasWide, kClusterCtas}) {
    if (ctas == kClusterCtasWide && (!wide_clusters_allowed() || tokens < 1024)) continue;
    const int rows = (tokens + ctas - 1) / ctas;
    const size_t smem = sinkhorn_smem(rows, experts, kClusterThreads, ctas, true);
    if (smem <= 200 * 1024 && tokens >= 256) {
      p.rows_per_cta = rows;
      const bool probe = ctas == kClusterCtasWide;
      int rc;
      switch (logits_dtype) {
        case MOE_F16: rc = launch_sinkhorn_cluster<__half>(p, ctas, smem, s, probe); break;
        case MOE_BF16: rc = launch_sinkhorn_cluster<__nv_bfloat16>(p, ctas, smem, s, probe); break;
        case MOE_F32: rc = launch_sinkhorn_cluster<float>(p, ctas, smem, s, probe); break;
        default: return fail(MOE_ERR_ARG, "moe_sinkhorn: logits must be fp16/bf16/fp32");
      }
      if (!(probe && rc == MOE_ERR_UNSUPPORTED)) return rc;
    }
  }

  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  int grid = (tokens + 127) / 128;  // about 128 rows per CTA: few partials to add after each barrier
  if (grid > sms) grid = sms;
  if (grid > kMaxGridBlocks) grid = kMaxGridBlocks;
  const int rows_per_cta = (tokens + grid - 1) / grid;
  grid = (tokens + rows_per_cta - 1) / rows_per_cta;
  const size_t smem = sinkhorn_smem(rows_per_cta, experts, kThreads, grid, false);
  if (smem > 200 * 1024)
    return fail(MOE_ERR_UNSUPPORTED, "moe_sinkhorn: tokens*experts too large for the resident kernel (%d x %d)", tokens, experts);
  p.rows_per_cta = rows_per_cta;
  switch (logits_dtype) {
    case MOE_F16: return launch_sinkhorn<__half>(p, grid, smem, s);
    case MOE_BF16: return launch_sinkhorn<__nv_bfloat16>(p, grid, smem, s);
    case MOE_F32: return launch_sinkhorn<float>(p, grid, smem, s);
    default: return fail(MOE_ERR_ARG, "moe_sinkhorn: logits must be fp16/bf16/fp32");
  }
}

}  // namespace
}  // namespace moe

extern "C" int moe_sinkhorn(const void* logits, int logits_dtype, int tokens, int experts, int top_k, int iters,
                            float epsilon, float temperature, int32_t* idx, float* gates, void* workspace,
                            size_t workspace_bytes, void* stream) {
  return moe::sinkhorn_route(logits, logits_dtype, tokens, experts, top_k, iters, epsilon, temperature, idx, 0, gates,
                             MOE_F32, workspace, workspace_bytes, stream);
}

extern "C" int moe_sinkhorn_router(const void* logits, int logits_dtype, int tokens, int experts, int top_k, int iters,
                                   float epsilon, float temperature, int64_t* idx, void* weights, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  return moe::sinkhorn_route(logits, logits_dtype, tokens, experts, top_k, iters, epsilon, temperature, idx, 1, weights,
                             logits_dtype, workspace, workspace_bytes, stream);
}
