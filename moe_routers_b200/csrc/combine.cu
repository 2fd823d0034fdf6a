// Gate-weighted un-permute and sum over the top-k picks.
//
// Replaces `y_e = expert(x_e) * w_e; out.index_add_(0, tok_e, y_e)`
// (models/decoder_moe.py:270-271): out[t] = sum_j gates[t,j] * y[route_row[t*k+j]],
// accumulated in fp32 in ascending j and rounded once.  One warp per token,
// 128-bit loads and stores; HBM-bound (k rows read + one row written per token).  With few tokens the
// columns of a token are dealt to several warps (blockIdx.y), down to one load per lane and row.
#include "common.cuh"

namespace moe {
namespace {

constexpr int kWarps = 8;
constexpr int kFillCtas = 2 * 148;

template <typename T2>
__device__ __forceinline__ float2 unpack2(uint32_t u);
template <>
__device__ __forceinline__ float2 unpack2<__half2>(uint32_t u) {
  return __half22float2(*reinterpret_cast<__half2*>(&u));
}
template <>
__device__ __forceinline__ float2 unpack2<__nv_bfloat162>(uint32_t u) {
  return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
}
template <typename T2>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__half2>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat162>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Vector path: d % 8 == 0 and 16-byte aligned bases.  DENSE: the rows are those of all experts (`top_k_rt` of them,
// expert e's row of token t at e * tokens + t), `route_row` holds the token's `picks` experts, and a row's gate is
// that of the pick of its expert, or 0.  A pick of an expert that does not exist counts nowhere and is recorded in `status`.
template <typename T2, int TOPK, bool SPLIT, bool DENSE = false>
__global__ void __launch_bounds__(kWarps * 32)
combine_vec_kernel(const uint4* __restrict__ y, const float* __restrict__ gates,
                   const int32_t* __restrict__ route_row, uint4* __restrict__ out, int tokens,
                   int n_vec_total, int part_vec, int top_k_rt, int total_rows, int picks = 0, int32_t* status = nullptr) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * kWarps + (threadIdx.x >> 5);
  // launched with programmatic stream serialisation: everything in global memory is touched after this
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // The kernel behind (the next layer's router) may set itself up; it waits for this one before it reads anything.
  // Layers one behind the other: 16 x 576, 60 experts: 31.9 -> 31.3 us; 3330 x 768, 32 experts: 62.5 -> 61.8.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (t >= tokens) return;
  const int v_begin = SPLIT ? blockIdx.y * part_vec : 0;  // this warp's 16-byte pieces of the row
  const int n_vec = SPLIT ? min(n_vec_total, v_begin + part_vec) : n_vec_total;
  const int top_k = TOPK > 0 ? TOPK : top_k_rt;
  const uint4* src[8];
  float g[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j < top_k) {
      int row;
      if constexpr (DENSE) {
        row = j * tokens + t;
        g[j] = 0.f;
        for (int i = 0; i < picks; ++i)
          if (__ldg(route_row + (size_t)t * picks + i) == j) g[j] += __ldg(gates + (size_t)t * picks + i);
      } else {
        row = route_row[(size_t)t * top_k + j];
        g[j] = gates[(size_t)t * top_k + j];
      }
      if ((unsigned)row >= (unsigned)total_rows) { row = 0; g[j] = 0.f; }  // never read out of bounds
      src[j] = y + (size_t)row * n_vec_total;
    }
  }
  uint4* dst = out + (size_t)t * n_vec_total;
  constexpr int U = 4;
  for (int v0 = v_begin + lane; v0 < n_vec; v0 += U * 32) {
    float acc[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[u][i] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j < top_k) {
        uint4 r[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + u * 32 < n_vec) r[u] = __ldg(src[j] + v0 + u * 32);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (v0 + u * 32 < n_vec) {
            const uint32_t w[4] = {r[u].x, r[u].y, r[u].z, r[u].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f = unpack2<T2>(w[i]);
              acc[u][2 * i] = fmaf(g[j], f.x, acc[u][2 * i]);
              acc[u][2 * i + 1] = fmaf(g[j], f.y, acc[u][2 * i + 1]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (v0 + u * 32 < n_vec) {
        uint4 o;
        o.x = pack2<T2>(acc[u][0], acc[u][1]);
        o.y = pack2<T2>(acc[u][2], acc[u][3]);
        o.z = pack2<T2>(acc[u][4], acc[u][5]);
        o.w = pack2<T2>(acc[u][6], acc[u][7]);
        dst[v0 + u * 32] = o;
      }
    }
  }
  if constexpr (DENSE) {  // (at the end, where nothing waits for it)
    if (lane < picks && (unsigned)__ldg(route_row + (size_t)t * picks + lane) >= (unsigned)top_k) record_error(status, kErrBadIndex);
  }
}

// Scalar path for any d / alignment.
template <typename T>
__global__ void __launch_bounds__(kWarps * 32)
combine_scalar_kernel(const T* __restrict__ y, const float* __restrict__ gates,
                      const int32_t* __restrict__ route_row, T* __restrict__ out, int tokens, int d,
                      int top_k, int total_rows) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (t >= tokens) return;
  for (int c = lane; c < d; c += 32) {
    float acc = 0.f;
    for (int j = 0; j < top_k; ++j) {
      const int row = route_row[(size_t)t * top_k + j];
      if ((unsigned)row < (unsigned)total_rows)
        acc = fmaf(gates[(size_t)t * top_k + j], to_float(y[(size_t)row * d + c]), acc);
    }
    out[(size_t)t * d + c] = from_float<T>(acc);
  }
}

// The columns of a token are halved, down to one load per lane and row, until there are two CTAs for every SM.
inline int part_of(int n_vec, int grid) {
  int part = (n_vec + 127) & ~127;
  while (part > 32 && (long long)grid * ((n_vec + part - 1) / part) < kFillCtas) part = ((part / 2) + 31) & ~31;
  return part;
}
template <typename Kernel>
int launch_vec(Kernel kernel, const uint4* y, const float* gates, const int32_t* rows, uint4* out, int tokens, int n_vec,
                 int part, int top_k, int total_rows, int picks, int32_t* status, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((tokens + kWarps - 1) / kWarps, (n_vec + part - 1) / part, 1);
  cfg.blockDim = dim3(kWarps * 32, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, y, gates, rows, out, tokens, n_vec, part, top_k, total_rows, picks, status);
  if (e != cudaSuccess) return fail(MOE_ERR_LAUNCH, "combine_kernel: %s", cudaGetErrorString(e));
  note_launch();
  return MOE_OK;
}

template <typename T2>
int launch_combine_dense(const void* y, const int32_t* idx, const float* gates, int tokens, int d, int experts, int top_k,
                         void* out, int32_t* status, cudaStream_t s) {
  // One form for all sizes, split down to whole rows: the form without a split takes the same time where that is what part_of
  // gives (8 experts x 4096 tokens x 4096: 68.1 split, 68.3 us; 8 x 16387 x 1024: 58.5, 58.7; 2 x 2048 x 8192 alone is faster
  // without: 22.4, 21.4) and is slower below (8 x 1000 x 4096: 19.6, 26.6).  (With two picks per token it is otherwise, below.)
  const int n_vec = d / 8;
  return launch_vec(combine_vec_kernel<T2, 0, true, true>, static_cast<const uint4*>(y), gates, idx, static_cast<uint4*>(out),
                      tokens, n_vec, part_of(n_vec, (tokens + kWarps - 1) / kWarps), experts, experts * tokens, top_k, status, s);
}

template <typename T, typename T2>
int launch_combine(const void* y, const float* gates, const int32_t* route_row, int tokens, int d,
                   int top_k, void* out, cudaStream_t s) {
  const int grid = (tokens + kWarps - 1) / kWarps;
  const int total_rows = tokens * top_k;
  const uintptr_t align = reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(out);
  if ((align & 15) == 0 && d % 8 == 0) {
    const uint4* yy = static_cast<const uint4*>(y);
    uint4* oo = static_cast<uint4*>(out);
    const int n_vec = d / 8;
    // Set up under the GEMM in front of it in either form (layer of 3330 x 768: 67.5 -> 65.5 us).
    if (grid >= kFillCtas)
      return launch_vec(top_k == 2 ? combine_vec_kernel<T2, 2, false> : combine_vec_kernel<T2, 0, false>, yy, gates, route_row, oo,
                        tokens, n_vec, n_vec, top_k, total_rows, 0, nullptr, s);
    // Few tokens: the columns are dealt to several CTAs (4 x 4096: 5.5 -> 1.6 us; 600 x 2048, k 4: 5.1 -> 4.5; the same
    // code with whole rows was 6 % slower at 4096 and 16387 tokens, hence the template).
    return launch_vec(top_k == 2 ? combine_vec_kernel<T2, 2, true> : combine_vec_kernel<T2, 0, true>, yy, gates, route_row, oo,
                        tokens, n_vec, part_of(n_vec, grid), top_k, total_rows, 0, nullptr, s);
  } else {
    combine_scalar_kernel<T><<<grid, kWarps * 32, 0, s>>>(static_cast<const T*>(y), gates, route_row,
                                                         static_cast<T*>(out), tokens, d, top_k, total_rows);
  }
  return check_launch("combine_kernel");
}

}  // namespace
}  // namespace moe

extern "C" int moe_combine(const void* y, int dtype, const float* gates, const int32_t* route_row,
                           int tokens, int d, int top_k, void* out, void* stream) {
  using namespace moe;
  if (tokens < 0 || d <= 0) return fail(MOE_ERR_ARG, "moe_combine: bad shape");
  if (top_k < 1 || top_k > 8) return fail(MOE_ERR_UNSUPPORTED, "moe_combine: top_k must be in [1,8], got %d", top_k);
  if (tokens == 0) return MOE_OK;
  if (!y || !gates || !route_row || !out) return fail(MOE_ERR_ARG, "moe_combine: null pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case MOE_F16: return launch_combine<__half, __half2>(y, gates, route_row, tokens, d, top_k, out, s);
    case MOE_BF16: return launch_combine<__nv_bfloat16, __nv_bfloat162>(y, gates, route_row, tokens, d, top_k, out, s);
    default: return fail(MOE_ERR_ARG, "moe_combine: dtype must be fp16 or bf16");
  }
}

extern "C" int moe_combine_dense_checked(const void* y, int dtype, const int32_t* idx, const float* gates, int tokens, int d,
                                         int experts, int top_k, void* out, int32_t* device_status, void* stream) {
  using namespace moe;
  if (tokens < 0 || d <= 0 || d % 8 != 0) return fail(MOE_ERR_ARG, "moe_combine_dense: bad shape");
  if (experts < 1 || experts > 8) return fail(MOE_ERR_UNSUPPORTED, "moe_combine_dense: experts must be in [1,8], got %d", experts);
  if (top_k < 1 || top_k > 8) return fail(MOE_ERR_UNSUPPORTED, "moe_combine_dense: top_k must be in [1,8], got %d", top_k);
  if ((long long)experts * tokens > 0x7fffffffLL) return fail(MOE_ERR_UNSUPPORTED, "moe_combine_dense: too many rows");
  if (tokens == 0) return MOE_OK;
  if (!y || !idx || !gates || !out) return fail(MOE_ERR_ARG, "moe_combine_dense: null pointer");
  if ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(out)) & 15)
    return fail(MOE_ERR_ARG, "moe_combine_dense: y and out must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case MOE_F16: return launch_combine_dense<__half2>(y, idx, gates, tokens, d, experts, top_k, out, device_status, s);
    case MOE_BF16: return launch_combine_dense<__nv_bfloat162>(y, idx, gates, tokens, d, experts, top_k, out, device_status, s);
    default: return fail(MOE_ERR_ARG, "moe_combine_dense: dtype must be fp16 or bf16");
  }
}

extern "C" int moe_combine_dense(const void* y, int dtype, const int32_t* idx, const float* gates, int tokens, int d,
                                 int experts, int top_k, void* out, void* stream) {
  return moe_combine_dense_checked(y, dtype, idx, gates, tokens, d, experts, top_k, out, nullptr, stream);
}
