// Small fused kernels of the decode harness around the packed linears: residual add + RMSNorm,
// rotary embedding + KV-cache write, SiLU(gate) * up.  The reference leaves these to vLLM /
// transformers (inference_lib/inference_demo_vllm.py, inference_demo_transformers.py:141-173); they are
// here so that a decode step is a few launches per layer instead of dozens of elementwise ones.
// T is __half or __nv_bfloat16; arithmetic is fp32.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/matgptq_b200.h"
#include "helper_kernels.cuh"
#include "kernels.h"

namespace mg {

// x[row] += delta[row] (when delta != null), then h[row] = rmsnorm(x[row]) * weight.  One CTA per row.
template <typename T>
__global__ void __launch_bounds__(256) add_rmsnorm_kernel(T *__restrict__ x, const T *__restrict__ delta, const T *__restrict__ weight,
                                                          T *__restrict__ h, int hidden, float eps) {
  pdl_prologue();
  __shared__ float red[8];
  T *xr = x + static_cast<size_t>(blockIdx.x) * hidden;
  const T *dr = delta ? delta + static_cast<size_t>(blockIdx.x) * hidden : nullptr;
  float ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    float v = to_f(xr[i]);
    if (dr) {
      v = to_f(from_f<T>(v + to_f(dr[i])));  // the residual stream stays in the model dtype
      xr[i] = from_f<T>(v);
    }
    ss += v * v;
  }
  for (int off = 16; off >= 1; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) tot += red[i];
  const float inv = rsqrtf(tot / hidden + eps);
  T *hr = h + static_cast<size_t>(blockIdx.x) * hidden;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x)
    hr[i] = from_f<T>(to_f(from_f<T>(to_f(xr[i]) * inv)) * to_f(weight[i]));
}

// The same with 16-byte accesses and the row kept in registers: hidden % 8 == 0, hidden <= 512 * 8 * kRowVecs.
constexpr int kNormThreads = 512, kRowVecs = 4;
template <typename T>
__global__ void __launch_bounds__(kNormThreads) add_rmsnorm_vec_kernel(T *__restrict__ x, const T *__restrict__ delta,
                                                                       const T *__restrict__ weight, T *__restrict__ h, int hidden,
                                                                       float eps) {
  pdl_prologue();
  __shared__ float red[kNormThreads / 32];
  const int nvec = hidden >> 3;
  uint4 *xr = reinterpret_cast<uint4 *>(x + static_cast<size_t>(blockIdx.x) * hidden);
  const uint4 *dr = delta ? reinterpret_cast<const uint4 *>(delta + static_cast<size_t>(blockIdx.x) * hidden) : nullptr;
  const uint4 *wr = reinterpret_cast<const uint4 *>(weight);
  uint4 xv[kRowVecs], dv[kRowVecs], wv[kRowVecs];
#pragma unroll
  for (int j = 0; j < kRowVecs; ++j) {
    const int v = threadIdx.x + j * kNormThreads;
    if (v < nvec) {
      xv[j] = xr[v];
      if (dr) dv[j] = dr[v];
      wv[j] = wr[v];
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kRowVecs; ++j) {
    const int v = threadIdx.x + j * kNormThreads;
    if (v < nvec) {
      T *xe = reinterpret_cast<T *>(&xv[j]);
      const T *de = reinterpret_cast<const T *>(&dv[j]);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (dr) xe[e] = from_f<T>(to_f(xe[e]) + to_f(de[e]));
        const float f = to_f(xe[e]);
        ss += f * f;
      }
      if (dr) xr[v] = xv[j];
    }
  }
  for (int off = 16; off >= 1; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) tot += red[i];
  const float inv = rsqrtf(tot / hidden + eps);
  uint4 *hr = reinterpret_cast<uint4 *>(h + static_cast<size_t>(blockIdx.x) * hidden);
#pragma unroll
  for (int j = 0; j < kRowVecs; ++j) {
    const int v = threadIdx.x + j * kNormThreads;
    if (v < nvec) {
      uint4 o;
      T *oe = reinterpret_cast<T *>(&o);
      const T *xe = reinterpret_cast<const T *>(&xv[j]);
      const T *we = reinterpret_cast<const T *>(&wv[j]);
#pragma unroll
      for (int e = 0; e < 8; ++e) oe[e] = from_f<T>(to_f(from_f<T>(to_f(xe[e]) * inv)) * to_f(we[e]));
      hr[v] = o;
    }
  }
}

// The rotation with its roundings spelled out: left to the compiler, the two kernels below contracted the same expression
// differently, and a model whose layers amplify one flipped bit showed it.
__device__ __forceinline__ float rotated_even(float a, float c, float cs, float sn) { return __fmaf_rn(a, cs, -__fmul_rn(c, sn)); }
__device__ __forceinline__ float rotated_odd(float a, float c, float cs, float sn) { return __fmaf_rn(c, cs, __fmul_rn(a, sn)); }

// qkv [B, S, (H + 2*KV) * d] -> q_out [B, H, S, d] rotated; k rotated and v written into the caches
// [B, KV, max_seq, d] at positions[s].  cos/sin are [max_seq, d/2] fp32.  Pairs are (2i, 2i+1).
template <typename T>
__global__ void rope_kv_kernel(const T *__restrict__ qkv, const long long *__restrict__ positions, const float *__restrict__ cos_t,
                               const float *__restrict__ sin_t, T *__restrict__ q_out, T *__restrict__ k_cache, T *__restrict__ v_cache,
                               int B, int S, int H, int KV, int d, int max_seq) {
  pdl_prologue();
  const int heads = H + 2 * KV, half = d / 2;
  const long long total = static_cast<long long>(B) * S * heads * half;
  for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(idx % half);
    long long r = idx / half;
    const int head = static_cast<int>(r % heads);
    r /= heads;
    const int s = static_cast<int>(r % S), b = static_cast<int>(r / S);
    const long long pos = positions[s];
    const T *src = qkv + ((static_cast<size_t>(b) * S + s) * heads + head) * d + 2 * i;
    const float a = to_f(src[0]), c = to_f(src[1]);
    if (head < H + KV) {
      const float cs = cos_t[pos * half + i], sn = sin_t[pos * half + i];
      const T r0 = from_f<T>(rotated_even(a, c, cs, sn)), r1 = from_f<T>(rotated_odd(a, c, cs, sn));
      T *dst = (head < H) ? q_out + ((static_cast<size_t>(b) * H + head) * S + s) * d + 2 * i
                          : k_cache + ((static_cast<size_t>(b) * KV + (head - H)) * max_seq + pos) * d + 2 * i;
      dst[0] = r0;
      dst[1] = r1;
    } else {
      T *dst = v_cache + ((static_cast<size_t>(b) * KV + (head - H - KV)) * max_seq + pos) * d + 2 * i;
      dst[0] = src[0];
      dst[1] = src[1];
    }
  }
}

// The same with 16-byte accesses: a thread takes eight elements (four pairs) of one head, blockIdx.y walks the rows.
// head_dim % 8 == 0, everything 16-byte aligned.  Bound by latency for few rows and by memory for a prompt; one pair per
// thread spent its time on three 64-bit divisions and 2-byte accesses (with silu_mul below, four 8B layers: a prompt of 512
// tokens 1462 -> 1388 us, a decode step at batch 1 258 -> 253).
template <typename T>
__global__ void __launch_bounds__(256) rope_kv_vec_kernel(const T *__restrict__ qkv, const long long *__restrict__ positions,
                                                          const float *__restrict__ cos_t, const float *__restrict__ sin_t,
                                                          T *__restrict__ q_out, T *__restrict__ k_cache, T *__restrict__ v_cache,
                                                          int B, int S, int H, int KV, int d, int max_seq) {
  pdl_prologue();
  const int heads = H + 2 * KV, vecs = d >> 3;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= heads * vecs) return;
  const int head = idx / vecs, i = (idx - head * vecs) * 8;
  for (int row = blockIdx.y; row < B * S; row += gridDim.y) {
    const int b = row / S, s = row - b * S;
    const long long pos = positions[s];
    uint4 v = *reinterpret_cast<const uint4 *>(qkv + (static_cast<size_t>(row) * heads + head) * d + i);
    if (head < H + KV) {
      const float4 cs = *reinterpret_cast<const float4 *>(cos_t + pos * (d >> 1) + (i >> 1));
      const float4 sn = *reinterpret_cast<const float4 *>(sin_t + pos * (d >> 1) + (i >> 1));
      const float cv[4] = {cs.x, cs.y, cs.z, cs.w}, sv[4] = {sn.x, sn.y, sn.z, sn.w};
      T *e = reinterpret_cast<T *>(&v);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float a = to_f(e[2 * p]), c = to_f(e[2 * p + 1]);
        e[2 * p] = from_f<T>(rotated_even(a, c, cv[p], sv[p]));
        e[2 * p + 1] = from_f<T>(rotated_odd(a, c, cv[p], sv[p]));
      }
    }
    T *dst = head < H ? q_out + ((static_cast<size_t>(b) * H + head) * S + s) * d
             : head < H + KV ? k_cache + ((static_cast<size_t>(b) * KV + (head - H)) * max_seq + pos) * d
                             : v_cache + ((static_cast<size_t>(b) * KV + (head - H - KV)) * max_seq + pos) * d;
    *reinterpret_cast<uint4 *>(dst + i) = v;
  }
}

// gu [rows, 2*inter] -> out [rows, inter] = silu(gate) * up, both factors rounded to the model dtype first
template <typename T>
__global__ void silu_mul_kernel(const T *__restrict__ gu, T *__restrict__ out, long long rows, int inter) {
  pdl_prologue();
  const long long total = rows * inter;
  for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = idx / inter;
    const int c = static_cast<int>(idx - r * inter);
    const float gte = to_f(gu[r * 2 * inter + c]), up = to_f(gu[r * 2 * inter + inter + c]);
    const float act = to_f(from_f<T>(gte / (1.f + __expf(-gte))));
    out[idx] = from_f<T>(act * up);
  }
}

// The same with 16-byte accesses, eight outputs a thread, blockIdx.y walks the rows: inter % 8 == 0 and 16-byte aligned
// buffers.  Bound by memory for a prompt; one output per thread spent its time on a 64-bit division and 2-byte accesses.
template <typename T>
__global__ void __launch_bounds__(256) silu_mul_vec_kernel(const T *__restrict__ gu, T *__restrict__ out, long long rows, int inter) {
  pdl_prologue();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= inter) return;
  for (long long r = blockIdx.y; r < rows; r += gridDim.y) {
    const uint4 gv = *reinterpret_cast<const uint4 *>(gu + r * 2 * inter + c);
    const uint4 uv = *reinterpret_cast<const uint4 *>(gu + r * 2 * inter + inter + c);
    const T *ge = reinterpret_cast<const T *>(&gv);
    const T *ue = reinterpret_cast<const T *>(&uv);
    uint4 o;
    T *oe = reinterpret_cast<T *>(&o);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float gte = to_f(ge[k]);
      oe[k] = from_f<T>(to_f(from_f<T>(gte / (1.f + __expf(-gte)))) * to_f(ue[k]));
    }
    *reinterpret_cast<uint4 *>(out + r * inter + c) = o;
  }
}

// mask [S, keys] in the model dtype for scores that are added up: 0 where a key is at or before the query's position, -inf
// behind it.  Eight keys a thread with one 16-byte store where keys % 8 == 0.  Bound by latency (half a KB for a decode step):
// one launch in the chain for the four elementwise ones that torch made of it (four 8B layers: a decode step at batch 1
// 251 -> 247 us; at batch 32, 467 -> 463, within what runs differ by).
template <typename T>
__global__ void __launch_bounds__(128) causal_mask_kernel(const long long *__restrict__ positions, T *__restrict__ mask, int seq, int keys) {
  pdl_prologue();
  const T none = from_f<T>(0.f), hidden = from_f<T>(-INFINITY);
  const int first = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (first >= keys) return;
  for (int s = blockIdx.y; s < seq; s += gridDim.y) {
    const long long pos = positions[s];
    T *row = mask + static_cast<size_t>(s) * keys;
    alignas(16) T v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = first + k <= pos ? none : hidden;
    if (keys % 8 == 0) {
      *reinterpret_cast<uint4 *>(row + first) = *reinterpret_cast<const uint4 *>(v);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (first + k < keys) row[first + k] = v[k];
    }
  }
}

// Greedy sampling: index of the largest logit of every row (the first one on ties), one CTA per row.  Logits
// [rows, cols] in the model dtype; `cols` a multiple of 8 and rows 16-byte aligned for the vector loads.
template <typename T>
__global__ void __launch_bounds__(1024, 1) argmax_kernel(const T *__restrict__ logits, long long *__restrict__ out, int cols) {
  pdl_prologue();
  const T *row = logits + static_cast<long long>(blockIdx.x) * cols;
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  for (int c = threadIdx.x * 8; c < cols; c += blockDim.x * 8) {
    const uint4 v = *reinterpret_cast<const uint4 *>(row + c);
    const T *e = reinterpret_cast<const T *>(&v);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float f = to_f(e[k]);
      if (f > best) {  // strictly greater: within a thread the columns ascend, so the first maximum stays
        best = f;
        best_i = c + k;
      }
    }
  }
  __shared__ float s_val[32];
  __shared__ int s_idx[32];
  auto better = [](float a, int ai, float b, int bi) { return a > b || (a == b && ai < bi); };
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float ov = __shfl_down_sync(0xffffffffu, best, off);
    const int oi = __shfl_down_sync(0xffffffffu, best_i, off);
    if (better(ov, oi, best, best_i)) {
      best = ov;
      best_i = oi;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    s_val[threadIdx.x >> 5] = best;
    s_idx[threadIdx.x >> 5] = best_i;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = blockDim.x >> 5;
    best = threadIdx.x < nw ? s_val[threadIdx.x] : -INFINITY;
    best_i = threadIdx.x < nw ? s_idx[threadIdx.x] : 0x7fffffff;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float ov = __shfl_down_sync(0xffffffffu, best, off);
      const int oi = __shfl_down_sync(0xffffffffu, best_i, off);
      if (better(ov, oi, best, best_i)) {
        best = ov;
        best_i = oi;
      }
    }
    if (threadIdx.x == 0) out[blockIdx.x] = best_i == 0x7fffffff ? 0 : best_i;
  }
}

static unsigned grid_for(long long total, int threads) {
  long long blocks = (total + threads - 1) / threads;
  if (blocks > 148LL * 16) blocks = 148LL * 16;
  if (blocks < 1) blocks = 1;
  return static_cast<unsigned>(blocks);
}

// blockIdx.x over the vectors of a row, blockIdx.y over the rows (a few rows a block once the grid fills the GPU)
static dim3 rows_grid(long long vecs, long long rows) {
  const unsigned x = static_cast<unsigned>((vecs + 255) / 256);
  long long y = (148LL * 64 + x - 1) / x;
  if (y > rows) y = rows;
  if (y > 65535) y = 65535;
  return dim3(x, static_cast<unsigned>(y), 1);
}

}  // namespace mg

extern "C" {

int matgptq_b200_add_rmsnorm(void *x, const void *delta, const void *weight, void *h, int64_t rows, int64_t hidden,
                             float eps, uint32_t flags, void *stream) {
  if (!x || !weight || !h || rows < 0 || hidden <= 0) return MG_ERR_BAD_ARG;
  if (rows == 0) return MG_OK;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const bool vec = hidden % 8 == 0 && hidden <= static_cast<int64_t>(mg::kNormThreads) * 8 * mg::kRowVecs &&
                   (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(weight) |
                    reinterpret_cast<uintptr_t>(h)) % 16 == 0;
  const dim3 grid(static_cast<unsigned>(rows));
  const int hd = static_cast<int>(hidden);
  const bool pdl = (flags & MATGPTQ_B200_FLAG_PDL) != 0;
  if (flags & MATGPTQ_B200_FLAG_BF16) {
    using T = __nv_bfloat16;
    if (vec)
      return mg::launch_helper(mg::add_rmsnorm_vec_kernel<T>, grid, mg::kNormThreads, cs, pdl, static_cast<T *>(x),
                               static_cast<const T *>(delta), static_cast<const T *>(weight), static_cast<T *>(h), hd, eps);
    else
      return mg::launch_helper(mg::add_rmsnorm_kernel<T>, grid, 256, cs, pdl, static_cast<T *>(x), static_cast<const T *>(delta),
                               static_cast<const T *>(weight), static_cast<T *>(h), hd, eps);
  } else {
    using T = __half;
    if (vec)
      return mg::launch_helper(mg::add_rmsnorm_vec_kernel<T>, grid, mg::kNormThreads, cs, pdl, static_cast<T *>(x),
                               static_cast<const T *>(delta), static_cast<const T *>(weight), static_cast<T *>(h), hd, eps);
    else
      return mg::launch_helper(mg::add_rmsnorm_kernel<T>, grid, 256, cs, pdl, static_cast<T *>(x), static_cast<const T *>(delta),
                               static_cast<const T *>(weight), static_cast<T *>(h), hd, eps);
  }
  return cudaGetLastError() == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}

int matgptq_b200_rope_kv(const void *qkv, const int64_t *positions, const float *cos_table, const float *sin_table, void *q_out,
                         void *k_cache, void *v_cache, int64_t batch, int64_t seq, int64_t n_heads, int64_t n_kv_heads,
                         int64_t head_dim, int64_t max_seq, uint32_t flags, void *stream) {
  if (!qkv || !positions || !cos_table || !sin_table || !q_out || !k_cache || !v_cache || head_dim % 2) return MG_ERR_BAD_ARG;
  const long long total = batch * seq * (n_heads + 2 * n_kv_heads) * (head_dim / 2);
  if (total <= 0) return MG_OK;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const long long *pos = reinterpret_cast<const long long *>(positions);
  const bool vec = head_dim % 8 == 0 && batch * seq <= INT32_MAX && n_heads + 2 * n_kv_heads <= (1 << 16) && head_dim <= (1 << 12) &&
                   (reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(cos_table) | reinterpret_cast<uintptr_t>(sin_table) |
                    reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) % 16 == 0;
  const dim3 grid = vec ? mg::rows_grid((n_heads + 2 * n_kv_heads) * (head_dim / 8), batch * seq) : dim3(mg::grid_for(total, 256));
  auto go = [&](auto kernel, auto tag) {
    using T = decltype(tag);
    return mg::launch_helper(kernel, grid, 256, cs, (flags & MATGPTQ_B200_FLAG_PDL) != 0, static_cast<const T *>(qkv), pos, cos_table,
                             sin_table, static_cast<T *>(q_out), static_cast<T *>(k_cache), static_cast<T *>(v_cache),
                             static_cast<int>(batch), static_cast<int>(seq), static_cast<int>(n_heads), static_cast<int>(n_kv_heads),
                             static_cast<int>(head_dim), static_cast<int>(max_seq));
  };
  if (flags & MATGPTQ_B200_FLAG_BF16) {
    using T = __nv_bfloat16;
    return vec ? go(mg::rope_kv_vec_kernel<T>, T{}) : go(mg::rope_kv_kernel<T>, T{});
  }
  using T = __half;
  return vec ? go(mg::rope_kv_vec_kernel<T>, T{}) : go(mg::rope_kv_kernel<T>, T{});
}

int matgptq_b200_argmax(const void *logits, int64_t *out, int64_t rows, int64_t cols, uint32_t flags, void *stream) {
  if (!logits || !out || rows < 0 || cols <= 0 || cols % 8 != 0 || cols > (1 << 30)) return MG_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(logits) & 15u) return MG_ERR_ALIGNMENT;
  if (rows == 0) return MG_OK;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  static_assert(sizeof(long long) == sizeof(int64_t), "int64_t is long long here");
  if (flags & MATGPTQ_B200_FLAG_BF16)
    return mg::launch_helper(mg::argmax_kernel<__nv_bfloat16>, static_cast<unsigned>(rows), 1024, cs, (flags & MATGPTQ_B200_FLAG_PDL) != 0,
        static_cast<const __nv_bfloat16 *>(logits), reinterpret_cast<long long *>(out), static_cast<int>(cols));
  else
    return mg::launch_helper(mg::argmax_kernel<__half>, static_cast<unsigned>(rows), 1024, cs, (flags & MATGPTQ_B200_FLAG_PDL) != 0,
                             static_cast<const __half *>(logits), reinterpret_cast<long long *>(out), static_cast<int>(cols));
  return cudaGetLastError() == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}

int matgptq_b200_causal_mask(const int64_t *positions, void *mask, int64_t seq, int64_t max_seq, uint32_t flags, void *stream) {
  if (!positions || !mask || seq < 0 || seq > INT32_MAX || max_seq <= 0 || max_seq > (1 << 30)) return MG_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(mask) & 15u) return MG_ERR_ALIGNMENT;
  if (seq == 0) return MG_OK;
  const long long *pos = reinterpret_cast<const long long *>(positions);
  const dim3 grid(static_cast<unsigned>((max_seq + 1023) / 1024), static_cast<unsigned>(seq < 4096 ? seq : 4096), 1);
  const auto go = [&](auto kernel, auto tag) {
    using T = decltype(tag);
    return mg::launch_helper(kernel, grid, 128, static_cast<cudaStream_t>(stream), (flags & MATGPTQ_B200_FLAG_PDL) != 0, pos,
                             static_cast<T *>(mask), static_cast<int>(seq), static_cast<int>(max_seq));
  };
  return (flags & MATGPTQ_B200_FLAG_BF16) ? go(mg::causal_mask_kernel<__nv_bfloat16>, __nv_bfloat16{}) : go(mg::causal_mask_kernel<__half>, __half{});
}

int matgptq_b200_silu_mul(const void *gate_up, void *out, int64_t rows, int64_t intermediate, uint32_t flags, void *stream) {
  if (!gate_up || !out || rows < 0 || intermediate <= 0) return MG_ERR_BAD_ARG;
  if (rows == 0) return MG_OK;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const bool vec = intermediate % 8 == 0 && intermediate <= (1 << 24) &&
                   (reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
  const dim3 grid = vec ? mg::rows_grid(intermediate / 8, rows) : dim3(mg::grid_for(rows * intermediate, 256));
  auto go = [&](auto kernel, auto tag) {
    using T = decltype(tag);
    return mg::launch_helper(kernel, grid, 256, cs, (flags & MATGPTQ_B200_FLAG_PDL) != 0, static_cast<const T *>(gate_up),
                             static_cast<T *>(out), static_cast<long long>(rows), static_cast<int>(intermediate));
  };
  if (flags & MATGPTQ_B200_FLAG_BF16) {
    using T = __nv_bfloat16;
    return vec ? go(mg::silu_mul_vec_kernel<T>, T{}) : go(mg::silu_mul_kernel<T>, T{});
  }
  using T = __half;
  return vec ? go(mg::silu_mul_vec_kernel<T>, T{}) : go(mg::silu_mul_kernel<T>, T{});
}

}  // extern "C"
