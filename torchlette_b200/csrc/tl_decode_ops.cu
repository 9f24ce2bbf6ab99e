// The ops either side of the projections in one Qwen3 decode step, so that a step can run on this
// backend end to end (packages/qwen3-browser/src/model.ts:220-420): RMSNorm (hidden-wide and the
// per-head q / k norm) and rotary embedding.  (Attention is tl_attention.cu; the residual adds,
// silu(gate) * up and the cache append are tl_binary_op, the multiply epilogue and tl_copy2d.)  All
// small next to the projections: one pass each, f32 arithmetic, any of f32 / f16 / bf16 storage.
//
//   rmsnorm    y = x * rsqrt(mean(x^2) + eps) * w            src/ops/semantic/composite.ts:156-170
//   rope       half-split (GPT-NeoX / Llama) rotation         src/backend/webgpu/rope-kernel.ts:1-93
#include <algorithm>

#include "tl_common.cuh"

namespace {

__device__ __forceinline__ float ld_f32(const void* p, int dtype, int64_t i) {
  if (dtype == TL_F32) return reinterpret_cast<const float*>(p)[i];
  if (dtype == TL_F16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Rows of whole 8-element vectors: the row is read once and held in registers, a vector (or CH of them) a thread, so a
// row costs one round trip to memory and one reduction.
template <typename T> __device__ __forceinline__ void load8(const T* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const T* e = reinterpret_cast<const T*>(&u);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = DT<T>::to_f32(e[i]);
}
template <> __device__ __forceinline__ void load8<float>(const float* p, float (&v)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <typename T> __device__ __forceinline__ void store8(T* p, const float (&v)[8]) {
  T e[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) e[i] = DT<T>::from_f32(v[i]);
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(e);
}
template <> __device__ __forceinline__ void store8<float>(float* p, const float (&v)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void load8_any(const void* p, int dtype, int64_t i, float (&v)[8]) {
  if (dtype == TL_F32) load8(reinterpret_cast<const float*>(p) + i, v);
  else if (dtype == TL_F16) load8(reinterpret_cast<const __half*>(p) + i, v);
  else load8(reinterpret_cast<const __nv_bfloat16*>(p) + i, v);
}
// blockDim.x threads per row, blockDim.y rows per CTA (more than one only where a row is one warp's)
template <int CH>
__global__ void __launch_bounds__(1024) rmsnorm_vec_kernel(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                                                           int64_t rows, int cols, float eps) {
  __shared__ float part[32];
  tl_pdl_wait();
  const int64_t row = int64_t(blockIdx.x) * blockDim.y + threadIdx.y;
  const bool here = row < rows;
  const int64_t base = row * cols;
  float v[CH][8], g0[8], ss = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * int(blockDim.x) + int(threadIdx.x)) * 8;
    if (here && i < cols) {
      load8_any(x, x_dtype, base + i, v[c]);
      if (CH == 1) load8_any(w, w_dtype, i, g0);  // on its way during the reduction
#pragma unroll
      for (int e = 0; e < 8; ++e) ss = fmaf(v[c][e], v[c][e], ss);
    }
  }
  ss = warp_sum(ss);
  if (blockDim.x > 32) {
    const int warps = int(blockDim.x) >> 5;
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = warp_sum(int(threadIdx.x & 31) < warps ? part[threadIdx.x & 31] : 0.f);
  }
  const float inv = rsqrtf(ss / float(cols) + eps);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * int(blockDim.x) + int(threadIdx.x)) * 8;
    if (here && i < cols) {
      float g[8];
      if (CH > 1) load8_any(w, w_dtype, i, g);
#pragma unroll
      for (int e = 0; e < 8; ++e) g[e] = v[c][e] * inv * (CH == 1 ? g0[e] : g[e]);
      if (out_dtype == TL_F32) store8(reinterpret_cast<float*>(out) + base + i, g);
      else if (out_dtype == TL_F16) store8(reinterpret_cast<__half*>(out) + base + i, g);
      else store8(reinterpret_cast<__nv_bfloat16*>(out) + base + i, g);
    }
  }
}
// any row: one CTA per row (cols up to any size), 128 threads
__global__ void __launch_bounds__(128) rmsnorm_kernel(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                                                      int64_t rows, int cols, float eps) {
  __shared__ float part[4];
  tl_pdl_wait();
  const int64_t row = blockIdx.x;
  if (row >= rows) return;
  const int64_t base = row * cols;
  float ss = 0.f;
  for (int c = threadIdx.x; c < cols; c += 128) {
    const float v = ld_f32(x, x_dtype, base + c);
    ss = fmaf(v, v, ss);
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  const float total = part[0] + part[1] + part[2] + part[3];
  const float inv = rsqrtf(total / float(cols) + eps);
  for (int c = threadIdx.x; c < cols; c += 128) {
    const float v = ld_f32(x, x_dtype, base + c);
    tl_store_out(out, out_dtype, base + c, v * inv * ld_f32(w, w_dtype, c));
  }
}

// one thread per output element of qk [outer, S, D]
__global__ void __launch_bounds__(256) rope_kernel(const void* qk, int dtype, const float* cos_t, const float* sin_t, void* out,
                                                   int64_t total, int seq_len, int head_dim, float sin_scale, int64_t cos_offset,
                                                   int64_t sin_offset) {
  tl_pdl_wait();
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int half = head_dim >> 1;
  for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    const int d = int(idx % head_dim);
    const int s = int((idx / head_dim) % seq_len);
    const bool second = d >= half;
    const int dh = second ? d - half : d;
    const float qi = ld_f32(qk, dtype, idx), qp = ld_f32(qk, dtype, second ? idx - half : idx + half);
    const float c = cos_t[cos_offset + int64_t(s) * half + dh];
    const float sn = sin_t[sin_offset + int64_t(s) * half + dh] * sin_scale;
    tl_store_out(out, dtype, idx, qi * c + (second ? 1.f : -1.f) * qp * sn);
  }
}

}  // namespace

extern "C" {

int32_t tl_rmsnorm(tl_ctx* ctx, const void* x, int32_t x_dtype, const void* weight, int32_t weight_dtype, void* out, int32_t out_dtype,
                   int64_t rows, int64_t cols, float eps) {
  TL_CHECK_CTX(ctx);
  if (rows < 0 || cols < 1 || cols > INT32_MAX || (rows > 0 && (!x || !weight || !out)))
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_rmsnorm: null pointer or bad shape");
  if (!tl_dtype_valid(x_dtype) || !tl_dtype_valid(weight_dtype) || !tl_dtype_valid(out_dtype))
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_rmsnorm: unknown dtype");
  if (rows == 0) return TL_OK;
  if (rows > INT32_MAX) return tl_set_error(ctx, TL_ERR_UNSUPPORTED, "tl_rmsnorm: too many rows for one launch");
  DeviceGuard guard(ctx->device);
  const bool vec = cols % 8 == 0 && cols <= 8 * 4 * 1024 &&
                   ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (vec) {
    // One vector a thread as far as a CTA's 1024 threads go (2 rows x 4096: 18.7 us with 128 threads and scalar loads);
    // short rows (per-head norms) share a CTA once there are enough of them to fill the chip.
    const int vecs = int(cols / 8), threads = std::min(1024, (vecs + 31) / 32 * 32);
    const int per_cta = threads == 32 && rows >= 8 * int64_t(ctx->sm_count) ? 8 : 1;
    const dim3 block(threads, per_cta);
    const unsigned grid = unsigned((rows + per_cta - 1) / per_cta);
    TL_CUDA(ctx, tl_launch_waiting(vecs <= 1024 ? rmsnorm_vec_kernel<1> : rmsnorm_vec_kernel<4>, dim3(grid), block, ctx->stream, x, x_dtype, weight,
                                   weight_dtype, out, out_dtype, rows, cols, eps));
  } else {
    TL_CUDA(ctx, tl_launch_waiting(rmsnorm_kernel, dim3(unsigned(rows)), dim3(128), ctx->stream, x, x_dtype, weight, weight_dtype, out, out_dtype, rows,
                                   cols, eps));
  }
  ctx->counters[TL_COUNTER_KERNEL_LAUNCHES]++;
  tl_wrote(ctx, out, rows * cols * tl_dtype_size(out_dtype), true);
  return TL_OK;
}

int32_t tl_rope(tl_ctx* ctx, const void* qk, int32_t dtype, const float* cos_table, const float* sin_table, void* out, int64_t outer,
                int64_t seq_len, int64_t head_dim, float sin_scale, int64_t cos_offset, int64_t sin_offset) {
  TL_CHECK_CTX(ctx);
  if (outer < 0 || seq_len < 1 || head_dim < 2 || seq_len > INT32_MAX || head_dim > INT32_MAX || cos_offset < 0 || sin_offset < 0)
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_rope: bad shape");
  if (head_dim % 2 != 0) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "applyRoPE: headDim must be even, got %lld", (long long)head_dim);
  if (!tl_dtype_valid(dtype)) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_rope: unknown dtype");
  const int64_t total = outer * seq_len * head_dim;
  if (total == 0) return TL_OK;
  if (!qk || !cos_table || !sin_table || !out || qk == out)
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_rope: null or aliased pointers (an element reads its partner: not in place)");
  DeviceGuard guard(ctx->device);
  const int grid = int(std::min<int64_t>((total + 255) / 256, int64_t(ctx->sm_count) * 8));
  TL_CUDA(ctx, tl_launch_waiting(rope_kernel, dim3(unsigned(grid)), dim3(256), ctx->stream, qk, dtype, cos_table, sin_table, out, total, seq_len,
                                 head_dim, sin_scale, cos_offset, sin_offset));
  ctx->counters[TL_COUNTER_KERNEL_LAUNCHES]++;
  tl_wrote(ctx, out, total * tl_dtype_size(dtype), true);
  return TL_OK;
}

}  // extern "C"
