// Shared by the attention kernels (tl_attention.cu, tl_attention_tc.cu): one query row by one warp, over exactly the
// keys that row sees, and the 16-bit split of f32 probabilities for the tensor cores.
#pragma once

#include <cfloat>

#include "tl_common.cuh"

#ifdef __CUDACC__
constexpr float kLog2e = 1.4426950408889634f;

// The fast kernels multiply whole tiles and split probabilities into terms: a key hidden from a row (or past the end) has
// probability zero there, and zero times an infinite or NaN value would still poison the row; a visible infinite value meets
// a low term that is zero or negative, and infinity becomes NaN.  A row whose result is not finite is therefore done again
// here, over exactly the keys that it sees and with whole probabilities: two passes, f32, a lane per D / 32 dimensions.  Only
// the dimensions from 32 * first on, 32 * count of them, are stored.
template <typename AT, int D>
__device__ __noinline__ void attention_row_warp(const AT* q, const AT* k, const AT* v, AT* out, int keys, float scale, const float* mask,
                                                int first, int count) {
  constexpr int V = D / 32;
  const int lane = threadIdx.x & 31;
  float qf[V], o[V], mx = -FLT_MAX, sum = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) { qf[i] = DT<AT>::to_f32(q[lane + 32 * i]); o[i] = 0.f; }
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll 1
    for (int j = 0; j < keys; ++j) {
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < V; ++i) dot = fmaf(qf[i], DT<AT>::to_f32(k[int64_t(j) * D + lane + 32 * i]), dot);
#pragma unroll
      for (int w = 16; w > 0; w >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, w);
      dot = dot * scale + (mask ? mask[j] : 0.f);
      if (pass == 0) {
        mx = fmaxf(mx, dot);
      } else {
        const float e = expf(dot - mx);
        sum += e;
#pragma unroll
        for (int i = 0; i < V; ++i) o[i] = fmaf(e, DT<AT>::to_f32(v[int64_t(j) * D + lane + 32 * i]), o[i]);
      }
    }
  }
  const float inv = 1.f / sum;
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (i >= first && i < first + count) out[lane + 32 * i] = DT<AT>::from_f32(o[i] * inv);
}

// Two f32 operations in one instruction
__device__ __forceinline__ float2 fma_x2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)), "l"(reinterpret_cast<const uint64_t&>(c)));
  return d;
}
__device__ __forceinline__ float2 add_x2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
  return d;
}

// Two probabilities as 16-bit terms whose sum carries nearly or quite all 24 bits of each: p rounded, then what is left
// rounded, then again.  Two f16 terms (11 bits each and the sign of the second) carry 23, three bf16 ones (8 bits) all.
template <typename AT> struct ProbSplit;
template <> struct ProbSplit<__half> {
  static constexpr int kTerms = 2;
  __device__ static __forceinline__ void split(float2 p, uint32_t (&t)[2]) {
    const __half2 hi = __floats2half2_rn(p.x, p.y);
    const float2 rest = fma_x2(__half22float2(hi), make_float2(-1.f, -1.f), p);  // exact
    const __half2 lo = __floats2half2_rn(rest.x, rest.y);
    t[0] = *reinterpret_cast<const uint32_t*>(&hi);
    t[1] = *reinterpret_cast<const uint32_t*>(&lo);
  }
};
template <> struct ProbSplit<__nv_bfloat16> {
  static constexpr int kTerms = 3;
  __device__ static __forceinline__ void split(float2 p, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(p.x, p.y);
      t[i] = *reinterpret_cast<const uint32_t*>(&h);
      p = fma_x2(make_float2(__uint_as_float(t[i] << 16), __uint_as_float(t[i] & 0xffff0000u)), make_float2(-1.f, -1.f), p);  // exact
    }
  }
};
#endif  // __CUDACC__
