// Scaled dot-product attention over (a prefix of) a KV cache with grouped query heads
// (packages/qwen3-browser/src/model.ts:284-318): softmax(q k^T * scale + mask) v, decode (one query
// position per sequence) and the causal form for several.  q is [B, H, S, D], the caches are
// [B, kvH, capacity, D], the output is [B, S, H, D] -- the permute in front of o_proj folded into the store.
//
//   decode   up to 16 query rows per KV head (query positions x query heads that share it): attn_decode_mma_kernel
//            (f16 / bf16) and attn_decode_f32_kernel.  Bound: HBM (the cache is read once), by the loads that twelve warps
//            an SM have in flight (DRAM pipe 54 % busy, long scoreboard the first stall).  8 sequences x 8 KV heads x
//            4000 keys x 128 f16 (131 MB): 27.1 us = 4.8 TB/s, about 5 us of it launch, first loads and merging (964 us
//            one CTA per query head, which read the cache once per query head along a serial chain); 2 x 8 x 700: 6.9
//            us (171).
//   prefill  more query rows, f16 / bf16 without a mask tensor: tl_attention_tc.cu.
//   general  everything else: attention_kernel, one CTA per query row.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include <cooperative_groups.h>

#include "tl_attention.cuh"
#include "tl_mma_frag.cuh"

namespace cg = cooperative_groups;

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

// ---------------------------------------------------------------------------
// General form: one CTA per (batch, query head, query position); 4 warps; scores for the visible positions
// live in shared memory.  With `causal`, query s sees the keys up to position kv_len - q_len + s (the mask the
// reference builds with triu, model.ts:300-307).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) attention_kernel(const void* q, const void* kc, const void* vc, void* out, int dtype,
                                                        int n_heads, int n_kv_heads, int q_len, int head_dim, int kv_len_total,
                                                        int64_t kv_capacity, float scale, const float* mask, int causal) {
  extern __shared__ float scores[];  // [kv_len]
  __shared__ float red[4];
  const int sq = blockIdx.x % q_len;
  const int bh = blockIdx.x / q_len;
  const int b = bh / n_heads, h = bh - b * n_heads;
  const int kvh = h / (n_heads / n_kv_heads);  // repeat_kv order: head h reads kv head h / n_rep
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_len = causal ? kv_len_total - q_len + sq + 1 : kv_len_total;
  const int64_t q_base = ((int64_t(b) * n_heads + h) * q_len + sq) * head_dim;
  const int64_t o_base = ((int64_t(b) * q_len + sq) * n_heads + h) * head_dim;
  const int64_t kv_base = (int64_t(b) * n_kv_heads + kvh) * kv_capacity * head_dim;
  // scores: a warp per key position, lanes over the head dimension
  float wmax = -FLT_MAX;
  for (int j = warp; j < kv_len; j += 4) {
    float dot = 0.f;
    for (int d = lane; d < head_dim; d += 32) dot = fmaf(ld_f32(q, dtype, q_base + d), ld_f32(kc, dtype, kv_base + int64_t(j) * head_dim + d), dot);
    dot = warp_sum(dot) * scale + (mask ? mask[int64_t(sq) * kv_len_total + j] : 0.f);
    if (lane == 0) scores[j] = dot;
    wmax = fmaxf(wmax, dot);
  }
  if (lane == 0) red[warp] = wmax;
  __syncthreads();
  const float mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  __syncthreads();
  float sum = 0.f;
  for (int j = threadIdx.x; j < kv_len; j += 128) {
    const float e = expf(scores[j] - mx);
    scores[j] = e;
    sum += e;
  }
  sum = warp_sum(sum);
  if (lane == 0) red[warp] = sum;
  __syncthreads();
  const float inv = 1.f / (red[0] + red[1] + red[2] + red[3]);
  // output: thread d accumulates over all positions (coalesced over d for every position)
  for (int d = threadIdx.x; d < head_dim; d += 128) {
    float acc = 0.f;
    for (int j = 0; j < kv_len; ++j) acc = fmaf(scores[j], ld_f32(vc, dtype, kv_base + int64_t(j) * head_dim + d), acc);
    tl_store_out(out, dtype, o_base + d, acc * inv);
  }
}

// ---------------------------------------------------------------------------
// Decode.  A cluster of `splits` CTAs owns one (batch, KV head): each CTA takes a contiguous range of 16-key
// tiles, its four warps interleaved over them, every warp with its own online softmax (running maximum, sum
// and output in registers); the warps' partials are merged in shared memory, the CTAs' through distributed
// shared memory, so there is no scratch, no second launch and no atomic.
// ---------------------------------------------------------------------------
struct DecodeArgs {
  const void* q;
  const void* k;
  const void* v;
  void* out;
  int32_t n_heads, n_kv_heads, rep, q_len, rows, kv_len, splits;  // rows = rep * q_len: query rows of one KV head
  int64_t capacity;
  float scale;
  const float* mask;  // [q_len, kv_len] or null
  int32_t causal;
};

// Partials of this CTA's warps -> the cluster's result.  sm: [warps][R] maxima, [warps][R] sums, [warps][R][D]
// outputs, then the CTA's own merged [R], [R], [R][D].
template <typename AT, int D, int R, int WARPS>
__device__ __forceinline__ void decode_merge(const DecodeArgs& p, float* sm, int b, int kvh) {
  float* wm = sm;
  float* wl = wm + WARPS * R;
  float* wo = wl + WARPS * R;
  float* cm = wo + WARPS * R * D;
  float* cl = cm + R;
  float* co = cl + R;
  __syncthreads();
  for (int e = threadIdx.x; e < p.rows * D; e += WARPS * 32) {
    const int r = e / D, d = e - r * D;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) m = fmaxf(m, wm[w * R + r]);
    float l = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float mw = wm[w * R + r];
      const float f = mw == -INFINITY ? 0.f : exp2f((mw - m) * kLog2e);
      l = fmaf(wl[w * R + r], f, l);
      o = fmaf(wo[(w * R + r) * D + d], f, o);
    }
    co[r * D + d] = o;
    if (d == 0) { cm[r] = m; cl[r] = l; }
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (p.splits > 1) cluster.sync();
  else __syncthreads();
  const int rank = p.splits > 1 ? int(cluster.block_rank()) : 0;
  const int total = p.rows * D, per = ((total + p.splits - 1) / p.splits + 31) & ~31;  // a warp's 32 values are one row's
  for (int e = rank * per + threadIdx.x; e < min(total, (rank + 1) * per); e += WARPS * 32) {
    const int r = e / D, d = e - r * D;
    float m = -INFINITY;
    for (int s = 0; s < p.splits; ++s) m = fmaxf(m, p.splits > 1 ? cluster.map_shared_rank(cm, s)[r] : cm[r]);
    float l = 0.f, o = 0.f;
    for (int s = 0; s < p.splits; ++s) {
      const float* rm = p.splits > 1 ? cluster.map_shared_rank(cm, s) : cm;
      const float* rl = p.splits > 1 ? cluster.map_shared_rank(cl, s) : cl;
      const float* ro = p.splits > 1 ? cluster.map_shared_rank(co, s) : co;
      const float ms = rm[r];
      const float f = ms == -INFINITY ? 0.f : exp2f((ms - m) * kLog2e);
      l = fmaf(rl[r], f, l);
      o = fmaf(ro[r * D + d], f, o);
    }
    const int qi = r / p.rep, h = kvh * p.rep + (r - qi * p.rep);
    const int64_t at = ((int64_t(b) * p.q_len + qi) * p.n_heads + h) * D;
    const float v = o / l;
    // Not finite: a probability times an infinite value went through the split terms (or a key past the end, clamped to the
    // last one, met it with probability zero), or it is what the row sees.  The redo tells them apart.
    if (__any_sync(0xffffffffu, !isfinite(v))) {
      const int64_t kv = (int64_t(b) * p.n_kv_heads + kvh) * p.capacity * D;
      attention_row_warp<AT, D>(reinterpret_cast<const AT*>(p.q) + ((int64_t(b) * p.n_heads + h) * p.q_len + qi) * D,
                                reinterpret_cast<const AT*>(p.k) + kv, reinterpret_cast<const AT*>(p.v) + kv,
                                reinterpret_cast<AT*>(p.out) + at, p.causal ? p.kv_len - p.q_len + qi + 1 : p.kv_len, p.scale,
                                p.mask ? p.mask + int64_t(qi) * p.kv_len : nullptr, d >> 5, 1);
    } else {
      reinterpret_cast<AT*>(p.out)[at + d] = DT<AT>::from_f32(v);
    }
  }
  if (p.splits > 1) cluster.sync();  // no CTA leaves while another reads its shared memory
}
template <int D, int R, int WARPS> constexpr size_t decode_smem_bytes() {
  return sizeof(float) * (size_t(WARPS) + 1) * R * (D + 2);
}

// Probabilities are held times 2^10 in f16: the low term of their split stays clear of f16's subnormals.
template <typename AT> constexpr float kProbBias = 0.f;
template <> constexpr float kProbBias<__half> = 10.f;

__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// f16 / bf16.  Everything between the cache and the output stays in registers: the K rows of a 16-key tile are
// the A operand of S^T = K q^T (16-byte loads of a lane feed two MMAs, the same permutation of d on both
// operands), the probabilities are transposed in the register file (movmatrix) into the B operand of
// O^T = V^T p, and V^T is put together from 16-byte row loads by byte permutes.  Tensor cores do the products
// because the CUDA cores could not keep up with HBM: four query heads per KV head are 8 FMA per cache byte pair.
// NT = 1: up to 8 query rows, NT = 2: up to 16.
template <typename AT, int D, int NT>
__global__ void __launch_bounds__(128, NT == 1 ? 3 : 2) attn_decode_mma_kernel(DecodeArgs p) {
  constexpr int R = 8 * NT, KC = D / 32, VH = D / 64, TERMS = ProbSplit<AT>::kTerms;
  extern __shared__ float decode_sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int split = int(blockIdx.x) % p.splits, bkv = int(blockIdx.x) / p.splits;
  const int b = bkv / p.n_kv_heads, kvh = bkv - b * p.n_kv_heads;
  const AT* kb = reinterpret_cast<const AT*>(p.k) + int64_t(bkv) * p.capacity * D + 8 * t;
  const AT* vb = reinterpret_cast<const AT*>(p.v) + int64_t(bkv) * p.capacity * D + 8 * g;
  const int tiles = (p.kv_len + 15) >> 4;
  const int tile_end = int(int64_t(tiles) * (split + 1) / p.splits);
  int tile = int(int64_t(tiles) * split / p.splits) + warp;
  const int last = p.kv_len - 1;

  uint4 kf[2][KC];
  auto load_k = [&](int tl) {
    const AT* r0 = kb + int64_t(min(tl * 16 + g, last)) * D;
    const AT* r1 = kb + int64_t(min(tl * 16 + g + 8, last)) * D;
#pragma unroll
    for (int i = 0; i < KC; ++i) {
      kf[0][i] = __ldg(reinterpret_cast<const uint4*>(r0 + 32 * i));
      kf[1][i] = __ldg(reinterpret_cast<const uint4*>(r1 + 32 * i));
    }
  };
  if (tile < tile_end) load_k(tile);

  uint4 qf[NT][KC];
  int bound[NT][2];         // visible keys of the lane's two query rows
  const float* mrow[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int rq = min(nt * 8 + g, p.rows - 1), qi = rq / p.rep, h = kvh * p.rep + (rq - qi * p.rep);
    const AT* qp = reinterpret_cast<const AT*>(p.q) + ((int64_t(b) * p.n_heads + h) * p.q_len + qi) * D + 8 * t;
#pragma unroll
    for (int i = 0; i < KC; ++i) qf[nt][i] = __ldg(reinterpret_cast<const uint4*>(qp + 32 * i));
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int qc = min(nt * 8 + 2 * t + c, p.rows - 1) / p.rep;
      bound[nt][c] = p.causal ? p.kv_len - p.q_len + qc + 1 : p.kv_len;
      mrow[nt][c] = p.mask ? p.mask + int64_t(qc) * p.kv_len : nullptr;
    }
  }
  float o[NT][D / 16][4], m[NT][2], l[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int j = 0; j < D / 16; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[nt][j][e] = 0.f;
    m[nt][0] = m[nt][1] = -INFINITY;
    l[nt][0] = l[nt][1] = 0.f;
  }

  while (tile < tile_end) {
    const int key0 = tile * 16;
    uint4 vf[4][VH];  // keys 2t, 2t+1, 2t+8, 2t+9
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const AT* r = vb + int64_t(min(key0 + 2 * t + (i & 1) + (i >> 1) * 8, last)) * D;
#pragma unroll
      for (int h = 0; h < VH; ++h) vf[i][h] = __ldg(reinterpret_cast<const uint4*>(r + 64 * h));
    }
    float s[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        MmaOps<AT>::mma_free(s0, kf[0][i].x, kf[1][i].x, kf[0][i].y, kf[1][i].y, qf[nt][i].x, qf[nt][i].y);
        MmaOps<AT>::mma_free(s1, kf[0][i].z, kf[1][i].z, kf[0][i].w, kf[1][i].w, qf[nt][i].z, qf[nt][i].w);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) s[nt][e] = s0[e] + s1[e];
    }
    tile += 4;
    if (tile < tile_end) load_k(tile);  // the next tile's keys are in flight during the softmax and the second product
    uint32_t pf[NT][TERMS][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {  // element e: key g + 8 * (e >> 1), query row 2t + (e & 1)
        const int key = key0 + g + 8 * (e >> 1);
        // natural units up to the difference with the maximum: a mask may hold the lowest f32, which no factor fits
        const float x = fmaf(s[nt][e], p.scale, p.mask ? mrow[nt][e & 1][min(key, last)] : 0.f);
        s[nt][e] = key < bound[nt][e & 1] ? x : -INFINITY;
      }
      float nm[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float v = fmaxf(s[nt][c], s[nt][c + 2]);
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 8));
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
        nm[c] = fmaxf(m[nt][c], v);
      }
      if (__any_sync(0xffffffffu, nm[0] != m[nt][0] || nm[1] != m[nt][1])) {
        float f[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          f[c] = nm[c] == m[nt][c] ? 1.f : exp2f((m[nt][c] - nm[c]) * kLog2e);  // first keys: exp2(-inf) = 0 on zeros
          l[nt][c] *= f[c];
          m[nt][c] = nm[c];
        }
#pragma unroll
        for (int j = 0; j < D / 16; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[nt][j][e] *= f[e & 1];
      }
      float pr[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float mm = m[nt][e & 1];
        pr[e] = mm == -INFINITY ? 0.f : exp2f(fmaf(s[nt][e] - mm, kLog2e, kProbBias<AT>));  // no key visible yet: nothing to add
        l[nt][e & 1] += pr[e];
      }
      uint32_t a[TERMS], c[TERMS];
      ProbSplit<AT>::split(make_float2(pr[0], pr[1]), a);
      ProbSplit<AT>::split(make_float2(pr[2], pr[3]), c);
#pragma unroll
      for (int i = 0; i < TERMS; ++i) {
        pf[nt][i][0] = transpose8x8(a[i]);
        pf[nt][i][1] = transpose8x8(c[i]);
      }
    }
#pragma unroll
    for (int h = 0; h < VH; ++h) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {  // d = 64 h + 8 g + 2 e (rows 0-7 of the tile) and + 1 (rows 8-15)
        const uint32_t w0 = (&vf[0][h].x)[e], w1 = (&vf[1][h].x)[e], w2 = (&vf[2][h].x)[e], w3 = (&vf[3][h].x)[e];
        const uint32_t a0 = __byte_perm(w0, w1, 0x5410), a1 = __byte_perm(w0, w1, 0x7632);
        const uint32_t a2 = __byte_perm(w2, w3, 0x5410), a3 = __byte_perm(w2, w3, 0x7632);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int i = 0; i < TERMS; ++i) MmaOps<AT>::mma_free(o[nt][h * 4 + e], a0, a1, a2, a3, pf[nt][i][0], pf[nt][i][1]);
      }
    }
  }

  float* wm = decode_sm;
  float* wl = wm + 4 * R;
  float* wo = wl + 4 * R;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float v = l[nt][c];
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      const int r = nt * 8 + 2 * t + c;
      if (g == 0) { wm[warp * R + r] = m[nt][c]; wl[warp * R + r] = v; }
#pragma unroll
      for (int h = 0; h < VH; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          *reinterpret_cast<float2*>(&wo[(warp * R + r) * D + 64 * h + 8 * g + 2 * e]) = make_float2(o[nt][h * 4 + e][c], o[nt][h * 4 + e][c + 2]);
    }
  }
  decode_merge<AT, D, R, 4>(p, decode_sm, b, kvh);
}

template <int V> __device__ __forceinline__ void load_vec(const float* p, float (&x)[V]) {
  if (V == 4) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    x[0] = v.x; x[1] = v.y; x[V - 2] = v.z; x[V - 1] = v.w;
  } else {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    x[0] = v.x; x[V - 1] = v.y;
  }
}

// f32.  The same split; a lane owns D / 32 dimensions of every key and of all R query rows, four keys at a time.
template <int D, int R>
__global__ void __launch_bounds__(128) attn_decode_f32_kernel(DecodeArgs p) {
  constexpr int V = D / 32, KEYS = R <= 4 ? 4 : 2;
  extern __shared__ float decode_sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = int(blockIdx.x) % p.splits, bkv = int(blockIdx.x) / p.splits;
  const int b = bkv / p.n_kv_heads, kvh = bkv - b * p.n_kv_heads;
  const float* kb = reinterpret_cast<const float*>(p.k) + int64_t(bkv) * p.capacity * D + V * lane;
  const float* vb = reinterpret_cast<const float*>(p.v) + int64_t(bkv) * p.capacity * D + V * lane;
  float q[R][V], o[R][V], m[R], l[R];
  int bound[R];
  const float* mrow[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int rq = min(r, p.rows - 1), qi = rq / p.rep, h = kvh * p.rep + (rq - qi * p.rep);
    const float* qp = reinterpret_cast<const float*>(p.q) + ((int64_t(b) * p.n_heads + h) * p.q_len + qi) * D + V * lane;
    load_vec<V>(qp, q[r]);
#pragma unroll
    for (int i = 0; i < V; ++i) o[r][i] = 0.f;
    m[r] = -INFINITY;
    l[r] = 0.f;
    bound[r] = p.causal ? p.kv_len - p.q_len + qi + 1 : p.kv_len;
    mrow[r] = p.mask ? p.mask + int64_t(qi) * p.kv_len : nullptr;
  }
  const int tiles = (p.kv_len + KEYS - 1) / KEYS, last = p.kv_len - 1;
  const int tile_end = int(int64_t(tiles) * (split + 1) / p.splits);
  for (int tile = int(int64_t(tiles) * split / p.splits) + warp; tile < tile_end; tile += 4) {
    float kf[KEYS][V], vf[KEYS][V];
#pragma unroll
    for (int j = 0; j < KEYS; ++j) {
      const int64_t at = int64_t(min(tile * KEYS + j, last)) * D;
      load_vec<V>(kb + at, kf[j]);
      load_vec<V>(vb + at, vf[j]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float s[KEYS], nm = m[r];
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        float x = 0.f;
#pragma unroll
        for (int i = 0; i < V; ++i) x = fmaf(q[r][i], kf[j][i], x);
        const int key = tile * KEYS + j;
        x = fmaf(warp_sum(x), p.scale, p.mask ? mrow[r][min(key, last)] : 0.f);
        s[j] = key < bound[r] ? x : -INFINITY;
        nm = fmaxf(nm, s[j]);
      }
      if (nm != -INFINITY) {
        const float f = exp2f((m[r] - nm) * kLog2e);
        m[r] = nm;
        l[r] *= f;
#pragma unroll
        for (int i = 0; i < V; ++i) o[r][i] *= f;
#pragma unroll
        for (int j = 0; j < KEYS; ++j) {
          const float e = exp2f((s[j] - nm) * kLog2e);
          l[r] += e;
#pragma unroll
          for (int i = 0; i < V; ++i) o[r][i] = fmaf(e, vf[j][i], o[r][i]);
        }
      }
    }
  }
  float* wm = decode_sm;
  float* wl = wm + 4 * R;
  float* wo = wl + 4 * R;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (lane == 0) { wm[warp * R + r] = m[r]; wl[warp * R + r] = l[r]; }
#pragma unroll
    for (int i = 0; i < V; ++i) wo[(warp * R + r) * D + V * lane + i] = o[r][i];
  }
  decode_merge<float, D, R, 4>(p, decode_sm, b, kvh);
}

template <typename K>
cudaError_t launch_decode(K kernel, tl_ctx* ctx, const DecodeArgs& p, int64_t groups, size_t smem) {
  if (p.splits > 8) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(groups * p.splits));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(p.splits);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <typename AT, int D>
cudaError_t launch_decode_mma(tl_ctx* ctx, const DecodeArgs& p, int64_t groups) {
  return p.rows <= 8 ? launch_decode(attn_decode_mma_kernel<AT, D, 1>, ctx, p, groups, decode_smem_bytes<D, 8, 4>())
                     : launch_decode(attn_decode_mma_kernel<AT, D, 2>, ctx, p, groups, decode_smem_bytes<D, 16, 4>());
}
template <int D>
cudaError_t launch_decode_f32(tl_ctx* ctx, const DecodeArgs& p, int64_t groups) {
  if (p.rows == 1) return launch_decode(attn_decode_f32_kernel<D, 1>, ctx, p, groups, decode_smem_bytes<D, 1, 4>());
  if (p.rows == 2) return launch_decode(attn_decode_f32_kernel<D, 2>, ctx, p, groups, decode_smem_bytes<D, 2, 4>());
  if (p.rows <= 4) return launch_decode(attn_decode_f32_kernel<D, 4>, ctx, p, groups, decode_smem_bytes<D, 4, 4>());
  return launch_decode(attn_decode_f32_kernel<D, 8>, ctx, p, groups, decode_smem_bytes<D, 8, 4>());
}

}  // namespace

extern "C" {

int32_t tl_attention(tl_ctx* ctx, const void* q, const void* k_cache, const void* v_cache, void* out, int32_t dtype, int64_t batch,
                     int64_t n_heads, int64_t n_kv_heads, int64_t q_len, int64_t head_dim, int64_t kv_len, int64_t kv_capacity, float scale,
                     const float* mask, int32_t causal) {
  TL_CHECK_CTX(ctx);
  if (batch < 0 || n_heads < 1 || n_kv_heads < 1 || n_heads % n_kv_heads != 0 || head_dim < 1 || q_len < 1 || kv_len < q_len ||
      kv_capacity < kv_len)
    return tl_set_error(ctx, TL_ERR_INVALID_ARG,
                        "tl_attention: bad shape (heads %lld, kv heads %lld, q_len %lld, kv_len %lld, capacity %lld)", (long long)n_heads,
                        (long long)n_kv_heads, (long long)q_len, (long long)kv_len, (long long)kv_capacity);
  if (!tl_dtype_valid(dtype)) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_attention: unknown dtype");
  if (batch == 0) return TL_OK;
  if (!q || !k_cache || !v_cache || !out) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_attention: null pointer");
  const size_t smem = size_t(kv_len) * sizeof(float);
  if (smem > 200 * 1024 || batch * n_heads * q_len > INT32_MAX || head_dim > 1024)
    return tl_set_error(ctx, TL_ERR_UNSUPPORTED, "tl_attention: kv_len %lld exceeds the %d positions one launch keeps in shared memory",
                        (long long)kv_len, 200 * 1024 / 4);
  DeviceGuard guard(ctx->device);
  const int64_t rep = n_heads / n_kv_heads, rows = rep * q_len, groups = batch * n_kv_heads;
  const bool aligned = !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15);
  cudaError_t e = cudaSuccess;
  if ((head_dim == 64 || head_dim == 128) && aligned && rows <= (dtype == TL_F32 ? 8 : 16)) {
    DecodeArgs p{};
    p.q = q; p.k = k_cache; p.v = v_cache; p.out = out;
    p.n_heads = int32_t(n_heads); p.n_kv_heads = int32_t(n_kv_heads); p.rep = int32_t(rep); p.q_len = int32_t(q_len);
    p.rows = int32_t(rows); p.kv_len = int32_t(kv_len); p.capacity = kv_capacity;
    p.scale = scale; p.mask = mask; p.causal = causal ? 1 : 0;
    // Splits (CTAs of a cluster) per KV head: double them while there are fewer than two CTAs per SM and a warp has
    // more than two 16-key tiles; above 8, which needs a non-portable cluster, only if that leaves SMs idle (1
    // sequence, 8 KV heads, 4000 keys: 10.3 us with 8, 9.7 with 16).  Then keep the launch in one wave of three
    // resident CTAs per SM (two for 9 to 16 rows, by registers): 64 heads x 4000 keys measured 27.1 us with 6
    // splits, 38 with 8 (a second wave of a few CTAs), 28.3 with 4, 68 with 1.
    const int64_t sms = ctx->sm_count, wave = sms * (rows <= 8 ? 3 : 2);
    const int most = groups * 8 < sms ? 16 : 8;
    p.splits = 1;
    while (p.splits < most && groups * p.splits < 2 * sms && kv_len > int64_t(p.splits) * 2 * 64) p.splits *= 2;
    if (groups * p.splits > wave) p.splits = int(std::max<int64_t>(1, wave / groups));
    if (dtype == TL_F32) e = head_dim == 64 ? launch_decode_f32<64>(ctx, p, groups) : launch_decode_f32<128>(ctx, p, groups);
    else if (dtype == TL_F16) e = head_dim == 64 ? launch_decode_mma<__half, 64>(ctx, p, groups) : launch_decode_mma<__half, 128>(ctx, p, groups);
    else e = head_dim == 64 ? launch_decode_mma<__nv_bfloat16, 64>(ctx, p, groups) : launch_decode_mma<__nv_bfloat16, 128>(ctx, p, groups);
  } else if (tl_attention_tc_applicable(q, k_cache, v_cache, out, dtype, rows, head_dim, scale, mask)) {
    int32_t rc = tl_launch_attention_tc(ctx, q, k_cache, v_cache, out, dtype, batch, n_heads, n_kv_heads, q_len, head_dim, kv_len, kv_capacity,
                                        scale, causal);
    if (rc != TL_OK) return rc;
  } else {
    if (smem > 48 * 1024) cudaFuncSetAttribute(attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    attention_kernel<<<unsigned(batch * n_heads * q_len), 128, smem, ctx->stream>>>(q, k_cache, v_cache, out, dtype, int(n_heads), int(n_kv_heads),
                                                                                    int(q_len), int(head_dim), int(kv_len), kv_capacity, scale, mask,
                                                                                    causal ? 1 : 0);
    e = cudaGetLastError();
  }
  TL_CUDA(ctx, e);
  ctx->counters[TL_COUNTER_KERNEL_LAUNCHES]++;
  tl_wrote(ctx, out, batch * q_len * n_heads * head_dim * tl_dtype_size(dtype));
  return TL_OK;
}

int32_t tl_decode_attention(tl_ctx* ctx, const void* q, const void* k_cache, const void* v_cache, void* out, int32_t dtype, int64_t batch,
                            int64_t n_heads, int64_t n_kv_heads, int64_t head_dim, int64_t kv_len, int64_t kv_capacity, float scale,
                            const float* mask) {
  return tl_attention(ctx, q, k_cache, v_cache, out, dtype, batch, n_heads, n_kv_heads, 1, head_dim, kv_len, kv_capacity, scale, mask, 0);
}

}  // extern "C"
