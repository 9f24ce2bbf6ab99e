// Attention of many query rows on the 5th-generation tensor cores: softmax(q k^T * scale) v, causal or not, grouped
// query heads (packages/qwen3-browser/src/model.ts:284-318, the prefill of a prompt or of a chunk behind a filled
// cache).  f16 / bf16, head dimension 64 or 128, no mask tensor.
//
// A CTA owns one or two blocks of 128 query rows of one KV head; a row is a (position, head of the group) pair, so the
// heads that share keys share the K and V tiles.  Scores and output accumulate in TMEM (256 columns a block); the
// probabilities take the scores' place there as the A operand of the second product, two 16-bit terms in f16, three
// in bf16: 23 and all 24 of the bits they were computed with.  The maximum that a row is scaled by moves only when it is
// passed by 2^8 (the output is then rescaled in TMEM): a step rarely waits for that.  With two blocks one is multiplied
// while the other's softmax runs.
// Bound: the tensor core in principle (three units of work per score in f16: one for q k^T, two for p v), the chain
// scores -> softmax -> products in practice: tensor pipe 51 % busy, instruction issue 49 %.  1 x 32 (8 KV) heads x 2048
// x 2048 x 128 causal, in the kernel: f16 51 us = 680 TFLOP/s of the causal work, bf16 62 (10.3 ms one CTA per query row;
// 67 / 91 with the MMAs issued by one lane of a branch).  The products start on the first half of a step's
// probabilities and the softmax works on pairs (f32x2): 1000 rows bf16 32.9 -> 30.2, 100 rows x 2000 keys 37.5 -> 35.1.
#include <algorithm>
#include <cmath>

#include "tl_attention.cuh"
#include "tl_tcgen05.cuh"

namespace {

struct AttnTcArgs {
  const void* q;
  const void* k;
  const void* v;
  void* out;
  int32_t n_heads, n_kv_heads, rep, q_len, rows, kv_len, causal, m_blocks, groups;  // rows = rep * q_len of one KV head
  int64_t capacity;
  float scale, scale_log2;  // scale_log2 = scale * log2(e) > 0: the softmax runs in base 2
  int* status;
};

// Per storage type: keys per step, and where in a row block's 128 score columns the scores lie.  A 16-key slice of
// scores (16 columns) is replaced by its probabilities' terms (8 columns each): f16 fits in place; bf16 needs 24
// columns a slice, so its 64 scores lie in the upper half and the probabilities are written from column 0 -- slice
// c ends at 24 c + 24, below the next unread score at 64 + 16 (c + 1).
template <typename AT> struct AttnTc;
template <> struct AttnTc<__half> {
  static constexpr uint32_t kFmt = 0;
  static constexpr int kBN = 128, kScoreCol = 0;
  static constexpr float kBias = 7.f;  // probabilities are held times 2^7: the low term stays clear of f16's subnormals
};
template <> struct AttnTc<__nv_bfloat16> {
  static constexpr uint32_t kFmt = 1;
  static constexpr int kBN = 64, kScoreCol = 64;
  static constexpr float kBias = 0.f;
};
constexpr float kLazy = 8.f;  // log2 by which a maximum may be passed before the row is rescaled: 2^(7 + 8) is an f16

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// MT row blocks of 128 per CTA.
template <typename AT, int D, int MT>
__global__ void __launch_bounds__(64 + 256 * MT, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, AttnTcArgs p) {
  constexpr int BN = AttnTc<AT>::kBN, TERMS = ProbSplit<AT>::kTerms, SLOTS = 4 * (128 / BN), SLABS = D / 64;
  constexpr int kQBytes = 128 * D * 2, kSlotBytes = BN * D * 2;
  constexpr uint32_t kTmemCols = 256 * MT, kScore = 128 + AttnTc<AT>::kScoreCol, kProb = 128;
  constexpr uint32_t kFmtBits = (1u << 4) | (AttnTc<AT>::kFmt << 7) | (AttnTc<AT>::kFmt << 10) | (uint32_t(128 >> 4) << 24);
  constexpr uint32_t kIdescS = kFmtBits | (uint32_t(BN >> 3) << 17);               // q k^T: both K-major
  constexpr uint32_t kIdescO = kFmtBits | (uint32_t(D >> 3) << 17) | (1u << 16);   // p v: v as it lies, MN-major

  extern __shared__ uint8_t attn_smem_raw[];
  __shared__ uint64_t kv_full[SLOTS], kv_empty[SLOTS], q_full[MT], s_full[MT], p_full[MT][2], o_full[MT], drained;
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag, issued;  // issued: key and value tiles that were asked for
  __shared__ float row_half[MT][2][2][128];  // [row block][step parity][half][row]: what a row's two threads tell each other
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(attn_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* kv_sm = sm + MT * kQBytes;
  pdl_launch_dependents();
  const int warp = warp_index(), lane = threadIdx.x & 31;
  // longest rows first: with a causal mask the last row blocks see the most keys
  const int mblk = p.m_blocks - 1 - int(blockIdx.x) / p.groups, bkv = int(blockIdx.x) % p.groups;
  const int b = bkv / p.n_kv_heads, kvh = bkv - b * p.n_kv_heads;
  int steps[MT], most = 0;  // key steps of each row block
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    const int row0 = (mblk * MT + t) * 128;
    const int keys = row0 >= p.rows ? 0 : p.causal ? p.kv_len - p.q_len + min(row0 + 127, p.rows - 1) / p.rep + 1 : p.kv_len;
    steps[t] = (keys + BN - 1) / BN;
    most = max(most, steps[t]);
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    for (int t = 0; t < MT; ++t) {
      mbar_init(&q_full[t], 8);
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t][0], 8);
      mbar_init(&p_full[t][1], 8);
      mbar_init(&o_full[t], 1);
    }
    mbar_init(&drained, 1);
    abort_flag = 0;
    issued = 2 * most;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_smem, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  pdl_wait();

  if (warp == 0) {
    // ------------------------------ TMA producer: k 0, v 0, k 1, v 1, ... ------------------------------
    if (lane == 0) {
      tma_prefetch_desc(&kmap);
      tma_prefetch_desc(&vmap);
      for (int i = 0; i < 2 * most; ++i) {
        const int s = i % SLOTS;
        if (i >= SLOTS && !mbar_wait(&kv_empty[s], ((i / SLOTS) - 1) & 1, &abort_flag)) {
          if (!abort_flag) { abort_flag = 1; atomicExch(p.status, TL_DEV_TIMEOUT_EMPTY); }
          issued = i;
          break;
        }
        mbar_expect_tx(&kv_full[s], kSlotBytes);
#pragma unroll
        for (int h = 0; h < SLABS; ++h)
          tma_load_3d(kv_sm + s * kSlotBytes + h * BN * 128, (i & 1) ? &vmap : &kmap, h * 64, (i >> 1) * BN, bkv, &kv_full[s]);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer: the whole warp, one lane elected ------------------------------
    {
      const uint32_t elected = elect_one(), tb = __shfl_sync(0xffffffffu, tmem_base, 0);
      bool ok = true;
      auto wait = [&](uint64_t* bar, int parity, int code) {
        if (ok && !mbar_wait_warp(bar, parity, &abort_flag)) {
          if (lane == 0 && !abort_flag) { abort_flag = 1; atomicExch(p.status, code); }
          ok = false;
        }
        return ok;
      };
      auto slot = [&](int i) { return smem_u32(kv_sm + (i % SLOTS) * kSlotBytes); };
      auto scores = [&](int t, int j) {
        const uint64_t a = make_b_desc(smem_u32(sm + t * kQBytes)), bb = make_b_desc(slot(2 * j));
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          tc_mma_ss(tb + t * 256 + kScore, desc_at(a, (kk >> 2) * (128 * 128) + (kk & 3) * 32),
                    desc_at(bb, (kk >> 2) * (BN * 128) + (kk & 3) * 32), kIdescS, kk > 0 ? 1u : 0u, elected);
        tc_commit(&s_full[t], elected);
      };
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        if (steps[t] == 0 || !wait(&q_full[t], 0, TL_DEV_TIMEOUT_FULL) || !wait(&kv_full[0], 0, TL_DEV_TIMEOUT_FULL)) continue;
        tc_fence_after();
        scores(t, 0);
      }
      if (ok) tc_commit(&kv_empty[0], elected);
      for (int j = 0; j < most && ok; ++j) {
        const int iv = 2 * j + 1, ik = 2 * j + 2;
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          if (j >= steps[t] || !wait(&kv_full[iv % SLOTS], (iv / SLOTS) & 1, TL_DEV_TIMEOUT_FULL)) continue;
          const uint64_t vb = make_mn_desc(slot(iv), BN * 128);
          // the probabilities come in two parts, the first half of each thread's slices and the rest
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!wait(&p_full[t][h], j & 1, TL_DEV_TIMEOUT_TMEM)) break;
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < BN / 32; ++i) {
              const int c = (i / (BN / 64)) * (BN / 32) + h * (BN / 64) + i % (BN / 64);
#pragma unroll
              for (int term = 0; term < TERMS; ++term)
                tc_mma_ts(tb + t * 256, tb + t * 256 + kProb + (c * TERMS + term) * 8, desc_at(vb, c * 2048), kIdescO,
                          (j > 0 || h > 0 || i > 0 || term > 0) ? 1u : 0u, elected);
            }
          }
          if (!ok) continue;
          if (j + 1 == steps[t]) {
            tc_commit(&o_full[t], elected);
          } else if (wait(&kv_full[ik % SLOTS], (ik / SLOTS) & 1, TL_DEV_TIMEOUT_FULL)) {
            // the tensor core works in order: these scores land where the product above has read its probabilities
            tc_fence_after();
            scores(t, j + 1);
          }
        }
        if (!ok) break;
        tc_commit(&kv_empty[iv % SLOTS], elected);
        if (j + 1 < most) tc_commit(&kv_empty[ik % SLOTS], elected);
      }
    }
  } else {
    // ------------------------------ softmax: two threads per query row ------------------------------
    // Each takes half of a step's keys (a single warp per scheduler and row block could not hide its own latencies: the
    // tensor core waited for it two thirds of the time) and half of the output.  They agree on the row's maximum
    // through shared memory; the barrier they meet at for that also says that all scores are in registers, before any
    // probability is written over them.
    constexpr int HN = BN / 2, HD = D / 2;
    const int t = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1, quad = warp & 3;
    const int block_row0 = (mblk * MT + t) * 128, warp_row0 = block_row0 + quad * 32;
    const int nsteps = MT == 1 ? steps[0] : t == 0 ? steps[0] : steps[MT - 1];
    const uint32_t tm = tmem_base + t * 256 + (uint32_t(quad * 32) << 16);
    auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + quad) : "memory"); };
    if (nsteps > 0) {
      // this warp's half of 32 query rows to shared memory, 128-byte swizzled slabs of 64 dimensions
      uint8_t* qs = sm + t * kQBytes;
      constexpr int kChunks = D / 8, kRowsPer = 32 / kChunks;
#pragma unroll
      for (int i = 0; i < kChunks / 2; ++i) {
        const int r = quad * 32 + (half * (kChunks / 2) + i) * kRowsPer + lane / kChunks, c = lane % kChunks;
        const int gr = block_row0 + r;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (gr < p.rows) {
          const int pos = gr / p.rep, h = kvh * p.rep + (gr - pos * p.rep);
          x = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const AT*>(p.q) + ((int64_t(b) * p.n_heads + h) * p.q_len + pos) * D) + c);
        }
        *reinterpret_cast<uint4*>(qs + (c >> 3) * (128 * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = x;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full[t]);
    }
    const int bound = p.causal ? p.kv_len - p.q_len + min(warp_row0 + lane, p.rows - 1) / p.rep + 1 : p.kv_len;  // keys this row sees
    const int warp_bound = p.causal ? p.kv_len - p.q_len + min(warp_row0, p.rows - 1) / p.rep + 1 : p.kv_len;
    const float c2 = p.scale_log2, lazy = kLazy / c2;
    float m = -INFINITY;
    float2 l = make_float2(0.f, 0.f);
    bool ok = true;  // a wait that gave up: the loop runs on, so that the other warp of the rows is met, but nothing is stored
    for (int j = 0; j < nsteps; ++j) {
      if (ok && !mbar_wait(&s_full[t], j & 1, &abort_flag)) {
        if (lane == 0 && !abort_flag) { abort_flag = 1; atomicExch(p.status, TL_DEV_TIMEOUT_TMEM); }
        ok = false;
      }
      tc_fence_after();
      uint32_t su[HN];
#pragma unroll
      for (int i = 0; i < HN; i += 32) tmem_ld32(tm + kScore + half * HN + i, su + i);
      tmem_ld_wait();
      const int key0 = j * BN + half * HN;
      if (warp_bound - key0 < HN) {
#pragma unroll
        for (int i = 0; i < HN; ++i) su[i] = key0 + i < bound ? su[i] : 0xff800000u;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < HN; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(su[i]));
      float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      row_half[t][j & 1][half][quad * 32 + lane] = top;
      meet();
      top = fmaxf(top, row_half[t][j & 1][half ^ 1][quad * 32 + lane]);
      if (__any_sync(0xffffffffu, top > m + lazy)) {
        const float nm = fmaxf(m, top);
        if (j > 0) {  // the scores' arrival says that the products before them are done
          const float f = ex2((m - nm) * c2);
          l.x *= f;
          l.y *= f;
#pragma unroll 1
          for (int i = 0; i < HD; i += 16) {
            uint32_t o[16];
            tmem_ld16(tm + half * HD + i, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
            tmem_st16(tm + half * HD + i, o);
          }
        }
        m = nm;
      }
      const float off = AttnTc<AT>::kBias - m * c2;
      const float2 scale2 = make_float2(c2, c2), off2 = make_float2(off, off);
#pragma unroll
      for (int c = 0; c < HN / 16; ++c) {
        uint32_t w[TERMS][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 x = fma_x2(make_float2(__uint_as_float(su[c * 16 + 2 * i]), __uint_as_float(su[c * 16 + 2 * i + 1])), scale2, off2);
          const float2 pr = make_float2(ex2(x.x), ex2(x.y));
          l = add_x2(l, pr);
          uint32_t tt[TERMS];
          ProbSplit<AT>::split(pr, tt);
#pragma unroll
          for (int k = 0; k < TERMS; ++k) w[k][i] = tt[k];
        }
#pragma unroll
        for (int k = 0; k < TERMS; ++k) tmem_st8(tm + kProb + ((half * (HN / 16) + c) * TERMS + k) * 8, w[k]);
        if (c == HN / 32 - 1 || c == HN / 16 - 1) {  // half of the slices is enough for the product to start on
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0 && ok) mbar_arrive(&p_full[t][c == HN / 16 - 1]);
        }
      }
    }
    if (nsteps > 0) {
      float sum = l.x + l.y;
      row_half[t][nsteps & 1][half][quad * 32 + lane] = sum;
      meet();
      sum += row_half[t][nsteps & 1][half ^ 1][quad * 32 + lane];
      if (ok && mbar_wait(&o_full[t], 0, &abort_flag)) {
        tc_fence_after();
        uint32_t o[HD];
#pragma unroll
        for (int i = 0; i < HD; i += 32) tmem_ld32(tm + half * HD + i, o + i);
        tmem_ld_wait();
        const float inv = 1.f / sum;
        float odd = 0.f;
#pragma unroll
        for (int i = 0; i < HD; ++i) {
          const float x = __uint_as_float(o[i]) * inv;
          odd = fmaf(x, 0.f, odd);  // NaN as soon as one value is not finite
          o[i] = __float_as_uint(x);
        }
        const int row = min(warp_row0 + lane, p.rows - 1), qpos = row / p.rep, head = kvh * p.rep + (row - qpos * p.rep);
        const int64_t slice = int64_t(bkv) * p.capacity * D;
        const bool fine = odd == 0.f, row_ok = warp_row0 + lane < p.rows;
        if (row_ok && fine) {
          AT* op = reinterpret_cast<AT*>(p.out) + ((int64_t(b) * p.q_len + qpos) * p.n_heads + head) * D + half * HD;
#pragma unroll
          for (int i = 0; i < HD; i += 8) {
            AT pk[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) pk[e] = DT<AT>::from_f32(__uint_as_float(o[i + e]));
            *reinterpret_cast<uint4*>(op + i) = *reinterpret_cast<const uint4*>(pk);
          }
        }
        for (uint32_t redo = __ballot_sync(0xffffffffu, row_ok && !fine); redo != 0; redo &= redo - 1) {
          const int r = warp_row0 + __ffs(redo) - 1, pos = r / p.rep, h = kvh * p.rep + (r - pos * p.rep);
          attention_row_warp<AT, D>(reinterpret_cast<const AT*>(p.q) + ((int64_t(b) * p.n_heads + h) * p.q_len + pos) * D,
                                    reinterpret_cast<const AT*>(p.k) + slice, reinterpret_cast<const AT*>(p.v) + slice,
                                    reinterpret_cast<AT*>(p.out) + ((int64_t(b) * p.q_len + pos) * p.n_heads + h) * D,
                                    p.causal ? p.kv_len - p.q_len + pos + 1 : p.kv_len, p.scale, nullptr, half * (HD / 32), HD / 32);
        }
      } else if (lane == 0 && !abort_flag) {
        abort_flag = 1;
        atomicExch(p.status, TL_DEV_TIMEOUT_TMEM);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    if (warp == 0 && lane == 0) tma_drain(kv_full, SLOTS, issued);
    if (warp == 1) tc_drain(&drained);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <typename AT, int D, int MT>
cudaError_t launch(tl_ctx* ctx, const CUtensorMap& kmap, const CUtensorMap& vmap, AttnTcArgs p) {
  constexpr size_t smem = size_t(MT) * 128 * D * 2 + 4 * size_t(128) * D * 2 + 1024;
  p.m_blocks = (p.rows + 128 * MT - 1) / (128 * MT);
  auto kern = attn_tc_kernel<AT, D, MT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(p.m_blocks) * unsigned(p.groups));
  cfg.blockDim = dim3(64 + 256 * MT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1] = {tl_pdl_attribute()};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, kmap, vmap, p);
}
template <typename AT, int D>
cudaError_t launch_mt(tl_ctx* ctx, const CUtensorMap& kmap, const CUtensorMap& vmap, const AttnTcArgs& p) {
  return int64_t(p.groups) * ((p.rows + 255) / 256) >= ctx->sm_count ? launch<AT, D, 2>(ctx, kmap, vmap, p) : launch<AT, D, 1>(ctx, kmap, vmap, p);
}

}  // namespace

bool tl_attention_tc_applicable(const void* q, const void* k, const void* v, const void* out, int32_t dtype, int64_t rows, int64_t head_dim,
                                float scale, const float* mask) {
  if (dtype != TL_F16 && dtype != TL_BF16) return false;
  if ((head_dim != 64 && head_dim != 128) || mask || rows <= 16) return false;
  if (!(scale > 0.f) || !std::isfinite(scale)) return false;  // the running maximum is kept on unscaled products
  return !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out)) & 15);
}

int32_t tl_launch_attention_tc(tl_ctx* ctx, const void* q, const void* k, const void* v, void* out, int32_t dtype, int64_t batch,
                               int64_t n_heads, int64_t n_kv_heads, int64_t q_len, int64_t head_dim, int64_t kv_len, int64_t capacity,
                               float scale, int32_t causal) {
  AttnTcArgs p{};
  p.q = q; p.k = k; p.v = v; p.out = out;
  p.n_heads = int32_t(n_heads); p.n_kv_heads = int32_t(n_kv_heads); p.rep = int32_t(n_heads / n_kv_heads);
  p.q_len = int32_t(q_len); p.rows = int32_t(p.rep * q_len); p.kv_len = int32_t(kv_len); p.capacity = capacity;
  p.groups = int32_t(batch * n_kv_heads);
  p.scale = scale; p.scale_log2 = scale * kLog2e; p.causal = causal ? 1 : 0; p.status = ctx->dev_status;
  const uint32_t bn = dtype == TL_F16 ? AttnTc<__half>::kBN : AttnTc<__nv_bfloat16>::kBN;
  CUtensorMap kmap, vmap;  // one slice per (sequence, KV head), kv_len rows of it: what lies behind reads as zero
  if (!tl_encode_tmap_3d(&kmap, 2, k, uint64_t(head_dim), uint64_t(kv_len), uint64_t(p.groups), uint64_t(head_dim) * 2,
                         uint64_t(capacity) * head_dim * 2, 64, bn, 3) ||
      !tl_encode_tmap_3d(&vmap, 2, v, uint64_t(head_dim), uint64_t(kv_len), uint64_t(p.groups), uint64_t(head_dim) * 2,
                         uint64_t(capacity) * head_dim * 2, 64, bn, 3))
    return tl_set_error(ctx, TL_ERR_CUDA, "tl_attention: cuTensorMapEncodeTiled failed (kv_len=%lld capacity=%lld)", (long long)kv_len,
                        (long long)capacity);
  cudaError_t e;
  if (dtype == TL_F16) e = head_dim == 64 ? launch_mt<__half, 64>(ctx, kmap, vmap, p) : launch_mt<__half, 128>(ctx, kmap, vmap, p);
  else e = head_dim == 64 ? launch_mt<__nv_bfloat16, 64>(ctx, kmap, vmap, p) : launch_mt<__nv_bfloat16, 128>(ctx, kmap, vmap, p);
  TL_CUDA(ctx, e);
  return TL_OK;
}
