// int4-grouped: the second weight-only scheme, which the reference plans but does not implement
// (docs/quantization-design.md:69-75, 386-396: "8 int4 per u32 word, packed 8-along-K into [N, K/8] u32,
// ... unpacks a nibble ((word >> (4*j)) & 0xF, sign-extend from 4 bits)"; "a new VALUE on the format
// axis: a scheme entry + unpackInt4 in the kernel", reusing the seam).  Everything here follows the int8
// path with the range [-7, 7]: scales are the f16 bits of the group abs-max (w = (q / 7) * scale), or
// f32 "direct" scales (w = q * s).
//
//   host quantizer        tl_quantize_linear_weight_int4 (same arithmetic as the int8 quantizer)
//   explicit dequant      tl_dequant_int4 (f64 through a 16-entry table, one rounding: bit-exact)
//   small batch, m <= 16  qgemv_int4_ring_kernel (f16 / bf16 activations, K a multiple of 128, groups of 32, 64 or
//                         multiples of 128): mma.sync with the nibbles converted pairwise, see below; else
//                         qgemv_int4_kernel: warp per R rows, one packed word (8 weights) per lane and
//                         step -- a warp reads 128 contiguous bytes of each row per step -- nibbles to
//                         f32 by exponent stuffing, f32 FMA, group scale applied to the group's partial
//                         sum, warp-shuffle reduction, the common epilogue.  HBM-bound at m <= 2
//                         (0.5 byte per weight against 3 ALU ops per weight and one FMA per batch
//                         row); FMA-bound above that.
//   m > 16                explicit dequant into library scratch in the activation type, then the dense
//                         matmul (tl_matmul: tcgen05 when it applies) -- the reference's fallback for
//                         every m > 1 (src/backend/webgpu/ops/matmul-ops.ts:163-181).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <thread>
#include <vector>

#include "tl_common.cuh"
#include "tl_mma_frag.cuh"
#include "tl_tma.cuh"

namespace {

inline double round_half_up(double x) {  // JS Math.round
  const double f = std::floor(x);
  return (x - f >= 0.5) ? f + 1.0 : f;
}

void quantize_rows_int4(const float* weight, int64_t row0, int64_t row1, int64_t k, int32_t group, uint32_t* packed,
                        uint16_t* scales) {
  const int64_t groups = k / group, words = k / 8;
  for (int64_t row = row0; row < row1; ++row) {
    const float* w = weight + row * k;
    uint32_t* pw = packed + row * words;
    std::memset(pw, 0, size_t(words) * 4);
    for (int64_t g = 0; g < groups; ++g) {
      const float* wg = w + g * group;
      float amax = 0.f;
      for (int32_t j = 0; j < group; ++j) amax = std::max(amax, std::fabs(wg[j]));
      const uint32_t sbits = tl_f32_to_f16_bits(amax);
      scales[row * groups + g] = uint16_t(sbits);
      // the scale that is stored is the scale that quantizes: widen the f16 bits back exactly
      const double s = double(tl_f16_bits_to_f32(sbits));
      const double inv = s > 0 ? 7.0 / s : 0.0;
      for (int32_t j = 0; j < group; ++j) {
        double q = round_half_up(double(wg[j]) * inv);
        q = std::isnan(q) ? 0.0 : std::max(-7.0, std::min(7.0, q));
        const int64_t kk = g * group + j;
        pw[kk >> 3] |= (uint32_t(int32_t(q)) & 0xfu) << ((kk & 7) * 4);
      }
    }
  }
}

template <typename OutT>
__global__ void __launch_bounds__(256)
dequant_int4_kernel(const uint32_t* __restrict__ packed, const void* __restrict__ scales, OutT* __restrict__ out, int64_t n_words,
                    int32_t group, int32_t scales_dtype, int32_t convention, int vec) {
  __shared__ double lut[16];  // q/7 (snorm) or q (direct), indexed by the raw nibble
  if (threadIdx.x < 16) {
    const int q = threadIdx.x >= 8 ? int(threadIdx.x) - 16 : int(threadIdx.x);
    lut[threadIdx.x] = convention == TL_SCALE_SNORM127 ? double(q) / 7.0 : double(q);
  }
  __syncthreads();
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int wpg = group >> 3;  // words per group: a word lies in one group, and groups are contiguous across rows
  const int shift = (wpg & (wpg - 1)) == 0 ? 31 - __clz(wpg) : -1;
  for (int64_t wi = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; wi < n_words; wi += stride) {
    const uint32_t word = __ldg(packed + wi);
    const double s = double(tl_load_scale(scales, scales_dtype, shift >= 0 ? wi >> shift : wi / wpg));
    alignas(16) OutT o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = DT<OutT>::from_f32(float(lut[(word >> (4 * j)) & 0xfu] * s));
    if (vec) {
#pragma unroll
      for (int j = 0; j < int(sizeof(o) / 16); ++j) reinterpret_cast<uint4*>(out + wi * 8)[j] = reinterpret_cast<const uint4*>(o)[j];
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) out[wi * 8 + j] = o[j];
    }
  }
}

__global__ void __launch_bounds__(256) unpack_int4_kernel(const uint32_t* __restrict__ packed, int8_t* __restrict__ out, int64_t n_words) {
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t wi = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; wi < n_words; wi += stride) {
    const uint32_t w = __ldg(packed + wi);
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lo |= (uint32_t(int32_t(w << (28 - 4 * j)) >> 28) & 0xffu) << (8 * j);
      hi |= (uint32_t(int32_t(w << (12 - 4 * j)) >> 28) & 0xffu) << (8 * j);
    }
    reinterpret_cast<uint2*>(out)[wi] = make_uint2(lo, hi);
  }
}

struct Int4Args {
  const void* a;
  const uint32_t* packed;
  const void* scales;
  void* out;
  int32_t m, n, k, row0;     // this launch's batch rows are [row0, row0 + m)
  int32_t group, groups_per_row, scales_dtype, out_dtype;
  float wscale;              // 1/7 for the abs-max convention, 1 for direct scales
};

template <typename AT> __device__ __forceinline__ void load8(const AT* p, float (&x)[8]);
template <> __device__ __forceinline__ void load8<float>(const float* p, float (&x)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__half>(const __half* p, float (&x)[8]) {
  const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    x[2 * i] = f.x; x[2 * i + 1] = f.y;
  }
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&x)[8]) {
  const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { x[2 * i] = __uint_as_float(w[i] << 16); x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}

// warp per R rows; lane per packed word (8 weights, one group: group % 8 == 0)
template <typename AT, int MT, int R>
__global__ void __launch_bounds__(256) qgemv_int4_kernel(Int4Args p, EpiParams epi) {
  const int warps = blockDim.x >> 5, lane = threadIdx.x & 31;
  const int64_t row_base = (int64_t(blockIdx.x) * warps + (threadIdx.x >> 5)) * R;
  if (row_base >= p.n) return;
  const AT* a = reinterpret_cast<const AT*>(p.a);
  const int words = p.k >> 3;
  int64_t rows[R];
#pragma unroll
  for (int r = 0; r < R; ++r) rows[r] = min(row_base + r, int64_t(p.n) - 1);  // tail rows clamp, stores mask
  float acc[R][MT];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[r][i] = 0.f;
  for (int c = lane; c < words; c += 32) {
    uint32_t wv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) wv[r] = __ldg(p.packed + rows[r] * words + c);
    float x[MT][8];
#pragma unroll
    for (int i = 0; i < MT; ++i) load8<AT>(a + int64_t(i) * p.k + int64_t(c) * 8, x[i]);
    const int grp = (c * 8) / p.group;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t u = wv[r] ^ 0x88888888u;  // two's complement nibble -> q + 8
      float part[MT];
#pragma unroll
      for (int i = 0; i < MT; ++i) part[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // (q + 8) into the mantissa of 2^23, minus (2^23 + 8): q exactly
        const float q = __uint_as_float(((u >> (4 * j)) & 0xfu) | 0x4B000000u) - 8388616.f;
#pragma unroll
        for (int i = 0; i < MT; ++i) part[i] = fmaf(q, x[i][j], part[i]);
      }
      const float s = tl_load_scale(p.scales, p.scales_dtype, rows[r] * p.groups_per_row + grp);
#pragma unroll
      for (int i = 0; i < MT; ++i) acc[r][i] = fmaf(s, part[i], acc[r][i]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t row = row_base + r;
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      float v = acc[r][i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0 && row < p.n) {
        const float o = tl_apply_epilogue(epi, v * p.wscale, p.row0 + i, row, p.n);
        tl_store_out(p.out, p.out_dtype, int64_t(p.row0 + i) * p.n + row, o);
      }
    }
  }
}

constexpr int kSimtWarps = 8;
constexpr int simt_batch(int m) { return m >= 4 ? 4 : m >= 2 ? 2 : 1; }   // batch rows of a launch
constexpr int simt_rows(int batch) { return batch >= 4 ? 2 : 4; }         // weight rows of a warp

template <typename AT, int MT>
void launch_int4(tl_ctx* ctx, const Int4Args& p, const EpiParams& e) {
  constexpr int R = simt_rows(MT), kRows = kSimtWarps * R;
  qgemv_int4_kernel<AT, MT, R><<<(p.n + kRows - 1) / kRows, kSimtWarps * 32, 0, ctx->stream>>>(p, e);
}

template <typename AT>
void launch_int4_m(tl_ctx* ctx, Int4Args p, const EpiParams& epi, int m) {
  const uint8_t* a0 = static_cast<const uint8_t*>(p.a);
  // column tiles of 4, 2 and 1 batch rows (each launch re-reads the weights: FMA-bound territory anyway)
  for (int m0 = 0; m0 < m;) {
    const int mt = simt_batch(m - m0);
    p.a = a0 + size_t(m0) * p.k * sizeof(AT);
    p.row0 = m0; p.m = mt;
    if (mt == 4) launch_int4<AT, 4>(ctx, p, epi);
    else if (mt == 2) launch_int4<AT, 2>(ctx, p, epi);
    else launch_int4<AT, 1>(ctx, p, epi);
    ctx->counters[TL_COUNTER_KERNEL_LAUNCHES]++;
    m0 += mt;
  }
}

// ---------------------------------------------------------------------------
// Tensor-core form (f16 / bf16 activations, K % 128 == 0, group 32, 64 or a multiple of 128): CTA per 16 * RT weight
// rows, warps interleaved over 128-wide k blocks.  Every warp runs its own cp.async ring in shared memory: a stage
// holds one k block, 64 bytes of each of the tile's rows and 256 bytes of each activation row, so weights AND
// activations are asked for S blocks ahead and hold no registers while they travel.  A row's 64 bytes are four
// 16-byte chunks of 32 weights; lane (g, t) reads word t of chunk i of rows g and g + 8 and the matching eight
// activations, so a chunk's two MMAs cover 32 consecutive k -- one group of the smallest size -- and its sums are
// folded into the totals with the rows' scales where a group ends (FOLD times a block; 0: scales once at the end).
// Chunks are swapped by the row (w: (row >> 1) & 3, activations: 4 * (row & 1)) so that neither read has a bank conflict.
// A mask and an exclusive or with a magic exponent and the sign bits make the pair (q_x + 8, q_{x+4} + 8)
// 16-bit floats 1024 + . (f16) or 128 + . (bf16), and one subtraction -- or, for the nibbles taken at bits 4-7, one
// fused multiply-add -- gives (q_x, q_{x+4}) exactly (Nib::quad); the activations are paired the same way.
// Bound: instruction issue (66 % of the slots, the ALU pipe 59 %; 317 instructions a 16 x 128 block, 337 with a division and row
// arithmetic in every block) and a second wave that fills half the chip, ahead of HBM.  14336 x 4096, groups of 128, bias + gelu,
// replayed: 15.0 us at m = 1, 15.3 at 4, 21.7 at 16 (16.2, 16.4, 22.9 with that arithmetic; 20.3, 21.5, 33.5 with two blocks in registers
// and the activations met in the loop); groups of 32: 18.5, 18.9, 28.8 (they took the CUDA cores' form).
// ---------------------------------------------------------------------------
// quad(u, v): the four MMA operand registers of one packed word u; the exclusive or that sets the exponent also turns
// the two's complement nibble into n = q + 8:
//   v[0] = (q0, q4), v[1] = (q1, q5), v[2] = (q2, q6), v[3] = (q3, q7)
template <typename AT> struct Nib;
template <> struct Nib<__half> {
  // ONE shift per word: nibbles at bits 0-3 give 1024 + n, nibbles at bits 4-7 give 1024 + 16 n, which
  // one fused multiply-add turns into n - 8 exactly ((1024 + 16 n) / 16 - 72); the upper half of the
  // word goes through the same two masks after a shift by 8.
  __device__ static void quad(uint32_t u, uint32_t (&v)[4]) {
    const __half2 k1032 = __halves2half2(__ushort_as_half(0x6408), __ushort_as_half(0x6408));
    const __half2 k16th = __halves2half2(__ushort_as_half(0x2C00), __ushort_as_half(0x2C00));   // 1/16
    const __half2 km72 = __halves2half2(__ushort_as_half(0xD480), __ushort_as_half(0xD480));    // -72
    const uint32_t u8 = u >> 8;
    const uint32_t a = (u & 0x000F000Fu) ^ 0x64086408u, b = (u & 0x00F000F0u) ^ 0x64806480u;
    const uint32_t c = (u8 & 0x000F000Fu) ^ 0x64086408u, d = (u8 & 0x00F000F0u) ^ 0x64806480u;
    const __half2 r0 = __hsub2(*reinterpret_cast<const __half2*>(&a), k1032);
    const __half2 r1 = __hfma2(*reinterpret_cast<const __half2*>(&b), k16th, km72);
    const __half2 r2 = __hsub2(*reinterpret_cast<const __half2*>(&c), k1032);
    const __half2 r3 = __hfma2(*reinterpret_cast<const __half2*>(&d), k16th, km72);
    v[0] = *reinterpret_cast<const uint32_t*>(&r0); v[1] = *reinterpret_cast<const uint32_t*>(&r1);
    v[2] = *reinterpret_cast<const uint32_t*>(&r2); v[3] = *reinterpret_cast<const uint32_t*>(&r3);
  }
};
template <> struct Nib<__nv_bfloat16> {
  // seven mantissa bits hold 128 + n only for a nibble at bits 0-3: one shift per pair
  __device__ static void quad(uint32_t u, uint32_t (&v)[4]) {
    const uint32_t m = 0x43084308u;  // 136 | 136
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const uint32_t w = ((u >> (4 * x)) & 0x000F000Fu) ^ 0x43084308u;
      const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&w), *reinterpret_cast<const __nv_bfloat162*>(&m));
      v[x] = *reinterpret_cast<const uint32_t*>(&r);
    }
  }
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

template <typename AT, int NT, int RT, int FOLD, int S>
__global__ void __launch_bounds__(RT == 2 ? 256 : 512) qgemv_int4_ring_kernel(Int4Args p, EpiParams epi) {
  extern __shared__ __align__(128) uint8_t ring4[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t tile_row = int64_t(blockIdx.x) * (16 * RT);
  const int64_t row_bytes = p.k >> 1;
  const int kblocks = p.k >> 7, mrows = p.m;
  const uint32_t stage_bytes = uint32_t(RT * 1024 + mrows * 256);
  const uint32_t ring = smem_u32(ring4) + uint32_t(warp * S) * stage_bytes;
  // This lane's rows (tail rows clamp, stores mask), and where their weights and scales begin.  Scales that fold several times a block
  // leave no registers for the latter (groups of 32, 14336 x 4096: 18.7 -> 20.4 us with them); with groups of 128 they took 16.4 -> 15.4.
  constexpr bool kKeep = FOLD <= 1;
  int64_t rows[RT][2];
  const uint8_t* wrow[RT][2];
  int64_t srow[RT][2];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      rows[r][h] = min(tile_row + r * 16 + h * 8 + g, int64_t(p.n) - 1);
      wrow[r][h] = reinterpret_cast<const uint8_t*>(p.packed) + rows[r][h] * row_bytes + 16 * t;
      srow[r][h] = rows[r][h] * p.groups_per_row;
    }
  const uint32_t w_swz = uint32_t((g >> 1) & 3);
  auto issue_weights = [&](int s, int kb) {
    const uint8_t* w = reinterpret_cast<const uint8_t*>(p.packed) + int64_t(kb) * 64 + 16 * t;
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        cp_async16(ring + s * stage_bytes + (r * 16 + h * 8 + g) * 64 + ((t ^ w_swz) << 4), kKeep ? wrow[r][h] + kb * 64 : w + rows[r][h] * row_bytes);
  };
  const AT* a_lane = reinterpret_cast<const AT*>(p.a) + int64_t(lane >> 4) * p.k + 8 * (lane & 15);
  const uint32_t a_dst = uint32_t(RT * 1024 + (lane >> 4) * 256 + (((lane & 15) ^ ((lane >> 4) << 2)) << 4));
  auto issue_acts = [&](int s, int kb) {
    // lanes 0-15 take even rows, 16-31 odd ones, a 16-byte chunk each
    const AT* a = a_lane + int64_t(kb) * 128;
    uint32_t dst = ring + s * stage_bytes + a_dst;
#pragma unroll
    for (int r = 0; r < 8 * NT; r += 2) {
      if (r + (lane >> 4) < mrows) cp_async16(dst, a);
      a += 2 * int64_t(p.k);
      dst += 512;
    }
  };
  // group scales, one block ahead of their use
  constexpr int NF = FOLD > 0 ? FOLD : 1;
  float sc[RT][2][NF];
  const int group_blocks = p.group >> 7, group_shift = (group_blocks & (group_blocks - 1)) == 0 ? 31 - __clz(max(group_blocks, 1)) : -1;
  auto load_scales = [&](int kb) {
    if (FOLD == 0) return;
    const int grp = FOLD != 1 ? kb * FOLD : group_shift >= 0 ? kb >> group_shift : kb / group_blocks;
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int f = 0; f < NF; ++f) sc[r][h][f] = tl_load_scale(p.scales, p.scales_dtype, (kKeep ? srow[r][h] : rows[r][h] * p.groups_per_row) + grp + f);
  };
  // the weights do not depend on the kernel before this one: ask for them while it drains
#pragma unroll
  for (int s = 0; s < S; ++s)
    if (warp + s * warps < kblocks) issue_weights(s, warp + s * warps);
  asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
  for (int s = 0; s < S; ++s) {
    if (warp + s * warps < kblocks) issue_acts(s, warp + s * warps);
    cp_async_commit();
  }
  if (warp < kblocks) load_scales(warp);
  if (epi.fast_bias && threadIdx.x < 16 * RT && tile_row + threadIdx.x < p.n)
    asm volatile("prefetch.global.L1 [%0];" ::"l"(epi.fast_bias + tile_row + threadIdx.x));

  float total[RT][NT][4];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) total[r][nt][i] = 0.f;
  uint32_t a_off[NT], a_swz[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int r = min(nt * 8 + g, mrows - 1);
    a_off[nt] = uint32_t(RT * 1024 + r * 256);
    a_swz[nt] = uint32_t((r & 1) << 2);
  }
  int s = 0;
  for (int kb = warp; kb < kblocks; kb += warps) {
    cp_async_wait<S - 1>();
    __syncwarp();
    const uint32_t st = ring + s * stage_bytes;
    float cs[RT][2][NF];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int f = 0; f < NF; ++f) cs[r][h][f] = sc[r][h][f];
    if (kb + warps < kblocks) load_scales(kb + warps);
    // two accumulators a tile: half as long a chain of dependent MMAs
    float c[RT][NT][4], d[RT][NT][4];
#pragma unroll
    for (int i4 = 0; i4 < 4; ++i4) {
      if (i4 % (4 / NF) == 0) {
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) { c[r][nt][i] = FOLD ? 0.f : total[r][nt][i]; d[r][nt][i] = 0.f; }
      }
      uint32_t b[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint4 xv = lds128(st + a_off[nt] + (((i4 * 4 + t) ^ a_swz[nt]) << 4));  // x0..x7 of this word
        b[nt][0] = __byte_perm(xv.x, xv.z, 0x5410); b[nt][1] = __byte_perm(xv.x, xv.z, 0x7632);
        b[nt][2] = __byte_perm(xv.y, xv.w, 0x5410); b[nt][3] = __byte_perm(xv.y, xv.w, 0x7632);
      }
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const uint32_t w = st + (r * 16 + g) * 64 + ((i4 ^ w_swz) << 4) + 4 * t;
        uint32_t lo[4], hi[4];
        Nib<AT>::quad(lds32(w), lo);
        Nib<AT>::quad(lds32(w + 512), hi);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          MmaOps<AT>::mma_free(c[r][nt], lo[0], hi[0], lo[1], hi[1], b[nt][0], b[nt][1]);
          MmaOps<AT>::mma_free(d[r][nt], lo[2], hi[2], lo[3], hi[3], b[nt][2], b[nt][3]);
        }
      }
      if ((i4 + 1) % (4 / NF) == 0) {
        const int f = i4 / (4 / NF);
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float v = c[r][nt][i] + d[r][nt][i];
              total[r][nt][i] = FOLD ? fmaf(cs[r][i >> 1][f], v, total[r][nt][i]) : v;
            }
      }
    }
    __syncwarp();  // every lane has read the stage
    if (kb + S * warps < kblocks) {
      issue_weights(s, kb + S * warps);
      issue_acts(s, kb + S * warps);
    }
    cp_async_commit();
    s = (s + 1) % S;
  }
  cp_async_wait<0>();
  __syncthreads();  // the rings are done with: the partial tiles meet in their place
  float* red = reinterpret_cast<float*>(ring4);  // [warps][RT][NT][4][32]
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) red[(((warp * RT + r) * NT + nt) * 4 + i) * 32 + lane] = total[r][nt][i];
  __syncthreads();
  for (int o = threadIdx.x; o < RT * NT * 128; o += blockDim.x) {
    const int tile = o >> 7, i = (o >> 5) & 3, ln = o & 31, r = tile / NT, nt = tile - r * NT;
    const int64_t row = tile_row + r * 16 + (ln >> 2) + ((i & 2) ? 8 : 0);
    const int col = 8 * nt + 2 * (ln & 3) + (i & 1);
    if (row < p.n && col < p.m) {
      // four short sums instead of one long one, whatever the number of warps
      float part[4] = {0.f, 0.f, 0.f, 0.f};
      for (int w = 0; w < warps; w += 4)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (w + e < warps) part[e] += red[(((w + e) * RT * NT + tile) * 4 + i) * 32 + ln];
      const float v = (part[0] + part[1]) + (part[2] + part[3]);
      float f = p.wscale;
      if (FOLD == 0) f *= tl_load_scale(p.scales, p.scales_dtype, row);
      tl_store_out(p.out, p.out_dtype, int64_t(col) * p.n + row, tl_apply_epilogue(epi, v * f, col, row, p.n));
    }
  }
}

inline size_t int4_ring_smem(int warps, int rt, int s, int m) { return size_t(warps) * s * (rt * 1024 + m * 256); }

template <typename AT, int NT, int RT, int FOLD, int S>
cudaError_t int4_ring_at(tl_ctx* ctx, const Int4Args& p, const EpiParams& e, int warps) {
  auto kern = qgemv_int4_ring_kernel<AT, NT, RT, FOLD, S>;
  const size_t smem = int4_ring_smem(warps, RT, S, p.m);
  if (smem > 48 * 1024) {
    cudaError_t rc = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (rc != cudaSuccess) return rc;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned((p.n + 16 * RT - 1) / (16 * RT)));
  cfg.blockDim = dim3(warps * 32);
  cfg.dynamicSmemBytes = smem;
  const EarlyStream stream = tl_early_stream(ctx);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = stream.attrs;
  return cudaLaunchKernelEx(&cfg, kern, p, e);
}
template <typename AT, int NT, int RT, int FOLD>
cudaError_t int4_ring_s(tl_ctx* ctx, const Int4Args& p, const EpiParams& e, int warps, int s) {
  return s == 4 ? int4_ring_at<AT, NT, RT, FOLD, 4>(ctx, p, e, warps) : int4_ring_at<AT, NT, RT, FOLD, 2>(ctx, p, e, warps);
}
template <typename AT, int NT, int RT>
cudaError_t int4_ring_fold(tl_ctx* ctx, const Int4Args& p, const EpiParams& e, int warps, int s) {
  if (p.group == p.k) return int4_ring_s<AT, NT, RT, 0>(ctx, p, e, warps, s);
  if (p.group % 128 == 0) return int4_ring_s<AT, NT, RT, 1>(ctx, p, e, warps, s);
  if (p.group == 64) return int4_ring_s<AT, NT, RT, 2>(ctx, p, e, warps, s);
  return int4_ring_s<AT, NT, RT, 4>(ctx, p, e, warps, s);
}
template <typename AT>
cudaError_t int4_ring(tl_ctx* ctx, const Int4Args& p, const EpiParams& e, int warps, int rt, int s) {
  if (p.m > 8) return rt == 2 ? int4_ring_fold<AT, 2, 2>(ctx, p, e, warps, s) : int4_ring_fold<AT, 2, 1>(ctx, p, e, warps, s);
  return rt == 2 ? int4_ring_fold<AT, 1, 2>(ctx, p, e, warps, s) : int4_ring_fold<AT, 1, 1>(ctx, p, e, warps, s);
}

struct RingShape { int warps, row_tiles, stages; };

RingShape int4_ring_shape(const tl_ctx* ctx, int m, int64_t n, int64_t k, int group, int32_t out_dtype) {
  const int kblocks = int(k >> 7);
  // A warp takes about a microsecond a block whatever the rest of the chip does, so the fewer the tiles the more warps
  // share each one's k loop: sixteen up to two tiles an SM, with rings of four stages where shared memory leaves the
  // tiles resident; else eight with two.  Two token tiles want 32-row tiles, which share the activations, once every SM
  // has a tile -- with groups below 128, whose folds take the registers, up to two tiles an SM.  us, groups of 128: 1425 x 11008 m = 1
  // 16 warps 7.9, 8 warps 10.5; 4096 x 14336 m = 4 17.0, 22.9; 4096 x 4096 m = 16 32-row tiles 7.6, 16-row 9.6; 14336 x 4096 m = 16
  // 4 warps 21.8 to 22.9, 8 warps 29.5.  Groups of 32: 30000 x 1024 m = 1 4 warps 10.3, 8 warps 13.3, m = 16 16.6, 22.7; 14336 x 4096 m = 16 28.8,
  // 30.6; 4096 x 12288 m = 16 32-row tiles 22.8, sixteen warps 26.7.
  // Fewer warps are longer f32 sums (against 64 bits, 16 x 4096 x 12288 in groups of 32: 1.07e-7 with sixteen, 1.34e-7 with eight): an f32
  // output keeps the warps that the small groups and short k loops would give up; a 16-bit one, off by 2.1e-4 either way, does not.
  const int64_t tiles = (n + 15) / 16, sms = ctx->sm_count;
  int warps = 8, rt = 1, s = 2;
  const bool folds_once = group == k || group % 128 == 0, fewer = out_dtype != TL_F32;
  if (m > 8 && tiles > sms && (folds_once || (fewer && tiles <= 2 * sms))) {
    rt = 2;
    if (tiles > 4 * sms) warps = 4;
    else s = 4;
  } else if (fewer && tiles > 4 * sms && (m > 8 || kblocks <= 8)) {
    warps = 4;  // several waves: short k loops, or the registers of two token tiles whose scales fold several times a block
  } else if (tiles <= 2 * sms && kblocks >= 16) {
    warps = 16;
    if (int4_ring_smem(16, 1, 4, m) <= (tiles <= sms ? 220 : 110) * 1024) s = 4;
  } else if (tiles <= 2 * sms) {
    s = 4;
  }
  while (warps > 2 && warps > kblocks) warps >>= 1;
  // A/B hook: {TL_FAMILY_QGEMV, 9, warps, row tiles, stages}
  if (ctx->has_forced && ctx->forced.family == TL_FAMILY_QGEMV && ctx->forced.kernel == 9) {
    const tl_variant& f = ctx->forced;
    if (f.p1 == 1 || f.p1 == 2) rt = f.p1;
    if (f.p0 >= 1 && f.p0 <= (rt == 2 ? 8 : 16) && (f.p0 & (f.p0 - 1)) == 0) warps = f.p0;
    if (f.p2 == 2 || f.p2 == 4) s = f.p2;
    if (int4_ring_smem(warps, rt, s, m) > 220 * 1024) s = 2;  // sixteen warps of many tokens: what a CTA may have
  }
  return RingShape{warps, rt, s};
}

// The tensor-core form, when its layout conditions hold (and it is not switched off for A/B tests)
bool int4_ring_applies(const tl_ctx* ctx, int32_t a_dtype, int64_t k, int group) {
  const bool forced_simt = ctx->has_forced && ctx->forced.family == TL_FAMILY_QGEMV && ctx->forced.kernel == 1;
  return !forced_simt && a_dtype != TL_F32 && k % 128 == 0 && (group % 128 == 0 || group == 64 || group == 32);
}

template <typename AT>
cudaError_t launch_int4_mma(tl_ctx* ctx, const Int4Args& p, const EpiParams& e) {
  const RingShape r = int4_ring_shape(ctx, p.m, p.n, p.k, p.group, p.out_dtype);
  cudaError_t rc = int4_ring<AT>(ctx, p, e, r.warps, r.row_tiles, r.stages);
  ctx->counters[TL_COUNTER_KERNEL_LAUNCHES]++;
  return rc;
}

int32_t check_int4(tl_ctx* ctx, const char* who, const void* packed, const void* scales, int64_t n, int64_t k, const tl_quant_desc* q) {
  if (!packed || !scales) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: missing packing/scales on B operand", who);
  if (n < 0 || k < 0 || n > 0x7fffffffLL || k > 0x7fffffffLL) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: bad shape n=%lld k=%lld", who, (long long)n, (long long)k);
  if (k % 8 != 0) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: K=%lld must be divisible by 8 (eight int4 per word)", who, (long long)k);
  if (q->group_size <= 0 || q->group_size % 8 != 0 || (k > 0 && k % q->group_size != 0))
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: K=%lld must be divisible by groupSize=%d, itself a multiple of 8", who, (long long)k, q->group_size);
  if (q->scales_dtype != TL_F16 && q->scales_dtype != TL_F32) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: scales dtype must be f16 or f32", who);
  if (q->scale_convention != TL_SCALE_SNORM127 && q->scale_convention != TL_SCALE_DIRECT)
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: unknown scale convention %d", who, q->scale_convention);
  if ((reinterpret_cast<uintptr_t>(packed) & 3) || (reinterpret_cast<uintptr_t>(scales) & (tl_dtype_size(q->scales_dtype) - 1)))
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: misaligned weight or scales pointer", who);
  return TL_OK;
}

}  // namespace

extern "C" {

int32_t tl_quantize_linear_weight_int4(const float* weight, int64_t n, int64_t k, int32_t group_size, uint32_t* packed, uint16_t* scales) {
  if (!weight || !packed || !scales) return tl_set_error(nullptr, TL_ERR_INVALID_ARG, "quantize int4: null pointer");
  if (n < 0 || k < 0) return tl_set_error(nullptr, TL_ERR_INVALID_ARG, "quantize int4: negative shape");
  if (k % 8 != 0) return tl_set_error(nullptr, TL_ERR_INVALID_ARG, "quantize int4: K=%lld must be divisible by 8", (long long)k);
  if (group_size <= 0 || k % group_size != 0)
    return tl_set_error(nullptr, TL_ERR_INVALID_ARG, "quantize int4: K=%lld must be divisible by groupSize=%d", (long long)k, group_size);
  if (n == 0 || k == 0) return TL_OK;
  const unsigned hw = std::thread::hardware_concurrency();
  int64_t nthreads = std::max<int64_t>(1, std::min<int64_t>(hw ? hw : 1, (n * k) / (1 << 16)));
  nthreads = std::min<int64_t>(nthreads, n);
  if (nthreads <= 1) {
    quantize_rows_int4(weight, 0, n, k, group_size, packed, scales);
    return TL_OK;
  }
  std::vector<std::thread> pool;
  const int64_t per = (n + nthreads - 1) / nthreads;
  for (int64_t t = 0; t < nthreads; ++t) {
    const int64_t r0 = t * per, r1 = std::min(n, r0 + per);
    if (r0 >= r1) break;
    pool.emplace_back(quantize_rows_int4, weight, r0, r1, k, group_size, packed, scales);
  }
  for (auto& th : pool) th.join();
  return TL_OK;
}

int32_t tl_dequant_int4(tl_ctx* ctx, const void* packed, const void* scales, void* out, int32_t out_dtype, int64_t n, int64_t k,
                        const tl_quant_desc* qdesc) {
  TL_CHECK_CTX(ctx);
  if (!qdesc || qdesc->scheme != TL_SCHEME_INT4_GROUPED) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_dequant_int4: the descriptor's scheme must be int4-grouped");
  int32_t rc = check_int4(ctx, "tl_dequant_int4", packed, scales, n, k, qdesc);
  if (rc != TL_OK) return rc;
  if (!out || !tl_dtype_valid(out_dtype)) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_dequant_int4: null output or unknown dtype");
  ctx->counters[TL_COUNTER_DEQUANT]++;
  const int64_t n_words = n * (k / 8);
  if (n_words == 0) return TL_OK;
  DeviceGuard guard(ctx->device);
  const int grid = int(std::min<int64_t>((n_words + 255) / 256, int64_t(ctx->sm_count) * 16));
  const int vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  const uint32_t* pk = static_cast<const uint32_t*>(packed);
  if (out_dtype == TL_F32)
    dequant_int4_kernel<float><<<grid, 256, 0, ctx->stream>>>(pk, scales, static_cast<float*>(out), n_words, qdesc->group_size, qdesc->scales_dtype, qdesc->scale_convention, vec);
  else if (out_dtype == TL_F16)
    dequant_int4_kernel<__half><<<grid, 256, 0, ctx->stream>>>(pk, scales, static_cast<__half*>(out), n_words, qdesc->group_size, qdesc->scales_dtype, qdesc->scale_convention, vec);
  else
    dequant_int4_kernel<__nv_bfloat16><<<grid, 256, 0, ctx->stream>>>(pk, scales, static_cast<__nv_bfloat16*>(out), n_words, qdesc->group_size, qdesc->scales_dtype, qdesc->scale_convention, vec);
  TL_CUDA(ctx, cudaGetLastError());
  ctx->counters[TL_COUNTER_KERNEL_LAUNCHES]++;
  tl_wrote(ctx, out, n * k * tl_dtype_size(out_dtype), true);
  return TL_OK;
}

int32_t tl_unpack_int4(tl_ctx* ctx, const void* packed, void* out_i8, int64_t n, int64_t k) {
  TL_CHECK_CTX(ctx);
  if (!packed || !out_i8 || n < 0 || k < 0 || k % 8 != 0 || (reinterpret_cast<uintptr_t>(out_i8) & 7))
    return tl_set_error(ctx, TL_ERR_INVALID_ARG, "tl_unpack_int4: null pointer, K %% 8 != 0 or an output not 8-byte aligned");
  const int64_t n_words = n * (k / 8);
  if (n_words == 0) return TL_OK;
  DeviceGuard guard(ctx->device);
  const int grid = int(std::min<int64_t>((n_words + 255) / 256, int64_t(ctx->sm_count) * 16));
  unpack_int4_kernel<<<grid, 256, 0, ctx->stream>>>(static_cast<const uint32_t*>(packed), static_cast<int8_t*>(out_i8), n_words);
  ctx->fresh_weights = true;  // its bytes are a packed int8 weight
  TL_CUDA(ctx, cudaGetLastError());
  ctx->counters[TL_COUNTER_KERNEL_LAUNCHES]++;
  return TL_OK;
}

}  // extern "C"

// The seam's int4 branch (tl_qmatmul_nt / tl_qgemv_nt / tl_qgemm_nt with an int4 descriptor).
// route: 0 by m, 1 GEMV only, 2 dequant + dense only.
int32_t tl_int4_matmul(tl_ctx* ctx, const char* who, int route, const void* a, int32_t a_dtype, const void* packed, const void* scales,
                       void* out, int32_t out_dtype, int64_t m, int64_t n, int64_t k, const tl_quant_desc* q, float alpha,
                       const tl_epilogue* epilogue, tl_plan_receipt* receipt_only) {
  int32_t rc = check_int4(ctx, who, receipt_only ? (const void*)16 : packed, receipt_only ? (const void*)16 : scales, n, k, q);
  if (rc != TL_OK) return rc;
  if (!tl_dtype_valid(a_dtype) || !tl_dtype_valid(out_dtype)) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: unknown dtype", who);
  if (m < 0) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: negative m", who);
  if (!receipt_only && ((m > 0 && !a) || !out)) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: null activation or output", who);
  if (route == 1 && (m < 1 || m > 16)) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: m=%lld outside the GEMV range [1,16]", who, (long long)m);
  EpiParams epi;
  bool has_ops = false;
  rc = tl_make_epi(ctx, epilogue, alpha, &epi, &has_ops);
  if (rc != TL_OK) return rc;
  const bool gemv = route == 1 || (route == 0 && m <= 16);
  // vector loads of the activations: 8 values per lane and step
  const bool a_aligned = receipt_only || (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  if (receipt_only) {
    memset(receipt_only, 0, sizeof(*receipt_only));
    receipt_only->choice.family = gemv ? TL_FAMILY_QGEMV : TL_FAMILY_QGEMM;
    receipt_only->choice.kernel = gemv ? 9 : 2;  // "int4" / "dequant+dense"
    if (gemv && m > 0 && n > 0) {
      int64_t rows = 0;  // of a CTA
      if (int4_ring_applies(ctx, a_dtype, k, q->group_size)) {
        const RingShape r = int4_ring_shape(ctx, int(m), n, k, q->group_size, out_dtype);
        receipt_only->choice.p0 = r.warps; receipt_only->choice.p1 = r.row_tiles; receipt_only->choice.p2 = r.stages;
        rows = 16 * r.row_tiles;
        receipt_only->block = 32 * r.warps;
      } else {  // the first of its launches, if the batch rows take several
        rows = kSimtWarps * simt_rows(simt_batch(int(m)));
        receipt_only->block = 32 * kSimtWarps;
      }
      receipt_only->grid[0] = int32_t((n + rows - 1) / rows);
      receipt_only->grid[1] = receipt_only->grid[2] = 1;
    }
    receipt_only->split_k = 1;
    receipt_only->epilogue_engaged = has_ops ? 1 : 0;
    return TL_OK;
  }
  if (m == 0 || n == 0) return TL_OK;
  DeviceGuard guard(ctx->device);
  if (gemv) {
    if (!a_aligned) return tl_set_error(ctx, TL_ERR_INVALID_ARG, "%s: int4 GEMV needs 16-byte aligned activations", who);
    if ((size_t(k) * tl_dtype_size(a_dtype)) % 16 != 0) return tl_set_error(ctx, TL_ERR_UNSUPPORTED, "%s: int4 GEMV needs activation rows of whole 16-byte vectors", who);
    Int4Args p{};
    p.a = a; p.packed = static_cast<const uint32_t*>(packed); p.scales = scales; p.out = out;
    p.n = int32_t(n); p.k = int32_t(k);
    p.group = q->group_size; p.groups_per_row = int32_t(k / q->group_size);
    p.scales_dtype = q->scales_dtype; p.out_dtype = out_dtype;
    p.wscale = q->scale_convention == TL_SCALE_SNORM127 ? 1.0f / 7.0f : 1.0f;
    const bool mma_ok = int4_ring_applies(ctx, a_dtype, k, q->group_size) && (reinterpret_cast<uintptr_t>(packed) & 15) == 0;
    p.m = int32_t(m); p.row0 = 0;
    if (mma_ok && a_dtype == TL_F16) TL_CUDA(ctx, launch_int4_mma<__half>(ctx, p, epi));
    else if (mma_ok) TL_CUDA(ctx, launch_int4_mma<__nv_bfloat16>(ctx, p, epi));
    else if (a_dtype == TL_F32) launch_int4_m<float>(ctx, p, epi, int(m));
    else if (a_dtype == TL_F16) launch_int4_m<__half>(ctx, p, epi, int(m));
    else launch_int4_m<__nv_bfloat16>(ctx, p, epi, int(m));
    TL_CUDA(ctx, cudaGetLastError());
    ctx->counters[TL_COUNTER_QGEMV]++;
    tl_wrote(ctx, out, m * n * tl_dtype_size(out_dtype));
    if (has_ops) ctx->counters[TL_COUNTER_QGEMV_EPILOGUE]++;
    return TL_OK;
  }
  // m > 16: dequantize [N, K] into scratch in the activation type, then the dense NT product
  void* wbuf = nullptr;
  rc = tl_ensure_scratch(ctx, size_t(n) * size_t(k) * tl_dtype_size(a_dtype) + (size_t(1) << 20), &wbuf);
  if (rc != TL_OK) return rc;
  // the dense kernel may want scratch of its own (operand transposition: not for NT) -- keep ours at the front
  rc = tl_dequant_int4(ctx, packed, scales, wbuf, a_dtype, n, k, q);
  if (rc != TL_OK) return rc;
  rc = tl_matmul(ctx, a, wbuf, out, m, n, k, 1, 0, 0, m * n, 0, 1, alpha, a_dtype, a_dtype, out_dtype, -1, -1, epilogue, nullptr);
  if (rc == TL_OK) ctx->counters[TL_COUNTER_QGEMM]++;
  return rc;
}
