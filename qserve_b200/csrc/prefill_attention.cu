// qserve_b200 -- causal variable-length prefill attention on the sm_100a tensor cores (tcgen05 kind::f16, accumulators and P in tensor memory).
//
// Replaces the third-party call on the reference's prompt path: flash_attn_varlen_func(q, k, v, cu_seqlens, cu_seqlens, max_seqlen, max_seqlen,
// dropout_p=0, causal=True) in qserve/modeling/models/llama_w4a8_unpad.py:232-242, where q / k / v are strided views of the post-RoPE fp16 qkv
// buffer that fused_attention.apply_bias_rope_update_kv_cache has just rotated in place.
//
// One CTA = one (sequence, query head, block of 128 query rows).  Per block of 64 keys:
//     S = Q K^T      8 x tcgen05.mma 128x64x16, both operands K-major in shared memory (TMA, 128-byte swizzle), fp32 accumulators in TMEM
//     softmax        4 warps, thread = query row (TMEM lane): running max / sum in the log2 domain, P = exp2(..) rounded to fp16 and written
//                    into tensor memory (P is the A operand of the next MMA)
//     O += P V       4 x tcgen05.mma 128x128x16, A from tensor memory, B = the V tile exactly as TMA delivers it ([key][dim] rows: an MN-major
//                    operand), accumulating in a third TMEM region
// S, P and O share no TMEM columns (64 + 32 + 128 of the CTA's 256), so the next block's S is computed while this block's softmax goes on, and P V while
// the next softmax does.  Blocks of 128 keys left room for P only over S, so the next S waited for P V: 8 prompts of 539 .. 1024 tokens x 32 heads 103 us,
// then 89; with the longest query blocks of all sequences first and whole rows stored 86, with two blocks in the first step 3 % less.  2 x 4096 tokens
// 374 -> 271 us (0.73 -> 1.01 PFLOP/s), 8192 tokens 674 -> 489.
// The first step takes two blocks (S in 128 columns, P in 2 x 32: nothing is there to overlap with yet): sequences of 65 to 128 tokens have one step, as with
// blocks of 128 keys.  40 x 100 tokens x 32 heads: 31.3 us with blocks of 128, 34.6 with one block in every step, now 30.7; calls whose sequences all have one query
// block take a form without the walk.
// The O accumulator is rescaled only when a row's maximum has grown by more than 2^8 since the last rescale (the sum uses the same stale
// maximum, so the quotient is exact up to rounding); the decision is taken per warp because tcgen05.ld/st are warp-collective.
// 256 TMEM columns and 96 KB of shared memory per CTA: two CTAs per SM, one's softmax overlaps the other's MMAs.  K and V are double-buffered.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include <mutex>

#include "common.cuh"
#include "launch.h"

namespace qs {
namespace {

constexpr int kD = 128;         // head dim
constexpr int kBQ = 128;        // query rows per CTA (UMMA M)
constexpr int kBKV = 64;        // keys per block (UMMA N of S, K extent of PV)
constexpr int kThreads = 192;   // warps 0..3 softmax / epilogue, warp 4 TMA producer, warp 5 TMEM allocator + MMA issuer
constexpr int kTileBytes = kBQ * kD * 2;      // 32 KB: two swizzled [128 rows x 64 halfs] sub-tiles
constexpr int kSubBytes = kTileBytes / 2;     // 16 KB
constexpr int kKvBytes = kBKV * kD * 2;       // 16 KB: a K or V block, two sub-tiles of 64 rows
constexpr int kKvSub = kKvBytes / 2;          // a sub-tile's two buffers lie side by side: both blocks are the rows of one operand
constexpr int kOffQ = 0, kOffK = kTileBytes, kOffV = kOffK + 2 * kKvBytes, kOffBar = kOffV + 2 * kKvBytes;
constexpr int kSmemBytes = kOffBar + 128;
constexpr uint32_t kTmemCols = 256;
// S: columns [0, 64), of the first two blocks [0, 128); P: [64, 96), of the second block [96, 128); O: [128, 256)
constexpr uint32_t kColP = 64, kColP1 = 96, kColO = 128;
constexpr float kRescaleThreshold = 8.f;      // log2 units

// kind::f16 instruction descriptor: D = f32, A = B = f16, A K-major; B K-major (S = Q K^T) or MN-major (O = P V)
//   bits [4,6) c_format (1 = F32)   [7,10) a_format (0 = F16)   [10,13) b_format   [15] a_major   [16] b_major (1 = MN)
//   bits [17,23) N >> 3             [24,29) M >> 4
__host__ __device__ constexpr uint32_t umma_idesc_f16(uint32_t m, uint32_t n, uint32_t b_mn_major) {
  return (1u << 4) | (b_mn_major << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      :
      : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}

// 2^x on the SFU (MUFU.EX2), flush-to-zero: the argument is <= 8 here and -inf must give 0
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// MN-major shared-memory operand under the 128-byte swizzle: rows of 128 B are 64 contiguous elements of the M/N dimension, one row per K
// index.  In 16-byte units the canonical layout is ((8, n), (8, k)) : ((1, LBO), (8, SBO)): LBO = distance between 64-element column groups
// (here the second 16 KB sub-tile), SBO = distance between groups of 8 K-rows (1024 B).
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(uint32_t smem_addr, uint32_t lbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(lbo_bytes >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// thread i of the warp writes 32 consecutive 32-bit columns of ITS lane (lane = 32 * (warp % 4) + i)
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
      "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
        "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
struct PrefillAttnParams {
  const int* cu_seqlens;  // [B + 1]
  __half* out;            // [T, Hq * 128] rows of out_stride halfs
  long long out_stride;
  int num_heads, num_kv_heads;
  float scale_log2;       // softmax scale * log2(e)
  int q_blocks;           // query blocks of the longest sequence, as far as this launch goes
};

// ONE: no sequence of the call has more than one query block
template <bool ONE>
__global__ void __launch_bounds__(kThreads, 2)
prefill_attention_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                         const __grid_constant__ CUtensorMap tmap_v, const PrefillAttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int b = blockIdx.y, h = blockIdx.x;
  const int seq_start = __ldg(p.cu_seqlens + b);
  const int seq_len = __ldg(p.cu_seqlens + b + 1) - seq_start;
  const int n_qb = (seq_len + kBQ - 1) / kBQ;
  const int qb = p.q_blocks - 1 - static_cast<int>(blockIdx.z);  // the last query blocks see most keys: they are scheduled first
  if (qb >= n_qb) return;                                                        // uniform per CTA: nothing has been allocated yet
  if (threadIdx.x == 0 && (smem_u32(smem) & 1023u) != 0) __trap();
  const int hkv = h / (p.num_heads / p.num_kv_heads);
  // causal, q and k positions coincide: the key blocks up to the query block's last row, as far as the sequence goes
  const int n_kb = (min((qb + 1) * kBQ, seq_len) + kBKV - 1) / kBKV;
  const int n_steps = ONE ? 1 : max(1, n_kb - 1);  // the first one takes two blocks

  uint8_t* s_q = smem + kOffQ;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kOffBar);
  uint64_t* bar_q = bar + 0;       // Q tile landed
  uint64_t* bar_s = bar + 1;       // a step's S complete in tensor memory
  uint64_t* bar_read = bar + 2;    // S read by the four softmax warps (4 arrivals): the next one may follow
  uint64_t* bar_p = bar + 3;       // P written by the four softmax warps (4 arrivals)
  uint64_t* bar_o = bar + 4;       // O += P V retired: O may be rescaled / read, P overwritten
  uint64_t* bar_kfull = bar + 5;   // [2] K block landed
  uint64_t* bar_kfree = bar + 7;   // [2] S = Q K^T retired: the K buffer may be refilled
  uint64_t* bar_vfull = bar + 9;   // [2]
  uint64_t* bar_vfree = bar + 11;  // [2] O += P V retired: the V buffer may be refilled
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bar + 13);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    for (int i = 0; i < 13; ++i) mbar_init(&bar[i], i == 2 || i == 3 ? 4 : 1);
    fence_barrier_init();
  }
  if (warp == 5) tmem_alloc<kTmemCols>(s_tmem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = *s_tmem;
  if (threadIdx.x == 0) pdl_launch_dependents();

  if (warp == 4) {
    // ===================================== TMA producer =====================================
    if (lane == 0) {
      pdl_wait();  // q / k / v are written by the preceding kernel (RoPE + KV append)
      const int q_row = seq_start + qb * kBQ;
      mbar_expect_tx(bar_q, kTileBytes);
      tma_load_2d(s_q, &tmap_q, h * kD, q_row, bar_q);
      tma_load_2d(s_q + kSubBytes, &tmap_q, h * kD + 64, q_row, bar_q);
      auto ring = [&](int j, const CUtensorMap* map, int off, uint64_t* full, uint64_t* freed) {
        const int k_row = seq_start + j * kBKV, st = j & 1;
        uint8_t* buf = smem + off + st * kKvSub;
        mbar_wait(&freed[st], ((static_cast<uint32_t>(j) >> 1) & 1u) ^ 1u);  // a fresh barrier passes the wait on the "previous" phase
        mbar_expect_tx(&full[st], kKvBytes);
        tma_load_2d(buf, map, hkv * kD, k_row, &full[st]);
        tma_load_2d(buf + 2 * kKvSub, map, hkv * kD + 64, k_row, &full[st]);
      };
      ring(0, &tmap_k, kOffK, bar_kfull, bar_kfree);
      for (int j = 0; j < n_kb; ++j) {
        if (j + 1 < n_kb) ring(j + 1, &tmap_k, kOffK, bar_kfull, bar_kfree);
        ring(j, &tmap_v, kOffV, bar_vfull, bar_vfree);
      }
    }
  } else if (warp == 5) {
    // ===================================== MMA issuer =====================================
    if (lane == 0) {
      constexpr uint32_t idesc_qk = umma_idesc_f16(kBQ, kBKV, 0u), idesc_qk2 = umma_idesc_f16(kBQ, 2 * kBKV, 0u);
      constexpr uint32_t idesc_pv = umma_idesc_f16(kBQ, kD, 1u);
      auto products = [&](int st, uint32_t idesc) {  // Q K^T of the block in buffer st, or of the blocks in both
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks) {
          const uint64_t adesc = umma_desc_sw128(smem_u32(s_q + (ks >> 2) * kSubBytes)) + (ks & 3) * 2;
          const uint64_t bdesc = umma_desc_sw128(smem_u32(smem + kOffK + st * kKvSub + (ks >> 2) * 2 * kKvSub)) + (ks & 3) * 2;
          umma_f16_ss(tmem_s, adesc, bdesc, idesc, ks > 0 ? 1u : 0u);
        }
        umma_commit(bar_s);
      };
      // O += P V of block j: A = P (fp16 pairs, 8 TMEM columns per 16 keys), B = V rows [key][dim] = MN-major, 16 keys (2 KB) per instruction
      auto weighted = [&](int j, uint32_t weights) {
        const int st = j & 1;
        mbar_wait(&bar_vfull[st], (static_cast<uint32_t>(j) >> 1) & 1u);
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < kBKV / 16; ++kk) {
          const uint64_t bdesc = umma_desc_sw128_mn(smem_u32(smem + kOffV + st * kKvSub + kk * 2048), 2 * kKvSub);
          umma_f16_ts(tmem_s + kColO, weights + kk * 8, bdesc, idesc_pv, (j > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(&bar_vfree[st]);
      };
      mbar_wait(bar_q, 0);
      mbar_wait(&bar_kfull[0], 0);
      if (n_kb > 1) {
        mbar_wait(&bar_kfull[1], 0);
        products(0, idesc_qk2);
        umma_commit(&bar_kfree[1]);
      } else {
        products(0, idesc_qk);
      }
      umma_commit(&bar_kfree[0]);
      for (int i = 0; i < n_steps; ++i) {
        if (i + 1 < n_steps) {  // the next step's S (block i + 2), while this step's softmax goes on
          const int st = i & 1;
          mbar_wait(bar_read, static_cast<uint32_t>(i) & 1u);
          mbar_wait(&bar_kfull[st], ((static_cast<uint32_t>(i) + 2) >> 1) & 1u);
          products(st, idesc_qk);
          umma_commit(&bar_kfree[st]);
        }
        mbar_wait(bar_p, static_cast<uint32_t>(i) & 1u);
        if (i == 0) {
          weighted(0, tmem_s + kColP);
          if (n_kb > 1) weighted(1, tmem_s + kColP1);
        } else {
          weighted(i + 1, tmem_s + kColP);
        }
        umma_commit(bar_o);
      }
    }
  } else {
    // ===================================== softmax + epilogue: thread = query row =====================================
    const int row = warp * 32 + lane;
    const uint32_t t_s = tmem_s + (static_cast<uint32_t>(warp * 32) << 16), t_o = t_s + kColO;
    const int q_pos = qb * kBQ + row;  // position inside the sequence
    float m_used = -CUDART_INF_F;      // the maximum the accumulated O and l are expressed against (log2 domain, scaled)
    float l = 0.f;
    using Row = uint32_t[2][32];       // of S: 64 fp32
    Row r;
    uint32_t pk[32];                   // its weights
    auto fetch = [&](Row& x, uint32_t from) {
      tmem_ld_32x32b_x32(from, x[0]);
      tmem_ld_32x32b_x32(from + 32, x[1]);
    };
    auto fetched = [&]() {
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_read);
    };
    auto mask = [&](Row& x, int j) {
      if (j * kBKV + kBKV - 1 > qb * kBQ + warp * 32) {  // warp-uniform: the block reaches past the warp's first row
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (j * kBKV + c * 32 + i > q_pos) x[c][i] = 0xff800000u;  // -inf: exp2 turns it into an exact 0
      }
    };
    auto largest = [&](const Row& x, float m) {
      float top[4] = {m, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) top[i & 3] = fmaxf(top[i & 3], __uint_as_float(x[c][i]));
      return fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
    };
    auto weights = [&](const Row& x) {  // P = exp2(s * scale - m_used), rounded to fp16
#pragma unroll
      for (int i = 0; i < 64; i += 2) {
        const float p0 = ex2_approx(fmaf(__uint_as_float(x[i >> 5][i & 31]), p.scale_log2, -m_used));
        const float p1 = ex2_approx(fmaf(__uint_as_float(x[i >> 5][(i & 31) + 1]), p.scale_log2, -m_used));
        const __half2 h2 = __floats2half2_rn(p0, p1);
        // the row sum is taken over the ROUNDED probabilities: numerator (the MMA sees fp16 P) and denominator then agree
        const float2 f = __half22float2(h2);
        l += f.x + f.y;
        pk[i >> 1] = *reinterpret_cast<const uint32_t*>(&h2);
      }
    };
    auto stored = [&]() {
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p);
    };
    // The first step takes two blocks; the second one's scores lie where P will be (a warp has read its lanes of them before it writes P).  A row's largest
    // weight against the maximum that is used is exactly 1 and rounds to fp16 without an error; the first 128 keys hold it more often than the first 64
    // (error against 64 bits 0.6 % larger with the first block's own maximum).  With more steps to come the second block's scores are read twice, for their
    // maximum and for their weights: with both rows held (152 registers) a step of one long and many short prompts took up to 1.4 times as long (20 x 64 and
    // 2048 tokens: 130 us, 89 with 127 registers)
    mbar_wait(bar_s, 0);
    tc_fence_after();
    if constexpr (ONE) {
      Row r1;
      fetch(r, t_s);
      if (n_kb > 1) fetch(r1, t_s + kBKV);
      tmem_wait_ld();
      mask(r, 0);
      float m = largest(r, -CUDART_INF_F);
      if (n_kb > 1) {
        mask(r1, 1);
        m = largest(r1, m);
      }
      m_used = m * p.scale_log2;
      weights(r);
      tmem_st_32x32b_x32(t_s + kColP, pk);
      if (n_kb > 1) {
        weights(r1);
        tmem_st_32x32b_x32(t_s + kColP1, pk);
      }
    } else {
      float m = -CUDART_INF_F;
      if (n_kb > 1) {
        fetch(r, t_s + kBKV);
        tmem_wait_ld();
        mask(r, 1);
        m = largest(r, m);
      }
      fetch(r, t_s);
      fetched();
      mask(r, 0);
      m_used = largest(r, m) * p.scale_log2;
      weights(r);
      if (n_kb > 1) {
        fetch(r, t_s + kBKV);
        tmem_wait_ld();
        mask(r, 1);
        tmem_st_32x32b_x32(t_s + kColP, pk);
        weights(r);
        tmem_st_32x32b_x32(t_s + kColP1, pk);
      } else {
        tmem_st_32x32b_x32(t_s + kColP, pk);
      }
    }
    stored();
    for (int i = 1; i < n_steps; ++i) {
      const uint32_t ph = static_cast<uint32_t>(i) & 1u;
      mbar_wait(bar_s, ph);
      tc_fence_after();
      fetch(r, t_s);  // ONE TMEM round trip
      fetched();
      mask(r, i + 1);
      const float m_blk = largest(r, -CUDART_INF_F) * p.scale_log2;
      // ---- lazy rescale of O and l (warp-uniform decision) ----
      const bool grow = (m_blk - m_used) > kRescaleThreshold;
      auto retired = [&]() {  // the previous O += P V
        mbar_wait(bar_o, ph ^ 1u);
        tc_fence_after();
      };
      if (__any_sync(0xffffffffu, grow)) {
        retired();
        const float m_new = grow ? m_blk : m_used;
        const float alpha = (m_used == -CUDART_INF_F) ? 0.f : ex2_approx(m_used - m_new);  // 1 for rows that keep their maximum
#pragma unroll 1
        for (int c = 0; c < kD / 32; ++c) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(t_o + c * 32, o);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
          tmem_st_32x32b_x32(t_o + c * 32, o);
        }
        l *= alpha;
        m_used = m_new;
      }
      weights(r);
      retired();
      tmem_st_32x32b_x32(t_s + kColP, pk);
      stored();
    }
    // ---- epilogue: O / l -> fp16 ----
    mbar_wait(bar_o, static_cast<uint32_t>(n_steps - 1) & 1u);
    tc_fence_after();
    const float inv = 1.f / l;
    auto eight = [&](const uint32_t* x) {  // eight outputs
      uint4 o;
      uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __half2 h2 = __floats2half2_rn(__uint_as_float(x[2 * e]) * inv, __uint_as_float(x[2 * e + 1]) * inv);
        ow[e] = *reinterpret_cast<const uint32_t*>(&h2);
      }
      return o;
    };
    if (ONE && qb * kBQ + warp * 32 + 32 > seq_len) {
      // the warp's rows end with the sequence, as most do where sequences are this short: a lane stores its row (300
      // sequences of 30 tokens x 32 heads: 159 us through shared memory, so 139; where all 32 rows are there, 40 x 128 tokens, 39.8 and 37.6)
      __half* dst = p.out + static_cast<long long>(seq_start + q_pos) * p.out_stride + h * kD;
#pragma unroll 1
      for (int c = 0; c < kD / 32; ++c) {
        tmem_ld_32x32b_x32(t_o + c * 32, r[0]);
        tmem_wait_ld();
        if (q_pos < seq_len) {
#pragma unroll
          for (int v = 0; v < 4; ++v) *reinterpret_cast<uint4*>(dst + c * 32 + v * 8) = eight(r[0] + v * 8);
        }
      }
    } else {
      // through shared memory (every product has retired: the K and V buffers are free), so that half a warp stores a whole row; a lane per row touched 32
      // lines with every store
      constexpr int kPitch = kD * 2 + 16;
      uint8_t* mine = smem + kOffK + warp * 32 * kPitch;
      static_assert(4 * 32 * kPitch <= kOffBar - kOffK, "the rows fit the K and V buffers");
#pragma unroll 1
      for (int c = 0; c < kD / 32; c += 2) {
        fetch(r, t_o + c * 32);
        tmem_wait_ld();
#pragma unroll
        for (int v = 0; v < 8; ++v) *reinterpret_cast<uint4*>(mine + lane * kPitch + c * 64 + v * 16) = eight(r[v >> 2] + (v & 3) * 8);
      }
      __syncwarp();
      const int pos0 = qb * kBQ + warp * 32 + (lane >> 4);
      __half* dst = p.out + static_cast<long long>(seq_start + pos0) * p.out_stride + h * kD + (lane & 15) * 8;
#pragma unroll 8
      for (int k = 0; k < 32; k += 2)
        if (pos0 + k < seq_len)
          *reinterpret_cast<uint4*>(dst + static_cast<long long>(k) * p.out_stride) = *reinterpret_cast<const uint4*>(mine + (k + (lane >> 4)) * kPitch + (lane & 15) * 16);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc<kTmemCols>(tmem_s);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

PFN_encodeTiled get_encode() {
  static PFN_encodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && p) fn = reinterpret_cast<PFN_encodeTiled>(p);
  });
  return fn;
}

// fp16 [rows, cols] with a row pitch of `stride` elements; box = 64 columns (128 B, swizzled) x box_rows rows
int make_tmap_f16(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t stride, uint32_t box_rows) {
  PFN_encodeTiled enc = get_encode();
  if (!enc) return set_error(QS_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {stride * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(QS_ERR_CUDA, "cuTensorMapEncodeTiled(f16) failed (%d): ptr=%p rows=%llu cols=%llu stride=%llu", (int)r, ptr, (unsigned long long)rows,
                     (unsigned long long)cols, (unsigned long long)stride);
  return QS_OK;
}

}  // namespace

int prefill_attention(const PrefillAttnArgs& a) {
  QS_REQUIRE(a.head_dim == kD, "prefill_attention: head_dim=%d (only 128 is built, as in the reference)", a.head_dim);
  QS_REQUIRE(a.num_heads > 0 && a.num_kv_heads > 0 && a.num_heads % a.num_kv_heads == 0, "prefill_attention: heads=%d kv_heads=%d", a.num_heads, a.num_kv_heads);
  QS_REQUIRE(a.batch >= 0 && a.num_tokens >= 0 && a.max_seqlen >= 0, "prefill_attention: negative size");
  if (a.batch == 0 || a.num_tokens == 0 || a.max_seqlen == 0) return QS_OK;
  QS_REQUIRE(a.batch <= 65535 && a.num_heads <= 65535, "prefill_attention: batch=%d / heads=%d exceed the grid limits", a.batch, a.num_heads);
  QS_REQUIRE(a.q && a.k && a.v && a.out && a.cu_seqlens, "prefill_attention: null pointer");
  QS_REQUIRE(a.q_stride % 8 == 0 && a.k_stride % 8 == 0 && a.v_stride % 8 == 0 && a.out_stride % 8 == 0, "prefill_attention: row strides must be multiples of 8 halfs");
  QS_REQUIRE(((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v) | reinterpret_cast<uintptr_t>(a.out)) & 15) == 0,
             "prefill_attention: q, k, v, out must be 16-byte aligned");
  QS_REQUIRE(a.q_stride >= a.num_heads * kD && a.k_stride >= a.num_kv_heads * kD && a.v_stride >= a.num_kv_heads * kD && a.out_stride >= a.num_heads * kD,
             "prefill_attention: row stride smaller than the row");
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_f16(&tq, a.q, a.num_tokens, static_cast<uint64_t>(a.num_heads) * kD, a.q_stride, kBQ);
  if (rc) return rc;
  rc = make_tmap_f16(&tk, a.k, a.num_tokens, static_cast<uint64_t>(a.num_kv_heads) * kD, a.k_stride, kBKV);
  if (rc) return rc;
  rc = make_tmap_f16(&tv, a.v, a.num_tokens, static_cast<uint64_t>(a.num_kv_heads) * kD, a.v_stride, kBKV);
  if (rc) return rc;
  const bool one = a.max_seqlen <= kBQ;
  auto kern = one ? prefill_attention_kernel<true> : prefill_attention_kernel<false>;
  static bool attr_set[2][kMaxDevices] = {};
  bool& done = attr_set[one ? 1 : 0][device_ordinal()];
  if (!done) {
    rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes), "cudaFuncSetAttribute(prefill attention)");
    if (rc) return rc;
    done = true;
  }
  PrefillAttnParams p{};
  p.cu_seqlens = a.cu_seqlens;
  p.out = static_cast<__half*>(a.out);
  p.out_stride = a.out_stride;
  p.num_heads = a.num_heads;
  p.num_kv_heads = a.num_kv_heads;
  p.scale_log2 = a.softmax_scale * 1.4426950408889634f;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = static_cast<cudaStream_t>(a.stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  constexpr int kMaxZ = 65535;  // (8.4 M tokens)
  for (int left = (a.max_seqlen + kBQ - 1) / kBQ; left > 0; left -= kMaxZ) {
    p.q_blocks = left;
    cfg.gridDim = dim3(a.num_heads, a.batch, left < kMaxZ ? left : kMaxZ);
    rc = check_cuda(cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, p), "prefill attention launch");
    if (rc) return rc;
  }
  return QS_OK;
}

}  // namespace qs
