// qserve_b200 -- prompt portions of the hybrid decoders' softmax attention on tcgen05: heads of 128 + 128 numbers, bfloat16 storage, paged cache.
//
// One CTA = one 64-row tile of an entry x TWO query heads that share a key / value head (the 128 rows of the MMA: rows 0 .. 63 the first head's, 64 .. 127
// the second's) x one score map.  Keys are walked in blocks of 64 (a block lies in one page: page sizes are multiples of 64):
//     S = Q K^T      8 x tcgen05.mma 128 x 64 x 16, K as TMA delivers it (128-byte swizzle) and Q laid out alike, fp32 accumulators in tensor memory
//     softmax        4 warps, thread = row: mask, optional cap and distance bias, running maximum and sum in the base-2 domain, fp32
//     O += P V       the fp32 weights enter as three bfloat16 terms (p = hi + mid + lo, 24 mantissa bits), the first two in tensor memory, the last in
//                    shared memory laid out like Q; 3 x 4 x tcgen05.mma 128 x 128 x 16, B = the V block as TMA delivers it ([key][dim]: MN-major)
// S, the two terms and O fill the 256 tensor memory columns of a CTA without sharing any, so the next block's S is computed while this block's softmax goes
// on, and P V while the next softmax does.  O is rescaled only when a row's maximum has grown by more than 2^8 (numerator and denominator share the stale
// maximum).  112 KB of shared memory per CTA: two CTAs per SM.  Two key / value blocks are in flight per CTA.
//
// Why: mma.sync with register fragments left the tensor pipe 51 % busy at 260 TFLOP/s of executed work (keys loaded once per head, 4 warps x 168
// registers).  Both heads of the pair read one copy of K and V here, and the three terms cost issue slots only once.
// Measured: 4 prompts of 1297 .. 2048 tokens, 16 heads, 4 key / value heads, 2 maps: mma.sync 732 us; with all three terms in tensor memory, two of them
// over S, so that the next S waited for P V, 275; with columns of their own 210; with the tiles of all entries in order of length, the queries fetched ahead
// of the set-up and whole rows stored 192.  A step of 64 keys takes a CTA 1.56 us, two CTAs per SM: 0.85 of the tensor pipe's time for its products (S is 64
// wide); a tile's set-up (2.6 us: tables, queries, first keys) and end (2.5) come on top, for 13.6 steps on average.  Eight softmax warps per CTA: 239.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math_constants.h>

#include <mutex>

#include "../../include/qserve_b200.h"
#include "common.cuh"
#include "hybrid_common.cuh"
#include "launch.h"

namespace qs {
namespace {

using namespace hyb;

constexpr int kD = 128, kRows = 64, kKeys = 64;
constexpr int kThreads = 192;                    // warps 0 .. 3 softmax / epilogue, warp 4 TMA, warp 5 tensor memory + MMA issuer
constexpr int kSubQ = 128 * 128, kSubK = kKeys * 128;  // bytes of a swizzled sub-tile: rows of 64 numbers
constexpr int kBlock = 2 * kSubK;                // a K or V block
constexpr int kOffK = 2 * kSubQ, kOffV = kOffK + 2 * kBlock, kOffLo = kOffV + 2 * kBlock, kOffBar = kOffLo + kSubQ;
constexpr int kSmem = kOffBar + 128;
constexpr uint32_t kTmemCols = 256, kColHi = 64, kColMid = 96, kColO = 128;  // S [0, 64) | P hi [64, 96) | P mid [96, 128) | O [128, 256)
constexpr float kGrow = 8.f;                     // base-2 units

__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t m, uint32_t n, uint32_t b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn_major << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u)
      : "memory");
}
// MN-major operand, rows of 64 numbers per K index: column groups of 64 are `lbo` bytes apart, groups of 8 K rows 1024
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, uint32_t lbo) {
  return static_cast<uint64_t>((addr & 0x3FFFF) >> 4) | static_cast<uint64_t>(lbo >> 4) << 16 | static_cast<uint64_t>(1024 >> 4) << 32 |
         static_cast<uint64_t>(1) << 46 | static_cast<uint64_t>(2) << 61;
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
      "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

template <bool EXTRA>  // EXTRA: a score cap and / or a distance bias
__global__ void __launch_bounds__(kThreads, 2) umma_tile_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                                                               const UmmaTiles p) {
  extern __shared__ __align__(1024) uint8_t sm[];
  // the last tiles of the list are the longest (of an entry always, of the list where the caller has sorted it): they go first, all heads of a tile together
  const int tile = p.n_tiles - 1 - static_cast<int>(blockIdx.y), pairs = p.H >> 1;
  const int hp = blockIdx.x % pairs, m = blockIdx.x / pairs, h0 = hp * 2, g = h0 / (p.H / p.G);
  const int e = p.tile_entry[tile], r0 = p.tile_row0[tile];
  const int n_rows = min(kRows, p.entry_len[e] - r0);
  const int tok0 = p.entry_start[e] + r0, qpos0 = p.entry_pos0[e] + r0, last_qpos = qpos0 + n_rows - 1;
  const int first0 = first_key(qpos0, p.chunk, p.window);  // the tile's first row sees furthest back
  const int kt_lo = first0 / kKeys, n_pre = kept_tiles(first0, p.keep, kKeys), n_walk = n_pre + last_qpos / kKeys + 1 - kt_lo;
  auto block_at = [&](int i) { return i < n_pre ? i : kt_lo + i - n_pre; };

  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kOffBar);
  uint64_t *bar_q = bar, *bar_s = bar + 1, *bar_p = bar + 2, *bar_o = bar + 3, *k_full = bar + 4, *k_free = bar + 6, *v_full = bar + 8, *v_free = bar + 10;
  uint64_t* bar_read = bar + 12;  // S has been read
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bar + 13);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    for (int i = 0; i < 13; ++i) mbar_init(&bar[i], i == 0 || i == 2 || i == 12 ? 4 : 1);
    fence_barrier_init();
  }
  if (warp == 5) tmem_alloc<kTmemCols>(s_tmem);
  uint4 queries[16];  // on their way while the first keys are asked for
  if (warp < 4) {
    const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(p.q) + static_cast<long long>(tok0) * p.q_stride + (h0 * p.maps + m) * kD;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int r = (threadIdx.x >> 4) + j * 8, w = threadIdx.x & 15, qr = r & (kRows - 1);
      queries[j] = make_uint4(0u, 0u, 0u, 0u);
      if (qr < n_rows) queries[j] = *reinterpret_cast<const uint4*>(q + qr * p.q_stride + (r >> 6) * p.maps * kD + w * 8);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;

  if (warp == 4) {
    if (lane == 0) {
      const int* bt = p.block_table + static_cast<size_t>(p.entry_slot[e]) * p.max_blocks;
      auto cell = [&](int i) {
        const int pos = block_at(i) * kKeys;
        return bt[pos / p.page] * p.page + pos % p.page;
      };
      int next = cell(0);
      for (int i = 0; i < n_walk; ++i) {
        const int row = next, st = i & 1;
        const uint32_t ph = (static_cast<uint32_t>(i) >> 1) & 1u;
        if (i + 1 < n_walk) next = cell(i + 1);
        uint8_t *kb = sm + kOffK + st * kBlock, *vb = sm + kOffV + st * kBlock;
        mbar_wait(&k_free[st], ph ^ 1u);  // a fresh barrier passes
        mbar_expect_tx(&k_full[st], kBlock);
        for (int c = 0; c < 2; ++c) tma_load_2d(kb + c * kSubK, &map_k, (g * p.maps + m) * kD + c * 64, row, &k_full[st]);
        mbar_wait(&v_free[st], ph ^ 1u);
        mbar_expect_tx(&v_full[st], kBlock);
        for (int c = 0; c < 2; ++c) tma_load_2d(vb + c * kSubK, &map_v, g * kD + c * 64, row, &v_full[st]);
      }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      constexpr uint32_t qk = idesc_bf16(128, kKeys, 0u), pv = idesc_bf16(128, kD, 1u);
      auto scores = [&](int i) {  // S of block i
        const int st = i & 1;
        mbar_wait(&k_full[st], (static_cast<uint32_t>(i) >> 1) & 1u);
        if (i > 0) mbar_wait(bar_read, static_cast<uint32_t>(i - 1) & 1u);
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
          mma_ss(tmem, umma_desc_sw128(smem_u32(sm + (ks >> 2) * kSubQ)) + (ks & 3) * 2,
                 umma_desc_sw128(smem_u32(sm + kOffK + st * kBlock + (ks >> 2) * kSubK)) + (ks & 3) * 2, qk, ks > 0 ? 1u : 0u);
        umma_commit(bar_s);
        umma_commit(&k_free[st]);
      };
      mbar_wait(bar_q, 0);
      scores(0);
      for (int i = 0; i < n_walk; ++i) {
        if (i + 1 < n_walk) scores(i + 1);  // S and P share no columns: while the softmax of block i goes on
        const int st = i & 1;
        mbar_wait(bar_p, static_cast<uint32_t>(i) & 1u);
        mbar_wait(&v_full[st], (static_cast<uint32_t>(i) >> 1) & 1u);
        tc_fence_after();
        auto values = [&](int kk) { return desc_mn(smem_u32(sm + kOffV + st * kBlock + kk * 2048), kSubK); };
        // the small terms first
#pragma unroll
        for (int kk = 0; kk < kKeys / 16; ++kk)
          mma_ss(tmem + kColO, umma_desc_sw128(smem_u32(sm + kOffLo)) + kk * 2, values(kk), pv, (i > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
        for (int t = 1; t >= 0; --t)
#pragma unroll
          for (int kk = 0; kk < kKeys / 16; ++kk) mma_ts(tmem + kColO, tmem + (t ? kColMid : kColHi) + kk * 8, values(kk), pv, 1u);
        umma_commit(&v_free[st]);
        umma_commit(bar_o);
      }
    }
  } else {
    // the queries, into the layout TMA gives the keys.  Not by TMA: a tensor map would have to end at the last token's row, which only the entries' tables
    // on the device tell
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int r = (threadIdx.x >> 4) + j * 8, w = threadIdx.x & 15;
      *reinterpret_cast<uint4*>(sm + (w >> 3) * kSubQ + r * 128 + (((w & 7) ^ (r & 7)) << 4)) = queries[j];
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_q);
    const int row = (warp & 1) * 32 + lane, h = h0 + (warp >> 1);
    const uint32_t t_s = tmem + (static_cast<uint32_t>(warp * 32) << 16), t_o = t_s + kColO;
    const int qpos = qpos0 + row, fk = first_key(qpos, p.chunk, p.window);
    const int warp_pos = qpos0 + (warp & 1) * 32, warp_fk = first_key(min(last_qpos, warp_pos + 31), p.chunk, p.window);  // first row, largest first key
    const float slope2 = EXTRA && p.slopes != nullptr ? p.slopes[h] * 1.4426950408889634f : 0.f;
    // a capped score leaves cap_scores in the base-2 domain already
    const float scale = EXTRA && p.cap_in > 0.f ? 1.f : p.scale_log2;
    // a sink is one more term of the denominator without a value
    float m_used = p.sinks != nullptr ? p.sinks[h] * 1.4426950408889634f : -CUDART_INF_F, l = p.sinks != nullptr ? 1.f : 0.f;
    for (int i = 0; i < n_walk; ++i) {
      const uint32_t ph = static_cast<uint32_t>(i) & 1u;
      const int key0 = block_at(i) * kKeys;
      mbar_wait(bar_s, ph);
      tc_fence_after();
      float s[kKeys / 4][4];
      {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_s, r);
        uint32_t q[32];
        tmem_ld_32x32b_x32(t_s + 32, q);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          s[k >> 2][k & 3] = __uint_as_float(r[k]);
          s[8 + (k >> 2)][k & 3] = __uint_as_float(q[k]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_read);  // the next block's S may follow
      if (EXTRA) {
        if (p.cap_in > 0.f) cap_scores(s, p.cap_in, p.cap_out);
        if (slope2 != 0.f) {
          const float back = static_cast<float>(qpos - key0);  // whole numbers: back - k is exact
#pragma unroll
          for (int k = 0; k < kKeys; ++k) s[k >> 2][k & 3] = s[k >> 2][k & 3] * scale - slope2 * (back - static_cast<float>(k));
        }
      }
      const float sc = EXTRA && slope2 != 0.f ? 1.f : scale;
      if (key0 + kKeys - 1 > warp_pos || key0 < warp_fk) {  // warp-uniform: a block past the warp's first row, or ahead of a row's first key
#pragma unroll
        for (int k = 0; k < kKeys; ++k)
          if (!key_visible(key0 + k, qpos, fk, p.keep)) s[k >> 2][k & 3] = -CUDART_INF_F;
      }
      float top[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int k = 0; k < kKeys; ++k) top[k & 3] = fmaxf(top[k & 3], s[k >> 2][k & 3]);
      const float m_blk = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * sc;  // the scale is positive
      const bool grow = (m_blk - m_used) > kGrow;
      auto retired = [&]() {  // the previous O += P V: O may be rescaled, P overwritten
        if (i > 0) {
          mbar_wait(bar_o, ph ^ 1u);
          tc_fence_after();
        }
      };
      if (__any_sync(0xffffffffu, grow)) {
        retired();
        const float m_new = grow ? m_blk : m_used;
        const float alpha = !grow ? 1.f : m_used == -CUDART_INF_F ? 0.f : fast_exp2(m_used - m_new);
        if (i > 0) {
#pragma unroll 1
          for (int c = 0; c < kD / 32; ++c) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(t_o + c * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
            tmem_st32(t_o + c * 32, o);
          }
        }
        l *= alpha;
        m_used = m_new;
      }
      const float ref = m_used == -CUDART_INF_F ? 0.f : m_used;  // nothing visible yet: every weight is 2^-inf
      uint32_t hi[32], mid[32], lo[32];
      float sum[2] = {0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        float a = fast_exp2(fmaf(s[k >> 1][(k & 1) * 2], sc, -ref)), b = fast_exp2(fmaf(s[k >> 1][(k & 1) * 2 + 1], sc, -ref));
        sum[0] += a;
        sum[1] += b;
        hi[k] = split_bf16x2(a, b);
        mid[k] = split_bf16x2(a, b);
        lo[k] = pack_bf16(a, b);
      }
      l += sum[0] + sum[1];
      retired();
      tmem_st32(t_s + kColHi, hi);
      tmem_st32(t_s + kColMid, mid);
      {
        const int r = threadIdx.x;  // of 128, laid out like the queries
#pragma unroll
        for (int w = 0; w < 8; ++w)
          *reinterpret_cast<uint4*>(sm + kOffLo + r * 128 + ((w ^ (r & 7)) << 4)) = make_uint4(lo[4 * w], lo[4 * w + 1], lo[4 * w + 2], lo[4 * w + 3]);
        fence_proxy_async();
      }
      const int valid = last_qpos - key0 + 1;
      if (valid < kKeys) {  // the walk's last block: cells past the portion's end may hold anything, and 0 x NaN would enter O
        uint8_t* vb = sm + kOffV + (i & 1) * kBlock;
        mbar_wait(&v_full[i & 1], (static_cast<uint32_t>(i) >> 1) & 1u);
        for (int k = threadIdx.x; k < (kKeys - valid) * 16; k += 128)
          *reinterpret_cast<uint4*>(vb + (k >> 3 & 1) * kSubK + (valid + (k >> 4)) * 128 + (k & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p);
    }
    mbar_wait(bar_o, static_cast<uint32_t>(n_walk - 1) & 1u);
    tc_fence_after();
    const float inv = 1.f / l;
    const int row0 = (warp & 1) * 32;
    if (row0 + 32 > n_rows) {
      // the warp's rows end with the portion: a lane stores its row (64 portions of 16 tokens x 16 heads x 2 maps: 35.9 us through shared memory,
      // 33.3 so)
      float* dst = p.a_out + ((static_cast<size_t>(tok0 + row) * p.H + h) * p.maps + m) * kD;
#pragma unroll 1
      for (int c = 0; c < (row0 < n_rows ? kD / 32 : 0); ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_o + c * 32, r);
        tmem_wait_ld();
        if (row < n_rows) {
#pragma unroll
          for (int v = 0; v < 8; ++v)
            *reinterpret_cast<float4*>(dst + c * 32 + v * 4) = make_float4(__uint_as_float(r[v * 4]) * inv, __uint_as_float(r[v * 4 + 1]) * inv,
                                                                           __uint_as_float(r[v * 4 + 2]) * inv, __uint_as_float(r[v * 4 + 3]) * inv);
        }
      }
    } else {
      // Through shared memory (every product has retired: the buffers are free), so that a warp stores whole rows; a lane per row touched 32 lines with every
      // store
      constexpr int kPitch = kD * 4 + 16;
      uint8_t* mine = sm + kOffK + warp * 32 * kPitch;
      static_assert(4 * 32 * kPitch <= kOffBar - kOffK, "the rows fit the key, value and weight buffers");
#pragma unroll 1
      for (int c = 0; c < kD / 32; c += 2) {
        uint32_t r[2][32];
        tmem_ld_32x32b_x32(t_o + c * 32, r[0]);
        tmem_ld_32x32b_x32(t_o + c * 32 + 32, r[1]);
        tmem_wait_ld();
#pragma unroll
        for (int v = 0; v < 16; ++v) {
          const uint32_t* x = &r[v >> 3][(v & 7) * 4];
          *reinterpret_cast<float4*>(mine + lane * kPitch + c * 128 + v * 16) =
              make_float4(__uint_as_float(x[0]) * inv, __uint_as_float(x[1]) * inv, __uint_as_float(x[2]) * inv, __uint_as_float(x[3]) * inv);
        }
      }
      __syncwarp();
      float* dst = p.a_out + ((static_cast<size_t>(tok0 + row0) * p.H + h) * p.maps + m) * kD + lane * 4;
      const size_t step = static_cast<size_t>(p.H) * p.maps * kD;
#pragma unroll 16
      for (int r = 0; r < 32; ++r) *reinterpret_cast<float4*>(dst + r * step) = *reinterpret_cast<const float4*>(mine + r * kPitch + lane * 16);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc<kTmemCols>(tmem);
}

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

PFN_encodeTiled encoder() {
  static PFN_encodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && p) fn = reinterpret_cast<PFN_encodeTiled>(p);
  });
  return fn;
}

// bfloat16 [rows, cols], `stride` elements from row to row; box = 64 columns x 64 rows
int tensor_map(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t stride) {
  PFN_encodeTiled enc = encoder();
  if (!enc) return set_error(QS_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
  cuuint64_t dims[2] = {cols, rows}, strides[1] = {stride * 2};
  cuuint32_t box[2] = {64, 64}, estr[2] = {1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? QS_OK : set_error(QS_ERR_CUDA, "cuTensorMapEncodeTiled(bf16) failed (%d): ptr=%p cols=%llu stride=%llu", (int)r, ptr,
                                               (unsigned long long)cols, (unsigned long long)stride);
}

}  // namespace

// Heads of 128 and 128 numbers (one swizzled pair of sub-tiles each), an even number of query heads per key / value head (they share the MMA's rows), pages
// of whole key blocks, a positive scale (the maximum is taken ahead of it), 16-byte rows.
bool umma_tiles_supported(const UmmaTiles& p, int D, int Dv, float scale) {
  auto al16 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
  return D == kD && Dv == kD && p.G > 0 && p.H % (2 * p.G) == 0 && p.page % kKeys == 0 && scale > 0.f && p.q_stride % 8 == 0 && al16(p.q) && al16(p.kpool) &&
         al16(p.vpool) && al16(p.a_out) && p.n_tiles <= 65535;
}

int umma_tiles(const UmmaTiles& p, cudaStream_t s) {
  CUtensorMap k, v;
  // the pools' extent is not known here: every row that is addressed lies in a page of the block table
  const uint64_t cells = 0x7fffffff;
  int rc = tensor_map(&k, p.kpool, cells, static_cast<uint64_t>(p.G) * p.maps * kD, static_cast<uint64_t>(p.G) * p.maps * kD);
  if (!rc) rc = tensor_map(&v, p.vpool, cells, static_cast<uint64_t>(p.G) * kD, static_cast<uint64_t>(p.G) * kD);
  if (rc) return rc;
  const bool extra = p.cap_in > 0.f || p.slopes != nullptr;
  auto kern = extra ? umma_tile_kernel<true> : umma_tile_kernel<false>;
  static bool done[2][kMaxDevices] = {};
  if (!done[extra][device_ordinal()]) {
    if (int r = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem), "hyb tile attention smem")) return r;
    done[extra][device_ordinal()] = true;
  }
  kern<<<dim3(p.H / 2 * p.maps, p.n_tiles), kThreads, kSmem, s>>>(k, v, p);
  return check_cuda(cudaGetLastError(), "hyb_attention tiles");
}

}  // namespace qs
