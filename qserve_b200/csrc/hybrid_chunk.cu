// qserve_b200 -- recurrences over long runs of tokens in chunks of 64 on tcgen05 (hybrid decoders' prompt portions, heads of 128 state rows).
//
//   retention, state space:   S <- a S + g (b v)^T,  o = S^T q [+ skip v]             one decay a per token and head
//   gated delta rule:         S <- a S;  u = b (v - S^T g);  S <- S + g u^T;  o = S^T q   (g the key, b the write strength)
//
// Token by token, a step costs about 900 cycles whatever its arithmetic: the update, a sum over the state's rows through shuffles and the read-out follow
// one another (2048 tokens, 16 delta heads x 4 sequences: 971 us; 64 state space heads: 1177 us).  With S the state ahead of a chunk, gam_t = a_1 .. a_t,
// r(s, t) = a_(s+1) .. a_t and w_s = r(s, 64),
//   o_t = gam_t S^T q_t + sum_(s <= t) P[t][s] u_s,      P[t][s] = r(s, t) (g_s . q_t) [b_s]
//   S  <- gam_64 S + sum_s g_s (w_s u_s)^T
//   u_s = v_s (P and w take b_s);     delta rule: U = T R,  R = b v - b gam S^T g,  T = (I + L)^-1,  L[t][s] = b_t r(s, t) (g_s . g_t) below the diagonal
// so that everything is matrix products.  r is always a product of decays, never a quotient: decays of zero are exact.
//
// fp32 on the tensor cores: every operand enters as three bfloat16 terms (24 mantissa bits) and the six products whose weight is above 2^-26 are summed in
// fp32 accumulators.  Relative error against 64 bits over the same prepared rows, 4 prompts of up to 2048 tokens, 64 heads: o 1.5e-7 (token by token
// 0.6e-7), S 0.75e-7 (0.6e-7); with decays near 1: o 3.0e-7 (1.2e-7), S 2.9e-7 (3.7e-7);
// delta rule, 16 heads: o 1.8e-7 (0.7e-7), S 0.9e-7 (0.5e-7).  A tensor core sum drops bits where a CUDA core rounds, so S
// itself is kept summed by the CUDA cores and only a chunk's addition comes from the tensor cores.  The layer rounds o to 16 bits (2e-3); storage of
// 32 bits keeps the token-by-token scan.  A value that is not finite makes its whole chunk's outputs of that value column not finite.
//
// Kernel 1 (no state, all chunks at once): P (delta rule: P T, and T with its rows times w) of every (chunk, head), fp32, into the chunk's own rows of
// o_raw, which only the head's own block of kernel 2 reads before it writes its outputs there.
// Kernel 2: one block per (entry, 128 value rows: one head of 128 or two of 64), S^T [128 values][128 rows] in tensor memory.
//   8 row warps (thread = value row; two warps share the rows of a tensor memory quarter, half the columns each): add the chunk's products to S and split it
//   into terms, form and store the outputs, split the chunk's values
//   7 operand warps: q, g, v and P (T) rows from global memory -> bfloat16 terms in swizzled shared memory
//   1 warp issues the products
// Chain of a chunk: split S -> S q products -> split values -> update products; the rest runs beside it.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "hybrid_common.cuh"
#include "launch.h"
#include "umma_bf16.cuh"

namespace qs {
namespace {

using namespace hyb;

constexpr int kChunk = 64, kState = 128;
constexpr int kSub = kChunk * 128;           // bytes of a swizzled sub-tile: 64 rows of 64 numbers
constexpr int kPlane = 2 * kSub;             // one term of a [64][128] operand
constexpr int kThreads = 512;                // warps 0 .. 7 rows (two per tensor memory quarter), 8 .. 14 operands, 15 issuer
constexpr int kLongRun = kLongRunTokens;     // shorter runs of a batch stay with the token-by-token scans

// tensor memory columns: S^T fp32; the three terms of S^T (64 columns each), later the chunk's addition to S^T; S q; the products with P per head.  The
// values' three terms (32 columns each) lie behind the addition, the third over the columns of S q that have been read.
constexpr uint32_t kColS = 0, kColT = 128, kColV = 256, kColI = 320, kColA = 384;

// the six products of two operands in three terms, small ones first
__device__ __forceinline__ uint32_t term_a(int i) { return (0x001102u >> (4 * i)) & 3u; }
__device__ __forceinline__ uint32_t term_b(int i) { return (0x010120u >> (4 * i)) & 3u; }

// eight numbers (32 bytes) in one load that keeps no line: with 200 KB of shared memory the SM's L1 holds what is on its way and nothing more, and two
// 16-byte loads would claim every sector twice
__device__ __forceinline__ void load8(float (&x)[8], const float* p) {
  asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7])
               : "l"(p));
}
// eight consecutive numbers of row r, 16-byte word j of 16 -> the three terms' tiles (j >> 3: sub-tile)
__device__ __forceinline__ void store_terms(uint8_t* base, int plane_bytes, int half_bytes, int r, int j, float (&x)[8]) {
  uint8_t* dst = base + (j >> 3) * half_bytes + r * 128 + (((j & 7) ^ (r & 7)) << 4);
  uint4 t;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    t.x = split_bf16x2(x[0], x[1]);
    t.y = split_bf16x2(x[2], x[3]);
    t.z = split_bf16x2(x[4], x[5]);
    t.w = split_bf16x2(x[6], x[7]);
    *reinterpret_cast<uint4*>(dst + k * plane_bytes) = t;
  }
}

// An operand [64][8 << shift] in global memory: rows `row` numbers apart, of which the first `valid` numbers exist; in shared memory its terms are `plane`
// bytes apart and the halves of 64 columns `half`.
struct Operand {
  uint8_t* base;
  const float* src;
  size_t row;
  int plane, half, shift, valid;
  uint64_t *full, *free_;
};
// Rows 0 .. n - 1 as terms, zeros below.  Eight items (256 bytes) of a thread are in flight together, the first eight ahead of the wait for the buffer
// (four: 519 us where eight take 474).  One copy of this code for all operands, and rolled loops in the other warps: with everything unrolled the block's
// 80 KB of instructions did not stay in the instruction cache.
__device__ __forceinline__ void stage_terms(const Operand& o, int n, int tid, int threads, uint32_t parity, int lane) {
  constexpr int N = 8;
  const int items = kChunk << o.shift, mask = (1 << o.shift) - 1;
#pragma unroll 1
  for (int q0 = tid; q0 < items; q0 += N * threads) {
    float x[N][8];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int idx = q0 + q * threads, r = idx >> o.shift, j = (idx & mask) * 8;
#pragma unroll
      for (int k = 0; k < 8; ++k) x[q][k] = 0.f;
      if (r < n && j < o.valid) load8(x[q], o.src + r * o.row + j);
    }
    if (q0 == tid) mbar_wait(o.free_, parity);
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int idx = q0 + q * threads;
      if (idx < items) store_terms(o.base, o.plane, o.half, idx >> o.shift, idx & mask, x[q]);
    }
  }
  fence_proxy_async();
  __syncwarp();
  if (lane == 0) mbar_arrive(o.full);
}

// a warp's products over 64 numbers, two per lane (2 lane, 2 lane + 1): inclusive from the front, exclusive from the back
__device__ __forceinline__ void chunk_products(float a0, float a1, int lane, float (&front)[2], float (&back)[2]) {
  float f = a0 * a1, b = f;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float x = __shfl_up_sync(0xffffffffu, f, o), y = __shfl_down_sync(0xffffffffu, b, o);
    if (lane >= o) f *= x;
    if (lane + o < 32) b *= y;
  }
  const float before = __shfl_up_sync(0xffffffffu, f, 1), after = __shfl_down_sync(0xffffffffu, b, 1);
  front[0] = (lane > 0 ? before : 1.f) * a0;
  front[1] = f;
  back[1] = lane < 31 ? after : 1.f;
  back[0] = back[1] * a1;
}

// decay and write strength of token t of head h
__device__ __forceinline__ float decay_of(const LongScan& p, const float* row, int h) { return p.a_at < 0 ? p.head_num[h] : row[p.a_at + h]; }
__device__ __forceinline__ float strength_of(const LongScan& p, const float* row, int h) { return p.b_at < 0 ? 1.f : row[p.b_at + h]; }

// ---------------------------------------------------------------------------------------------------------------------------------
// kernel 1.  One block per (chunk, vectors g / q shared by a run of heads): the 64 x 64 products g_s . q_t (and g_s . g_t) once, then every head's P (or
// P T and w T) with its own decays.  64 x 64 fp32 products on the CUDA cores, 4 x 4 per thread.
// ---------------------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool find_chunk(const LongScan& p, int E, int idx, int& e, int& c) {
  for (e = 0; e < E; ++e) {
    const int n = p.entry_len[e] >= kLongRun ? (p.entry_len[e] + kChunk - 1) / kChunk : 0;
    if (idx < n) { c = idx; return true; }
    idx -= n;
  }
  return false;
}

constexpr int kPairLd = kChunk + 4;  // floats per row of the transposed operands and of the products in shared memory

template <bool DELTA>
__global__ void __launch_bounds__(256) chunk_pairs_kernel(const LongScan p, int E) {
  extern __shared__ __align__(1024) uint8_t sm[];
  float *gT = reinterpret_cast<float*>(sm), *qT = gT + kState * kPairLd, *prod = qT + kState * kPairLd;  // [128][68] each; prod: g.q [64][68] (, g.g [64][68])
  float* prod2 = prod + kChunk * kPairLd;
  __shared__ float s_a[4][kChunk], s_b[4][kChunk], s_w[DELTA ? 4 : 1][kChunk];
  int e, c;
  if (!find_chunk(p, E, blockIdx.x, e, c)) return;
  const int n = min(kChunk, p.entry_len[e] - c * kChunk), row0 = p.entry_start[e] + c * kChunk, kh = blockIdx.y, tid = threadIdx.x;
  for (int idx = tid; idx < kChunk * kState / 4; idx += 256) {
    const int t = idx & 63, i = (idx >> 6) * 4;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f), q = g;
    if (t < n && i < p.D) {
      const float* r = p.prep + (size_t)(row0 + t) * p.P;
      g = ld4(r + p.g_at + kh * p.D + i);
      q = ld4(r + p.q_at + kh * p.D + i);
    }
    gT[i * kPairLd + t] = g.x; gT[(i + 1) * kPairLd + t] = g.y; gT[(i + 2) * kPairLd + t] = g.z; gT[(i + 3) * kPairLd + t] = g.w;
    qT[i * kPairLd + t] = q.x; qT[(i + 1) * kPairLd + t] = q.y; qT[(i + 2) * kPairLd + t] = q.z; qT[(i + 3) * kPairLd + t] = q.w;
  }
  __syncthreads();
  {
    const int t0 = (tid >> 4) * 4, s0 = (tid & 15) * 4;
    float x[4][4] = {}, y[4][4] = {};
    if (s0 <= t0 + 3) {
      for (int i = 0; i < p.D; ++i) {
        const float4 gs = ld4(gT + i * kPairLd + s0), qt = ld4(qT + i * kPairLd + t0);
        const float a[4] = {qt.x, qt.y, qt.z, qt.w}, b[4] = {gs.x, gs.y, gs.z, gs.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) x[j][k] = fmaf(a[j], b[k], x[j][k]);
        if (DELTA) {
          const float4 gt = ld4(gT + i * kPairLd + t0);
          const float d[4] = {gt.x, gt.y, gt.z, gt.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) y[j][k] = fmaf(d[j], b[k], y[j][k]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      st4(prod + (t0 + j) * kPairLd + s0, make_float4(x[j][0], x[j][1], x[j][2], x[j][3]));
      if (DELTA) st4(prod2 + (t0 + j) * kPairLd + s0, make_float4(y[j][0], y[j][1], y[j][2], y[j][3]));
    }
  }
  // four heads at a time: thread (head, s) walks down its column
  const int hl = tid >> 6, s = tid & 63;
  for (int h0 = 0; h0 < p.head_div; h0 += 4) {
    const int h = kh * p.head_div + h0 + hl;
    const bool on = h0 + hl < p.head_div;
    __syncthreads();
    if (on) {
      const float* r = p.prep + (size_t)(row0 + min(s, n - 1)) * p.P;
      s_a[hl][s] = s < n ? decay_of(p, r, h) : 1.f;
      s_b[hl][s] = s < n ? strength_of(p, r, h) : 0.f;
    }
    __syncthreads();
    float* o = p.o_raw + (size_t)row0 * p.H * p.Dv + (size_t)h * p.Dv + s;
    const size_t step = (size_t)p.H * p.Dv;
    if constexpr (!DELTA) {
      if (on) {
        const float bs = s_b[hl][s];
        float r = 1.f;
        for (int t = 0; t < n; ++t) {
          if (t > s) r *= s_a[hl][t];
          o[t * step] = t >= s ? r * prod[t * kPairLd + s] * bs : 0.f;
        }
      }
    } else {
      // L of this head over gT / qT (free by now), column s; r ends as w_s
      float* L = (hl < 2 ? gT : qT) + (hl & 1) * kChunk * kPairLd;
      if (on) {
        float r = 1.f;
        for (int t = 0; t < kChunk; ++t) {
          if (t > s) r *= s_a[hl][t];
          L[t * kPairLd + s] = t > s && t < n ? s_b[hl][t] * r * prod2[t * kPairLd + s] : 0.f;
        }
        s_w[hl][s] = r;
      }
      __syncthreads();
      // column s of the inverse by forward substitution; every thread of a head reads the same word of L, whose entries from column t on are zero
      float x[kChunk];
      if (on) {
#pragma unroll
        for (int t = 0; t < kChunk; ++t) {
          float acc[4] = {t == s ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int k = 0; k < t; k += 4) {
            const float4 l = ld4(L + t * kPairLd + k);
            acc[0] = fmaf(-l.x, x[k], acc[0]);
            if (k + 1 < t) acc[1] = fmaf(-l.y, x[k + 1], acc[1]);
            if (k + 2 < t) acc[2] = fmaf(-l.z, x[k + 2], acc[2]);
            if (k + 3 < t) acc[3] = fmaf(-l.w, x[k + 3], acc[3]);
          }
          x[t] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        }
#pragma unroll
        for (int t = 0; t < kChunk; ++t)
          if (t < n) o[t * step + kChunk] = s_w[hl][t] * x[t];
      }
      __syncthreads();  // L has been read: P in its place
      if (on) {
        float r = 1.f;
        for (int t = 0; t < kChunk; ++t) {
          if (t > s) r *= s_a[hl][t];
          L[t * kPairLd + s] = t >= s && t < n ? r * prod[t * kPairLd + s] : 0.f;
        }
      }
      __syncthreads();
      if (on) {
        // column s of P T; a row of P ends at the diagonal: sixteen rows at a time take the columns that they can have
#pragma unroll
        for (int t0 = 0; t0 < kChunk; t0 += 16)
#pragma unroll 1
          for (int t = t0; t < min(t0 + 16, n); ++t) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < t0 + 16; k += 4) {
              const float4 l = ld4(L + t * kPairLd + k);
              acc[0] = fmaf(l.x, x[k], acc[0]);
              acc[1] = fmaf(l.y, x[k + 1], acc[1]);
              acc[2] = fmaf(l.z, x[k + 2], acc[2]);
              acc[3] = fmaf(l.w, x[k + 3], acc[3]);
            }
            o[t * step] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
          }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// kernel 2: what the row warps of both forms do with S^T (thread = value row, `half` of the 128 columns)
// ---------------------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void load_state(uint32_t t_row, int half, const float* Sg, const LongScan& p, bool fresh) {
#pragma unroll 1
  for (int d0 = half * 64; d0 < half * 64 + 64; d0 += 32) {
    uint32_t x[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) x[k] = __float_as_uint(!fresh && d0 + k < p.D ? Sg[(size_t)(d0 + k) * p.Dv] : 0.f);
    tmem_st32(t_row + kColS + d0, x);
  }
  tmem_wait_st();
}
__device__ __forceinline__ void store_state(uint32_t t_row, int half, float* Sg, const LongScan& p) {
#pragma unroll 1
  for (int d0 = half * 64; d0 < half * 64 + 64; d0 += 32) {
    uint32_t x[32];
    tmem_ld_32x32b_x32(t_row + kColS + d0, x);
    tmem_wait_ld();
#pragma unroll
    for (int k = 0; k < 32; ++k)
      if (d0 + k < p.D) Sg[(size_t)(d0 + k) * p.Dv] = __uint_as_float(x[k]);
  }
}
// S <- g S + the chunk's addition: the tensor cores' accumulators truncate, so the running state is summed here, rounded to nearest
__device__ __forceinline__ void add_chunk(uint32_t t_row, int half, float g) {
#pragma unroll 1
  for (int d0 = half * 64; d0 < half * 64 + 64; d0 += 32) {
    uint32_t a[32], b[32];
    tmem_ld_32x32b_x32(t_row + kColS + d0, a);
    tmem_ld_32x32b_x32(t_row + kColT + d0, b);
    tmem_wait_ld();
#pragma unroll
    for (int k = 0; k < 32; ++k) a[k] = __float_as_uint(fmaf(g, __uint_as_float(a[k]), __uint_as_float(b[k])));
    tmem_st32(t_row + kColS + d0, a);
  }
  tmem_wait_st();
}
__device__ __forceinline__ void split_state(uint32_t t_row, int half) {
#pragma unroll 1
  for (int d0 = half * 64; d0 < half * 64 + 64; d0 += 32) {
    uint32_t s[32], t[16];
    tmem_ld_32x32b_x32(t_row + kColS + d0, s);
    tmem_wait_ld();
    float y[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) y[k] = __uint_as_float(s[k]);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
      for (int k = 0; k < 16; ++k) t[k] = split_bf16x2(y[2 * k], y[2 * k + 1]);
      tmem_st16(t_row + kColT + q * 64 + d0 / 2, t);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// kernel 2, retention and state space
// ---------------------------------------------------------------------------------------------------------------------------------
template <int HEADS>  // heads per block: 1 of 128 values or 2 of 64
struct LinearSmem {
  static constexpr int kOffQ = 0, kOffG = 3 * kPlane, kOffV = 6 * kPlane, kOffP = 9 * kPlane;  // three terms each; P: [term][head][64][64]
  static constexpr int kOffNum = kOffP + HEADS * 3 * kSub;                                    // per row warp: gam [64], w b [64]
  static constexpr int kOffBar = kOffNum + 8 * 2 * kChunk * 4;
  static constexpr int kBytes = kOffBar + 128;
};

template <int HEADS>
__global__ void __launch_bounds__(kThreads, 1) linear_chunk_kernel(const LongScan p) {
  using SM = LinearSmem<HEADS>;
  extern __shared__ __align__(1024) uint8_t sm[];
  constexpr int DV = 128 / HEADS;
  const int e = blockIdx.x, h0 = blockIdx.y * HEADS, kh = h0 / p.head_div;
  const int len = p.entry_len[e], s0 = p.entry_start[e];
  if (len < kLongRun) return;
  const int n_chunks = (len + kChunk - 1) / kChunk;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SM::kOffBar);
  uint64_t *full = bar, *free_ = bar + 4;                                                                    // operands v, q, g, P in shared memory
  uint64_t *st_full = bar + 8, *i_full = bar + 9, *vt_full = bar + 10, *s_full = bar + 11;                   // tensor memory
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bar + 12);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    const int counts[12] = {3, 2, 2, 3 * HEADS, 1, 1, 1, 1, 8, 1, 8, 1};  // three warps bring every head's P
    for (int i = 0; i < 12; ++i) mbar_init(&bar[i], counts[i]);
    fence_barrier_init();
  }
  if (warp == 15) tmem_alloc<512>(s_tmem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;

  if (warp == 15) {
    if (lane == 0) {
      constexpr uint32_t d_intra = idesc_bf16(128, HEADS * kChunk, 0u, 1u), d_inter = idesc_bf16(128, kChunk, 0u), d_update = idesc_bf16(128, kState, 1u);
      const uint64_t v_desc = desc_mn(smem_u32(sm + SM::kOffV), kSub), p_desc = umma_desc_sw128(smem_u32(sm + SM::kOffP));
      const uint64_t q_desc = umma_desc_sw128(smem_u32(sm + SM::kOffQ)), g_desc = desc_mn(smem_u32(sm + SM::kOffG), kSub);
      for (int c = 0; c < n_chunks; ++c) {
        const uint32_t ph = static_cast<uint32_t>(c) & 1u;
        mbar_wait(&full[0], ph);
        mbar_wait(&full[3], ph);
        tc_fence_after();
        // both heads' P beside each other: a row warp reads its own head's columns
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint64_t a = v_desc + term_a(i) * (kPlane / 16), b = p_desc + term_b(i) * (HEADS * kSub / 16);
#pragma unroll
          for (int ks = 0; ks < kChunk / 16; ++ks) mma_ss(tmem + kColA, a + ks * 128, b + ks * 2, d_intra, (i > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(&free_[0]);
        umma_commit(&free_[3]);
        mbar_wait(&full[1], ph);
        mbar_wait(st_full, ph);
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t a = tmem + kColT + term_a(i) * 64;
          const uint64_t b = q_desc + term_b(i) * (kPlane / 16);
#pragma unroll
          for (int ks = 0; ks < kState / 16; ++ks)
            mma_ts(tmem + kColI, a + ks * 8, b + ((ks >> 2) * kSub + (ks & 3) * 32) / 16, d_inter, (i > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(&free_[1]);
        umma_commit(i_full);
        mbar_wait(&full[2], ph);
        mbar_wait(vt_full, ph);
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t t = term_a(i), a = tmem + (t == 2 ? kColI : kColV + t * 32), step = t == 2 ? 16 : 8;
          const uint64_t b = g_desc + term_b(i) * (kPlane / 16);
#pragma unroll
          for (int ks = 0; ks < kChunk / 16; ++ks) mma_ts(tmem + kColT, a + ks * step, b + ks * 128, d_update, (i > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(&free_[2]);
        umma_commit(s_full);
      }
    }
  } else if (warp >= 8) {
    // warps 8 .. 10: v, then P of every head; 11, 12: q; 13, 14: g
    const int op = warp < 11 ? 0 : warp < 13 ? 1 : 2, tid = threadIdx.x - (op == 0 ? 256 : op == 1 ? 352 : 416), threads = op == 0 ? 96 : 64;
    const size_t step = (size_t)p.H * p.Dv;
    Operand first{sm + (op == 0 ? SM::kOffV : op == 1 ? SM::kOffQ : SM::kOffG),
                  p.prep + (size_t)s0 * p.P + (op == 0 ? p.v_at + h0 * p.Dv : (op == 1 ? p.q_at : p.g_at) + kh * p.D), (size_t)p.P, kPlane, kSub, 4,
                  op == 0 ? 128 : p.D, &full[op], &free_[op]};
    const Operand pairs{sm + SM::kOffP, p.o_raw + s0 * step + (size_t)h0 * p.Dv, step, HEADS * kSub, kSub, 3, kChunk, &full[3], &free_[3]};
#pragma unroll 1
    for (int i = 0; i < n_chunks * (op == 0 ? 1 + HEADS : 1); ++i) {
      const int c = op == 0 ? i / (1 + HEADS) : i, job = op == 0 ? i - c * (1 + HEADS) : 0;
      Operand o = first;
      o.src += (size_t)c * kChunk * p.P;
      if (job > 0) {
        o = pairs;
        o.src += (size_t)c * kChunk * step + (size_t)(job - 1) * p.Dv;
        o.base += (job - 1) * kSub;
      }
      stage_terms(o, min(kChunk, len - c * kChunk), tid, threads, (static_cast<uint32_t>(c) & 1u) ^ 1u, lane);
    }
  } else {
    const int half = warp >> 2, r = (warp & 3) * 32 + lane, hh = r / DV, h = h0 + hh, v = r % DV;
    const uint32_t t_row = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    float* gam = reinterpret_cast<float*>(sm + SM::kOffNum) + warp * 2 * kChunk;
    float* wb = gam + kChunk;
    float* Sg = p.state + ((size_t)p.entry_slot[e] * p.H + h) * (size_t)p.D * p.Dv + v;
    const bool fresh = p.entry_pos0[e] == 0;
    const float skip = p.skip ? p.head_num[h] : 0.f;
    load_state(t_row, half, Sg, p, fresh);
    float g_all = 1.f;
    for (int c = 0; c < n_chunks; ++c) {
      const uint32_t ph = static_cast<uint32_t>(c) & 1u;
      const int n = min(kChunk, len - c * kChunk);
      const float* rows = p.prep + (size_t)(s0 + c * kChunk) * p.P;
      // ---- the chunk's decays; loads are out before the wait for the state ----
      float f[2], w[2], b[2];
      {
        float a[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int t = 2 * lane + k;
          a[k] = t < n ? decay_of(p, rows + (size_t)t * p.P, h) : 1.f;
          b[k] = t < n ? strength_of(p, rows + (size_t)t * p.P, h) : 0.f;
        }
        chunk_products(a[0], a[1], lane, f, w);
      }
      if (c > 0) {
        mbar_wait(s_full, ph ^ 1u);
        tc_fence_after();
        add_chunk(t_row, half, g_all);
        named_bar_sync(1, 256);  // the terms of S go over the addition, which the other half's warp reads too
      }
      __syncwarp();  // the previous chunk's numbers have been read
      *reinterpret_cast<float2*>(gam + 2 * lane) = make_float2(f[0], f[1]);
      *reinterpret_cast<float2*>(wb + 2 * lane) = make_float2(w[0] * b[0], w[1] * b[1]);
      __syncwarp();
      g_all = gam[kChunk - 1];
      split_state(t_row, half);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(st_full);
      // ---- sixteen tokens at a time: outputs, and w_s b_s x_s in terms (the values are read again, one piece ahead) ----
      const float* xp = rows + (size_t)half * 32 * p.P + p.v_at + h * p.Dv + v;
      float* o = p.o_raw + (size_t)(s0 + c * kChunk + half * 32) * p.H * p.Dv + (size_t)h * p.Dv + v;
      const int step = p.H * p.Dv;
      float next[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) next[k] = half * 32 + k < n ? xp[(size_t)k * p.P] : 0.f;
      mbar_wait(i_full, ph);
      tc_fence_after();
#pragma unroll 1
      for (int t0 = half * 32; t0 < half * 32 + 32; t0 += 16, o += (size_t)16 * step) {
        uint32_t yi[16], ya[16];
        tmem_ld_32x32b_x16(t_row + kColI + t0, yi);
        tmem_ld_32x32b_x16(t_row + kColA + hh * kChunk + t0, ya);
        float x[16], gm[16], ww[16];  // the shared numbers ahead of the stores, which the compiler must take for writers of them
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = next[k];
        xp += (size_t)16 * p.P;
        if ((t0 & 16) == 0) {
#pragma unroll
          for (int k = 0; k < 16; ++k) next[k] = t0 + 16 + k < n ? xp[(size_t)k * p.P] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 16; k += 4) {
          *reinterpret_cast<float4*>(gm + k) = *reinterpret_cast<const float4*>(gam + t0 + k);
          *reinterpret_cast<float4*>(ww + k) = *reinterpret_cast<const float4*>(wb + t0 + k);
        }
        tmem_wait_ld();
        uint32_t hi[8], mid[8], lo[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float y0 = x[2 * k] * ww[2 * k], y1 = x[2 * k + 1] * ww[2 * k + 1];
          hi[k] = split_bf16x2(y0, y1);
          mid[k] = split_bf16x2(y0, y1);
          lo[k] = pack_bf16(y0, y1);
        }
        tmem_st8(t_row + kColV + t0 / 2, hi);
        tmem_st8(t_row + kColV + 32 + t0 / 2, mid);
        tmem_st8(t_row + kColI + t0, lo);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float y = fmaf(skip, x[k], fmaf(gm[k], __uint_as_float(yi[k]), __uint_as_float(ya[k])));
          if (t0 + k < n) o[(size_t)k * step] = y;
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(vt_full);
    }
    mbar_wait(s_full, static_cast<uint32_t>(n_chunks - 1) & 1u);
    tc_fence_after();
    add_chunk(t_row, half, g_all);
    store_state(t_row, half, Sg, p);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 15) tmem_dealloc<512>(tmem);
}

// ---------------------------------------------------------------------------------------------------------------------------------
// kernel 2, gated delta rule: one block per (entry, head of 128 values).  A chunk's chain: split S^T -> [S^T g | S^T q] -> split R -> [R (w T) | R (P T)]
// = [w U | outputs] -> split w U -> addition to S.  g and q, and w T and P T, lie beside each other, so that each product is 128 wide.
// ---------------------------------------------------------------------------------------------------------------------------------
struct DeltaSmem {
  static constexpr int kOffK = 0, kOffT = 6 * kPlane;  // three terms each: [half of 64 numbers][64 g, 64 q rows], then [64 rows of w T, 64 of P T]
  static constexpr int kOffNum = kOffT + 3 * kPlane;   // per row warp: gam [64], b [64]
  static constexpr int kOffBar = kOffNum + 8 * 2 * kChunk * 4;
  static constexpr int kBytes = kOffBar + 128;
};
// tensor memory columns: S^T; its three terms, later (first 128) the chunk's addition; both 128-wide products; three terms of R, later of w U, the first two
// over the third term of S^T
constexpr uint32_t kColProd = 320;
__device__ __forceinline__ uint32_t col_r(uint32_t term) { return term == 2 ? 448u : 256u + term * 32u; }

__global__ void __launch_bounds__(kThreads, 1) delta_chunk_kernel(const LongScan p) {
  using SM = DeltaSmem;
  extern __shared__ __align__(1024) uint8_t sm[];
  const int e = blockIdx.x, h = blockIdx.y, kh = h / p.head_div;
  const int len = p.entry_len[e], s0 = p.entry_start[e];
  if (len < kLongRun) return;
  const int n_chunks = (len + kChunk - 1) / kChunk;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SM::kOffBar);
  uint64_t *full = bar, *free_ = bar + 3;                                                                                        // g, q, w T and P T
  uint64_t *st_full = bar + 6, *d1_full = bar + 7, *r_full = bar + 8, *d2_full = bar + 9, *u_full = bar + 10, *s_full = bar + 11;  // tensor memory
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bar + 12);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    const int counts[12] = {4, 3, 6, 1, 1, 1, 8, 1, 8, 1, 8, 1};
    for (int i = 0; i < 12; ++i) mbar_init(&bar[i], counts[i]);
    fence_barrier_init();
  }
  if (warp == 15) tmem_alloc<512>(s_tmem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;

  if (warp == 15) {
    if (lane == 0) {
      constexpr uint32_t d_wide = idesc_bf16(128, 128, 0u), d_update = idesc_bf16(128, kState, 1u);
      const uint64_t kq_desc = umma_desc_sw128(smem_u32(sm + SM::kOffK)), t_desc = umma_desc_sw128(smem_u32(sm + SM::kOffT));
      const uint64_t g_desc = desc_mn(smem_u32(sm + SM::kOffK), 2 * kSub);
      for (int c = 0; c < n_chunks; ++c) {
        const uint32_t ph = static_cast<uint32_t>(c) & 1u;
        mbar_wait(&full[0], ph);
        mbar_wait(&full[1], ph);
        mbar_wait(st_full, ph);
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t a = tmem + kColT + term_a(i) * 64;
          const uint64_t b = kq_desc + term_b(i) * (2 * kPlane / 16);
#pragma unroll
          for (int ks = 0; ks < kState / 16; ++ks)
            mma_ts(tmem + kColProd, a + ks * 8, b + ((ks >> 2) * 2 * kSub + (ks & 3) * 32) / 16, d_wide, (i > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(&free_[1]);
        umma_commit(d1_full);
        mbar_wait(&full[2], ph);
        mbar_wait(r_full, ph);
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t a = tmem + col_r(term_a(i));
          const uint64_t b = t_desc + term_b(i) * (kPlane / 16);
#pragma unroll
          for (int ks = 0; ks < kChunk / 16; ++ks) mma_ts(tmem + kColProd, a + ks * 8, b + ks * 2, d_wide, (i > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(&free_[2]);
        umma_commit(d2_full);
        mbar_wait(u_full, ph);
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t a = tmem + col_r(term_a(i));
          const uint64_t b = g_desc + term_b(i) * (2 * kPlane / 16);
#pragma unroll
          for (int ks = 0; ks < kChunk / 16; ++ks) mma_ts(tmem + kColT, a + ks * 8, b + ks * 128, d_update, (i > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(&free_[0]);
        umma_commit(s_full);
      }
    }
  } else if (warp >= 8) {
    // warps 8 .. 11: g, which the next chunk needs first and the last product gives back last; 12 .. 14: q, w T, P T
    const bool key = warp < 12;
    const int tid = threadIdx.x - (key ? 256 : 384), threads = key ? 128 : 96;
    const size_t step = (size_t)p.H * p.Dv;
    const Operand rows{sm + SM::kOffK + (key ? 0 : kSub), p.prep + (size_t)s0 * p.P + (key ? p.g_at : p.q_at) + kh * p.D, (size_t)p.P, 2 * kPlane, 2 * kSub, 4,
                       p.D, &full[key ? 0 : 1], &free_[key ? 0 : 1]};
    const Operand pairs{sm + SM::kOffT, p.o_raw + s0 * step + (size_t)h * p.Dv, step, kPlane, kSub, 3, kChunk, &full[2], &free_[2]};
#pragma unroll 1
    for (int i = 0; i < n_chunks * (key ? 1 : 3); ++i) {
      const int c = key ? i : i / 3, job = key ? 0 : i - c * 3;
      Operand o = rows;
      o.src += (size_t)c * kChunk * p.P;
      if (job > 0) {
        o = pairs;
        o.src += (size_t)c * kChunk * step + (job == 1 ? kChunk : 0);
        o.base += (job - 1) * kSub;
      }
      stage_terms(o, min(kChunk, len - c * kChunk), tid, threads, (static_cast<uint32_t>(c) & 1u) ^ 1u, lane);
    }
  } else {
    const int half = warp >> 2, v = (warp & 3) * 32 + lane;
    const uint32_t t_row = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    float* gam = reinterpret_cast<float*>(sm + SM::kOffNum) + warp * 2 * kChunk;
    float* bs = gam + kChunk;
    float* Sg = p.state + ((size_t)p.entry_slot[e] * p.H + h) * (size_t)p.D * p.Dv + v;
    const bool fresh = p.entry_pos0[e] == 0;
    load_state(t_row, half, Sg, p, fresh);
    float g_all = 1.f;
    for (int c = 0; c < n_chunks; ++c) {
      const uint32_t ph = static_cast<uint32_t>(c) & 1u;
      const int n = min(kChunk, len - c * kChunk);
      const float* rows = p.prep + (size_t)(s0 + c * kChunk) * p.P;
      float f[2], b[2];
      {
        float a[2], w[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int t = 2 * lane + k;
          a[k] = t < n ? decay_of(p, rows + (size_t)t * p.P, h) : 1.f;
          b[k] = t < n ? strength_of(p, rows + (size_t)t * p.P, h) : 0.f;
        }
        chunk_products(a[0], a[1], lane, f, w);
      }
      if (c > 0) {
        mbar_wait(s_full, ph ^ 1u);
        tc_fence_after();
        add_chunk(t_row, half, g_all);
        named_bar_sync(1, 256);  // the terms of S go over the addition, which the other half's warp reads too
      }
      __syncwarp();  // the previous chunk's numbers have been read
      *reinterpret_cast<float2*>(gam + 2 * lane) = make_float2(f[0], f[1]);
      *reinterpret_cast<float2*>(bs + 2 * lane) = make_float2(b[0], b[1]);
      __syncwarp();
      g_all = gam[kChunk - 1];
      split_state(t_row, half);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(st_full);
      // ---- R of this warp's 32 tokens in terms; S^T q stays in registers, its columns are the next product's ----
      const int first = half * 32;
      const float* xp = rows + (size_t)first * p.P + p.v_at + h * p.Dv + v;
      float y[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) y[k] = first + k < n ? xp[(size_t)k * p.P] : 0.f;
      mbar_wait(d1_full, ph);
      tc_fence_after();
      {
        uint32_t kS[32], t[16];
        tmem_ld_32x32b_x32(t_row + kColProd + first, kS);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k) y[k] = bs[first + k] * fmaf(-gam[first + k], __uint_as_float(kS[k]), y[k]);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
#pragma unroll
          for (int k = 0; k < 16; ++k) t[k] = split_bf16x2(y[2 * k], y[2 * k + 1]);
          tmem_st16(t_row + col_r(q) + first / 2, t);
        }
      }
      float yq[32];
      {
        uint32_t qS[32];
        tmem_ld_32x32b_x32(t_row + kColProd + kChunk + first, qS);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k) yq[k] = gam[first + k] * __uint_as_float(qS[k]);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(r_full);
      // ---- w U in terms, then the outputs ----
      mbar_wait(d2_full, ph);
      tc_fence_after();
      {
        uint32_t u[32], t[16];
        tmem_ld_32x32b_x32(t_row + kColProd + first, u);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k) y[k] = __uint_as_float(u[k]);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
#pragma unroll
          for (int k = 0; k < 16; ++k) t[k] = split_bf16x2(y[2 * k], y[2 * k + 1]);
          tmem_st16(t_row + col_r(q) + first / 2, t);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(u_full);
      {
        float* o = p.o_raw + (size_t)(s0 + c * kChunk + first) * p.H * p.Dv + (size_t)h * p.Dv + v;
        const int step = p.H * p.Dv;
        uint32_t ou[32];
        tmem_ld_32x32b_x32(t_row + kColProd + kChunk + first, ou);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k)
          if (first + k < n) o[(size_t)k * step] = yq[k] + __uint_as_float(ou[k]);
      }
      tc_fence_before();
    }
    mbar_wait(s_full, static_cast<uint32_t>(n_chunks - 1) & 1u);
    tc_fence_after();
    add_chunk(t_row, half, g_all);
    store_state(t_row, half, Sg, p);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 15) tmem_dealloc<512>(tmem);
}

}  // namespace

// Two heads of 64 values share their q and g; a row's pieces begin on 32-byte words.  Which is faster: token by token a run costs 0.4 us a token, and 5 ns
// a token for every 128 value rows of the batch when those fill the machine; chunks cost 50 us for the second kernel and the wait for the longest chain, and
// 8 us a chunk for every 148 of them.  The host knows the runs' average only.  Measured (whole call, us, token by token / chunks): 16 delta heads of 128 x 128
//   1 x 256 121 / 101, 2 x 128 74 / 83, 4 x 64 59 / 75, 8 x 32 54 / 70, 32 x 32 149 / 128, 32 x 64 275 / 159, 60 single tokens and 2000 1195 / 437,
//   1 x 2048 846 / 363, 4 x about 1500 1279 / 495
// 64 state space heads of 128 x 64
//   1 x 32 31 / 49, 1 x 64 41 / 54, 1 x 128 64 / 64, 32 x 32 197 / 176, 32 x 64 338 / 208, 60 single tokens and 2000 1131 / 400, 1 x 2048 702 / 315,
//   4 x about 1500 1343 / 474
bool long_chunks_supported(const LongScan& p, int T, int E, bool delta) {
  auto al32 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 31) == 0; };
  const bool heads = p.Dv == 128 || (!delta && p.Dv == 64 && p.head_div % 2 == 0);
  if (!(heads && p.D > 64 && p.D <= kState && p.D % 8 == 0 && p.P % 8 == 0 && p.q_at % 8 == 0 && p.g_at % 8 == 0 && p.v_at % 8 == 0 && al32(p.prep) &&
        al32(p.o_raw) && p.H <= 65535 && E > 0 && T / E >= kLongRun))
    return false;
  const long long run = T / E, blocks = static_cast<long long>(E) * p.H * p.Dv / 128;
  const long long tokens_ns = run * std::max(400ll, 5 * blocks), chunks_ns = 50000 + 8000 * ((run + kChunk - 1) / kChunk) * ((blocks + 147) / 148);
  return chunks_ns < tokens_ns;
}

int long_chunks(const LongScan& p, int T, int E, bool delta, cudaStream_t s) {
  const int pairs_smem = (2 * kState + (delta ? 2 : 1) * kChunk) * kPairLd * (int)sizeof(float);
  auto pairs = delta ? chunk_pairs_kernel<true> : chunk_pairs_kernel<false>;
  auto scan = delta ? delta_chunk_kernel : p.Dv == 64 ? linear_chunk_kernel<2> : linear_chunk_kernel<1>;
  const int scan_smem = delta ? DeltaSmem::kBytes : p.Dv == 64 ? LinearSmem<2>::kBytes : LinearSmem<1>::kBytes;
  static bool done[3][kMaxDevices] = {};
  bool& set = done[delta ? 2 : p.Dv == 64][device_ordinal()];
  if (!set) {
    if (int rc = check_cuda(cudaFuncSetAttribute(pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, pairs_smem), "hyb chunk pairs smem")) return rc;
    if (int rc = check_cuda(cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, scan_smem), "hyb chunk scan smem")) return rc;
    set = true;
  }
  pairs<<<dim3(T / kChunk + E, p.H / p.head_div), 256, pairs_smem, s>>>(p, E);
  scan<<<dim3(E, p.H * p.Dv / 128), kThreads, scan_smem, s>>>(p);
  return check_cuda(cudaGetLastError(), "hyb long chunks");
}

}  // namespace qs
