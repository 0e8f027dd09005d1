// qserve_b200 -- the token-by-token recurrences over heads of 65 to 128 state rows (hybrid_linear.cu and hybrid.cu describe the layers): per head a
// [D, Dv] fp32 state whose columns are independent of one another.
//
//   kScanHeadDecay     S <- decay_h S + g v^T                        o = S^T q
//   kScanChannelGate   S <- v + g (S - v)            (row by row)    o = S^T q
//   kScanChannelDecay  S <- diag(a) S + g v^T                        o = S^T q
//   kScanTokenDecay    S <- a S + g (dt v)^T                         o = S^T q + skip_h v
//   kScanDelta         u = beta (v - a S^T g),  S <- a S + g u^T     o = S^T q
//
// What bounds it.  A step costs three fp32 operations per state element (delta rule: four), 0.30 ms for the 6758 tokens of 64 heads of 128 x 64 at the
// chip's rate, and the state never leaves the registers; all else is overhead of a warp's step: reading q and g from shared memory, summing products over
// the lanes, and waiting.  The scan before this one gave a thread 16 rows of two columns, read q and g for those alone, summed every token by itself and
// waited for it (1.20 ms; delta rule over 16 heads of 128 x 128: 0.99).  Here
//  - a thread holds 16 rows of CPT adjacent columns, 1 to 4 by the number of units,
//  - the arithmetic goes in pairs of rows (fma.rn.f32x2: the rate per element is the same, the issue slots half; in single operations 10 % slower),
//  - the products of two tokens are summed in one tree that halves its values at each level (7 shuffles for 2 tokens x 4 columns in place of 24) and goes on
//    between the steps of the next two; the delta rule reads a token out while the sums of the next one are on their way, and every step's operands are read
//    ahead of it,
//  - units are dealt to the SMs by length (10 to 15 % of the cases below).
// Measured: 0.59 ms (6758 tokens, 64 heads of 128 x 64), delta rule 0.49 (16 heads of 128 x 128).  A warp's instructions other than the arithmetic and the
// register ports they share with it are what is left (340 cycles per step of 64 elements a thread where the arithmetic is 192).
//
// Every variant adds in the same order, which is that of the general kernels in hybrid_linear.cu and hybrid.cu: eight parts of 16 neighbouring rows, in
// each four chains by row mod 4, (0 + 1) + (2 + 3), then a tree over the parts.  The variant is therefore free to follow the step's shape: a result does
// not depend on where a prompt was cut or on what else is in the step.
#include <cuda_bf16.h>
#include <math.h>

#include <algorithm>
#include <atomic>

#include "../../include/qserve_b200.h"
#include "common.cuh"
#include "hybrid_common.cuh"
#include "launch.h"

namespace qs {
namespace {

using namespace hyb;

constexpr int kParts = 8, kRows = 16, kSeg = kRows + 4;  // a part's segment of a staged row vector is padded: the parts hit different banks
constexpr int kVec = kParts * kSeg;                      // floats of a staged row vector
constexpr int kThreads = 128, kSms = 148;  // (the device deals the units by kSms as well: a B200's)

constexpr int scan_vectors(int mode) { return mode == kScanChannelDecay ? 3 : 2; }
// Tokens of a staged chunk, two of which are in shared memory.  A chunk costs its barrier, the wait for its copies and the first token's reads: 6 % of the time where
// two blocks share an SM, 20 % where a block is alone.  us of the layer with 12 / 16 / 24 tokens: state space, 4 x 2048 tokens, 64 heads (4 columns a thread) 691 / 681 /
// 690, 32 heads (2) 417 / 403 / 409, 1 x 2048, 64 heads (1) 341 / 347 / 337; delta rule, 8 heads (1) 393 / 391 / 385, 16 heads (2) 559 / 562 / 577, retention (2) 438 / 447 / 463.
constexpr int scan_chunk(int mode, int cpt) {
  return mode == kScanChannelDecay ? 8 : mode == kScanTokenDecay ? (cpt == 1 ? 24 : 16) : mode == kScanDelta && cpt == 1 ? 24 : 12;
}
constexpr bool scan_numbers(int mode) { return mode == kScanTokenDecay || mode == kScanDelta; }
constexpr int scan_token_floats(int mode, int cpt) { return scan_vectors(mode) * kVec + 16 * cpt + 4; }

// Sums over the parts of N values per lane (lane bits 2 .. 4 are the part), neighbouring parts first.  A level leaves each lane half of its values while
// there are several, so that log2(N) of the part's bits come to say which of the values a lane ends with, and lanes that differ in the other bits end
// with the same.  A level is in two halves, so that work that does not wait for the shuffles can stand between them.
template <int N>
struct Tree {
  float v[N], got[(N + 1) / 2];
  static constexpr int kLevels = N == 8 ? 3 : N == 4 ? 2 : N == 2 ? 1 : 0;
  static constexpr int left(int level) { return level >= kLevels ? 1 : N >> level; }  // values ahead of a level
  template <int L>
  __device__ __forceinline__ void send(int lane) {
    constexpr int n = left(L), bit = 4 << L;
    const bool up = (lane & bit) != 0;
    if constexpr (n == 1) {
      got[0] = __shfl_xor_sync(0xffffffffu, v[0], bit);
    } else {
#pragma unroll
      for (int i = 0; i < n / 2; ++i) {
        const float keep = up ? v[i + n / 2] : v[i], give = up ? v[i] : v[i + n / 2];
        got[i] = __shfl_xor_sync(0xffffffffu, give, bit);
        v[i] = keep;
      }
    }
  }
  template <int L>
  __device__ __forceinline__ void take() {
    constexpr int n = left(L);
#pragma unroll
    for (int i = 0; i < (n + 1) / 2; ++i) v[i] += got[i];
  }
  __device__ __forceinline__ float sum(int lane) {
    send<0>(lane); take<0>(); send<1>(lane); take<1>(); send<2>(lane); take<2>();
    return v[0];
  }
  // which of the N values the lane ends with; `store`: the lane is the first of those that end with it
  __device__ __forceinline__ static int index(int lane, bool& store) {
    int idx = 0;
#pragma unroll
    for (int l = 0; l < kLevels; ++l) idx = idx * 2 + ((lane >> (2 + l)) & 1);
    store = (lane >> (2 + kLevels)) == 0;
    return idx;
  }
};

// Which (entry, head, columns) a block takes.  Blocks go out to the SMs in rounds of one each, so the units are dealt in order of length, every other
// round backwards: an SM that got one of the longest runs gets one of the shortest next.  (Up to 32 entries; with more there are units enough.)
__device__ __forceinline__ void scan_unit(const ScanArgs& p, int lane, int cols, int& e, int& h, int& base) {
  const int groups = (p.Dv + cols - 1) / cols, per = p.H * groups, units = p.E * per, b = blockIdx.x;
  int u = b;
  if (p.E > 1 && p.E <= 32) {
    const int lo = b / kSms * kSms, size = min(kSms, units - lo);
    if (b / kSms & 1) u = lo + size - 1 - (b - lo);
    const int len = lane < p.E ? p.entry_len[lane] : 0;
    int rank = 0;
    for (int i = 0; i < p.E; ++i) {
      const int other = __shfl_sync(0xffffffffu, len, i);
      rank += other > len || (other == len && i < lane);
    }
    e = __ffs(__ballot_sync(0xffffffffu, lane < p.E && rank == u / per)) - 1;
  } else {
    e = u / per;
  }
  const int rest = u % per;
  h = rest / groups;
  base = rest % groups * cols;
}

// One block per (entry, head, 16 CPT columns): warp w has columns 4 w CPT .. of them, lane = 4 part + column group.  Tokens are staged in chunks with
// cp.async into a double buffer: q | g [| a] in padded segments, v of the block's columns, the head's two numbers.
template <int MODE, int CPT>
__global__ void __launch_bounds__(kThreads, CPT == 1 ? 2 : 0) column_scan_kernel(const ScanArgs p) {
  constexpr int NV = scan_vectors(MODE), CH = scan_chunk(MODE, CPT), COLS = 16 * CPT, ROW = scan_token_floats(MODE, CPT), VAL = NV * kVec, NUM = VAL + COLS;
  constexpr bool DELTA = MODE == kScanDelta, TOKEN = MODE == kScanTokenDecay;
  extern __shared__ __align__(16) float sm[];  // [2][CH][ROW]
  const int tid = threadIdx.x, lane = tid & 31, part = lane >> 2;
  int e, h, base;
  scan_unit(p, lane, COLS, e, h, base);
  const int cl = ((tid >> 5) * 4 + (lane & 3)) * CPT, col0 = base + cl;
  const int n = p.entry_len[e], s0 = p.entry_start[e], D = p.D, Dv = p.Dv;
  const bool fresh = p.entry_pos0[e] == 0, live = col0 < Dv;  // Dv is a multiple of 4, CPT divides it
  const float number = p.head_number != nullptr ? p.head_number[h] : 0.f;  // kScanHeadDecay: the decay, kScanTokenDecay: the skip factor
  float* Sg = p.state + ((size_t)p.entry_slot[e] * p.H + h) * (size_t)D * Dv + col0;

  // rows part * 16 + 2 j, + 1 of column col0 + c
  f2 S[CPT][kRows / 2];
#pragma unroll
  for (int j = 0; j < kRows / 2; ++j) {
    float x[2][CPT];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = part * kRows + 2 * j + k;
      const bool have = live && !fresh && i < D;
      if constexpr (CPT == 4) {
        const float4 f = have ? *reinterpret_cast<const float4*>(Sg + (size_t)i * Dv) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[k][0] = f.x; x[k][1] = f.y; x[k][2] = f.z; x[k][3] = f.w;
      } else if constexpr (CPT == 2) {
        const float2 f = have ? *reinterpret_cast<const float2*>(Sg + (size_t)i * Dv) : make_float2(0.f, 0.f);
        x[k][0] = f.x; x[k][1] = f.y;
      } else {
        x[k][0] = have ? Sg[(size_t)i * Dv] : 0.f;
      }
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) S[c][j] = pack2(x[0][c], x[1][c]);
  }

  // Staging: a row vector is 32 words of 16 bytes, so a word's place depends on the thread alone.  Places past the head's rows or columns hold zero
  // throughout.
  const float* rows = p.prep + (size_t)s0 * p.row;
  const int gh = h / p.heads_per_vec;
  if (D < kParts * kRows || base + COLS > Dv) {
    for (int i = tid; i < 2 * CH * ROW; i += kThreads) sm[i] = 0.f;
    __syncthreads();
  }
  auto stage = [&](int chunk) {
    const int cnt = min(CH, n - chunk * CH);
    float* buf = sm + (size_t)(chunk & 1) * CH * ROW;
    const float* src = rows + (size_t)chunk * CH * p.row;
    {
      const int w = tid & 31;
      const int dst = (w >> 2) * kSeg + (w & 3) * 4;
      if (w * 4 < D) {
        for (int tk = tid >> 5; tk < cnt; tk += kThreads / 32) {
          const float* r = src + (size_t)tk * p.row + gh * D + w * 4;
          float* b = buf + tk * ROW + dst;
          cp_async16(b, r + p.q);
          cp_async16(b + kVec, r + p.g);
          if (NV == 3) cp_async16(b + 2 * kVec, r + p.a);
        }
      }
    }
    {
      constexpr int W = COLS / 4, PER = kThreads / W;  // words of a token's values, tokens at a time
      const int w = tid % W;
      if (base + w * 4 < Dv)
        for (int tk = tid / W; tk < cnt; tk += PER) cp_async16(buf + tk * ROW + VAL + w * 4, src + (size_t)tk * p.row + p.v + h * Dv + base + w * 4);
    }
    if (scan_numbers(MODE) && tid < 2 * cnt) {
      const int tk = tid >> 1;
      cp_async4(buf + tk * ROW + NUM + (tid & 1), src + (size_t)tk * p.row + ((tid & 1) ? p.n1 : p.n0) + h);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  struct Vec { f2 w[kRows / 2]; };
  auto vec = [&](const float* r, int which) {
    Vec x;
    const ulonglong2* s = reinterpret_cast<const ulonglong2*>(r + which * kVec + part * kSeg);
#pragma unroll
    for (int j = 0; j < kRows / 4; ++j) {
      const ulonglong2 t = s[j];
      x.w[2 * j] = t.x;
      x.w[2 * j + 1] = t.y;
    }
    return x;
  };
  auto values = [&](float (&v)[CPT], const float* r) {
    const float* s = r + VAL + cl;
    if constexpr (CPT == 4) {
      const float4 f = *reinterpret_cast<const float4*>(s);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else if constexpr (CPT == 2) {
      const float2 f = *reinterpret_cast<const float2*>(s);
      v[0] = f.x; v[1] = f.y;
    } else {
      v[0] = s[0];
    }
  };
  // the part's share of every column's product with x
  auto products = [&](const Vec& x, float (&sum)[CPT]) {
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      f2 a = mul2(S[c][0], x.w[0]), b = mul2(S[c][1], x.w[1]);
#pragma unroll
      for (int j = 2; j < kRows / 2; j += 2) {
        a = fma2(S[c][j], x.w[j], a);
        b = fma2(S[c][j + 1], x.w[j + 1], b);
      }
      const float2 s = unpack2(a), t = unpack2(b);
      sum[c] = (s.x + s.y) + (t.x + t.y);
    }
  };
  // what a step needs of a token apart from q
  struct Token { Vec g, a; float v[CPT], n0, n1; };
  auto token = [&](const float* r) {
    Token t;
    t.g = vec(r, 1);
    if constexpr (NV == 3) t.a = vec(r, 2);
    values(t.v, r);
    t.n0 = scan_numbers(MODE) ? r[NUM] : 1.f;
    t.n1 = scan_numbers(MODE) ? r[NUM + 1] : number;
    return t;
  };
  auto update = [&](const Token& t, const float (&x)[CPT]) {  // x: what the token writes, by column
    const f2 decay = pack2(t.n1, t.n1);
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const f2 x2 = pack2(x[c], x[c]), neg = pack2(-x[c], -x[c]);
#pragma unroll
      for (int j = 0; j < kRows / 2; ++j) {
        if constexpr (MODE == kScanChannelGate) S[c][j] = fma2(t.g.w[j], add2(S[c][j], neg), x2);
        else S[c][j] = fma2(S[c][j], MODE == kScanChannelDecay ? t.a.w[j] : decay, mul2(t.g.w[j], x2));
      }
    }
  };
  auto step = [&](const Token& t) {
    float x[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) x[c] = TOKEN ? t.v[c] * t.n0 : t.v[c];
    update(t, x);
  };
  float* out = p.o_raw + (size_t)s0 * p.H * Dv + (size_t)h * Dv + base;
  const size_t out_row = (size_t)p.H * Dv;
  using One = Tree<CPT>;
  using Two = Tree<2 * CPT>;  // by column, then token

  const int chunks = (n + CH - 1) / CH;
  stage(0);
  if constexpr (DELTA) {
    bool store;
    const int mine = cl + One::index(lane, store);
    store = store && base + mine < Dv;
    Vec q;  // of the token before
#pragma unroll
    for (int j = 0; j < kRows / 2; ++j) q.w[j] = 0;
    float* dst = out + mine - out_row;
    bool any = false;
    for (int ch = 0; ch < chunks; ++ch) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // the chunk is there for every thread, and every thread has left the buffer that the next one goes to
      if (ch + 1 < chunks) stage(ch + 1);
      const int cnt = min(CH, n - ch * CH);
      const float* r = sm + (size_t)(ch & 1) * CH * ROW;
      Token t = token(r);
#pragma unroll 2
      for (int tk = 0; tk < cnt; ++tk, dst += out_row) {
        float ks[CPT], got[CPT];
        One o;
        auto send = [&](int bit) {
#pragma unroll
          for (int c = 0; c < CPT; ++c) got[c] = __shfl_xor_sync(0xffffffffu, ks[c], bit);
        };
        auto take = [&]() {
#pragma unroll
          for (int c = 0; c < CPT; ++c) ks[c] += got[c];
        };
        products(t.g, ks);
        send(4);
        // while those sums travel: the read-out of the token before
        products(q, o.v);
        take();
        send(8);
        o.template send<0>(lane);
        q = vec(r, 0);
        r += tk + 1 < cnt ? ROW : 0;
        take();
        send(16);
        o.template take<0>();
        o.template send<1>(lane);
        const Token next = token(r);
        take();
        float u[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) u[c] = t.n0 * (t.v[c] - ks[c] * t.n1);
        o.template take<1>();
        o.template send<2>(lane);
        update(t, u);
        o.template take<2>();
        if (any && store) *dst = o.v[0];
        any = true;
        t = next;
      }
    }
    if (n > 0) {
      One o;
      products(q, o.v);
      const float x = o.sum(lane);
      if (store) *dst = x;
    }
  } else {
    bool store;
    const int idx = Two::index(lane, store), mine = cl + (idx >> 1), k = idx & 1;
    store = store && base + mine < Dv;
    float* dst = out + mine + (k - 2) * (ptrdiff_t)out_row;  // of the pair of tokens whose sums are on their way
    Two o;
#pragma unroll
    for (int i = 0; i < 2 * CPT; ++i) o.v[i] = 0.f;
    float pass = 0.f;
    bool any = false;
    for (int ch = 0; ch < chunks; ++ch) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // the chunk is there for every thread, and every thread has left the buffer that the next one goes to
      if (ch + 1 < chunks) stage(ch + 1);
      const int cnt = min(CH, n - ch * CH);
      const float* r = sm + (size_t)(ch & 1) * CH * ROW;
      Token t = token(r);
      int tk = 0;
      for (; tk + 2 <= cnt; tk += 2, dst += 2 * out_row) {
        // the tree of the pair before goes on between the steps of this one
        o.template send<0>(lane);
        step(t);
        const Vec q0 = vec(r, 0);
        const Token t1 = token(r + ROW);
        o.template take<0>();
        o.template send<1>(lane);
        float first[CPT];
        products(q0, first);
        o.template take<1>();
        o.template send<2>(lane);
        step(t1);
        const Vec q1 = vec(r + ROW, 0);
        o.template take<2>();
        if (any && store) *dst = TOKEN ? __fmaf_rn(number, pass, o.v[0]) : o.v[0];
        any = true;
        if (TOKEN) pass = r[k * ROW + VAL + mine];
        r += tk + 2 < cnt ? 2 * ROW : 0;
        t = token(r);
        float second[CPT];
        products(q1, second);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          o.v[2 * c] = first[c];
          o.v[2 * c + 1] = second[c];
        }
      }
      if (tk < cnt) {  // the last token of a run of odd length (a chunk is even)
        step(t);
        const Vec q0 = vec(r, 0);
        One last;
        products(q0, last.v);
        bool store1;
        const int m1 = cl + One::index(lane, store1);
        float x = last.sum(lane);
        if (TOKEN) x = __fmaf_rn(number, r[VAL + m1], x);
        if (store1 && base + m1 < Dv) out[(size_t)(n - 1) * out_row + m1] = x;
      }
    }
    const float x = o.sum(lane);
    if (any && store) *dst = TOKEN ? __fmaf_rn(number, pass, x) : x;
  }

#pragma unroll
  for (int j = 0; j < kRows / 2; ++j) {
    float x[2][CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const float2 f = unpack2(S[c][j]);
      x[0][c] = f.x;
      x[1][c] = f.y;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = part * kRows + 2 * j + k;
      if (!live || i >= D) continue;
      float* dst = Sg + (size_t)i * Dv;
      if constexpr (CPT == 4) *reinterpret_cast<float4*>(dst) = make_float4(x[k][0], x[k][1], x[k][2], x[k][3]);
      else if constexpr (CPT == 2) *reinterpret_cast<float2*>(dst) = make_float2(x[k][0], x[k][1]);
      else dst[0] = x[k][0];
    }
  }
}

template <int MODE, int CPT>
int launch(const ScanArgs& p, cudaStream_t s) {
  constexpr size_t smem = (size_t)2 * scan_chunk(MODE, CPT) * scan_token_floats(MODE, CPT) * sizeof(float);
  static_assert(smem <= 68 * 1024, "three blocks per SM");
  if constexpr (smem > 48 * 1024) {
    static std::atomic<bool> done[kMaxDevices] = {};  // the attribute is a device's own
    std::atomic<bool>& d = done[device_ordinal()];
    if (!d.load(std::memory_order_relaxed)) {
      if (int rc = check_cuda(cudaFuncSetAttribute(column_scan_kernel<MODE, CPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "column scan smem")) return rc;
      d.store(true, std::memory_order_relaxed);
    }
  }
  column_scan_kernel<MODE, CPT><<<p.E * p.H * ((p.Dv + 16 * CPT - 1) / (16 * CPT)), kThreads, smem, s>>>(p);
  return check_cuda(cudaGetLastError(), "hyb column scan");
}

template <int MODE>
int launch_mode(const ScanArgs& p, cudaStream_t s) {
  auto blocks = [&](int cpt) { return (long long)p.E * p.H * ((p.Dv + 16 * cpt - 1) / (16 * cpt)); };
  // The narrowest blocks of which each SM holds two.  A step costs a warp about 140 cycles and 110 more per column of a thread: few units want short
  // steps, many want few instructions per element.  us of the whole layer with 1 / 2 / 4 columns (chunks of 12 tokens), width 2048 unless said: delta rule, 1 x 2048 tokens of
  // width 1024: 355 / 439 / 648, 2 x 1000: 280 / 292 / 396, 4 x 2048: 869 / 771 / 878, 8 x 1000: 838 / 703 / 654; state space, 1 x 2048 of width 1024:
  // 290 / 339 / 502, 2 x 1000: 372 / 312 / 357, 4 x 2048: 1180 / 1105 / 1035.  The delta rule's single tokens take the same rule; the kernel before this one
  // and this one, 16 heads of 128 x 128: 8 tokens 17.1 / 13.7, 64 61.8 / 42.0, 256 210 / 126 (no other width has been measured for them).
  if (blocks(1) <= 2 * kSms) return launch<MODE, 1>(p, s);
  if (blocks(2) <= 2 * kSms) return launch<MODE, 2>(p, s);
  return launch<MODE, 4>(p, s);
}

}  // namespace

bool column_scan_takes(const ScanArgs& p) {
  auto words = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return p.D > 64 && p.D <= kParts * kRows && p.Dv >= 64 && p.D % 4 == 0 && p.Dv % 4 == 0 && p.row % 4 == 0 && p.q % 4 == 0 && p.g % 4 == 0 && p.a % 4 == 0 &&
         p.v % 4 == 0 && words(p.prep) && words(p.state);
}

int column_scan(const ScanArgs& p, int mode, cudaStream_t s) {
  switch (mode) {
    case kScanHeadDecay: return launch_mode<kScanHeadDecay>(p, s);
    case kScanChannelGate: return launch_mode<kScanChannelGate>(p, s);
    case kScanChannelDecay: return launch_mode<kScanChannelDecay>(p, s);
    case kScanTokenDecay: return launch_mode<kScanTokenDecay>(p, s);
    default: return launch_mode<kScanDelta>(p, s);
  }
}

}  // namespace qs
