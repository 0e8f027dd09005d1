// qserve_b200 -- short causal convolutions over the flat token batch (hybrid decoders): the convolution's inputs of a token come from the rows ahead of
// it, from the sequence's convolution state (fp32 [slots][taps - 1][channels], oldest input first) ahead of a portion, and are zero ahead of the
// sequence.
#pragma once
#include "hybrid_common.cuh"

namespace qs {
namespace hyb {

// The convolution's inputs of one token, channels c .. c + V - 1: `back` tokens before row t.  Inputs ahead of the portion come from the
// convolution state, inputs ahead of the sequence are zero; `in_bias` (may be null) belongs to the inputs.
template <typename ST, int V>
__device__ __forceinline__ void conv_input(float (&x)[V], const ST* __restrict__ in, long long stride, const float* __restrict__ in_bias,
                                           const float* st, int t, int local, int pos, int back, int taps, int C, int c) {
#pragma unroll
  for (int v = 0; v < V; ++v) x[v] = 0.f;
  if (pos - back < 0) return;
  if (local - back >= 0) {
    const ST* p = in + (size_t)(t - back) * stride + c;
    if constexpr (V == 4) {
      const float4 q = ld4(p);
      x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
    } else {
      x[0] = ldf(p);
    }
    if (in_bias != nullptr) {
#pragma unroll
      for (int v = 0; v < V; ++v) x[v] += in_bias[c + v];
    }
  } else {
    const float* p = st + (size_t)(taps - 1 + local - back) * C + c;
#pragma unroll
    for (int v = 0; v < V; ++v) x[v] = p[v];
  }
}

// Convolution of row t at channels c .. c + V - 1 (bias included).  In a step of single tokens the thread is the only reader of its channels'
// state and shifts the token's input in (`shift`); other steps do that in conv_state_kernel afterwards.
template <typename ST, int V>
__device__ __forceinline__ void conv_row(float (&y)[V], const ST* __restrict__ in, long long stride, const float* __restrict__ in_bias, float* st,
                                         const float* __restrict__ w, const float* __restrict__ b, int t, int local, int pos, int taps, int C, int c,
                                         bool shift) {
#pragma unroll
  for (int v = 0; v < V; ++v) y[v] = b != nullptr ? b[c + v] : 0.f;
  for (int j = 0; j < taps; ++j) {
    float x[V];
    conv_input<ST, V>(x, in, stride, in_bias, st, t, local, pos, taps - 1 - j, taps, C, c);
#pragma unroll
    for (int v = 0; v < V; ++v) y[v] += w[(size_t)(c + v) * taps + j] * x[v];
    if (shift && j > 0) {  // input j is slot j - 1 of the next token's state; slot j is read before slot j is written
#pragma unroll
      for (int v = 0; v < V; ++v) st[(size_t)(j - 1) * C + c + v] = x[v];
    }
  }
}

// tables of a walk: convolution states, the batch, channels, taps
struct ConvTables {
  float* state;
  const int *tok_entry, *tok_pos, *entry_start, *entry_slot;
  int C, taps;
};

// The same for a walk over neighbouring rows, `TAPS` known: the channels' weights and the window of inputs stay in registers.
template <typename ST, int V, int TAPS>
struct ConvWalk {
  float w[V][TAPS], b[V], xb[V], x[TAPS][V];
  float* st = nullptr;
  int entry = -1;

  __device__ __forceinline__ ConvWalk(const float* __restrict__ cw, const float* __restrict__ cb, const float* __restrict__ in_bias, int c) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      b[v] = cb != nullptr ? cb[c + v] : 0.f;
      xb[v] = in_bias != nullptr ? in_bias[c + v] : 0.f;
#pragma unroll
      for (int j = 0; j < TAPS; ++j) w[v][j] = cw[(size_t)(c + v) * TAPS + j];
    }
  }
  // row t's own input, ahead of its use
  __device__ __forceinline__ void fetch(float (&q)[V], const ST* __restrict__ in, long long stride, int t, int c) const {
    const ST* p = in + (size_t)t * stride + c;
    if constexpr (V == 4) {
      const float4 f = ld4(p);
      q[0] = f.x; q[1] = f.y; q[2] = f.z; q[3] = f.w;
    } else {
      q[0] = ldf(p);
    }
  }
  __device__ __forceinline__ void row(float (&y)[V], const float (&own)[V], const ST* __restrict__ in, long long stride, const float* __restrict__ in_bias,
                                      const ConvTables& tab, int t, int e, int pos, int c, bool shift) {
    if (e != entry) {
      st = tab.state + (size_t)tab.entry_slot[e] * (TAPS - 1) * tab.C;
      const int local = t - tab.entry_start[e];
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) conv_input<ST, V>(x[j], in, stride, in_bias, st, t, local, pos, TAPS - 1 - j, TAPS, tab.C, c);
      entry = e;
    } else {
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j)
#pragma unroll
        for (int v = 0; v < V; ++v) x[j][v] = x[j + 1][v];
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      x[TAPS - 1][v] = own[v] + xb[v];
      y[v] = b[v];
#pragma unroll
      for (int j = 0; j < TAPS; ++j) y[v] += w[v][j] * x[j][v];
    }
    if (shift) {
#pragma unroll
      for (int j = 1; j < TAPS; ++j)
#pragma unroll
        for (int v = 0; v < V; ++v) st[(size_t)(j - 1) * tab.C + c + v] = x[j][v];
    }
  }
};
// any number of taps
template <typename ST, int V>
struct ConvWalk<ST, V, 0> {
  const float *cw, *cb;
  int taps;
  __device__ __forceinline__ ConvWalk(const float* w, const float* b, int n) : cw(w), cb(b), taps(n) {}
  __device__ __forceinline__ void fetch(float (&)[V], const ST* __restrict__, long long, int, int) const {}
  __device__ __forceinline__ void row(float (&y)[V], const float (&)[V], const ST* __restrict__ in, long long stride, const float* __restrict__ in_bias,
                                      const ConvTables& tab, int t, int e, int pos, int c, bool shift) {
    conv_row<ST, V>(y, in, stride, in_bias, tab.state + (size_t)tab.entry_slot[e] * (taps - 1) * tab.C, cw, cb, t, t - tab.entry_start[e], pos, taps, tab.C, c,
                    shift);
  }
};
template <typename ST, int V, int TAPS>
__device__ __forceinline__ ConvWalk<ST, V, TAPS> conv_walk(const float* w, const float* b, const float* in_bias, int taps, int c) {
  if constexpr (TAPS == 0) return ConvWalk<ST, V, 0>(w, b, taps);
  else return ConvWalk<ST, V, TAPS>(w, b, in_bias, c);
}

// Rows t0 .. t1 - 1 at channels c .. c + V - 1 in order, `use(t, y)` takes each.  The inputs and tables of N rows are fetched together: one at a time,
// every row waited for its own load.  A walk of one row (conv_run) takes N = 1: the other rows' code costs registers (256 rows of 6144 channels: 21 us
// with N = 4, 19 with 1; single tokens of 64 sequences 6.9).  Prompts wait for memory with few warps in flight: the walks of four rows with four taps, which
// take 92 to 96 registers by themselves, ask for six blocks per SM (80 registers; five: 6758 rows of 6144 channels 81 us, six 75, eight spill; the next four
// rows ahead of these: 83 to 99).  The others do not: they need fewer, and where six blocks are asked for the compiler spends up to 85 on them.
template <typename ST, int V, int N = 4, typename Walk, typename Use>
__device__ __forceinline__ void conv_rows(Walk& walk, const ST* __restrict__ in, long long stride, const float* __restrict__ in_bias, const ConvTables& tab,
                                          int t0, int t1, int c, bool shift, Use use) {
  for (int t = t0; t < t1; t += N) {
    int e[N], pos[N];
    float own[N][V];
#pragma unroll
    for (int q = 0; q < N; ++q)
      if (q == 0 || t + q < t1) {
        e[q] = tab.tok_entry[t + q];
        pos[q] = tab.tok_pos[t + q];
        walk.fetch(own[q], in, stride, t + q, c);
      }
#pragma unroll
    for (int q = 0; q < N; ++q)
      if (t + q < t1) {
        float y[V];
        walk.row(y, own[q], in, stride, in_bias, tab, t + q, e[q], pos[q], c, shift);
        use(t + q, y);
      }
  }
}

// tokens a block of a convolution kernel walks: neighbours find each other's rows in the cache once there are blocks enough
inline int conv_run(int T) { return T >= 2048 ? 16 : T >= 512 ? 4 : 1; }

}  // namespace hyb
}  // namespace qs
