// Kernels of the mixers that carry a state of fixed size per request instead of (or beside) cached
// keys: short causal convolutions, decays and step sizes, the recurrence itself, the norm and gate
// that follow it, and the activation of the dense feed-forward.
//
// A step is a packed ragged batch: entry e owns rows cu_seqlens[e] .. cu_seqlens[e + 1] - 1, its
// request sits in slot entry_slot[e] and had entry_start[e] tokens before this step.  State lives in
// one float32 row per slot (`state + slot * state_stride + offset`); a request at position 0 starts
// from zeros whatever the row holds, so a slot needs no clearing when it changes hands.  Everything a
// recurrence consumes (decays, step sizes, gates, unit vectors, the state) is float32 in both engine
// precisions.  The recurrence runs token by token in a fixed order, so a row's result does not depend
// on how the tokens were cut into steps or on what else is in the batch; in 16-bit engines long entries
// are walked in pieces or taken in blocks of tokens (scan_blocks.cu), whose order of sums depends on the entry's length in the
// step and on nothing else in it.
//
// Pointers to what an earlier kernel of the same step wrote (activations, the state) carry no `__restrict__`:
// a load through a const restrict pointer counts as invariant and may be moved above the wait for the
// kernel before (seen: a convolution that read its rows before the product that writes them had finished,
// once its loads no longer depended on anything else).  Weights and the step's uploaded metadata keep it.
#include <type_traits>

#include "common.cuh"
#include "scan_blocks.cuh"

namespace rl {

__device__ __forceinline__ float softplus_f(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }

constexpr int kMaxTaps = 16;

// ------------------------------------------------------------ short causal convolution
// out[t, c] = silu(bias[c] + sum_d taps[c, K - 1 - d] * x[t - d, c]) over the request's own tokens:
// those of this step from the rows of x, the K - 1 before them from the slot's tail (float32,
// [K - 1, C], oldest first), zeros before position 0.  x is columns col0 .. col0 + C - 1 of rows of
// length x_stride.
constexpr int kConvRows = 8;

template <typename T>
__device__ __forceinline__ float2 load_pair(const T* p);
template <>
__device__ __forceinline__ float2 load_pair<float>(const float* p) { return *reinterpret_cast<const float2*>(p); }
template <>
__device__ __forceinline__ float2 load_pair<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}

// Four neighbouring elements as floats, 8 or 16 bytes at once.
__device__ __forceinline__ void load_four(const float* p, float (&v)[4]) {
  const float4 four = *reinterpret_cast<const float4*>(p);
  v[0] = four.x; v[1] = four.y; v[2] = four.z; v[3] = four.w;
}
__device__ __forceinline__ void load_four(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  const float2 lo = __bfloat1622float2(h[0]), hi = __bfloat1622float2(h[1]);
  v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
}
__device__ __forceinline__ void store_four(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store_four(__nv_bfloat16* p, const float (&v)[4]) {
  __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
}

// A thread owns kLanes (1 or 2) neighbouring channels over kConvRows consecutive packed rows and slides the taps'
// window down them, so a row of x is fetched once, not once per tap.  kLanes == 2 wants even C, col0 and x_stride.
// kTaps > 0: the taps' number is known when compiling and the window lives in registers; 0: any number up to kMaxTaps.
template <typename T, int kLanes, int kTaps>
__global__ void causal_conv_silu_kernel(const T* x, int x_stride, int col0,
                                        const float* __restrict__ taps, const float* __restrict__ bias,
                                        const float* state, long long state_stride, int state_off,
                                        float* __restrict__ out, const int* __restrict__ cu_seqlens,
                                        const int* __restrict__ entry_slot, const int* __restrict__ entry_start,
                                        int entries, int tokens, int C, int taps_given, int slots, int* __restrict__ fault,
                                        int act) {
  pdl_trigger();
  const int K = kTaps > 0 ? kTaps : taps_given;
  constexpr int kHeld = kTaps > 0 ? kTaps : kMaxTaps;
  const int groups = C / kLanes, tiles = (tokens + kConvRows - 1) / kConvRows;
  const long long total = static_cast<long long>(tiles) * groups;
  const long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (idx >= total) {
    pdl_wait();
    return;
  }
  const int tile = static_cast<int>(idx / groups), c = static_cast<int>(idx - static_cast<long long>(tile) * groups) * kLanes;
  float w[kLanes][kHeld], b[kLanes];
#pragma unroll
  for (int l = 0; l < kLanes; ++l) {
    b[l] = bias ? bias[c + l] : 0.0f;
#pragma unroll
    for (int d = 0; d < kHeld; ++d)
      if (d < K) w[l][d] = taps[static_cast<size_t>(c + l) * K + d];     // w[K - 1] is the current token's
  }
  const int t0 = tile * kConvRows;
  int e = entry_of(cu_seqlens, entries, t0);
  pdl_wait();
  // this tile's own rows, asked for at once (every row needs its own input, whatever entry it belongs to)
  float own[kLanes][kConvRows];
#pragma unroll
  for (int r = 0; r < kConvRows; ++r) {
    if (t0 + r < tokens) {
      if constexpr (kLanes == 2) {
        const float2 v = load_pair(x + static_cast<size_t>(t0 + r) * x_stride + col0 + c);
        own[0][r] = v.x; own[1][r] = v.y;
      } else {
        own[0][r] = to_float(x[static_cast<size_t>(t0 + r) * x_stride + col0 + c]);
      }
    }
  }
  // the window: hist[d] is the input d rows back (hist[0] the current row's)
  float hist[kLanes][kHeld];
  int filled_for = -1;      // the entry the window was filled for
#pragma unroll
  for (int r = 0; r < kConvRows; ++r) {
    const int t = t0 + r;
    if (t >= tokens) break;
    while (t >= cu_seqlens[e + 1]) ++e;
    const int local = t - cu_seqlens[e], start = entry_start[e];
    if (filled_for != e) {      // first row of this tile that belongs to entry e: fetch the K - 1 inputs before it
      int slot = entry_slot[e];
      if (slot < 0 || slot >= slots) {
        atomicOr(fault, kFaultSlot);
        slot = 0;
      }
      const float* tail = state + slot * state_stride + state_off;
#pragma unroll
      for (int d = 1; d < kHeld; ++d) {
        if (d >= K) break;
        const int at = local - d;
#pragma unroll
        for (int l = 0; l < kLanes; ++l) hist[l][d] = 0.0f;
        if (at >= 0) {
          if constexpr (kLanes == 2) {
            const float2 v = load_pair(x + static_cast<size_t>(t - d) * x_stride + col0 + c);
            hist[0][d] = v.x; hist[1][d] = v.y;
          } else {
            hist[0][d] = to_float(x[static_cast<size_t>(t - d) * x_stride + col0 + c]);
          }
        } else if (start + at >= 0) {
#pragma unroll
          for (int l = 0; l < kLanes; ++l) hist[l][d] = tail[static_cast<size_t>(K - 1 + at) * C + c + l];
        }
      }
      filled_for = e;
    }
#pragma unroll
    for (int l = 0; l < kLanes; ++l) hist[l][0] = own[l][r];
    float acc[kLanes];
#pragma unroll
    for (int l = 0; l < kLanes; ++l) {
      acc[l] = b[l];
#pragma unroll
      for (int d = 0; d < kHeld; ++d)
        if (d < K) acc[l] += w[l][K - 1 - d] * hist[l][d];
      if (act) acc[l] = silu_f(acc[l]);      // act 0: the convolution's plain result
    }
    if constexpr (kLanes == 2) {
      *reinterpret_cast<float2*>(out + static_cast<size_t>(t) * C + c) = make_float2(acc[0], acc[1]);
    } else {
      out[static_cast<size_t>(t) * C + c] = acc[0];
    }
#pragma unroll
    for (int l = 0; l < kLanes; ++l) {
#pragma unroll
      for (int d = kHeld - 1; d > 0; --d)
        if (d < K) hist[l][d] = hist[l][d - 1];
    }
  }
}

// The slot's tail after the step: the last K - 1 inputs of the request, taken from this step's rows
// and, where the step brought fewer, from the old tail.  A thread reads all it needs before it writes.
template <typename T>
__global__ void conv_tail_update_kernel(const T* x, int x_stride, int col0,
                                        float* __restrict__ state, long long state_stride, int state_off,
                                        const int* __restrict__ cu_seqlens, const int* __restrict__ entry_slot,
                                        const int* __restrict__ entry_start, int entries, int C, int K, int slots) {
  pdl_trigger();
  pdl_wait();
  const long long total = static_cast<long long>(entries) * C;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int e = static_cast<int>(idx / C), c = static_cast<int>(idx - static_cast<long long>(e) * C);
    const int slot = entry_slot[e];
    if (slot < 0 || slot >= slots) continue;
    const int first = cu_seqlens[e], length = cu_seqlens[e + 1] - first, start = entry_start[e];
    float* tail = state + slot * state_stride + state_off;
    float fresh[kMaxTaps];
    for (int j = 0; j < K - 1; ++j) {
      const int at = length - (K - 1) + j;      // index among this step's tokens of the request
      float v = 0.0f;
      if (at >= 0) {
        v = to_float(x[static_cast<size_t>(first + at) * x_stride + col0 + c]);
      } else if (start + at >= 0) {
        v = tail[static_cast<size_t>(K - 1 + at) * C + c];
      }
      fresh[j] = v;
    }
    for (int j = 0; j < K - 1; ++j) tail[static_cast<size_t>(j) * C + c] = fresh[j];
  }
}

// ------------------------------------------------------------ activation into float32 rows
// out[t, c] = act(x[t, col0 + c]) as float32 (act 0: the value itself, 1: SiLU): what a mixer without a
// convolution feeds into its recurrence.
template <typename T>
__global__ void activate_rows_kernel(const T* x, int x_stride, int col0, float* __restrict__ out, int tokens, int C,
                                     int act) {
  pdl_trigger();
  pdl_wait();
  const long long total = static_cast<long long>(tokens) * C;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = idx / C;
    const int c = static_cast<int>(idx - t * C);
    const float v = to_float(x[static_cast<size_t>(t) * x_stride + col0 + c]);
    out[idx] = act ? silu_f(v) : v;
  }
}

// The same for rows that can be fetched four columns at a time: four rows a thread, their loads in flight together.  Bound by
// its bytes: 2,048 rows of 12,288, 16 bits in, 32 out, 81 -> 27 us (5.6 TB/s).
constexpr int kActivateRows = 4;
template <typename T>
__global__ void __launch_bounds__(256) activate_rows_wide_kernel(const T* x, int x_stride, int col0, float* out, int tokens, int C,
                                                                 int act) {
  pdl_trigger();
  const int c = (blockIdx.x * 256 + threadIdx.x) * 4, t0 = blockIdx.y * kActivateRows;
  pdl_wait();
  if (c >= C) return;
  float v[kActivateRows][4];
#pragma unroll
  for (int i = 0; i < kActivateRows; ++i)
    if (t0 + i < tokens) load_four(x + static_cast<size_t>(t0 + i) * x_stride + col0 + c, v[i]);
#pragma unroll
  for (int i = 0; i < kActivateRows; ++i) {
    if (t0 + i >= tokens) break;
    if (act) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = silu_f(v[i][j]);
    }
    store_four(out + static_cast<size_t>(t0 + i) * C + c, v[i]);
  }
}

// ------------------------------------------------------------ decays and step sizes
// step[t, c] = softplus(x[t, c] + bias[c]); decay[t, c] = exp(-rate[c / per] * step[t, c]), rate = exp(A_log)
// (taken once when the weights are loaded).  kWide: four columns a thread, 8- and 16-byte accesses.
template <typename T, bool kWide>
__global__ void decay_gate_kernel(const T* x, int x_stride, int col0, const float* __restrict__ rate,
                                  const float* __restrict__ bias, int per, float* __restrict__ decay,
                                  float* __restrict__ step, int tokens, int C) {
  pdl_trigger();
  pdl_wait();
  constexpr int kEach = kWide ? 4 : 1;
  const int per_row = C / kEach;
  const long long total = static_cast<long long>(tokens) * per_row;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(idx / per_row), c = static_cast<int>(idx - static_cast<long long>(t) * per_row) * kEach;
    const T* in = x + static_cast<size_t>(t) * x_stride + col0 + c;
    float raw[kEach], dt[kEach], d[kEach];
    if constexpr (kWide && sizeof(T) == 2) {
      const uint2 packed = *reinterpret_cast<const uint2*>(in);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&packed);
      const float2 lo = __bfloat1622float2(h[0]), hi = __bfloat1622float2(h[1]);
      raw[0] = lo.x; raw[1] = lo.y; raw[2] = hi.x; raw[3] = hi.y;
    } else if constexpr (kWide) {
      const float4 f = *reinterpret_cast<const float4*>(in);
      raw[0] = f.x; raw[1] = f.y; raw[2] = f.z; raw[3] = f.w;
    } else {
      raw[0] = to_float(in[0]);
    }
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
      dt[j] = softplus_f(raw[j] + (bias ? bias[c + j] : 0.0f));
      d[j] = expf(-rate[(c + j) / per] * dt[j]);
    }
    float* to = decay + static_cast<size_t>(t) * C + c;
    if constexpr (kWide) {
      *reinterpret_cast<float4*>(to) = make_float4(d[0], d[1], d[2], d[3]);
      if (step) *reinterpret_cast<float4*>(step + static_cast<size_t>(t) * C + c) = make_float4(dt[0], dt[1], dt[2], dt[3]);
    } else {
      to[0] = d[0];
      if (step) step[static_cast<size_t>(t) * C + c] = dt[0];
    }
  }
}

// ------------------------------------------------------------ decay from a double exponential
// decay[t, c] = exp(-exp(x[t, c] + bias[c])), float32: a decay per token and channel that stays inside (0, 1).
template <typename T>
__global__ void exp_decay_kernel(const T* x, int x_stride, int col0, const float* __restrict__ bias,
                                 float* __restrict__ decay, int tokens, int C) {
  pdl_trigger();
  pdl_wait();
  const long long total = static_cast<long long>(tokens) * C;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = idx / C;
    const int c = static_cast<int>(idx - t * C);
    const float v = to_float(x[static_cast<size_t>(t) * x_stride + col0 + c]) + (bias ? bias[c] : 0.0f);
    decay[idx] = expf(-expf(v));
  }
}

// ------------------------------------------------------------ decay from a low-rank product
// decay[t, c] = sigmoid(bias[c] + sum_r w[c, r] low[t, r]) ^ (1 / tau), taken as exp(-softplus(-z) / tau): the second
// product of a low-rank pair, its bias and the decay in one pass, in float32 from the stored numbers on (z is never
// rounded).  Beside it the mixer's q, k and v columns as float32 rows, which the recurrence reads.  low and the copied
// columns are columns of the same rows x.
// A block takes kDecayTokens rows and kDecayThreads decays or 4 * kDecayThreads copied columns (the later blocks of the
// y dimension); a decay's weight row is read once for its tokens.
constexpr int kDecayThreads = 128;
constexpr int kDecayTokens = 8;
constexpr int kDecayRankStep = 16;      // numbers of a weight row held in registers at a time

template <typename T>
__global__ void __launch_bounds__(kDecayThreads) low_rank_decay_kernel(
    const T* x, int x_stride, int copied, int low_col0, const T* __restrict__ w, int rank, const float* __restrict__ bias,
    float inv_tau, float* rows, int channels, float* decay, int tokens, int decay_blocks, int vector_rows) {
  __shared__ __align__(16) float low[kDecayTokens][kDecayRankStep];
  pdl_trigger();
  const int t0 = blockIdx.x * kDecayTokens, count = min(kDecayTokens, tokens - t0);
  if (static_cast<int>(blockIdx.y) >= decay_blocks) {
    const int c0 = ((blockIdx.y - decay_blocks) * kDecayThreads + threadIdx.x) * 4;
    pdl_wait();
    if (c0 >= copied) return;
    if (vector_rows) {
      // (eight loads in flight, then eight stores)
      float4 v[kDecayTokens];
#pragma unroll
      for (int i = 0; i < kDecayTokens; ++i) {
        if (i >= count) break;
        const T* from = x + static_cast<size_t>(t0 + i) * x_stride + c0;
        if constexpr (sizeof(T) == 2) {
          const uint2 packed = *reinterpret_cast<const uint2*>(from);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&packed);
          const float2 lo = __bfloat1622float2(h[0]), hi = __bfloat1622float2(h[1]);
          v[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
        } else {
          v[i] = *reinterpret_cast<const float4*>(from);
        }
      }
#pragma unroll
      for (int i = 0; i < kDecayTokens; ++i) {
        if (i >= count) break;
        *reinterpret_cast<float4*>(rows + static_cast<size_t>(t0 + i) * copied + c0) = v[i];
      }
      return;
    }
    for (int i = 0; i < count; ++i)
      for (int c = c0; c < min(c0 + 4, copied); ++c)
        rows[static_cast<size_t>(t0 + i) * copied + c] = to_float(x[static_cast<size_t>(t0 + i) * x_stride + c]);
    return;
  }
  const int c = blockIdx.y * kDecayThreads + threadIdx.x;
  const bool mine = c < channels;
  float sum[kDecayTokens];
#pragma unroll
  for (int i = 0; i < kDecayTokens; ++i) sum[i] = mine ? bias[c] : 0.0f;
  bool waited = false;
  for (int r0 = 0; r0 < rank; r0 += kDecayRankStep) {
    const int here = min(kDecayRankStep, rank - r0);
    float wr[kDecayRankStep];
    const T* from = w + static_cast<size_t>(mine ? c : 0) * rank + r0;
    if (here == kDecayRankStep && rank % 8 == 0) {      // rows of whole 16-byte pieces (weights are aligned)
#pragma unroll
      for (int r = 0; r < kDecayRankStep; r += 8) {
        float eight[8];
        load8(from + r, eight);
#pragma unroll
        for (int j = 0; j < 8; ++j) wr[r + j] = eight[j];
      }
    } else {
#pragma unroll
      for (int r = 0; r < kDecayRankStep; ++r) wr[r] = r < here ? to_float(from[r]) : 0.0f;
    }
    if (!waited) {
      pdl_wait();
      waited = true;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < kDecayTokens * kDecayRankStep; idx += kDecayThreads) {
      const int i = idx / kDecayRankStep, r = idx - i * kDecayRankStep;
      low[i][r] = i < count && r < here ? to_float(x[static_cast<size_t>(t0 + i) * x_stride + low_col0 + r0 + r]) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kDecayTokens; ++i) {
      if (i < count) {
#pragma unroll
        for (int r = 0; r < kDecayRankStep; r += 4) {
          const float4 four = *reinterpret_cast<const float4*>(&low[i][r]);
          sum[i] = fmaf(wr[r], four.x, sum[i]);
          sum[i] = fmaf(wr[r + 1], four.y, sum[i]);
          sum[i] = fmaf(wr[r + 2], four.z, sum[i]);
          sum[i] = fmaf(wr[r + 3], four.w, sum[i]);
        }
      }
    }
  }
  if (!mine) return;
#pragma unroll
  for (int i = 0; i < kDecayTokens; ++i)
    if (i < count) decay[static_cast<size_t>(t0 + i) * channels + c] = expf(-softplus_f(-sum[i]) * inv_tau);
}

// ------------------------------------------------------------ tanh of rows, in the rows' own type
// out[i] = tanh(x[i]) in float32, rounded once: the activation between the two halves of a low-rank product.
template <typename T>
__global__ void tanh_rows_kernel(const T* x, T* out, long long total) {
  pdl_trigger();
  pdl_wait();
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x)
    out[idx] = from_float<T>(tanhf(to_float(x[idx])));
}

// ------------------------------------------------------------ blends of a row with the row before it
// out[s][t][c] = x[t][c] + (before[t][c] - x[t][c]) * mu[s][c] for `mixes` vectors mu, float32 arithmetic, one
// rounding at the store; out is `mixes` planes of [tokens, C].  `before` is the request's previous row: row t - 1 of
// the same entry, the slot's kept row (float32) for the entry's first row, zeros at position 0.  The block of an
// entry's first row also brings the kept row up to date (the entry's last row), each thread after it has read
// what it needs; no other block touches the slot's row.
template <typename T>
__global__ void shift_mix_kernel(const T* x, int x_stride, const float* __restrict__ mu, int mixes, T* out,
                                 float* kept, long long kept_stride, int kept_off,
                                 const int* __restrict__ cu_seqlens, const int* __restrict__ entry_slot,
                                 const int* __restrict__ entry_start, int entries, int tokens, int C, int slots,
                                 int* __restrict__ fault) {
  pdl_trigger();
  const int t = blockIdx.x;
  const int e = entry_of(cu_seqlens, entries, t);
  const int first = cu_seqlens[e], last = cu_seqlens[e + 1] - 1;
  int slot = entry_slot[e];
  const bool slot_ok = slot >= 0 && slot < slots;
  if (!slot_ok) {
    if (threadIdx.x == 0) atomicOr(fault, kFaultSlot);
    slot = 0;
  }
  const bool opens = t == first;
  const bool from_kept = opens && entry_start[e] > 0;
  float* kr = kept + slot * kept_stride + kept_off;
  const T* xr = x + static_cast<size_t>(t) * x_stride;
  const T* pr = xr - x_stride;
  const T* lr = x + static_cast<size_t>(last) * x_stride;
  const size_t plane = static_cast<size_t>(tokens) * C;
  pdl_wait();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    const float now = to_float(xr[c]);
    float before = 0.0f;
    if (from_kept) before = kr[c];
    else if (!opens) before = to_float(pr[c]);
    if (opens && slot_ok) kr[c] = to_float(lr[c]);
    const float step = before - now;
    for (int s = 0; s < mixes; ++s)
      out[s * plane + static_cast<size_t>(t) * C + c] = from_float<T>(fmaf(step, mu[static_cast<size_t>(s) * C + c], now));
  }
}

// ------------------------------------------------------------ unit vectors per head, write strengths
// Heads of `dim` floats, `heads` of them side by side from column col0 of a float32 row: each becomes
// x / sqrt(sum(x^2) + eps) times scale_low (heads below `split`) or scale_high.  One warp a head.
// Beside it, sigmoid of `gates` columns of a row of the engine's dtype into a float32 [T, gates].
template <typename T>
__global__ void unit_heads_kernel(float* __restrict__ rows, int stride, int col0, int heads, int dim, float eps,
                                  int split, float scale_low, float scale_high, const T* gate_in,
                                  int gate_stride, int gate_col0, int gates, float* __restrict__ gate_out, int tokens) {
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int t = blockIdx.x;
  if (t >= tokens) return;
  for (int head = warp; head < heads; head += warps) {
    float* v = rows + static_cast<size_t>(t) * stride + col0 + static_cast<size_t>(head) * dim;
    float sum_sq = 0.0f;
    for (int i = lane; i < dim; i += 32) sum_sq += v[i] * v[i];
    sum_sq = warp_sum(sum_sq);
    const float factor = (head < split ? scale_low : scale_high) / sqrtf(sum_sq + eps);
    for (int i = lane; i < dim; i += 32) v[i] *= factor;
  }
  for (int i = threadIdx.x; i < gates; i += blockDim.x)
    gate_out[static_cast<size_t>(t) * gates + i] =
        sigmoid_f(to_float(gate_in[static_cast<size_t>(t) * gate_stride + gate_col0 + i]));
}

// The same with kLanes lanes of a warp per head, four entries a lane, read and written once; blocks behind the heads' form
// the gates.  2,048 tokens, 32 heads of 128: 22.5 -> 17 us.
template <typename T, int kLanes>
__global__ void __launch_bounds__(256) unit_heads_wide_kernel(float* rows, int stride, int col0, int heads, int dim, float eps,
                                                              int split, float scale_low, float scale_high, const T* gate_in,
                                                              int gate_stride, int gate_col0, int gates, float* gate_out,
                                                              int tokens, int head_blocks) {
  pdl_trigger();
  if (static_cast<int>(blockIdx.x) >= head_blocks) {
    const long long idx = (static_cast<long long>(blockIdx.x) - head_blocks) * 256 + threadIdx.x;
    pdl_wait();
    if (idx >= static_cast<long long>(tokens) * gates) return;
    const long long t = idx / gates;
    const int i = static_cast<int>(idx - t * gates);
    gate_out[idx] = sigmoid_f(to_float(gate_in[static_cast<size_t>(t) * gate_stride + gate_col0 + i]));
    return;
  }
  const int lane = threadIdx.x % kLanes;
  const long long index = blockIdx.x * static_cast<long long>(256 / kLanes) + threadIdx.x / kLanes;
  const bool mine = index < static_cast<long long>(tokens) * heads;
  const long long t = mine ? index / heads : 0;
  const int head = mine ? static_cast<int>(index - t * heads) : 0;
  float* p = rows + static_cast<size_t>(t) * stride + col0 + static_cast<size_t>(head) * dim + lane * 4;
  const bool reads = mine && lane * 4 < dim;
  pdl_wait();
  float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (reads) load_four(p, v);
  float sum_sq = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
#pragma unroll
  for (int off = kLanes / 2; off >= 1; off >>= 1) sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, off);
  const float factor = (head < split ? scale_low : scale_high) / sqrtf(sum_sq + eps);
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] *= factor;
  if (reads) store_four(p, v);
}

// ------------------------------------------------------------ rotation for heads without a cache
// in: a row of the engine's dtype with `heads` query heads of `dim` from column q_col0, as many key
// heads from k_col0 and `heads * vdim` values from v_col0.  out (float32): [q | k | v]; q and k with
// their first `rot` entries rotated by position (entry i paired with i + rot / 2, angle = position *
// inv_freq[i], all float32), k times k_scale after the rotation.
template <typename T>
__global__ void rotate_heads_kernel(const T* in, int in_stride, int q_col0, int k_col0, int v_col0,
                                    float* __restrict__ out, const int* __restrict__ positions,
                                    const float* __restrict__ inv_freq, int heads, int dim, int vdim, int rot,
                                    float k_scale, int tokens, int wide) {
  extern __shared__ __align__(16) float angles[];      // cos, then sin, of the token's rot / 2 angles: the same for every head
  pdl_trigger();
  const int t = blockIdx.x;
  const int qk = heads * dim, half = rot >> 1;
  const float pos = static_cast<float>(positions[t]);
  for (int i = threadIdx.x; i < half; i += blockDim.x) sincosf(pos * inv_freq[i], &angles[half + i], &angles[i]);
  pdl_wait();
  __syncthreads();
  const T* row = in + static_cast<size_t>(t) * in_stride;
  float* o = out + static_cast<size_t>(t) * (2 * qk + heads * vdim);
  if (wide) {
    // four neighbouring entries of a head and their partners at once: every input is read once, 8 or 16 bytes at a time
    auto load4 = [](const T* p, float (&v)[4]) {
      if constexpr (sizeof(T) == 2) {
        const uint2 packed = *reinterpret_cast<const uint2*>(p);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&packed);
        const float2 lo = __bfloat1622float2(h[0]), hi = __bfloat1622float2(h[1]);
        v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
      } else {
        const float4 f = *reinterpret_cast<const float4*>(p);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      }
    };
    const int quads_rot = half >> 2, quads_rest = (dim - rot) >> 2, per_head = quads_rot + quads_rest;
    for (int idx = threadIdx.x; idx < 2 * heads * per_head; idx += blockDim.x) {
      const int head2 = idx / per_head, j = idx - head2 * per_head;      // head2: query heads, then key heads
      const bool is_k = head2 >= heads;
      const int head = is_k ? head2 - heads : head2;
      const T* src = row + (is_k ? k_col0 : q_col0) + head * dim;
      float* dst = o + (is_k ? qk : 0) + head * dim;
      const float scale = is_k ? k_scale : 1.0f;
      if (j < quads_rot) {
        const int i = j << 2;
        float x1[4], x2[4];
        load4(src + i, x1);
        load4(src + i + half, x2);
        const float4 c = *reinterpret_cast<const float4*>(angles + i), sn = *reinterpret_cast<const float4*>(angles + half + i);
        const float cs[4] = {c.x, c.y, c.z, c.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
        float o1[4], o2[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          o1[n] = (x1[n] * cs[n] - x2[n] * ss[n]) * scale;
          o2[n] = (x2[n] * cs[n] + x1[n] * ss[n]) * scale;
        }
        *reinterpret_cast<float4*>(dst + i) = make_float4(o1[0], o1[1], o1[2], o1[3]);
        *reinterpret_cast<float4*>(dst + i + half) = make_float4(o2[0], o2[1], o2[2], o2[3]);
      } else {
        const int i = rot + ((j - quads_rot) << 2);
        float v[4];
        load4(src + i, v);
        *reinterpret_cast<float4*>(dst + i) = make_float4(v[0] * scale, v[1] * scale, v[2] * scale, v[3] * scale);
      }
    }
    for (int idx = threadIdx.x * 4; idx < heads * vdim; idx += blockDim.x * 4) {
      float v[4];
      load4(row + v_col0 + idx, v);
      *reinterpret_cast<float4*>(o + 2 * qk + idx) = make_float4(v[0], v[1], v[2], v[3]);
    }
    return;
  }
  for (int idx = threadIdx.x; idx < 2 * qk; idx += blockDim.x) {
    const bool is_k = idx >= qk;
    const int within = is_k ? idx - qk : idx;
    const int i = within % dim;
    const T* src = row + (is_k ? k_col0 : q_col0) + (within - i);
    float v = to_float(src[i]);
    if (i < rot) {
      const int pair = i < half ? i : i - half;
      const float c = angles[pair], sn = angles[half + pair];
      v = i < half ? v * c - to_float(src[i + half]) * sn : v * c + to_float(src[i - half]) * sn;
    }
    o[idx] = is_k ? v * k_scale : v;
  }
  for (int idx = threadIdx.x; idx < heads * vdim; idx += blockDim.x) o[2 * qk + idx] = to_float(row[v_col0 + idx]);
}

// ------------------------------------------------------------ the recurrence
// Per head a state S of dim x vdim floats; per token, in this order:
//   S <- decay * S                  decay: one number per head (mode 0), per token and head (mode 1),
//                                   or per token, head and row of S (mode 2)
//   u = beta * (v - S^T k)          with beta (the delta rule), else u = v_scale * v (v_scale may be null)
//   S <- S + k u^T
//   out = S^T q (+ skip * v)
// With `bonus` (one number per head and row of S) the read-out comes first and the token's own pair enters it
// weighed, before the state decays and takes the pair:
//   out = (S + diag(bonus) k v^T)^T q;   S <- decay * S + k v^T
// Query/key head of head h is h / (heads / kv_heads).
//
// A block owns (entry, head, a tile of columns of S) and walks the entry's tokens in order.
//
// A column of S is shared by kPartners lanes of one warp, a lane holds kRows of its rows in registers (pieces of four,
// kPartners pieces apart) for kCols neighbouring columns; sums over rows run down a lane's rows and then over lanes in a
// fixed tree of exchanges (offsets from kPartners / 2 down), so in a walk a token's result depends on nothing but the tokens
// before it: not on the step it came in, the group of tokens it was walked in, or kCols.  In the slot's row a head's state lies
// column by column (S^T, [vdim][dim]).
//
// What bounds the walk: a token's k, q and row decays are wanted by every column, and shared memory hands a multiprocessor
// 128 bytes a cycle, broadcasts included: with one column a lane the fetches took four times as long as the multiply-adds.
// Then the instructions a token takes (about 90 a warp) with one warp a scheduler to issue them (0.3 a cycle): a walk from
// end to end cannot use the rest of the GPU, so in 16-bit engines long prompts are walked in pieces (below).
// A correction (beta) makes a token wait for the sum over the whole column of the token before it: there a column has
// few lanes with many rows each, since an exchange between lanes waits as long as eight multiply-adds, and prompts are
// walked from end to end (in pieces the state has to go through a matrix per piece, which costs digits) or, where that is
// ahead, taken in blocks of tokens.
// 2,048 tokens, us, before / from end to end / in pieces: 16 heads of 128, fixed decay 432 / 284 / 199; 32 heads of 64, row
// decays 383 / 252 / 140; with a bonus 334 / 258 / 154; 32 heads of 128, fixed, 570 / 398 / 341; with a
// correction, 16 heads of 128, 632 / 571.  64 single tokens: 64 heads of 64, row decays 54 / 31 (4.3 TB/s), 16 heads of
// 128, fixed 53 / 31 (see the kernel).  Root mean square error against 64 bits, 1,300 tokens of 16 heads of 128, before /
// from end to end / in pieces: fixed decays 3.52e-7 / 3.52e-7 / 2.50e-7, row decays 1.836e-7 / 1.838e-7 / 1.806e-7, with a
// correction 1.646e-7 / 1.646e-7; their states 4.06e-7 / 4.06e-7 / 2.18e-7, 1.71e-7 / 1.71e-7 / 1.64e-7, 1.46e-7 / 1.47e-7.
struct ScanArgs {
  const float* q; int q_stride;
  const float* k; int k_stride;
  const float* v; int v_stride;
  const float* decay; int decay_mode;
  const float* beta;
  const float* v_scale;
  const float* skip;
  const float* bonus;   // [heads, dim] or null: the read-out comes before the update and weighs the token's own pair
  float* out; int out_stride;
  float* state; long long state_stride; int state_off;
  const int* cu_seqlens; const int* entry_slot; const int* entry_start;
  int heads, kv_heads, dim, vdim, slots;
  int run;
  int wide_in;      // q, k, v (and row decays) can be fetched 16 bytes at a time
  int* fault;
  int entries;
  int segment;            // 0: a block walks its entry from end to end; else at most so many tokens, from a state of its own
  int from;               // entries of so many tokens and more are cut into pieces, the others walked (0: none is cut)
  float* seg_states;      // [pieces, heads, vdim, dim]: what a piece alone leaves, then what it starts from
  float* seg_decays;      // [pieces, heads, dim]: the product of a piece's decays
  int in_blocks;          // entries of so many tokens and more are taken in blocks of tokens (scan_blocks.cu) and left out here (0: none)
};

// The piece that block `index` owns: of which entry, which one of the entry's, its tokens, its place in the arrays of
// pieces; false behind the last, and for a walk (segment 0) of an entry that is cut.
struct ScanPiece { int entry, number, first, length, of, place; };
__device__ __forceinline__ bool scan_piece(const ScanArgs& a, int index, ScanPiece& s) {
  if (a.segment == 0) {
    s = {index, 0, a.cu_seqlens[index], a.cu_seqlens[index + 1] - a.cu_seqlens[index], 1, 0};
    return (a.from == 0 || s.length < a.from) && (a.in_blocks == 0 || s.length < a.in_blocks);
  }
  int at = 0;
  for (int e = 0; e < a.entries; ++e) {
    const int first = a.cu_seqlens[e], length = a.cu_seqlens[e + 1] - first;
    const int count = length >= a.from ? (length + a.segment - 1) / a.segment : 0;
    if (index < at + count) {
      const int number = index - at, skipped = number * a.segment;
      s = {e, number, first + skipped, min(a.segment, length - skipped), count, index};
      return true;
    }
    at += count;
  }
  return false;
}
// The pieces of entry `e` (none where it is walked) and the place of its first.
__device__ __forceinline__ int scan_pieces_of(const ScanArgs& a, int e, int& place) {
  place = 0;
  int count = 0;
  for (int i = 0; i <= e; ++i) {
    const int length = a.cu_seqlens[i + 1] - a.cu_seqlens[i];
    place += count;
    count = length >= a.from ? (length + a.segment - 1) / a.segment : 0;
  }
  return count;
}

constexpr int kScanThreads = 128, kScanWarps = kScanThreads / 32;
constexpr int kScanPlain = 0, kScanDelta = 1, kScanBonus = 2;

// Two neighbouring rows and their arithmetic, each half rounded by itself: packed into one instruction for the walks, plain
// where what counts is the loads in flight (packed, the register pairs cost the single tokens' kernel 5 to 20 us of 35).
struct PackedPair {
  unsigned long long both;
};
struct PlainPair {
  float x, y;
};
template <typename P>
__device__ __forceinline__ P pair_of(float x, float y) {
  if constexpr (std::is_same_v<P, PlainPair>) {
    return {x, y};
  } else {
    PackedPair out;
    asm("mov.b64 %0, {%1, %2};" : "=l"(out.both) : "f"(x), "f"(y));
    return out;
  }
}
__device__ __forceinline__ float2 pair_halves(PlainPair a) { return make_float2(a.x, a.y); }
__device__ __forceinline__ float2 pair_halves(PackedPair a) {
  float2 out;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(out.x), "=f"(out.y) : "l"(a.both));
  return out;
}
__device__ __forceinline__ PlainPair pair_fma(PlainPair a, PlainPair b, PlainPair c) { return {fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
__device__ __forceinline__ PlainPair pair_mul(PlainPair a, PlainPair b) { return {__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)}; }
__device__ __forceinline__ PlainPair pair_add(PlainPair a, PlainPair b) { return {__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)}; }
__device__ __forceinline__ PackedPair pair_fma(PackedPair a, PackedPair b, PackedPair c) {
  PackedPair out;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(out.both) : "l"(a.both), "l"(b.both), "l"(c.both));
  return out;
}
__device__ __forceinline__ PackedPair pair_mul(PackedPair a, PackedPair b) {
  PackedPair out;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(out.both) : "l"(a.both), "l"(b.both));
  return out;
}
__device__ __forceinline__ PackedPair pair_add(PackedPair a, PackedPair b) {
  PackedPair out;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(out.both) : "l"(a.both), "l"(b.both));
  return out;
}
template <typename P>
__device__ __forceinline__ float pair_sum(P a) {
  const float2 both = pair_halves(a);
  return __fadd_rn(both.x, both.y);
}

__device__ __forceinline__ void copy_async4(float* shared, const float* global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(shared))),
               "l"(global) : "memory");
}
__device__ __forceinline__ void copy_async16(float* shared, const float* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(shared))),
               "l"(global) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }

// The numbers of one token that a lane works with.
template <int kRows, int kCols, bool kRowDecay, typename P>
struct ScanToken {
  P k[kRows / 2], q[kRows / 2], g[kRowDecay ? kRows / 2 : 1];
  float v[kCols];
  float strength;
};

// A lane's share of S and what it does to it, one token at a time.
template <int kRows, int kPartners, int kCols, int kKind, bool kRowDecay, bool kRead, typename P>
struct ScanColumns {
  P S[kCols][kRows / 2];
  P bonus[kKind == kScanBonus ? kRows / 2 : 1];

  __device__ __forceinline__ void take(const ScanToken<kRows, kCols, kRowDecay, P>& t, float decay, bool scaled, float (&o)[kCols]) {
    const P d2 = pair_of<P>(decay, decay);
    if constexpr (kKind == kScanDelta) {
      float seen[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        P sum[2] = {pair_of<P>(0.0f, 0.0f), pair_of<P>(0.0f, 0.0f)};
#pragma unroll
        for (int r = 0; r < kRows / 2; ++r) {
          S[c][r] = pair_mul(S[c][r], kRowDecay ? t.g[r] : d2);
          sum[r & 1] = pair_fma(S[c][r], t.k[r], sum[r & 1]);
        }
        seen[c] = pair_sum(pair_add(sum[0], sum[1]));
      }
#pragma unroll
      for (int off = kPartners / 2; off >= 1; off >>= 1) {
#pragma unroll
        for (int c = 0; c < kCols; ++c) seen[c] += __shfl_xor_sync(0xffffffffu, seen[c], off);
      }
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const float u = t.strength * (t.v[c] - seen[c]);
        const P u2 = pair_of<P>(u, u);
        P sum[2] = {pair_of<P>(0.0f, 0.0f), pair_of<P>(0.0f, 0.0f)};
#pragma unroll
        for (int r = 0; r < kRows / 2; ++r) {
          S[c][r] = pair_fma(t.k[r], u2, S[c][r]);
          if constexpr (kRead) sum[r & 1] = pair_fma(S[c][r], t.q[r], sum[r & 1]);
        }
        if constexpr (kRead) o[c] = pair_sum(pair_add(sum[0], sum[1]));
      }
    } else {
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const float u = scaled ? t.strength * t.v[c] : t.v[c];
        const P u2 = pair_of<P>(u, u);
        // one chain of up to four pairs: a chain's first product is rounded by itself, so two chains would lose digits
        constexpr int kChains = kRows > 8 ? 2 : 1;
        P sum[kChains];
#pragma unroll
        for (int i = 0; i < kChains; ++i) sum[i] = pair_of<P>(0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < kRows / 2; ++r) {
          const P kv = pair_mul(t.k[r], u2);
          if constexpr (kKind == kScanBonus) {
            // read the state as the tokens before left it, the token's own pair weighed by the bonus; then decay and add
            sum[r % kChains] = pair_fma(pair_fma(bonus[r], kv, S[c][r]), t.q[r], sum[r % kChains]);
            S[c][r] = pair_fma(S[c][r], kRowDecay ? t.g[r] : d2, kv);
          } else {
            S[c][r] = pair_fma(S[c][r], kRowDecay ? t.g[r] : d2, kv);
            if constexpr (kRead) sum[r % kChains] = pair_fma(S[c][r], t.q[r], sum[r % kChains]);
          }
        }
        if constexpr (kRead) o[c] = pair_sum(kChains == 2 ? pair_add(sum[0], sum[kChains - 1]) : sum[0]);
      }
    }
  }

  // Column c of the lane's columns at `home`; `left` columns exist.
  __device__ __forceinline__ void load(const float* home, int dim, int part, int left, bool wide) {
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
#pragma unroll
      for (int j = 0; j < kRows / 4; ++j) {
        const int row = (j * kPartners + part) * 4;
        float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (c < left) {
          const float* p = home + static_cast<size_t>(c) * dim + row;
          if (wide) {
            if (row < dim) {
              const float4 four = *reinterpret_cast<const float4*>(p);
              x[0] = four.x; x[1] = four.y; x[2] = four.z; x[3] = four.w;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (row + e < dim) x[e] = p[e];
          }
        }
        S[c][2 * j] = pair_of<P>(x[0], x[1]);
        S[c][2 * j + 1] = pair_of<P>(x[2], x[3]);
      }
    }
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int c = 0; c < kCols; ++c)
#pragma unroll
      for (int r = 0; r < kRows / 2; ++r) S[c][r] = pair_of<P>(0.0f, 0.0f);
  }
  __device__ __forceinline__ void store(float* home, int dim, int part, int left, bool wide) const {
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
      if (c >= left) break;
#pragma unroll
      for (int j = 0; j < kRows / 4; ++j) {
        const int row = (j * kPartners + part) * 4;
        float* p = home + static_cast<size_t>(c) * dim + row;
        const float2 lower = pair_halves(S[c][2 * j]), upper = pair_halves(S[c][2 * j + 1]);
        const float x[4] = {lower.x, lower.y, upper.x, upper.y};
        if (wide) {
          if (row < dim) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (row + e < dim) p[e] = x[e];
        }
      }
    }
  }
};

// Sums kCount values over the kPartners lanes of a column, value i of every lane with value i of the others.  Where there
// are more values than one, each exchange also halves the values a lane keeps: the result is values[0 .. kept - 1], which
// are the sums of values `first` (returned) and up.  The tree is the same for any kCount.
template <int kPartners, int kCount>
__device__ __forceinline__ int scan_sums(float (&values)[kCount], int part) {
  int first = 0;
#pragma unroll
  for (int off = kPartners / 2, count = kCount; off >= 1; off >>= 1) {
    const bool upper = part & off;
    if (count > 1) {
      count >>= 1;
#pragma unroll
      for (int i = 0; i < kCount / 2; ++i) {
        if (i < count) {
          const float keep = upper ? values[i + count] : values[i], send = upper ? values[i] : values[i + count];
          values[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
      first += upper ? count : 0;
    } else {
      values[0] += __shfl_xor_sync(0xffffffffu, values[0], off);
    }
  }
  return first;
}

// Floats of shared memory a token takes.
template <int kRows, int kPartners, int kCols, bool kRowDecay, bool kRead>
__host__ __device__ constexpr int scan_token_floats() {
  return ((kRowDecay ? 2 : 1) + (kRead ? 1 : 0)) * kPartners * kRows + kScanWarps * (32 / kPartners) * kCols + 2;
}

// Walks an entry's tokens; q, k, row decays, v and the per-token numbers of a run of tokens are brought into shared memory
// by asynchronous copies while the run before is walked, and a token's numbers into registers while the one before is taken.
// With `segment` a prompt's tokens are walked in pieces side by side: every piece from zeros without its read-outs
// (kRead false; scan_join_kernel then makes each piece's true start out of them), and again from its true start.
template <int kRows, int kPartners, int kCols, int kKind, bool kRowDecay, bool kRead>
__global__ void __launch_bounds__(kScanThreads) linear_scan_kernel(const ScanArgs a) {
  extern __shared__ __align__(16) float staged[];
  // Its successor is let in only when the walk is over (below): a kernel that waits at its start still holds
  // warp slots, and the walk is bound by its own latencies, which more resident warps do not shorten.
  const int head = blockIdx.y;
  ScanPiece seg;
  // the last piece of an entry is walked once: nothing starts from what it leaves
  if (!scan_piece(a, blockIdx.x, seg) || (!kRead && seg.number == seg.of - 1)) {
    pdl_wait();
    return;
  }
  const int e = seg.entry;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = lane % kPartners;
  constexpr int kSpread = 32 / kPartners;      // groups of kCols columns a warp has
  constexpr int kTile = kScanWarps * kSpread * kCols;
  constexpr int kPadded = kPartners * kRows;
  const int col_in_tile = (warp * kSpread + lane / kPartners) * kCols;
  const int col = blockIdx.z * kTile + col_in_tile;
  const int left = a.vdim - col;      // columns of this lane that exist
  const int kv_head = head / (a.heads / a.kv_heads);

  const int first = seg.first, length = seg.length, start = a.entry_start[e];
  int slot = a.entry_slot[e];
  const bool slot_ok = slot >= 0 && slot < a.slots;
  if (!slot_ok) {
    if (threadIdx.x == 0) atomicOr(a.fault, kFaultSlot);
    slot = 0;
  }
  const size_t in_head = static_cast<size_t>(left > 0 ? col : 0) * a.dim;
  float* home = a.state + slot * a.state_stride + a.state_off + static_cast<size_t>(head) * a.dim * a.vdim + in_head;
  const bool wide = (a.dim & 3) == 0 && (reinterpret_cast<uintptr_t>(home) & 15) == 0;
  const size_t own = (static_cast<size_t>(seg.place) * a.heads + head) * a.dim;      // of this piece in the three arrays

  // two buffers, each: k, q (and row decays) [run][kPadded]; v [run][kTile]; write strength, decay [run]
  const int run = a.run;
  constexpr int kPerToken = scan_token_floats<kRows, kPartners, kCols, kRowDecay, kRead>();
  const int buffer_floats = (run * kPerToken + 3) & ~3;      // both buffers start on 16 bytes
  const float fixed_decay = a.decay_mode == 0 ? a.decay[head] : 1.0f;
  const float skip = a.skip ? a.skip[head] : 0.0f;
  const float* strength = a.beta ? a.beta : a.v_scale;

  auto stage = [&](int base, float* buffer) {
    const int count = min(run, length - base);
    float* sk = buffer;
    float* sq = sk + run * kPadded;
    float* sg = sq + (kRead ? run * kPadded : 0);
    float* sv = sg + (kRowDecay ? run * kPadded : 0);
    float* sbeta = sv + run * kTile;
    float* sdecay = sbeta + run;
    // a row decay that is not one per row is spread over the rows here
    auto spread = [&](size_t t) { return a.decay_mode == 1 ? a.decay[t * a.heads + head] : fixed_decay; };
    if (a.wide_in) {
      constexpr int quads = kPadded / 4, tile_quads = kTile / 4;
      for (int idx = threadIdx.x; idx < count * quads; idx += kScanThreads) {
        const int tt = idx / quads, i = (idx - tt * quads) << 2;
        const size_t t = static_cast<size_t>(first + base + tt);
        const int at = tt * kPadded + i;
        if (i < a.dim) {
          copy_async16(sk + at, a.k + t * a.k_stride + kv_head * a.dim + i);
          if constexpr (kRead) copy_async16(sq + at, a.q + t * a.q_stride + kv_head * a.dim + i);
        } else {
          *reinterpret_cast<float4*>(sk + at) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if constexpr (kRead) *reinterpret_cast<float4*>(sq + at) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        if constexpr (kRowDecay) {
          if (a.decay_mode != 2) {
            const float d = spread(t);
            *reinterpret_cast<float4*>(sg + at) = make_float4(d, d, d, d);
          } else if (i < a.dim) {
            copy_async16(sg + at, a.decay + (t * a.heads + head) * a.dim + i);
          } else {
            *reinterpret_cast<float4*>(sg + at) = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
          }
        }
      }
      for (int idx = threadIdx.x; idx < count * tile_quads; idx += kScanThreads) {
        const int tt = idx / tile_quads, j = (idx - tt * tile_quads) << 2;
        const int c = blockIdx.z * kTile + j;
        float* to = sv + tt * kTile + j;
        if (c < a.vdim) copy_async16(to, a.v + static_cast<size_t>(first + base + tt) * a.v_stride + head * a.vdim + c);
        else *reinterpret_cast<float4*>(to) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    } else {
      for (int idx = threadIdx.x; idx < count * kPadded; idx += kScanThreads) {
        const int tt = idx / kPadded, i = idx - tt * kPadded;
        const size_t t = static_cast<size_t>(first + base + tt);
        if (i < a.dim) {
          copy_async4(sk + idx, a.k + t * a.k_stride + kv_head * a.dim + i);
          if constexpr (kRead) copy_async4(sq + idx, a.q + t * a.q_stride + kv_head * a.dim + i);
        } else {
          sk[idx] = 0.0f;
          if constexpr (kRead) sq[idx] = 0.0f;
        }
        if constexpr (kRowDecay) {
          if (a.decay_mode != 2) sg[idx] = spread(t);
          else if (i < a.dim) copy_async4(sg + idx, a.decay + (t * a.heads + head) * a.dim + i);
          else sg[idx] = 1.0f;
        }
      }
      for (int idx = threadIdx.x; idx < count * kTile; idx += kScanThreads) {
        const int tt = idx / kTile, j = idx - tt * kTile;
        const int c = blockIdx.z * kTile + j;
        if (c < a.vdim) copy_async4(sv + idx, a.v + static_cast<size_t>(first + base + tt) * a.v_stride + head * a.vdim + c);
        else sv[idx] = 0.0f;
      }
    }
    for (int tt = threadIdx.x; tt < count; tt += kScanThreads) {
      const size_t at = static_cast<size_t>(first + base + tt) * a.heads + head;
      if (strength) copy_async4(sbeta + tt, strength + at); else sbeta[tt] = 1.0f;
      if (a.decay_mode == 1) copy_async4(sdecay + tt, a.decay + at); else sdecay[tt] = fixed_decay;
    }
    copy_async_commit();
  };

  pdl_wait();
  if (length > 0) stage(0, staged);
  using P = PackedPair;
  ScanColumns<kRows, kPartners, kCols, kKind, kRowDecay, kRead, P> mine;
  if constexpr (!kRead) {
    mine.clear();
  } else if (seg.of == 1) {
    if (start > 0) mine.load(home, a.dim, part, left, wide); else mine.clear();
  } else if (start > 0 || seg.number > 0) {
    mine.load(a.seg_states + own * a.vdim + in_head, a.dim, part, left, true);
  } else {
    mine.clear();
  }
  // The product of the piece's decays, for the one warp that stores it: two floats a row, product - rest, so that it is
  // rounded once and not at every token (slow decays would lose digits: the state is multiplied by what is left of 1).
  constexpr int kFactors = kRowDecay ? kRows / 2 : 1;
  const bool multiplies = !kRead && blockIdx.z == 0 && warp == 0;
  P product[kFactors], rest[kFactors];
#pragma unroll
  for (int r = 0; r < kFactors; ++r) {
    product[r] = pair_of<P>(1.0f, 1.0f);
    rest[r] = pair_of<P>(0.0f, 0.0f);
  }
  if constexpr (kKind == kScanBonus) {
#pragma unroll
    for (int r = 0; r < kRows / 2; ++r) {
      const int row = ((r / 2) * kPartners + part) * 4 + (r & 1) * 2;
      const float* p = a.bonus + static_cast<size_t>(head) * a.dim + row;
      mine.bonus[r] = pair_of<P>(row < a.dim ? p[0] : 0.0f, row + 1 < a.dim ? p[1] : 0.0f);
    }
  }
  const bool scaled = strength != nullptr;

  int flip = 0;
  for (int base = 0; base < length; base += run, flip ^= 1) {
    const int count = min(run, length - base);
    float* buffer = staged + flip * buffer_floats;
    if (base + run < length) {
      stage(base + run, staged + (flip ^ 1) * buffer_floats);   // the next run, while this one is walked
      copy_async_wait<1>();
    } else {
      copy_async_wait<0>();
    }
    __syncthreads();
    const float* sk = buffer;
    const float* sq = sk + run * kPadded;
    const float* sg = sq + (kRead ? run * kPadded : 0);
    const float* sv = sg + (kRowDecay ? run * kPadded : 0);
    const float* sbeta = sv + run * kTile;
    const float* sdecay = sbeta + run;
    auto fetch = [&](ScanToken<kRows, kCols, kRowDecay, P>& t, int tt) {
      const int at = tt * kPadded + part * 4;
      auto two = [&](const float* from, P& lower, P& upper) {
        const ulonglong2 four = *reinterpret_cast<const ulonglong2*>(from);
        lower.both = four.x;
        upper.both = four.y;
      };
#pragma unroll
      for (int j = 0; j < kRows / 4; ++j) {
        two(sk + at + j * kPartners * 4, t.k[2 * j], t.k[2 * j + 1]);
        if constexpr (kRead) two(sq + at + j * kPartners * 4, t.q[2 * j], t.q[2 * j + 1]);
        if constexpr (kRowDecay) two(sg + at + j * kPartners * 4, t.g[2 * j], t.g[2 * j + 1]);
      }
      const float* pv = sv + tt * kTile + col_in_tile;
      if constexpr (kCols == 4) {
        const float4 v4 = *reinterpret_cast<const float4*>(pv);
        t.v[0] = v4.x; t.v[1] = v4.y; t.v[2] = v4.z; t.v[3] = v4.w;
      } else if constexpr (kCols == 2) {
        const float2 v2 = *reinterpret_cast<const float2*>(pv);
        t.v[0] = v2.x; t.v[1] = v2.y;
      } else {
        t.v[0] = pv[0];
      }
      t.strength = scaled ? sbeta[tt] : 1.0f;
    };
    // Read-outs of kGroup tokens are summed over lanes together after the group: their exchanges run side by side and
    // a lane ends up with its share of the sums.
    auto finish = [&](auto group, float (&o)[decltype(group)::value * kCols], int tt) {
      constexpr int kCount = decltype(group)::value * kCols;
      const int at0 = scan_sums<kPartners, kCount>(o, part);
      constexpr int kKept = kCount > kPartners ? kCount / kPartners : 1;
      // lanes that hold the same sum: the last exchanges' offsets tell them apart
      constexpr int kSame = kPartners > kCount ? kPartners / kCount : 1;
      if (part % kSame != 0) return;
#pragma unroll
      for (int i = 0; i < kKept; ++i) {
        const int g = (at0 + i) / kCols, c = (at0 + i) % kCols;
        if (c < left) {
          float sum = o[i];
          if (a.skip) sum += skip * sv[(tt + g) * kTile + col_in_tile + c];
          a.out[static_cast<size_t>(first + base + tt + g) * a.out_stride + head * a.vdim + col + c] = sum;
        }
      }
    };
    auto multiply = [&](const ScanToken<kRows, kCols, kRowDecay, P>& t, float decay) {
      if (!multiplies) return;
      const P minus_one = pair_of<P>(-1.0f, -1.0f);
#pragma unroll
      for (int r = 0; r < kFactors; ++r) {
        const P d = kRowDecay ? t.g[r] : pair_of<P>(decay, decay), rounded = pair_mul(product[r], d);
        rest[r] = pair_fma(rest[r], d, pair_fma(product[r], pair_mul(d, minus_one), rounded));
        product[r] = rounded;
      }
    };
    constexpr int kGroup = 4;
    const int whole = count / kGroup * kGroup;
    ScanToken<kRows, kCols, kRowDecay, P> next;
    if (whole) fetch(next, 0);
    for (int tt = 0; tt < whole; tt += kGroup) {
      float o[kGroup * kCols];
#pragma unroll
      for (int g = 0; g < kGroup; ++g) {
        const ScanToken<kRows, kCols, kRowDecay, P> now = next;
        fetch(next, min(tt + g + 1, count - 1));      // the next token's numbers are on their way during this one's sums
        float one[kCols];
        const float decay = kRowDecay ? 1.0f : sdecay[tt + g];
        mine.take(now, decay, scaled, one);
        if constexpr (kRead) {
#pragma unroll
          for (int c = 0; c < kCols; ++c) o[g * kCols + c] = one[c];
        } else {
          multiply(now, decay);
        }
      }
      if constexpr (kRead) finish(std::integral_constant<int, kGroup>{}, o, tt);
    }
    for (int tt = whole; tt < count; ++tt) {
      ScanToken<kRows, kCols, kRowDecay, P> now;
      fetch(now, tt);
      float o[kCols];
      const float decay = kRowDecay ? 1.0f : sdecay[tt];
      mine.take(now, decay, scaled, o);
      if constexpr (kRead) finish(std::integral_constant<int, 1>{}, o, tt);
      else multiply(now, decay);
    }
    __syncthreads();     // the buffer is free for the run after the next
  }
  pdl_trigger();
  if (left <= 0) return;
  if constexpr (!kRead) {
    mine.store(a.seg_states + own * a.vdim + in_head, a.dim, part, left, true);
    if (blockIdx.z == 0 && threadIdx.x < kPartners) {
#pragma unroll
      for (int r = 0; r < kRows / 2; ++r) {
        const int row = ((r / 2) * kPartners + part) * 4 + (r & 1) * 2;
        const float2 both = pair_halves(product[kRowDecay ? r : 0]), off = pair_halves(rest[kRowDecay ? r : 0]);
        if (row < a.dim) a.seg_decays[own + row] = both.x - off.x;
        if (row + 1 < a.dim) a.seg_decays[own + row + 1] = both.y - off.y;
      }
    }
  } else if (slot_ok && seg.number == seg.of - 1) {
    mine.store(home, a.dim, part, left, wide);
  }
}

// What each piece starts from, in place of what it left: start' = decays * start + left, from the slot's state on.
// A thread owns four rows of a column and goes through the entry's pieces in order; their loads do not wait for one another.
__global__ void __launch_bounds__(256) scan_join_kernel(const ScanArgs a) {
  const int e = blockIdx.x, head = blockIdx.y;
  const int quads = a.dim >> 2, at = blockIdx.z * blockDim.x + threadIdx.x;
  const int col = at / quads, row = (at - col * quads) * 4;
  int place;
  const int pieces = scan_pieces_of(a, e, place);
  int slot = a.entry_slot[e];
  if (slot < 0 || slot >= a.slots) slot = 0;      // the walk says so in the fault word
  pdl_wait();
  if (col >= a.vdim || pieces == 0) return;
  float4 S = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (a.entry_start[e] > 0) {
    const float* home = a.state + slot * a.state_stride + a.state_off + static_cast<size_t>(head) * a.dim * a.vdim +
                        static_cast<size_t>(col) * a.dim + row;
    S = make_float4(home[0], home[1], home[2], home[3]);
  }
  const size_t step = static_cast<size_t>(a.heads) * a.dim;
  size_t own = (static_cast<size_t>(place) * a.heads + head) * a.dim;
#pragma unroll 4
  for (int p = 0; p < pieces; ++p, own += step) {
    float4* state = reinterpret_cast<float4*>(a.seg_states + own * a.vdim + static_cast<size_t>(col) * a.dim + row);
    if (p == pieces - 1) {
      *state = S;
      break;
    }
    const float4 left = *state, d = *reinterpret_cast<const float4*>(a.seg_decays + own + row);
    *state = S;
    S.x = fmaf(S.x, d.x, left.x); S.y = fmaf(S.y, d.y, left.y); S.z = fmaf(S.z, d.z, left.z); S.w = fmaf(S.w, d.w, left.w);
  }
}

// A step of single tokens: bound by the states' way through memory, so nothing is staged.  A lane's numbers of the token
// come straight from the rows; with four columns a lane it has four 16-byte pieces of the state on their way.
template <int kRows, int kPartners, int kCols, int kKind, bool kRowDecay>
__global__ void __launch_bounds__(kScanThreads) linear_scan_single_kernel(const ScanArgs a) {
  pdl_trigger();
  const int e = blockIdx.x, head = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = lane % kPartners;
  constexpr int kSpread = 32 / kPartners, kTile = kScanWarps * kSpread * kCols;
  const int col = blockIdx.z * kTile + (warp * kSpread + lane / kPartners) * kCols;
  const int left = a.vdim - col;
  const int kv_head = head / (a.heads / a.kv_heads);
  const int first = a.cu_seqlens[e], length = a.cu_seqlens[e + 1] - first, start = a.entry_start[e];
  int slot = a.entry_slot[e];
  const bool slot_ok = slot >= 0 && slot < a.slots;
  if (!slot_ok) {
    if (threadIdx.x == 0) atomicOr(a.fault, kFaultSlot);
    slot = 0;
  }
  float* home = a.state + slot * a.state_stride + a.state_off + static_cast<size_t>(head) * a.dim * a.vdim +
                static_cast<size_t>(left > 0 ? col : 0) * a.dim;
  const bool wide = (reinterpret_cast<uintptr_t>(home) & 15) == 0;
  const float* strength = a.beta ? a.beta : a.v_scale;
  const bool scaled = strength != nullptr;
  const float skip = a.skip ? a.skip[head] : 0.0f;
  const float fixed_decay = a.decay_mode == 0 ? a.decay[head] : 1.0f;
  using P = PlainPair;
  ScanColumns<kRows, kPartners, kCols, kKind, kRowDecay, true, P> mine;
  if constexpr (kKind == kScanBonus) {
#pragma unroll
    for (int j = 0; j < kRows / 4; ++j) {
      const int row = (j * kPartners + part) * 4;
      const float* p = a.bonus + static_cast<size_t>(head) * a.dim + row;
      mine.bonus[2 * j] = row < a.dim ? pair_of<P>(p[0], p[1]) : pair_of<P>(0.0f, 0.0f);
      mine.bonus[2 * j + 1] = row < a.dim ? pair_of<P>(p[2], p[3]) : pair_of<P>(0.0f, 0.0f);
    }
  }
  pdl_wait();
  if (start > 0) mine.load(home, a.dim, part, left, wide); else mine.clear();
  for (int i = 0; i < length; ++i) {
    const size_t t = static_cast<size_t>(first) + i;
    ScanToken<kRows, kCols, kRowDecay, P> now;
    const float decay = a.decay_mode == 1 ? a.decay[t * a.heads + head] : fixed_decay;
    auto rows = [&](const float* p, int j, float otherwise, P& lower, P& upper) {
      const int row = (j * kPartners + part) * 4;
      float4 four = make_float4(otherwise, otherwise, otherwise, otherwise);
      if (row < a.dim) four = *reinterpret_cast<const float4*>(p + row);
      lower = pair_of<P>(four.x, four.y);
      upper = pair_of<P>(four.z, four.w);
    };
#pragma unroll
    for (int j = 0; j < kRows / 4; ++j) {
      rows(a.k + t * a.k_stride + kv_head * a.dim, j, 0.0f, now.k[2 * j], now.k[2 * j + 1]);
      rows(a.q + t * a.q_stride + kv_head * a.dim, j, 0.0f, now.q[2 * j], now.q[2 * j + 1]);
      if constexpr (kRowDecay) {
        if (a.decay_mode == 2) rows(a.decay + (t * a.heads + head) * a.dim, j, 1.0f, now.g[2 * j], now.g[2 * j + 1]);
        else now.g[2 * j] = now.g[2 * j + 1] = pair_of<P>(decay, decay);
      }
    }
    const float* v = a.v + t * a.v_stride + head * a.vdim + col;
#pragma unroll
    for (int c = 0; c < kCols; ++c) now.v[c] = c < left ? v[c] : 0.0f;
    now.strength = scaled ? strength[t * a.heads + head] : 1.0f;
    float o[kCols];
    mine.take(now, decay, scaled, o);
    const int at0 = scan_sums<kPartners, kCols>(o, part);
    constexpr int kSame = kPartners > kCols ? kPartners / kCols : 1, kKept = kCols > kPartners ? kCols / kPartners : 1;
    if (part % kSame == 0) {
#pragma unroll
      for (int c = 0; c < kKept; ++c) {
        const int at = at0 + c;
        if (at < left) {
          float sum = o[c];
          if (a.skip) sum += skip * v[at];
          a.out[t * a.out_stride + head * a.vdim + col + at] = sum;
        }
      }
    }
  }
  if (slot_ok && left > 0) mine.store(home, a.dim, part, left, wide);
}

// ------------------------------------------------------------ norm and gate after a mixer
// y: [T, C] in groups of `group` columns.  gate = act(g[t, g_col0 + c]) with act 0 none, 1 sigmoid,
// 2 SiLU.  With `gate_first` the gate multiplies before the norm, else after it.  The norm (if `norm`)
// divides a group by sqrt(mean(z^2) + eps) and multiplies by weight[c % weight_period] (or nothing).
// One block per (token, group); float32 arithmetic, one rounding at the store.
template <typename TY, typename T>
__global__ void gated_norm_kernel(const TY* y, int y_stride, const T* g, int g_stride,
                                  int g_col0, int act, int gate_first, int norm, const float* __restrict__ weight,
                                  int weight_period, float eps, T* __restrict__ out, int group, int groups) {
  __shared__ float scratch[32];
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, part = blockIdx.y;
  const TY* yr = y + static_cast<size_t>(t) * y_stride + static_cast<size_t>(part) * group;
  const T* gr = g ? g + static_cast<size_t>(t) * g_stride + g_col0 + static_cast<size_t>(part) * group : nullptr;
  T* o = out + (static_cast<size_t>(t) * groups + part) * group;
  auto gate_at = [&](int i) {
    if (!gr || act == 0) return 1.0f;
    const float raw = to_float(gr[i]);
    return act == 1 ? sigmoid_f(raw) : silu_f(raw);
  };
  float inv = 1.0f;
  if (norm) {
    float sum_sq = 0.0f;
    for (int i = threadIdx.x; i < group; i += blockDim.x) {
      float z = to_float(yr[i]);
      if (gate_first) z *= gate_at(i);
      sum_sq += z * z;
    }
    sum_sq = block_sum(sum_sq, scratch);
    inv = 1.0f / sqrtf(sum_sq / static_cast<float>(group) + eps);
  }
  for (int i = threadIdx.x; i < group; i += blockDim.x) {
    const float gate = gate_at(i);
    float z = to_float(yr[i]);
    if (gate_first) z *= gate;
    z *= inv;
    if (norm && weight) z *= weight[(part * group + i) % weight_period];
    if (!gate_first) z *= gate;
    o[i] = from_float<T>(z);
  }
}

// What the two kernels below share: a thread's columns (runs of four, `apart` columns from one to the next) and their gates,
// read once, from the loads to the sum of squares and from the norm to the store.  `wide`: every run of four starts on a
// vector's boundary.
template <typename TY, typename T, int kPer>
struct GatedColumns {
  float z[kPer][4], gate[kPer][4];

  __device__ __forceinline__ float take(const TY* yr, const T* gr, int first, int apart, int group, int act, int gate_first, int wide) {
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int i = first + p * apart;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        z[p][j] = 0.0f;
        gate[p][j] = 1.0f;
      }
      if (i >= group) continue;
      if (wide) {
        load_four(yr + i, z[p]);
        if (gr) load_four(gr + i, gate[p]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          z[p][j] = to_float(yr[i + j]);
          if (gr) gate[p][j] = to_float(gr[i + j]);
        }
      }
    }
    float sum_sq = 0.0f;
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (gr) gate[p][j] = act == 1 ? sigmoid_f(gate[p][j]) : silu_f(gate[p][j]);
        if (gate_first) z[p][j] *= gate[p][j];
        sum_sq += z[p][j] * z[p][j];
      }
    }
    return sum_sq;
  }
  __device__ __forceinline__ void give(T* o, float inv, const float* weight, int weight_at, int weight_period, int first, int apart,
                                       int group, int gate_first, int wide) {
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int i = first + p * apart;
      if (i >= group) break;
      int at = weight ? (weight_at + i) % weight_period : 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        z[p][j] *= inv;
        if (weight) {
          z[p][j] *= weight[at];
          at = at + 1 == weight_period ? 0 : at + 1;
        }
        if (!gate_first) z[p][j] *= gate[p][j];
      }
      if (wide) {
        store_four(o + i, z[p]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i + j] = from_float<T>(z[p][j]);
      }
    }
  }
};

// The same with kLanes lanes of a warp per (token, group), for groups of at most kLanes * 4 * kPer columns, a multiple of 4.
// 2,048 tokens, us: 32 heads of 64 33 -> 15 (half a warp idled), 16 heads of 128 18 -> 15.
template <typename TY, typename T, int kLanes, int kPer>
__global__ void __launch_bounds__(256) gated_norm_warp_kernel(
    const TY* y, int y_stride, const T* g, int g_stride, int g_col0, int act, int gate_first, int norm,
    const float* __restrict__ weight, int weight_period, float eps, T* out, int group, int groups, long long total, int wide) {
  pdl_trigger();
  const int lane = threadIdx.x % kLanes;
  const long long index = blockIdx.x * static_cast<long long>(256 / kLanes) + threadIdx.x / kLanes;
  const bool mine = index < total;
  const long long t = mine ? index / groups : 0;
  const int part = mine ? static_cast<int>(index - t * groups) : 0;
  const int columns = mine ? group : 0;
  const T* gr = (g && act != 0) ? g + static_cast<size_t>(t) * g_stride + g_col0 + static_cast<size_t>(part) * group : nullptr;
  GatedColumns<TY, T, kPer> own;
  pdl_wait();
  float sum_sq = own.take(y + static_cast<size_t>(t) * y_stride + static_cast<size_t>(part) * group, gr, lane * 4, kLanes * 4, columns,
                          act, gate_first, wide);
  float inv = 1.0f;
  if (norm) {
#pragma unroll
    for (int off = kLanes / 2; off >= 1; off >>= 1) sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, off);
    inv = 1.0f / sqrtf(sum_sq / static_cast<float>(group) + eps);
  }
  const int weight_at = weight ? static_cast<int>(static_cast<long long>(part) * group % weight_period) : 0;
  own.give(out + (static_cast<size_t>(t) * groups + part) * group, inv, norm ? weight : nullptr, weight_at, weight_period, lane * 4,
           kLanes * 4, columns, gate_first, wide);
}

// One block per (token, group) for groups of thousands of columns, up to 256 * 4 * kPer.  2,048 rows of 4,096: 48 -> 21 us.
template <typename TY, typename T, int kPer>
__global__ void __launch_bounds__(256) gated_norm_row_kernel(
    const TY* y, int y_stride, const T* g, int g_stride, int g_col0, int act, int gate_first, int norm,
    const float* __restrict__ weight, int weight_period, float eps, T* out, int group, int groups) {
  __shared__ float scratch[32];
  pdl_trigger();
  const int t = blockIdx.x, part = blockIdx.y, first = threadIdx.x * 4;
  const T* gr = (g && act != 0) ? g + static_cast<size_t>(t) * g_stride + g_col0 + static_cast<size_t>(part) * group : nullptr;
  GatedColumns<TY, T, kPer> own;
  pdl_wait();
  const float sum_sq = own.take(y + static_cast<size_t>(t) * y_stride + static_cast<size_t>(part) * group, gr, first, 1024, group, act,
                                gate_first, 1);
  const float inv = norm ? 1.0f / sqrtf(block_sum(sum_sq, scratch) / static_cast<float>(group) + eps) : 1.0f;
  const int weight_at = weight ? static_cast<int>(static_cast<long long>(part) * group % weight_period) : 0;
  own.give(out + (static_cast<size_t>(t) * groups + part) * group, inv, norm ? weight : nullptr, weight_at, weight_period, first, 1024,
           group, gate_first, 1);
}

// ------------------------------------------------------------ xIELU
// z > 0: softplus(p) z^2 + z / 2;  z <= 0: (1/2 + softplus(q)) (exp(z) - 1 - z) + z / 2;  pq = {p, q}.
template <typename T>
__global__ void xielu_kernel(const T* in, T* __restrict__ out, const float* __restrict__ pq, size_t n,
                             int vector) {
  pdl_trigger();
  const float up = softplus_f(pq[0]), down = 0.5f + softplus_f(pq[1]);
  pdl_wait();
  auto one = [&](float z) {
    // exp(z) - 1 - z loses digits for small |z|, but beside z / 2 what is lost is below a sixteen-bit result's last
    // place; the 32-bit engine takes expm1f
    const float grown = sizeof(T) == 2 ? __expf(z) - 1.0f : expm1f(z);
    return z > 0.0f ? up * z * z + 0.5f * z : down * (grown - z) + 0.5f * z;
  };
  const size_t quads = vector ? n >> 2 : 0;      // four at a time where both rows start on 16 bytes
  for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < quads;
       idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
    float z[4];
    if constexpr (sizeof(T) == 2) {
      const uint2 raw = *reinterpret_cast<const uint2*>(in + idx * 4);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
      const float2 lo = __bfloat1622float2(h[0]), hi = __bfloat1622float2(h[1]);
      z[0] = lo.x; z[1] = lo.y; z[2] = hi.x; z[3] = hi.y;
      uint2 packed;
      __nv_bfloat162* ph = reinterpret_cast<__nv_bfloat162*>(&packed);
      ph[0] = __floats2bfloat162_rn(one(z[0]), one(z[1]));
      ph[1] = __floats2bfloat162_rn(one(z[2]), one(z[3]));
      *reinterpret_cast<uint2*>(out + idx * 4) = packed;
    } else {
      const float4 v = *reinterpret_cast<const float4*>(in + idx * 4);
      *reinterpret_cast<float4*>(out + idx * 4) = make_float4(one(v.x), one(v.y), one(v.z), one(v.w));
    }
  }
  for (size_t idx = (quads << 2) + blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < n;
       idx += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[idx] = from_float<T>(one(to_float(in[idx])));
}

// weighted sum of two results: out = a_scale * a + b_scale * b (float32 arithmetic)
template <typename T>
__global__ void scaled_sum_kernel(const T* a, const T* b, float a_scale, float b_scale,
                                  T* __restrict__ out, size_t n) {
  pdl_trigger();
  pdl_wait();
  for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < n;
       idx += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[idx] = from_float<T>(a_scale * to_float(a[idx]) + b_scale * to_float(b[idx]));
}

inline unsigned flat_blocks(long long total, int threads) {
  long long blocks = (total + threads - 1) / threads;
  if (blocks > 148 * 32) blocks = 148 * 32;
  return static_cast<unsigned>(blocks < 1 ? 1 : blocks);
}

}  // namespace rl

namespace rl {

// A group of up to 512 columns takes the lanes of a warp that hold four columns each (a warp's part, so that no lane idles at
// heads of 64 and 32), one of thousands a block; odd sizes go element by element.
template <typename TY, typename T>
static int launch_gated_norm(const TY* y, int y_stride, const T* g, int g_stride, int g_col0, int act, int gate_first, int norm,
                             const float* weight, int weight_period, float eps, T* out, int tokens, int group, int groups,
                             int pdl, cudaStream_t stream) {
  const bool wide = ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
                    y_stride % 4 == 0 && g_stride % 4 == 0 && g_col0 % 4 == 0;
  const long long total = static_cast<long long>(tokens) * groups;
  auto warps = [&](auto kernel, int lanes) {
    const long long per = 256 / lanes;
    return launch_kernel(kernel, dim3(static_cast<unsigned>((total + per - 1) / per)), dim3(256), 0, stream, pdl != 0, y, y_stride,
                         g, g_stride, g_col0, act, gate_first, norm, weight, weight_period, eps, out, group, groups, total,
                         static_cast<int>(wide));
  };
  if (group % 4 == 0 && group <= 512) {
    if (group <= 32) return warps(gated_norm_warp_kernel<TY, T, 8, 1>, 8);
    if (group <= 64) return warps(gated_norm_warp_kernel<TY, T, 16, 1>, 16);
    if (group <= 128) return warps(gated_norm_warp_kernel<TY, T, 32, 1>, 32);
    if (group <= 256) return warps(gated_norm_warp_kernel<TY, T, 32, 2>, 32);
    return warps(gated_norm_warp_kernel<TY, T, 32, 4>, 32);
  }
  auto rows = [&](auto kernel, int threads) {
    return launch_kernel(kernel, dim3(tokens, groups), dim3(threads), 0, stream, pdl != 0, y, y_stride, g, g_stride, g_col0, act,
                         gate_first, norm, weight, weight_period, eps, out, group, groups);
  };
  if (group % 4 == 0 && wide && group <= 8192) {
    if (group <= 2048) return rows(gated_norm_row_kernel<TY, T, 2>, 256);
    if (group <= 4096) return rows(gated_norm_row_kernel<TY, T, 4>, 256);
    return rows(gated_norm_row_kernel<TY, T, 8>, 256);
  }
  int threads = 32;
  while (threads < 256 && threads * 2 <= group) threads *= 2;
  return rows(gated_norm_kernel<TY, T>, threads);
}

template <int kRows, int kPartners, int kCols, int kKind, bool kRowDecay, bool kRead = true>
static int launch_scan(ScanArgs a, int blocks, int pdl, cudaStream_t stream) {
  constexpr int kTile = kScanWarps * (32 / kPartners) * kCols;
  constexpr int kPerToken = scan_token_floats<kRows, kPartners, kCols, kRowDecay, kRead>();
  constexpr int kRun = 20 * 1024 / 4 / kPerToken;      // two buffers of a run each within 40 KB
  a.run = kRun > 16 ? 16 : (kRun < 1 ? 1 : kRun);
  const size_t smem = 2 * static_cast<size_t>((a.run * kPerToken + 3) & ~3) * sizeof(float);
  const dim3 grid(blocks, a.heads, (a.vdim + kTile - 1) / kTile);
  return launch_kernel(linear_scan_kernel<kRows, kPartners, kCols, kKind, kRowDecay, kRead>, grid, dim3(kScanThreads), smem,
                       stream, pdl != 0, a);
}

// Rows a lane and lanes a column are a matter of the head's size alone, since they fix the order of a column's sums.
template <int kKind, bool kRowDecay>
static int launch_plain_scan(const ScanArgs& a, int blocks, int pdl, cudaStream_t stream) {
  const int dim = a.dim;
  if (dim <= 4) return launch_scan<4, 1, 2, kKind, kRowDecay>(a, blocks, pdl, stream);
  if (dim <= 8) return launch_scan<4, 2, 2, kKind, kRowDecay>(a, blocks, pdl, stream);
  if (dim <= 16) return launch_scan<4, 4, 2, kKind, kRowDecay>(a, blocks, pdl, stream);
  if (dim <= 32) return launch_scan<4, 8, 2, kKind, kRowDecay>(a, blocks, pdl, stream);
  if (dim <= 64) return launch_scan<4, 16, 2, kKind, kRowDecay>(a, blocks, pdl, stream);
  if (dim <= 128) return launch_scan<4, 32, 2, kKind, kRowDecay>(a, blocks, pdl, stream);
  if (dim <= 256) return launch_scan<8, 32, 2, kKind, kRowDecay>(a, blocks, pdl, stream);
  if (dim <= 512) return launch_scan<16, 32, 1, kKind, kRowDecay>(a, blocks, pdl, stream);
  return launch_scan<32, 32, 1, kKind, kRowDecay>(a, blocks, pdl, stream);
}

static int launch_delta_scan(const ScanArgs& a, int blocks, int pdl, cudaStream_t stream) {
  const int dim = a.dim;
  if (dim <= 4) return launch_scan<4, 1, 2, kScanDelta, true>(a, blocks, pdl, stream);
  if (dim <= 8) return launch_scan<4, 2, 2, kScanDelta, true>(a, blocks, pdl, stream);
  if (dim <= 16) return launch_scan<4, 4, 2, kScanDelta, true>(a, blocks, pdl, stream);
  if (dim <= 32) return launch_scan<8, 4, 2, kScanDelta, true>(a, blocks, pdl, stream);
  if (dim <= 64) return launch_scan<16, 4, 2, kScanDelta, true>(a, blocks, pdl, stream);
  if (dim <= 128) return launch_scan<16, 8, 2, kScanDelta, true>(a, blocks, pdl, stream);
  if (dim <= 256) return launch_scan<16, 16, 2, kScanDelta, true>(a, blocks, pdl, stream);
  if (dim <= 512) return launch_scan<16, 32, 1, kScanDelta, true>(a, blocks, pdl, stream);
  return launch_scan<32, 32, 1, kScanDelta, true>(a, blocks, pdl, stream);
}

// In pieces there are blocks enough: more rows a lane and four columns, fewer exchanges and fetches a column.
template <int kKind, bool kRowDecay, bool kRead>
static int launch_pieces(const ScanArgs& a, int blocks, int pdl, cudaStream_t stream) {
  return a.dim <= 64 ? launch_scan<8, 8, 4, kKind, kRowDecay, kRead>(a, blocks, pdl, stream)
                     : launch_scan<8, 16, 4, kKind, kRowDecay, kRead>(a, blocks, pdl, stream);
}

template <int kRows, int kPartners, int kCols, int kKind, bool kRowDecay>
static int launch_single_scan(const ScanArgs& a, int pdl, cudaStream_t stream) {
  constexpr int kTile = kScanWarps * (32 / kPartners) * kCols;
  return launch_kernel(linear_scan_single_kernel<kRows, kPartners, kCols, kKind, kRowDecay>,
                       dim3(a.entries, a.heads, (a.vdim + kTile - 1) / kTile), dim3(kScanThreads), 0, stream, pdl != 0, a);
}

}  // namespace rl

extern "C" {

// out = silu(conv(x)) for every row of the step, then the slots' tails are brought up to date.
int rl_causal_conv_silu(int dtype, const void* x, int x_stride, int col0, const float* taps, const float* bias,
                        float* state, long long state_stride, int state_off, float* out, const int* cu_seqlens,
                        const int* entry_slot, const int* entry_start, int entries, int tokens, int channels,
                        int width, int slots, int* fault, int act, int pdl, cudaStream_t stream) {
  if (tokens == 0 || channels == 0) return 0;
  if (width < 1 || width > rl::kMaxTaps || entries < 1 || act < 0 || act > 1) return static_cast<int>(cudaErrorInvalidValue);
  RL_DISPATCH_DTYPE(dtype, {
    const bool pairs = channels % 2 == 0 && col0 % 2 == 0 && x_stride % 2 == 0 &&
                       (reinterpret_cast<uintptr_t>(x) & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    const long long tiles = (tokens + rl::kConvRows - 1) / rl::kConvRows;
    const long long threads = tiles * (pairs ? channels / 2 : channels);
    auto kernel = pairs ? rl::causal_conv_silu_kernel<scalar_t, 2, 0> : rl::causal_conv_silu_kernel<scalar_t, 1, 0>;
    if (pairs && width == 4) kernel = rl::causal_conv_silu_kernel<scalar_t, 2, 4>;
    if (pairs && width == 3) kernel = rl::causal_conv_silu_kernel<scalar_t, 2, 3>;
    if (pairs && width == 2) kernel = rl::causal_conv_silu_kernel<scalar_t, 2, 2>;
    int code = rl::launch_kernel(kernel, dim3(static_cast<unsigned>((threads + 127) / 128)), dim3(128), 0,
                                 stream, pdl != 0, static_cast<const scalar_t*>(x), x_stride, col0, taps, bias,
                                 static_cast<const float*>(state), state_stride, state_off, out, cu_seqlens,
                                 entry_slot, entry_start, entries, tokens, channels, width, slots, fault, act);
    if (code != 0 || width == 1) return code;
    return rl::launch_kernel(rl::conv_tail_update_kernel<scalar_t>,
                             dim3(rl::flat_blocks(static_cast<long long>(entries) * channels, 256)), dim3(256), 0,
                             stream, pdl != 0, static_cast<const scalar_t*>(x), x_stride, col0, state, state_stride,
                             state_off, cu_seqlens, entry_slot, entry_start, entries, channels, width, slots);
  });
  return 0;
}

int rl_activate_rows(int dtype, const void* x, int x_stride, int col0, float* out, int tokens, int channels, int act,
                     int pdl, cudaStream_t stream) {
  if (tokens == 0 || channels == 0) return 0;
  if (act < 0 || act > 1) return static_cast<int>(cudaErrorInvalidValue);
  const int row_blocks = (tokens + rl::kActivateRows - 1) / rl::kActivateRows;
  const bool wide = channels % 4 == 0 && col0 % 4 == 0 && x_stride % 4 == 0 && row_blocks <= 65535 &&
                    ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  RL_DISPATCH_DTYPE(dtype, {
    if (wide)
      return rl::launch_kernel(rl::activate_rows_wide_kernel<scalar_t>, dim3((channels + 1023) / 1024, row_blocks), dim3(256), 0,
                               stream, pdl != 0, static_cast<const scalar_t*>(x), x_stride, col0, out, tokens, channels, act);
    return rl::launch_kernel(rl::activate_rows_kernel<scalar_t>,
                             dim3(rl::flat_blocks(static_cast<long long>(tokens) * channels, 256)), dim3(256), 0, stream,
                             pdl != 0, static_cast<const scalar_t*>(x), x_stride, col0, out, tokens, channels, act);
  });
  return 0;
}

int rl_decay_gate(int dtype, const void* x, int x_stride, int col0, const float* rate, const float* bias, int per,
                  float* decay, float* step, int tokens, int channels, int pdl, cudaStream_t stream) {
  if (tokens == 0 || channels == 0) return 0;
  if (per < 1) return static_cast<int>(cudaErrorInvalidValue);
  const bool wide = channels % 4 == 0 && x_stride % 4 == 0 && col0 % 4 == 0 &&
                    ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(decay) | reinterpret_cast<uintptr_t>(step)) & 15) == 0;
  RL_DISPATCH_DTYPE(dtype, {
    auto kernel = wide ? rl::decay_gate_kernel<scalar_t, true> : rl::decay_gate_kernel<scalar_t, false>;
    return rl::launch_kernel(kernel, dim3(rl::flat_blocks(static_cast<long long>(tokens) * channels / (wide ? 4 : 1), 256)),
                             dim3(256), 0, stream, pdl != 0, static_cast<const scalar_t*>(x), x_stride, col0, rate, bias,
                             per, decay, step, tokens, channels);
  });
  return 0;
}

int rl_exp_decay(int dtype, const void* x, int x_stride, int col0, const float* bias, float* decay, int tokens,
                 int channels, int pdl, cudaStream_t stream) {
  if (tokens == 0 || channels == 0) return 0;
  RL_DISPATCH_DTYPE(dtype, {
    return rl::launch_kernel(rl::exp_decay_kernel<scalar_t>,
                             dim3(rl::flat_blocks(static_cast<long long>(tokens) * channels, 256)), dim3(256), 0, stream,
                             pdl != 0, static_cast<const scalar_t*>(x), x_stride, col0, bias, decay, tokens, channels);
  });
  return 0;
}

int rl_low_rank_decay(int dtype, const void* x, int x_stride, int copied, int low_col0, const void* w, int rank,
                      const float* bias, float tau, float* rows, int channels, float* decay, int tokens, int pdl,
                      cudaStream_t stream) {
  if (tokens == 0) return 0;
  if (rank < 1 || channels < 1 || copied < 0 || copied > x_stride || low_col0 < 0 || low_col0 + rank > x_stride || !(tau > 0.0f) ||
      bias == nullptr || w == nullptr || (reinterpret_cast<uintptr_t>(w) & 15))
    return static_cast<int>(cudaErrorInvalidValue);
  const int decay_blocks = (channels + rl::kDecayThreads - 1) / rl::kDecayThreads;
  const int copy_blocks = (copied + 4 * rl::kDecayThreads - 1) / (4 * rl::kDecayThreads);
  const int vector_rows = copied % 4 == 0 && x_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                          (reinterpret_cast<uintptr_t>(rows) & 15) == 0;
  const dim3 grid((tokens + rl::kDecayTokens - 1) / rl::kDecayTokens, decay_blocks + copy_blocks);
  RL_DISPATCH_DTYPE(dtype, {
    return rl::launch_kernel(rl::low_rank_decay_kernel<scalar_t>, grid, dim3(rl::kDecayThreads), 0, stream, pdl != 0,
                             static_cast<const scalar_t*>(x), x_stride, copied, low_col0, static_cast<const scalar_t*>(w), rank, bias,
                             1.0f / tau, rows, channels, decay, tokens, decay_blocks, vector_rows);
  });
  return 0;
}

int rl_tanh_rows(int dtype, const void* x, void* out, long long total, int pdl, cudaStream_t stream) {
  if (total == 0) return 0;
  RL_DISPATCH_DTYPE(dtype, {
    return rl::launch_kernel(rl::tanh_rows_kernel<scalar_t>, dim3(rl::flat_blocks(total, 256)), dim3(256), 0, stream,
                             pdl != 0, static_cast<const scalar_t*>(x), static_cast<scalar_t*>(out), total);
  });
  return 0;
}

int rl_shift_mix(int dtype, const void* x, int x_stride, const float* mu, int mixes, void* out, float* kept,
                 long long kept_stride, int kept_off, const int* cu_seqlens, const int* entry_slot,
                 const int* entry_start, int entries, int tokens, int channels, int slots, int* fault, int pdl,
                 cudaStream_t stream) {
  if (tokens == 0 || channels == 0) return 0;
  if (mixes < 1 || entries < 1) return static_cast<int>(cudaErrorInvalidValue);
  RL_DISPATCH_DTYPE(dtype, {
    return rl::launch_kernel(rl::shift_mix_kernel<scalar_t>, dim3(tokens), dim3(channels >= 1024 ? 256 : 128), 0, stream,
                             pdl != 0, static_cast<const scalar_t*>(x), x_stride, mu, mixes, static_cast<scalar_t*>(out),
                             kept, kept_stride, kept_off, cu_seqlens, entry_slot, entry_start, entries, tokens, channels,
                             slots, fault);
  });
  return 0;
}

int rl_unit_heads(int dtype, float* rows, int stride, int col0, int heads, int dim, float eps, int split,
                  float scale_low, float scale_high, const void* gate_in, int gate_stride, int gate_col0, int gates,
                  float* gate_out, int tokens, int pdl, cudaStream_t stream) {
  if (tokens == 0) return 0;
  const bool wide = dim % 4 == 0 && dim <= 128 && heads > 0 && stride % 4 == 0 && col0 % 4 == 0 && (reinterpret_cast<uintptr_t>(rows) & 15) == 0;
  RL_DISPATCH_DTYPE(dtype, {
    if (wide) {
      const int lanes = dim <= 32 ? 8 : dim <= 64 ? 16 : 32, per = 256 / lanes;
      const long long head_blocks = (static_cast<long long>(tokens) * heads + per - 1) / per;
      const long long gate_blocks = (static_cast<long long>(tokens) * gates + 255) / 256;
      auto kernel = lanes == 8 ? rl::unit_heads_wide_kernel<scalar_t, 8>
                               : lanes == 16 ? rl::unit_heads_wide_kernel<scalar_t, 16> : rl::unit_heads_wide_kernel<scalar_t, 32>;
      return rl::launch_kernel(kernel, dim3(static_cast<unsigned>(head_blocks + gate_blocks)), dim3(256), 0, stream, pdl != 0,
                               rows, stride, col0, heads, dim, eps, split, scale_low, scale_high,
                               static_cast<const scalar_t*>(gate_in), gate_stride, gate_col0, gates, gate_out, tokens,
                               static_cast<int>(head_blocks));
    }
    return rl::launch_kernel(rl::unit_heads_kernel<scalar_t>, dim3(tokens), dim3(128), 0, stream, pdl != 0, rows,
                             stride, col0, heads, dim, eps, split, scale_low, scale_high,
                             static_cast<const scalar_t*>(gate_in), gate_stride, gate_col0, gates, gate_out, tokens);
  });
  return 0;
}

int rl_rotate_heads(int dtype, const void* in, int in_stride, int q_col0, int k_col0, int v_col0, float* out,
                    const int* positions, const float* inv_freq, int heads, int dim, int vdim, int rot, float k_scale,
                    int tokens, int pdl, cudaStream_t stream) {
  if (tokens == 0) return 0;
  if (rot < 0 || rot > dim || (rot & 1)) return static_cast<int>(cudaErrorInvalidValue);
  const bool wide = rot % 8 == 0 && dim % 4 == 0 && vdim % 4 == 0 && in_stride % 4 == 0 && q_col0 % 4 == 0 &&
                    k_col0 % 4 == 0 && v_col0 % 4 == 0 &&
                    ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  RL_DISPATCH_DTYPE(dtype, {
    return rl::launch_kernel(rl::rotate_heads_kernel<scalar_t>, dim3(tokens), dim3(256), rot * sizeof(float), stream, pdl != 0,
                             static_cast<const scalar_t*>(in), in_stride, q_col0, k_col0, v_col0, out, positions,
                             inv_freq, heads, dim, vdim, rot, k_scale, tokens, static_cast<int>(wide));
  });
  return 0;
}

int rl_linear_scan(const float* q, int q_stride, const float* k, int k_stride, const float* v, int v_stride,
                   const float* decay, int decay_mode, const float* beta, const float* v_scale, const float* skip,
                   const float* bonus, float* out, int out_stride, float* state, long long state_stride, int state_off,
                   const int* cu_seqlens, const int* entry_slot, const int* entry_start, int entries, int tokens, int heads,
                   int kv_heads, int dim, int vdim, int slots, int* fault, int segment, int from, int segments, int others,
                   float* seg_states, float* seg_decays, int blocks_from, int blocks, int taken, float* records, int record_floats, int pdl,
                   cudaStream_t stream) {
  if (entries == 0) return 0;
  if (heads < 1 || kv_heads < 1 || heads % kv_heads || dim < 1 || dim > 1024 || vdim < 1 || decay_mode < 0 ||
      decay_mode > 2 || decay == nullptr || (bonus != nullptr && beta != nullptr))
    return static_cast<int>(cudaErrorInvalidValue);
  rl::ScanArgs a;
  a.q = q; a.q_stride = q_stride; a.k = k; a.k_stride = k_stride; a.v = v; a.v_stride = v_stride;
  a.decay = decay; a.decay_mode = decay_mode; a.beta = beta; a.v_scale = v_scale; a.skip = skip; a.bonus = bonus;
  a.out = out; a.out_stride = out_stride; a.state = state; a.state_stride = state_stride; a.state_off = state_off;
  a.cu_seqlens = cu_seqlens; a.entry_slot = entry_slot; a.entry_start = entry_start;
  a.heads = heads; a.kv_heads = kv_heads; a.dim = dim; a.vdim = vdim; a.slots = slots;
  a.fault = fault;
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  a.wide_in = dim % 4 == 0 && vdim % 4 == 0 && q_stride % 4 == 0 && k_stride % 4 == 0 && v_stride % 4 == 0 &&
              aligned(q) && aligned(k) && aligned(v) && (decay_mode != 2 || aligned(decay));
  a.entries = entries;
  a.segment = segment;
  a.from = segment ? from : 0;
  a.seg_states = seg_states; a.seg_decays = seg_decays;
  a.in_blocks = blocks_from;
  using namespace rl;
  if (blocks_from > 0) {
    // An entry's own length says how it is taken, so that its sums are in the same order whatever else is in the step.
    if (segment != 0 || record_floats != scan_record_floats(dim, beta != nullptr)) return static_cast<int>(cudaErrorInvalidValue);
    const ScanBlockArgs in_blocks = {q, q_stride, k, k_stride, v, v_stride, decay, decay_mode, beta, v_scale, skip, bonus, out, out_stride,
                                     state + state_off, state_stride, cu_seqlens, entry_slot, entry_start, heads, kv_heads, dim, vdim, slots,
                                     entries, blocks_from, a.wide_in, records, fault};
    const int e = scan_blocks(in_blocks, blocks, taken, stream);
    if (e || !others) return e;
  }
  // single tokens of the common head sizes: the same rows a lane and lanes a column as the walk, so the same sums
  if (segment == 0 && blocks_from == 0 && tokens == entries && a.wide_in && dim > 32 && dim <= 128) {
    if (beta)
      return dim <= 64 ? launch_single_scan<16, 4, 2, kScanDelta, true>(a, pdl, stream)
                       : launch_single_scan<16, 8, 2, kScanDelta, true>(a, pdl, stream);
    if (bonus)
      return dim <= 64 ? launch_single_scan<4, 16, 4, kScanBonus, true>(a, pdl, stream)
                       : launch_single_scan<4, 32, 4, kScanBonus, true>(a, pdl, stream);
    if (decay_mode == 2)
      return dim <= 64 ? launch_single_scan<4, 16, 4, kScanPlain, true>(a, pdl, stream)
                       : launch_single_scan<4, 32, 4, kScanPlain, true>(a, pdl, stream);
    return dim <= 64 ? launch_single_scan<4, 16, 4, kScanPlain, false>(a, pdl, stream)
                     : launch_single_scan<4, 32, 4, kScanPlain, false>(a, pdl, stream);
  }
  if (segment == 0) {
    if (beta) return launch_delta_scan(a, entries, pdl, stream);
    if (bonus) return launch_plain_scan<kScanBonus, true>(a, entries, pdl, stream);
    if (decay_mode == 2) return launch_plain_scan<kScanPlain, true>(a, entries, pdl, stream);
    return launch_plain_scan<kScanPlain, false>(a, entries, pdl, stream);
  }
  // in pieces side by side: sizes and pieces the kernels are made for (an entry that is cut has two pieces at least)
  if (segment < 0 || from <= segment || beta != nullptr || dim <= 32 || dim > 128 || dim % 4 || vdim % 4 || segments < 1 || seg_states == nullptr ||
      seg_decays == nullptr || !aligned(seg_states) || !aligned(seg_decays))
    return static_cast<int>(cudaErrorInvalidValue);
  // An entry's own length says whether it is cut, so that its sums are in the same order whatever else is in the step; the
  // others are walked by themselves.
  int e = 0;
  if (others) {
    ScanArgs walked = a;
    walked.segment = 0;
    e = bonus ? launch_plain_scan<kScanBonus, true>(walked, entries, pdl, stream)
              : decay_mode == 2 ? launch_plain_scan<kScanPlain, true>(walked, entries, pdl, stream)
                                : launch_plain_scan<kScanPlain, false>(walked, entries, pdl, stream);
    if (e) return e;
  }
  // with a bonus the state moves as without one
  e = bonus || decay_mode == 2 ? launch_pieces<kScanPlain, true, false>(a, segments, pdl, stream)
                                   : launch_pieces<kScanPlain, false, false>(a, segments, pdl, stream);
  if (e == 0)
    e = launch_kernel(scan_join_kernel, dim3(entries, heads, (vdim * (dim / 4) + 255) / 256), dim3(256), 0, stream, pdl != 0, a);
  if (e) return e;
  if (bonus) return launch_pieces<kScanBonus, true, true>(a, segments, pdl, stream);
  if (decay_mode == 2) return launch_pieces<kScanPlain, true, true>(a, segments, pdl, stream);
  return launch_pieces<kScanPlain, false, true>(a, segments, pdl, stream);
}

// y_f32: y is float32 whatever the engine's dtype (the result of a recurrence); else y has the engine's dtype.
int rl_gated_norm(int dtype, int y_f32, const void* y, int y_stride, const void* g, int g_stride, int g_col0, int act,
                  int gate_first, int norm, const float* weight, int weight_period, float eps, void* out, int tokens,
                  int group, int groups, int pdl, cudaStream_t stream) {
  if (tokens == 0 || groups == 0) return 0;
  if (group < 1 || act < 0 || act > 2 || (weight != nullptr && weight_period < 1))
    return static_cast<int>(cudaErrorInvalidValue);
  RL_DISPATCH_DTYPE(dtype, {
    if (y_f32)
      return rl::launch_gated_norm<float, scalar_t>(static_cast<const float*>(y), y_stride, static_cast<const scalar_t*>(g),
                                                    g_stride, g_col0, act, gate_first, norm, weight, weight_period, eps,
                                                    static_cast<scalar_t*>(out), tokens, group, groups, pdl, stream);
    return rl::launch_gated_norm<scalar_t, scalar_t>(static_cast<const scalar_t*>(y), y_stride, static_cast<const scalar_t*>(g),
                                                     g_stride, g_col0, act, gate_first, norm, weight, weight_period, eps,
                                                     static_cast<scalar_t*>(out), tokens, group, groups, pdl, stream);
  });
  return 0;
}

int rl_xielu(int dtype, const void* in, void* out, const float* pq, long long n, int pdl, cudaStream_t stream) {
  if (n == 0) return 0;
  RL_DISPATCH_DTYPE(dtype, {
    return rl::launch_kernel(rl::xielu_kernel<scalar_t>, dim3(rl::flat_blocks((n + 3) / 4, 256)), dim3(256), 0, stream, pdl != 0,
                             static_cast<const scalar_t*>(in), static_cast<scalar_t*>(out), pq, static_cast<size_t>(n),
                             static_cast<int>(((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0));
  });
  return 0;
}

int rl_scaled_sum(int dtype, const void* a, const void* b, float a_scale, float b_scale, void* out, long long n,
                  int pdl, cudaStream_t stream) {
  if (n == 0) return 0;
  RL_DISPATCH_DTYPE(dtype, {
    return rl::launch_kernel(rl::scaled_sum_kernel<scalar_t>, dim3(rl::flat_blocks(n, 256)), dim3(256), 0, stream,
                             pdl != 0, static_cast<const scalar_t*>(a), static_cast<const scalar_t*>(b), a_scale,
                             b_scale, static_cast<scalar_t*>(out), static_cast<size_t>(n));
  });
  return 0;
}

}  // extern "C"
