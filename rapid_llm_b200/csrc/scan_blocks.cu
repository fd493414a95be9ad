// The recurrence over blocks of 32 tokens, for long prompts of 16-bit engines.
//
// With G_t the product of a block's decays up to and with token t, and the state S the block starts from,
//   R = V - (G k) S,  U = T R         with a correction: T = (I + diag(beta) M)^-1 diag(beta), M[t][j] = k_t (G_t / G_j) k_j, j < t
//   U = v_scale V                     without one
//   out = (G q) S + P U               P[t][j] = q_t (G_t / G_j) k_j, j <= t
//   S <- G_32 S + ((G_32 / G) k)^T U
// (a bonus reads before the token's own decay and weighs the diagonal of P).  The products from the block's start and to its
// end run in float64 and are rounded once.  U and T are the WY form of a product of factors I - beta k k^T (Bischof and Van Loan
// 1987), which the published chunked forms of the delta rule rest on.
//
// scan_prepare_kernel makes what does not depend on S, all blocks side by side: a record of G k, G q, (G_32 / G) k, P, T, G_32.
// scan_blocks_kernel walks an entry's blocks in order, a CTA per head and kCols columns of S; the records come by bulk copies
// a block ahead.  Its products run on mma.sync with every float32 as three bfloat16 parts (tile_products).
//
// The parts of an infinity add up to NaN, those of a number that rounds to one, too, and a sum over a block's tokens lets it into
// the read-outs before it.  So where q, k, V, beta, the bonus, the decays' products, R, U or the state an entry starts from are not
// finite or beyond 2^60, the rest of the entry's tokens are walked one after the other, with the walk's infinities (2,048 tokens
// that are not finite from the first on: 1.7 to 2.1 ms, a walk 0.4 to 0.6).  A record says whether its block is one of those, so that
// the blocks themselves look at no more than V, R and U.
//
// An entry's sums depend on its own tokens in this step alone: not on the step's other entries.
//
// What bounds it: a block's chain of dependent steps (rows times S, with a correction R and U, the update, barriers between
// them), some 5,500 cycles with a correction and a CTA a multiprocessor, at 0.4 instructions a cycle and scheduler; the records'
// kernel by its instructions.  us (records + blocks; walked or in pieces): 2,048 tokens, 16 heads of 128 with a correction
// 48 + 198 (552); 32 heads of 64 61 + 160 (465); 700 + 333 + 1,015 tokens of 32 heads of 128, fixed decays, 59 + 225 (404).
// Float32 multiply-adds would be bound by shared memory (an 8 x 8 patch a thread takes as long to fetch as to multiply),
// tcgen05 by its latencies at these sizes.  Root mean square error against 64 bits, 1,300 tokens of 16 heads of 128, here (read-
// outs and states; walked): with a correction 1.24e-7, 9.3e-8 (1.65e-7, 1.47e-7); row decays 1.02e-7, 7.1e-8 (1.84e-7, 1.71e-7).
// Those are decays near one, as the timed calls have them; where they are small a walk is nearer: drawn from 0.05 to 0.95, 900 tokens of
// 8 heads, with a correction 1.14e-7, 7.0e-8 (8.8e-8, 4.9e-8), without one 9.0e-8, 4.4e-8 (8.3e-8, 4.0e-8).
#include <cuda.h>

#include <cuda_bf16.h>

#include <type_traits>

#include "scan_blocks.cuh"
#include "tc_common.cuh"

namespace rl {

constexpr int kBlockPlain = 0, kBlockDelta = 1, kBlockBonus = 2;
constexpr int kTokenStride = kScanBlock + 8;      // floats between rows of 32 tokens: four neighbouring rows of pairs meet in no bank

// Where things lie in a record, in floats.
template <int kDim, bool kDelta>
struct BlockRecord {
  static constexpr int kRowStride = kDim + 8;
  static constexpr int kRows = 0;                                                  // G k of 32 tokens (with a correction), then G q
  static constexpr int kQ = kDelta ? kScanBlock * kRowStride : 0;
  static constexpr int kEnd = kQ + kScanBlock * kRowStride;                        // (G_32 / G) k, [kDim][40]
  static constexpr int kP = kEnd + kDim * kTokenStride;                            // [32][40]
  static constexpr int kT = kP + kScanBlock * kTokenStride;
  static constexpr int kG = kT + (kDelta ? kScanBlock * kTokenStride : 0);         // G_32
  static constexpr int kOdd = kG + kDim;                                           // not zero: the parts cannot say what is in the block
  static constexpr int kSize = kOdd + 4;
  static_assert(kSize % 4 == 0, "records are copied 16 bytes at a time");
};

int scan_record_floats(int dim, bool corrected) {
  if (dim <= 64) return corrected ? BlockRecord<64, true>::kSize : BlockRecord<64, false>::kSize;
  return corrected ? BlockRecord<128, true>::kSize : BlockRecord<128, false>::kSize;
}

__device__ __forceinline__ int blocks_of(const ScanBlockArgs& a, int e) {
  const int length = a.cu_seqlens[e + 1] - a.cu_seqlens[e];
  return length >= a.from ? (length + kScanBlock - 1) / kScanBlock : 0;
}

// What the products are made for: sums of such numbers stay finite.
constexpr float kScanLargest = 0x1p60f;
__device__ __forceinline__ bool is_plain(float x) { return fabsf(x) < kScanLargest; }

// ------------------------------------------------------------------ float32 products on the tensor cores
// Two neighbouring numbers as three pairs of bfloat16 each, every one what the ones before leave, rounded to nearest.
__device__ __forceinline__ void bf16_parts(float x, float y, uint32_t (&parts)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 both = __floats2bfloat162_rn(x, y);
    parts[i] = *reinterpret_cast<const uint32_t*>(&both);
    if (i < 2) {
      x -= __uint_as_float(parts[i] << 16);
      y -= __uint_as_float(parts[i] & 0xffff0000u);
    }
  }
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_bf16_begin(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {      // C = 0
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.0f));
}
// Columns of numbers along the inner dimension, as they are or cut into parts once where they are written: a word holds a part of
// two neighbours, the parts lie `part` words apart.
struct FloatColumns {
  const float* at;
  int stride;
  __device__ __forceinline__ void fetch(int column, int k, uint32_t (&lower)[3], uint32_t (&upper)[3]) const {
    const float2 x = *reinterpret_cast<const float2*>(at + column * stride + k), y = *reinterpret_cast<const float2*>(at + column * stride + k + 8);
    bf16_parts(x.x, x.y, lower);
    bf16_parts(y.x, y.y, upper);
  }
};
struct PartColumns {
  const uint32_t* at;
  int stride, part;
  __device__ __forceinline__ void fetch(int column, int k, uint32_t (&lower)[3], uint32_t (&upper)[3]) const {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      lower[i] = at[i * part + column * stride + (k >> 1)];
      upper[i] = at[i * part + column * stride + (k >> 1) + 4];
    }
  }
};

// sums[n] += A (16 x 16 kSteps) B_n, kTiles tiles of eight columns: `a` at this lane's group's row.  The products of the leading
// parts have a sum of their own per step, which their 16 bits leave all but exact; the five that are smaller by 2^8 and more have
// another, and both are added in float32: the tensor core cuts off what lies below its last bit, which on one sum of all would
// cost 2^-24 a step, one way (two tf32 parts a number, whose leading products fill the sum, were 1.4 times as far off).
// Products of several steps and tiles are formed side by side: one waits 30 cycles for the one before it in its own sum.
template <int kSteps, int kTiles, typename Columns>
__device__ __forceinline__ void tile_products(float (&sums)[kTiles][4], const float* a, int a_stride, const Columns b) {
  constexpr int kGroup = kTiles >= 4 ? 1 : 2;
  static_assert(kSteps % kGroup == 0, "whole groups");
  const int group = (threadIdx.x >> 2) & 7, two = (threadIdx.x & 3) * 2;
#pragma unroll
  for (int step = 0; step < kSteps; step += kGroup) {
    uint32_t x[kGroup][3][4], y[kGroup][kTiles][3][2];
    float leading[kGroup][kTiles][4], small[kGroup][kTiles][4];
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
      const int k = (step + i) * 16 + two;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 pair = *reinterpret_cast<const float2*>(a + (j & 1) * 8 * a_stride + k + (j >> 1) * 8);
        uint32_t parts[3];
        bf16_parts(pair.x, pair.y, parts);
        x[i][0][j] = parts[0]; x[i][1][j] = parts[1]; x[i][2][j] = parts[2];
      }
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
        uint32_t lower[3], upper[3];
        b.fetch(n * 8 + group, k, lower, upper);
#pragma unroll
        for (int part = 0; part < 3; ++part) { y[i][n][part][0] = lower[part]; y[i][n][part][1] = upper[part]; }
      }
    }
    constexpr int kA[5] = {2, 0, 1, 1, 0}, kB[5] = {0, 2, 1, 0, 1};
#pragma unroll
    for (int product = 0; product < 5; ++product) {
#pragma unroll
      for (int i = 0; i < kGroup; ++i) {
#pragma unroll
        for (int n = 0; n < kTiles; ++n) {
          if (product == 0) {
            mma_bf16_begin(small[i][n], x[i][2], y[i][n][0]);
            mma_bf16_begin(leading[i][n], x[i][0], y[i][n][0]);
          } else {
            mma_bf16(small[i][n], x[i][kA[product]], y[i][n][kB[product]]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
#pragma unroll
        for (int j = 0; j < 4; ++j) sums[n][j] += leading[i][n][j] + small[i][n][j];
      }
    }
  }
}
// A 16 x 8 tile of results (this lane's group's rows and two columns) into columns of parts along the rows: neighbouring rows
// lie in lanes four apart, which swap one column each, so that a word is one lane's to write.
__device__ __forceinline__ void show_tile(const float (&x)[4], uint32_t* at, int stride, int part, int column0, int row0) {
  const int group = (threadIdx.x >> 2) & 7, two = (threadIdx.x & 3) * 2, odd = group & 1;
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const float got = __shfl_xor_sync(0xffffffffu, odd ? x[i] : x[i + 1], 4);
    uint32_t parts[3];
    if (odd) bf16_parts(got, x[i + 1], parts);
    else bf16_parts(x[i], got, parts);
    uint32_t* to = at + (column0 + two + odd) * stride + ((row0 + i * 4 + group) >> 1);
#pragma unroll
    for (int j = 0; j < 3; ++j) to[j * part] = parts[j];
  }
}

__device__ __forceinline__ void lane_channels(const float* from, float (&x)[4]) {
  const float4 four = *reinterpret_cast<const float4*>(from);
  x[0] = four.x; x[1] = four.y; x[2] = four.z; x[3] = four.w;
}
__device__ __forceinline__ void lane_channels(const float* from, float (&x)[2]) {
  const float2 two = *reinterpret_cast<const float2*>(from);
  x[0] = two.x; x[1] = two.y;
}

template <int kDim, int kKind>
constexpr int prepare_smem() { return (3 * kScanBlock * (kDim + 8) + 2 * kScanBlock * kTokenStride + kScanBlock) * 4; }

// A CTA makes one block's record of one head.  Where the products of decays to the block's end, E_t = G_32 / G_t, lie within
// 2^-40 and 2^40, P = (q / E) (E k)^T and M = (k / E) (E k)^T on the tensor cores; else by running products: a warp owns four
// keys and carries each along the tokens behind it, a lane with kDim / 32 channels, and sums over channels of four tokens are
// exchanged together.
template <int kDim, int kKind>
__global__ void __launch_bounds__(256) scan_prepare_kernel(const ScanBlockArgs a) {
  constexpr bool kDelta = kKind == kBlockDelta;
  using Record = BlockRecord<kDim, kDelta>;
  constexpr int kC = kDim / 32, kStride = kDim + 8;
  extern __shared__ __align__(16) float prepare_floats[];
  float* sq = prepare_floats;
  float* sk = sq + kScanBlock * kStride;
  float* sg = sk + kScanBlock * kStride;
  float* sp = sg + kScanBlock * kStride;                    // P, then M
  float* sm = sp + kScanBlock * kTokenStride;
  float* sbeta = sm + kScanBlock * kTokenStride;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, head = blockIdx.y;
  int e = 0, at = blockIdx.x;
  for (; e < a.entries; ++e) {
    const int count = blocks_of(a, e);
    if (at < count) break;
    at -= count;
  }
  if (e == a.entries) return;
  const int first = a.cu_seqlens[e] + at * kScanBlock, length = min(kScanBlock, a.cu_seqlens[e + 1] - first);
  const int kv_head = head / (a.heads / a.kv_heads);
  float* record = a.records + (static_cast<size_t>(blockIdx.x) * a.heads + head) * Record::kSize;
  __shared__ int odd_flag;
  if (tid == 0) odd_flag = 0;
  bool odd = false, grows = false;      // grows: decays above one, whose products may get anywhere

  for (int idx = tid; idx < kScanBlock * kDim / 4; idx += 256) {
    const int t = idx / (kDim / 4), c = (idx - t * (kDim / 4)) * 4;
    float q[4] = {0.0f, 0.0f, 0.0f, 0.0f}, k[4] = {0.0f, 0.0f, 0.0f, 0.0f}, g[4] = {1.0f, 1.0f, 1.0f, 1.0f};
    if (t < length && c < a.dim) {                       // dim is a multiple of four
      const size_t row = static_cast<size_t>(first) + t;
      const float* pq = a.q + row * a.q_stride + kv_head * a.dim + c;
      const float* pk = a.k + row * a.k_stride + kv_head * a.dim + c;
      const float* pg = a.decay + (a.decay_mode == 0 ? head : a.decay_mode == 1 ? row * a.heads + head : (row * a.heads + head) * a.dim + c);
      if (a.wide_in) {
        *reinterpret_cast<float4*>(q) = *reinterpret_cast<const float4*>(pq);
        *reinterpret_cast<float4*>(k) = *reinterpret_cast<const float4*>(pk);
        if (a.decay_mode == 2) *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(pg);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          q[i] = pq[i];
          k[i] = pk[i];
          if (a.decay_mode == 2) g[i] = pg[i];
        }
      }
      if (a.decay_mode != 2) g[0] = g[1] = g[2] = g[3] = pg[0];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      odd = odd || !is_plain(q[i]) || !is_plain(k[i]);
      grows = grows || !(fabsf(g[i]) <= 1.0f);
    }
    *reinterpret_cast<float4*>(sq + t * kStride + c) = *reinterpret_cast<const float4*>(q);
    *reinterpret_cast<float4*>(sk + t * kStride + c) = *reinterpret_cast<const float4*>(k);
    *reinterpret_cast<float4*>(sg + t * kStride + c) = *reinterpret_cast<const float4*>(g);
  }
  for (int idx = tid; idx < 2 * kScanBlock * kTokenStride; idx += 256) sp[idx] = 0.0f;
  if (kDelta && tid < kScanBlock) {
    sbeta[tid] = tid < length ? a.beta[(static_cast<size_t>(first) + tid) * a.heads + head] : 0.0f;
    odd = odd || !is_plain(sbeta[tid]);
  }
  if (__syncthreads_or(grows) && tid < kDim) {
    double product = 1.0;
    for (int t = 0; t < kScanBlock; ++t) {
      product *= static_cast<double>(sg[t * kStride + tid]);
      odd = odd || !is_plain(static_cast<float>(product));
    }
    product = 1.0;
    for (int t = kScanBlock - 1; t > 0; --t) {
      product *= static_cast<double>(sg[t * kStride + tid]);
      odd = odd || !is_plain(static_cast<float>(product));
    }
  }

  // ---- products of decays from the start and to the end, a thread per channel each
  float to_end[kScanBlock];
  bool wide_range = false;
  if (tid < kDim) {
    double product = 1.0;
#pragma unroll 4
    for (int t = 0; t < kScanBlock; ++t) {
      const double g = static_cast<double>(sg[t * kStride + tid]);
      if (kKind != kBlockBonus) product *= g;
      const float from_start = static_cast<float>(product);
      record[Record::kQ + t * Record::kRowStride + tid] = sq[t * kStride + tid] * from_start;
      if (kDelta) record[Record::kRows + t * Record::kRowStride + tid] = sk[t * kStride + tid] * from_start;
      if (kKind == kBlockBonus) product *= g;
    }
    record[Record::kG + tid] = static_cast<float>(product);
  } else if (tid < 2 * kDim) {
    const int c = tid - kDim;
    double product = 1.0;
#pragma unroll
    for (int t = kScanBlock - 1; t >= 0; --t) {
      to_end[t] = static_cast<float>(product);
      product *= static_cast<double>(sg[t * kStride + c]);
      wide_range = wide_range || !(to_end[t] >= 0x1p-40f && to_end[t] <= 0x1p40f);
    }
    wide_range = wide_range || !(static_cast<float>(product) >= 0x1p-40f && static_cast<float>(product) <= 0x1p40f);
#pragma unroll
    for (int t0 = 0; t0 < kScanBlock; t0 += 4)
      *reinterpret_cast<float4*>(record + Record::kEnd + c * kTokenStride + t0) =
          make_float4(sk[t0 * kStride + c] * to_end[t0], sk[(t0 + 1) * kStride + c] * to_end[t0 + 1], sk[(t0 + 2) * kStride + c] * to_end[t0 + 2],
                      sk[(t0 + 3) * kStride + c] * to_end[t0 + 3]);
  }
  if (odd) odd_flag = 1;
  if (__syncthreads_or(wide_range)) {
  {
    float w[4][kC], bonus[kC];
#pragma unroll
    for (int c = 0; c < kC; ++c)
    {
      bonus[c] = kKind == kBlockBonus && lane * kC + c < a.dim ? a.bonus[static_cast<size_t>(head) * a.dim + lane * kC + c] : 0.0f;
      if (!is_plain(bonus[c])) odd_flag = 1;
    }
    auto four_tokens = [&](int j0, int t0, auto own) {   // own: the keys' own four tokens
      constexpr bool kOwn = decltype(own)::value;
      constexpr int kValues = kDelta ? 32 : 16, kEach = kDelta ? 2 : 1;
      float values[kValues];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float q[kC], k[kC], g[kC];
        const int at = (t0 + i) * kStride + lane * kC;
        lane_channels(sq + at, q);
        lane_channels(sk + at, k);
        lane_channels(sg + at, g);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float p = 0.0f, m = 0.0f;
          if (kOwn && i == j) {
#pragma unroll
            for (int c = 0; c < kC; ++c) {
              w[j][c] = k[c];
              p = fmaf(kKind == kBlockBonus ? q[c] * bonus[c] : q[c], k[c], p);
            }
          } else if (!kOwn || i > j) {
#pragma unroll
            for (int c = 0; c < kC; ++c) {
              if (kKind != kBlockBonus) w[j][c] *= g[c];
              p = fmaf(q[c], w[j][c], p);
              if (kDelta) m = fmaf(k[c], w[j][c], m);
              if (kKind == kBlockBonus) w[j][c] *= g[c];
            }
          }
          values[(i * 4 + j) * kEach] = p;
          if (kDelta) values[(i * 4 + j) * kEach + kEach - 1] = m;
        }
      }
      // every exchange halves the values a lane keeps; the last one, where there are sixteen, only adds
#pragma unroll
      for (int off = 16, count = kValues; off >= 1; off >>= 1) {
        const bool upper = lane & off;
        if (count > 1) {
          count >>= 1;
#pragma unroll
          for (int i = 0; i < kValues / 2; ++i) {
            if (i < count) {
              const float keep = upper ? values[i + count] : values[i], send = upper ? values[i] : values[i + count];
              values[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
            }
          }
        } else {
          values[0] += __shfl_xor_sync(0xffffffffu, values[0], off);
        }
      }
      const int index = lane >> 1;
      float* to = (kDelta && (lane & 1)) ? sm : sp;
      if (kDelta || (lane & 1) == 0) to[(t0 + (index >> 2)) * kTokenStride + j0 + (index & 3)] = values[0];
    };
    // The first four groups of keys have 8 to 5 groups of tokens before them: their warps stop after five, and the warp of the
    // group opposite, which has few of its own, takes the rest from where the keys' running products have got to by then.
    constexpr int kMost = 20;
    const int own = warp * 4, left = (7 - warp) * 4, own_end = min(kScanBlock, own + kMost);
    four_tokens(own, own, std::true_type{});
    int keys = own;
    for (int t0 = own + 4;; t0 += 4) {
      if (keys == own && t0 == own_end) {
        if (warp < 4 || left + kMost >= kScanBlock) break;
        keys = left;
        t0 = left + kMost;
#pragma unroll
        for (int j = 0; j < 4; ++j) lane_channels(sk + (left + j) * kStride + lane * kC, w[j]);
#pragma unroll 1
        for (int t = left + 1; t < t0; ++t) {
          float g[kC];
          lane_channels(sg + t * kStride + lane * kC, g);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (t > left + j) {
#pragma unroll
              for (int c = 0; c < kC; ++c) w[j][c] *= g[c];
            }
          }
        }
      }
      if (t0 >= kScanBlock) break;
      four_tokens(keys, t0, std::false_type{});
    }
  }
  } else {
    // the bonus weighs the token's own pair, and its read-outs come before the token's own decay
    if (kKind == kBlockBonus) {
      float bonus[kC];
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        bonus[c] = lane * kC + c < a.dim ? a.bonus[static_cast<size_t>(head) * a.dim + lane * kC + c] : 0.0f;
        if (!is_plain(bonus[c])) odd_flag = 1;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = warp * 4 + i;
        float q[kC], k[kC], sum = 0.0f;
        lane_channels(sq + t * kStride + lane * kC, q);
        lane_channels(sk + t * kStride + lane * kC, k);
#pragma unroll
        for (int c = 0; c < kC; ++c) sum = fmaf(q[c] * bonus[c], k[c], sum);
        sum = warp_sum(sum);
        if (lane == 0) sbeta[t] = sum;
      }
      __syncthreads();
    }
    if (tid >= kDim && tid < 2 * kDim) {
      const int c = tid - kDim;
#pragma unroll
      for (int t = 0; t < kScanBlock; ++t) {
        const int at = t * kStride + c;
        const float k = sk[at], over = __frcp_rn(kKind == kBlockBonus ? to_end[t] * sg[at] : to_end[t]);
        sq[at] *= over;
        if (kDelta) sk[at] = k * over;
        sg[at] = k * to_end[t];
      }
    }
    __syncthreads();
    // tiles of 16 tokens by 8 keys, a warp's beside one another: with a correction four of rows (P, then M) by two pairs of
    // columns, else two of rows by four columns
    constexpr int kTiles = kDelta ? 2 : 1, kRowTiles = kDelta ? 4 : 2;
    const int row_tile = warp % kRowTiles, first_key = warp / kRowTiles * kTiles * 8, token = (row_tile & 1) * 16;
    if (first_key <= token + 15) {
      const int group = lane >> 2, two = (lane & 3) * 2;
      float sums[kTiles][4] = {};
      tile_products<kDim / 16, kTiles>(sums, (row_tile < 2 ? sq : sk) + (token + group) * kStride, kStride, FloatColumns{sg + first_key * kStride, kStride});
      float* to = row_tile < 2 ? sp : sm;
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = token + group + (i >> 1) * 8, j = first_key + n * 8 + two + (i & 1);
          if (j < t || (j == t && row_tile < 2)) to[t * kTokenStride + j] = kKind == kBlockBonus && j == t ? sbeta[t] : sums[n][i];
        }
      }
    }
  }
  __syncthreads();
  if (tid == 255) record[Record::kOdd] = odd_flag ? 1.0f : 0.0f;
  if (kDelta && warp == 0) {
    // column `lane` of T: forward substitution, the sums over the tokens before in four chains
    float x[kScanBlock];
#pragma unroll
    for (int t = 0; t < kScanBlock; ++t) {
      float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int s = 0; s < t; s += 4) {
        const float4 m = *reinterpret_cast<const float4*>(sm + t * kTokenStride + s);
        sum[0] = fmaf(m.x, x[s], sum[0]);
        if (s + 1 < t) sum[1] = fmaf(m.y, x[s + 1], sum[1]);
        if (s + 2 < t) sum[2] = fmaf(m.z, x[s + 2], sum[2]);
        if (s + 3 < t) sum[3] = fmaf(m.w, x[s + 3], sum[3]);
      }
      const float beta = sbeta[t];
      x[t] = t == lane ? beta : (t > lane ? -beta * ((sum[0] + sum[1]) + (sum[2] + sum[3])) : 0.0f);
      record[Record::kT + t * kTokenStride + lane] = x[t];
    }
  } else {
    for (int idx = tid - (kDelta ? 32 : 0); idx < kScanBlock * kTokenStride; idx += kDelta ? 224 : 256) record[Record::kP + idx] = sp[idx];
  }
}

// Tokens one after the other, as the walk takes them, for what the products cannot say.
// `S`: a CTA's columns at the start, [kCols][kDim] in shared memory, afterwards those at the end; a lane holds kRows rows of one.
template <int kDim, int kKind, int kCols, int kThreads>
__device__ __noinline__ void walk_tokens(const ScanBlockArgs& args, float* S, int head, int col0, int first, int length) {
  constexpr int kLanes = kThreads / kCols, kRows = kDim / kLanes;
  static_assert(kLanes <= 32 && 32 % kLanes == 0 && kDim % kLanes == 0, "a column's lanes are neighbours in a warp");
  const ScanBlockArgs a = args;      // (what is written below could lie anywhere)
  const int col = static_cast<int>(threadIdx.x) / kLanes, part = static_cast<int>(threadIdx.x) % kLanes;
  const bool inside = col0 + col < a.vdim;
  const size_t kv_col = static_cast<size_t>(head / (a.heads / a.kv_heads)) * a.dim;
  float* column = S + col * kDim;
  auto column_sum = [](float x) {
#pragma unroll
    for (int off = kLanes / 2; off >= 1; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    return x;
  };
  float s[kRows], bonus[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int r = part + i * kLanes;
    s[i] = column[r];
    bonus[i] = kKind == kBlockBonus && r < a.dim ? a.bonus[static_cast<size_t>(head) * a.dim + r] : 0.0f;
  }
#pragma unroll 1
  for (int t = 0; t < length; ++t) {
    const size_t row = static_cast<size_t>(first) + t, own = row * a.heads + head;
    const float* decay = a.decay + (a.decay_mode == 0 ? head : a.decay_mode == 1 ? own : own * a.dim);
    const float v = inside ? a.v[row * a.v_stride + static_cast<size_t>(head) * a.vdim + col0 + col] : 0.0f;
    const float strength = kKind == kBlockDelta ? a.beta[own] : a.v_scale ? a.v_scale[own] : 1.0f;
    float q[kRows], k[kRows], g[kRows], seen = 0.0f, read = 0.0f;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int r = part + i * kLanes;
      const bool good = r < a.dim;
      q[i] = good ? a.q[row * a.q_stride + kv_col + r] : 0.0f;
      k[i] = good ? a.k[row * a.k_stride + kv_col + r] : 0.0f;
      g[i] = good ? decay[a.decay_mode == 2 ? r : 0] : 1.0f;
    }
    if (kKind == kBlockDelta) {
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        s[i] *= g[i];
        if (part + i * kLanes < a.dim) seen = fmaf(s[i], k[i], seen);
      }
      seen = column_sum(seen);
    }
    const float u = kKind == kBlockDelta ? strength * (v - seen) : a.v_scale ? strength * v : v;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      if (part + i * kLanes >= a.dim) continue;      // (rows that are not there take no part, whatever u is)
      const float pair = k[i] * u, kept = s[i];
      s[i] = kKind == kBlockDelta ? fmaf(k[i], u, kept) : fmaf(kept, g[i], pair);
      read = fmaf(kKind == kBlockBonus ? fmaf(bonus[i], pair, kept) : s[i], q[i], read);
    }
    read = column_sum(read);
    if (inside && part == 0) a.out[row * a.out_stride + static_cast<size_t>(head) * a.vdim + col0 + col] = a.skip ? read + a.skip[head] * v : read;
  }
#pragma unroll
  for (int i = 0; i < kRows; ++i) column[part + i * kLanes] = s[i];
}

// Warps of a CTA: for every 16 rows times 16 columns of S two, half of the channels each; then the tiles of S are dealt to them.
template <int kDim, int kKind>
struct BlockShape {
  static constexpr bool kDelta = kKind == kBlockDelta;
  static constexpr int kCols = kDim == 128 && !kDelta ? 32 : 16;          // columns of S a CTA owns
  static constexpr int kBuffers = 2;                                      // of records
  static constexpr int kRowTiles = kDelta ? 4 : 2, kTasks = kRowTiles * kCols / 16, kWarps = 2 * kTasks, kThreads = 32 * kWarps;
  static constexpr int kStateTiles = kDim / 16, kOwn = kStateTiles * (kCols / 8) / kWarps;      // tiles of S a warp owns
  static_assert(kWarps % kStateTiles == 0 && (kDelta || kThreads * 4 == kScanBlock * kCols), "work for every warp");
  static constexpr int kRecord = BlockRecord<kDim, kDelta>::kSize;
  static constexpr int kStateStride = kDim / 2 + 4, kValueStride = kScanBlock / 2 + 4;      // words of two numbers' parts in a column
  static constexpr int kStatePart = kCols * kStateStride, kValuePart = kCols * kValueStride, kState = 3 * kStatePart, kValues = 3 * kValuePart;
  static constexpr int kFloats = kBuffers * kRecord + 2 * kState + 2 * kValues + kTasks * 256;
};

__device__ __forceinline__ void bulk_copy(uint32_t to, const float* from, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(from), "r"(bytes),
               "r"(bar) : "memory");
}

// Registers for one CTA a multiprocessor where shared memory holds no more (with a correction, keys of 128: 267 us with 128 registers a
// thread, 256 with 164, 2,048 tokens of 16 heads); without a correction more of them are slower (290 us, 313 with 186).
template <int kDim, int kKind>
__global__ void __launch_bounds__(BlockShape<kDim, kKind>::kThreads, kDim == 128 && kKind == kBlockDelta ? 1 : 2) scan_blocks_kernel(const __grid_constant__ ScanBlockArgs a) {
  using Shape = BlockShape<kDim, kKind>;
  constexpr bool kDelta = Shape::kDelta;
  using Record = BlockRecord<kDim, kDelta>;
  constexpr int kCols = Shape::kCols;
  extern __shared__ __align__(128) float block_floats[];
  __shared__ __align__(8) uint64_t full_bar[Shape::kBuffers];
  __shared__ int aborted_flag;
  volatile int* aborted = &aborted_flag;
  uint32_t* states = reinterpret_cast<uint32_t*>(block_floats + Shape::kBuffers * Shape::kRecord);      // columns of S, of this block and the next
  uint32_t* values = states + 2 * Shape::kState;                         // of U, of this block and of the next, or of U and of R
  float4* halves = reinterpret_cast<float4*>(values + 2 * Shape::kValues);      // [task][tile][lane]
  const int head = blockIdx.x, col0 = blockIdx.y * kCols;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // The longest entries first: the last ones to start are short (700, 333 and 1,015 tokens of 32 heads of 128: 228 us in their
  // order).  So the first CTAs have all the work there is, and entries that are not taken here get none: beside 600 tokens of 32
  // heads of 128, 64 single ones had 8,192, each with 155 KB of shared memory: 284 us, now 204.
  __shared__ int entry;
  if (tid == 0) entry = -1;
  __syncthreads();
  for (int i = tid; i < a.entries; i += Shape::kThreads) {
    const int own = blocks_of(a, i);
    if (own == 0) continue;
    int longer = 0;
    for (int j = 0; j < a.entries; ++j) {
      const int other = blocks_of(a, j);
      longer += other > own || (other == own && j < i);
    }
    if (longer == static_cast<int>(blockIdx.z)) entry = i;
  }
  __syncthreads();
  const int e = entry;
  if (e < 0) return;
  const int blocks = blocks_of(a, e);
  int before = 0;
  for (int i = 0; i < e; ++i) before += blocks_of(a, i);
  const int first = a.cu_seqlens[e], length = a.cu_seqlens[e + 1] - first;
  int slot = a.entry_slot[e];
  const bool slot_ok = slot >= 0 && slot < a.slots;
  if (!slot_ok) {
    if (tid == 0) atomicOr(a.fault, kFaultSlot);
    slot = 0;
  }
  float* home = a.state + slot * a.state_stride + static_cast<size_t>(head) * a.dim * a.vdim;
  const float* records = a.records + (static_cast<size_t>(before) * a.heads + head) * Record::kSize;
  int fetched = 0;
  auto fetch = [&](int block) {      // one thread
    ++fetched;
    const uint32_t bar = smem_addr(&full_bar[block % Shape::kBuffers]);
    mbar_expect_tx(bar, Record::kSize * 4);
    bulk_copy(smem_addr(block_floats + (block % Shape::kBuffers) * Shape::kRecord), records + static_cast<size_t>(block) * a.heads * Record::kSize,
              Record::kSize * 4, bar);
  };
  if (tid == 0) {
    for (int b = 0; b < Shape::kBuffers; ++b) mbar_init(smem_addr(&full_bar[b]), 1);
    aborted_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int b = 0; b < Shape::kBuffers - 1 && b < blocks; ++b) fetch(b);
  }
  // this warp's tile of rows (with a correction the first two of four make R, the others the read-outs) and its tiles of S
  const int task = warp >> 1, half = warp & 1, row_tile = task % Shape::kRowTiles, task_col = task / Shape::kRowTiles * 16;
  const bool reads = !kDelta || row_tile >= 2;
  const int token_tile = (kDelta ? row_tile & 1 : row_tile) * 16, my_col = task_col + half * 8;
  float4* shared_half = halves + task * 64 + lane;
  const int s_row = warp % Shape::kStateTiles * 16 + g, s_col = warp / Shape::kStateTiles * Shape::kOwn * 8;
  float S[Shape::kOwn][4];
#pragma unroll
  for (int n = 0; n < Shape::kOwn; ++n) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = s_row + (i >> 1) * 8, col = col0 + s_col + n * 8 + 2 * t + (i & 1);
      S[n][i] = a.entry_start[e] > 0 && row < a.dim && col < a.vdim ? home[static_cast<size_t>(col) * a.dim + row] : 0.0f;
    }
  }
  auto show_state = [&](int block) {
    uint32_t* state = states + (block & 1) * Shape::kState;
#pragma unroll
    for (int n = 0; n < Shape::kOwn; ++n) show_tile(S[n], state, Shape::kStateStride, Shape::kStatePart, s_col + n * 8, s_row - g);
  };
  auto value_columns = [&](int which, int col) { return PartColumns{values + which * Shape::kValues + col * Shape::kValueStride, Shape::kValueStride, Shape::kValuePart}; };
  // V a block ahead: with a correction what this warp's tile of R wants, else two columns of two tokens a thread.  What lies
  // outside is loaded from inside and made zero where it is used: a choice at the load would wait for it.
  float v[4], v_scale[2] = {1.0f, 1.0f};
  const int v_token = tid / (kCols / 2) * 2, v_col = tid % (kCols / 2) * 2;
  auto fetch_values = [&](int block) {
    const int last = length - 1 - block * kScanBlock;
    const float* base = a.v + (static_cast<size_t>(first) + block * kScanBlock) * a.v_stride + head * a.vdim;
    if constexpr (kDelta) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        v[i] = base[static_cast<size_t>(min(token_tile + g + (i >> 1) * 8, last)) * a.v_stride + min(col0 + my_col + 2 * t + (i & 1), a.vdim - 1)];
    } else {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int token = min(v_token + i, last);
        const float* from = base + static_cast<size_t>(token) * a.v_stride + min(col0 + v_col, a.vdim - 2);
        if (a.wide_in) {
          const float2 two = *reinterpret_cast<const float2*>(from);
          v[2 * i] = two.x; v[2 * i + 1] = two.y;
        } else {
          v[2 * i] = from[0]; v[2 * i + 1] = from[1];
        }
        if (a.v_scale) v_scale[i] = a.v_scale[(static_cast<size_t>(first) + block * kScanBlock + token) * a.heads + head];
      }
    }
  };
  auto show_values = [&](int block) {      // without a correction: columns of U; true if one of them is not plain
    bool odd = false;
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool inside = block * kScanBlock + v_token + (i >> 1) < length && col0 + v_col < a.vdim;      // vdim is a multiple of four
      x[i] = inside ? (a.v_scale ? v[i] * v_scale[i >> 1] : v[i]) : 0.0f;
      odd = odd || !is_plain(x[i]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t parts[3];
      bf16_parts(x[i], x[2 + i], parts);
#pragma unroll
      for (int j = 0; j < 3; ++j) values[(block & 1) * Shape::kValues + j * Shape::kValuePart + (v_col + i) * Shape::kValueStride + (v_token >> 1)] = parts[j];
    }
    return odd;
  };
  const float skip = a.skip ? a.skip[head] : 0.0f;
  // Blocks whose record says so are not taken here, nor those behind them.
  __shared__ int first_odd;
  if (tid == 0) first_odd = blocks;
  __syncthreads();
  for (int i = tid; i < blocks; i += Shape::kThreads)
    if (records[static_cast<size_t>(i) * a.heads * Record::kSize + Record::kOdd] != 0.0f) atomicMin(&first_odd, i);
  __syncthreads();
  const int plain_blocks = first_odd;
  bool odd = false;
  int walk_from = -1;      // the block from whose start on the tokens are walked, with its state in registers
#pragma unroll
  for (int n = 0; n < Shape::kOwn; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) odd = odd || !is_plain(S[n][i]);
  show_state(0);
  fetch_values(0);
  if constexpr (!kDelta) {
    odd = show_values(0) || odd;
    if (blocks > 1) fetch_values(1);
  }
  for (int block = 0; block < plain_blocks; ++block) {
    const float* record = block_floats + (block % Shape::kBuffers) * Shape::kRecord;
    const uint32_t* state = states + (block & 1) * Shape::kState;
    __syncwarp();
    if (__syncthreads_or(odd)) {      // S and, without a correction, U are there; the record before is done with
      walk_from = block;
      break;
    }
    // Once a record did not come nothing more is asked for (a barrier with bytes outstanding takes no others): what follows ends at
    // once, and nothing of it is kept.  The threads do not agree on that block by block, which would take 5 % of a block's time.
    if (tid == 0 && block + Shape::kBuffers - 1 < blocks && !*aborted) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      fetch(block + Shape::kBuffers - 1);
    }
    __syncwarp();
    mbar_wait(smem_addr(&full_bar[block % Shape::kBuffers]), (block / Shape::kBuffers) & 1, aborted, a.fault);
    __syncwarp();      // the products below are the whole warp's
    float sums[2][4] = {};
    tile_products<kDim / 32, 2>(sums, record + (row_tile * 16 + g) * Record::kRowStride + half * (kDim / 2), Record::kRowStride,
                                PartColumns{state + task_col * Shape::kStateStride + half * (kDim / 4), Shape::kStateStride, Shape::kStatePart});
    // the two halves' warps give each other one tile's sums, so that each ends up with one whole tile
    float mine[1][4];
    shared_half[(half ^ 1) * 32] = half ? make_float4(sums[0][0], sums[0][1], sums[0][2], sums[0][3])
                                        : make_float4(sums[1][0], sums[1][1], sums[1][2], sums[1][3]);
    __syncthreads();
    {
      const float4 other = shared_half[half * 32];
      const float others[4] = {other.x, other.y, other.z, other.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) mine[0][i] = (half ? sums[1][i] : sums[0][i]) + others[i];
    }
    const int u = kDelta ? 0 : block & 1;      // which of the two
    if constexpr (kDelta) {
      if (!reads) {
        float left[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int token = block * kScanBlock + token_tile + g + (i >> 1) * 8, col = col0 + my_col + 2 * t + (i & 1);
          left[i] = (token < length && col < a.vdim ? v[i] : 0.0f) - mine[0][i];
          odd = odd || !is_plain(left[i]);
        }
        __syncwarp();
        show_tile(left, values + Shape::kValues, Shape::kValueStride, Shape::kValuePart, my_col, token_tile);
        if (block + 1 < blocks) fetch_values(block + 1);
      }
      __syncwarp();
      if (__syncthreads_or(odd)) {      // R is there
        walk_from = block;
        break;
      }
      if (!reads) {
        float rows[1][4] = {};
        tile_products<kScanBlock / 16, 1>(rows, record + Record::kT + (token_tile + g) * kTokenStride, kTokenStride, value_columns(1, my_col));
        show_tile(rows[0], values, Shape::kValueStride, Shape::kValuePart, my_col, token_tile);
#pragma unroll
        for (int i = 0; i < 4; ++i) odd = odd || !is_plain(rows[0][i]);
      }
      __syncwarp();
      if (__syncthreads_or(odd)) {      // U is there
        walk_from = block;
        break;
      }
    }
    float added[Shape::kOwn][4] = {};
    tile_products<kScanBlock / 16, Shape::kOwn>(added, record + Record::kEnd + s_row * kTokenStride, kTokenStride, value_columns(u, s_col));
    const float decay[2] = {record[Record::kG + s_row], record[Record::kG + s_row + 8]};
#pragma unroll
    for (int n = 0; n < Shape::kOwn; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) S[n][i] = fmaf(S[n][i], decay[i >> 1], added[n][i]);
    show_state(block + 1);      // (the other of the two: this block's is still being read)
    if constexpr (!kDelta) {
      if (block + 1 < blocks) odd = show_values(block + 1);
      if (block + 2 < blocks) fetch_values(block + 2);
    }
    if (reads) {
      __syncwarp();      // (keeps these loads behind the state's products: 2 % of the kernel without a correction)
      tile_products<kScanBlock / 16, 1>(mine, record + Record::kP + (token_tile + g) * kTokenStride, kTokenStride, value_columns(u, my_col));
      const int col = col0 + my_col + 2 * t;
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const int token = block * kScanBlock + token_tile + g + i * 4;
        if (token < length && col < a.vdim) {      // vdim is a multiple of four: both columns
          const size_t at = static_cast<size_t>(first) + token;
          float* to = a.out + at * a.out_stride + head * a.vdim + col;
          const float* from = a.v + at * a.v_stride + head * a.vdim + col;
#pragma unroll
          for (int j = 0; j < 2; ++j) to[j] = a.skip ? mine[0][i + j] + skip * from[j] : mine[0][i + j];
        }
      }
    }
  }
  __syncthreads();
  const bool gave_up = *aborted;
  if (walk_from < 0 && plain_blocks < blocks) walk_from = plain_blocks;
  if (walk_from >= 0 && !gave_up) {
    float* plain = reinterpret_cast<float*>(states);      // the parts that lie there are done with
    static_assert(kCols * kDim <= 2 * Shape::kState, "room for the state");
    auto each = [&](auto act) {
#pragma unroll
      for (int n = 0; n < Shape::kOwn; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) act(S[n][i], plain + (s_col + n * 8 + 2 * t + (i & 1)) * kDim + s_row + (i >> 1) * 8);
    };
    each([](float& x, float* at) { *at = x; });
    __syncthreads();
    walk_tokens<kDim, kKind, kCols, Shape::kThreads>(a, plain, head, col0, first + walk_from * kScanBlock, length - walk_from * kScanBlock);
    __syncthreads();
    each([](float& x, float* at) { x = *at; });
  }
  if (slot_ok && !gave_up) {
#pragma unroll
    for (int n = 0; n < Shape::kOwn; ++n) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = s_row + (i >> 1) * 8, col = col0 + s_col + n * 8 + 2 * t + (i & 1);
        if (row < a.dim && col < a.vdim) home[static_cast<size_t>(col) * a.dim + row] = S[n][i];
      }
    }
  }
  if ((gave_up || walk_from >= 0) && tid == 0) {      // copies land before the shared memory goes
    volatile int go_on = 0;
    for (int b = 0; b < Shape::kBuffers; ++b) {
      const int fills = (fetched - b + Shape::kBuffers - 1) / Shape::kBuffers;
      if (fills > 0) mbar_wait(smem_addr(&full_bar[b]), (fills - 1) & 1, &go_on, a.fault);
    }
  }
}

template <int kDim, int kKind>
static int launch_blocks(const ScanBlockArgs& a, int blocks, int taken, cudaStream_t stream) {
  using Shape = BlockShape<kDim, kKind>;
  static std::atomic<unsigned long long> prepared, configured;
  auto prepare = scan_prepare_kernel<kDim, kKind>;
  cudaError_t e = allow_shared(prepare, prepare_smem<kDim, kKind>(), prepared);
  if (e != cudaSuccess) return static_cast<int>(e);
  prepare<<<dim3(blocks, a.heads), 256, prepare_smem<kDim, kKind>(), stream>>>(a);
  int r = launch_status();
  if (r) return r;
  auto walk = scan_blocks_kernel<kDim, kKind>;
  e = allow_shared(walk, Shape::kFloats * 4, configured);
  if (e != cudaSuccess) return static_cast<int>(e);
  walk<<<dim3(a.heads, (a.vdim + Shape::kCols - 1) / Shape::kCols, taken), Shape::kThreads, Shape::kFloats * 4, stream>>>(a);
  return launch_status();
}

int scan_blocks(const ScanBlockArgs& a, int blocks, int taken, cudaStream_t stream) {
  const int least = a.beta ? 32 : 64;      // smaller heads without a correction are ahead in pieces
  if (a.dim <= least || a.dim > 128 || a.dim % 4 || a.vdim % 4 || blocks < 1 || taken < 1 || taken > 65535 || a.from < 1 || a.records == nullptr ||
      reinterpret_cast<uintptr_t>(a.records) % 16)
    return static_cast<int>(cudaErrorInvalidValue);
  if (a.beta) return a.dim <= 64 ? launch_blocks<64, kBlockDelta>(a, blocks, taken, stream) : launch_blocks<128, kBlockDelta>(a, blocks, taken, stream);
  return a.bonus ? launch_blocks<128, kBlockBonus>(a, blocks, taken, stream) : launch_blocks<128, kBlockPlain>(a, blocks, taken, stream);
}

}  // namespace rl
