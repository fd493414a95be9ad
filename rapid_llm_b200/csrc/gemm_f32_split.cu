// 32-bit matrix products on the tensor cores: C[M, N] = A[M, K] * W[N, K]^T (+ bias), float32 in, float32 out.
//
// A float32 number is exactly the sum of three bfloat16 ones, each what the ones before leave, rounded to nearest (Dekker's
// splitting, in three): the second is at most 2^-8 of the number's leading power of two, the third 2^-17.  Of the nine products
// of two such sums six are formed, each exact in the tensor core's float32:
//   w0 x0                                          summed over 256 columns, then added to a float32 sum in registers
//   w0 x1, w1 x0, w1 x1, w0 x2, w2 x0              summed over all columns in an accumulator of their own
// What is left out, w1 x2 + w2 x1 + w2 x2, stays within 2^-24 of a product, either way (parts that are cut off instead of rounded
// leave out up to 2^-21 of it, always towards zero).  The tensor core cuts off what lies below its accumulator's last bit; 256
// columns at a time, and with the small products apart, that costs less than the roundings of one fused multiply-add after the
// other.  Relative error, multiply-adds / here, inner extent 4,096: operands of mean zero 1.15e-6 / 2.4e-7, all positive 8.4e-7 /
// 3.1e-7; rows with few numbers that are not zero, 1 2.54e-8 / 2.6e-8, 2 3.0e-8 / 3.6e-8 (each segment's sum is rounded), 4
// 3.9e-8 / 4.4e-8, 8 5.3e-8 / 5.3e-8, 32 1.0e-7 / 6.1e-8.  Forming w1 x2 and w2 x1 too brings a single number's to 2.54e-8, the
// others nowhere, for 7 to 17 % of the time at 64 rows and more.
//
// An output is a sum in an order that n and k alone decide (256 columns, then the columns of a segment, then the segments,
// whose number `split_segments` takes from n and k): not M, the tile it falls in, or what else is in the batch.
// A product of an infinity's or a NaN's parts is not finite; such outputs are formed again from the numbers themselves.
//
// A CTA owns 128 weight rows (the lanes of the accumulators), up to 208 tokens and a segment of the columns.  TMA brings the
// weights 32 columns at a time; eight warps cut them into their parts, which go to tensor memory: there they are an operand
// that costs no shared memory (read from it six times a step they were the bound: 54 of 94 KB a step at 16 tokens).  The
// tokens' parts come by TMA too, cut once per product by split_rows_kernel; few tokens are cut beside the weights.  The
// workers add finished sums to their registers while the small products of the columns after them run.  The CTAs of a cluster
// hold the segments of a tile and add them up through each other's shared memory.
#include <cuda.h>

#include "tc_common.cuh"

namespace rl {

constexpr int kSplitM = 128;          // weight rows per CTA
constexpr int kSplitK = 32;           // columns per buffer: rows of 64 bytes
constexpr int kSplitSum = 8;          // buffers whose main products are summed before they go to the registers
constexpr int kSplitWorkers = 256;
constexpr int kSplitMaxTokens = 208;  // two accumulators of as many columns beside 96 for the weights' parts fill tensor memory
constexpr int kSplitPartColumns = kSplitK / 2;      // of tensor memory, two bfloat16 each

// What a token tile's size decides: two CTAs a multiprocessor up to 64 tokens, one above.
template <int kTokens, bool kCopied>
struct SplitShape {
  static constexpr int kPerMultiprocessor = kTokens <= 64 ? 2 : 1;
  static constexpr int kThreads = kSplitWorkers + (kCopied ? 96 : 64);
  // of parts: what hides the way from a buffer's last product to the next one written and back, some 1,000 cycles
  static constexpr int kBuffers = kTokens <= 32 || kTokens == 128 ? 4 : 2;
  static constexpr int kUsedColumns = 2 * kTokens + kBuffers * 3 * kSplitPartColumns;
  static constexpr int kColumns = kUsedColumns <= 128 ? 128 : kUsedColumns <= 256 ? 256 : 512;
  static constexpr int kBufferBytes = 3 * kTokens * kSplitK * 2;                          // the tokens' parts
  static constexpr int kRawBytes = (kSplitM + (kCopied ? 0 : kTokens)) * kSplitK * 4;     // weights (and few tokens) as they lie in memory
  static constexpr int kRaw = kTokens > 64 ? 6 : 4;
  static_assert(kRaw % 2 == 0 && kBuffers % 2 == 0, "a place of a ring belongs to one of the two groups: a wait knows a fill from the one before it only");
  static constexpr int kSmem = kBuffers * kBufferBytes + kRaw * kRawBytes + 1024;
};

struct SplitArgs {
  const float* a;
  const float* w;
  const float* bias;
  float* c;
  int m, n, k, lda, ldc;
  int tile_tokens;        // a multiple of 16
  int segment;            // columns a CTA takes: a multiple of 256
  int a_in_fours;         // rows of A can be fetched 16 bytes at a time
  int* fault;
};

// K-major rows of 64 bytes, 64-byte swizzle, groups of eight rows 512 bytes apart.
__device__ __forceinline__ uint64_t operand_desc_64(uint32_t smem_address) {
  return static_cast<uint64_t>((smem_address & 0x3FFFFu) >> 4) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}

// Takes the next part off two neighbouring numbers, side by side in a word: rounded to nearest, which leaves exactly what the
// parts behind it have to hold.
__device__ __forceinline__ uint32_t next_parts(float& x, float& y) {
  const __nv_bfloat162 both = __floats2bfloat162_rn(x, y);
  const uint32_t word = *reinterpret_cast<const uint32_t*>(&both);
  x -= __uint_as_float(word << 16);
  y -= __uint_as_float(word & 0xffff0000u);
  return word;
}

// Eight columns of a row into the three parts' buffers, 16 bytes each.
__device__ __forceinline__ void store_parts(uint32_t at, uint32_t part_bytes, float (&v)[8]) {
#pragma unroll
  for (int part = 0; part < 3; ++part)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + part * part_bytes), "r"(next_parts(v[0], v[1])),
                 "r"(next_parts(v[2], v[3])), "r"(next_parts(v[4], v[5])), "r"(next_parts(v[6], v[7])) : "memory");
}
// Four columns (the `quad`th) of a row of 32 in the 128-byte-swizzled layout.
__device__ __forceinline__ void load_raw(uint32_t base, int row, int quad, float* v) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(base + row * 128 + ((quad ^ (row & 7)) << 4)) : "memory");
}

// Four numbers where `good`, without a branch, so that many loads are on their way at once.
__device__ __forceinline__ void load_four_or_zeros(float (&v)[4], const float* from, bool good) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n mov.f32 %2, 0f00000000;\n"
      " mov.f32 %3, 0f00000000;\n @p ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n}\n"
      : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3]) : "l"(from), "r"(static_cast<int>(good)));
}

__device__ __forceinline__ bool split_finite(float sum) { return fabsf(sum) <= 3.402823466e38f; }

// A warp's outputs of one token that are not finite, formed from the numbers themselves, for what the parts cannot say: NaN where
// the token's row has one, else a sum over the columns that the lanes share out.  24,576 x 4,096, us: one of 64 rows with a NaN 231 (with
// none 103; every output down the columns by a lane of its own 4,139), 203 rows of them 1,562 (249; 86,158), one of 64 with an infinity
// 4,400.
__device__ __noinline__ void split_again(const SplitArgs& args, float (&sums)[4], int token, int row0) {
  const int lane = threadIdx.x & 31, k = args.k;
  const float* a = args.a + static_cast<size_t>(token) * args.lda;
  bool nan = false;
#pragma unroll 8
  for (int i = lane; i < k; i += 32) nan = nan || a[i] != a[i];
  if (__any_sync(0xffffffffu, nan)) {
#pragma unroll
    for (int j = 0; j < 4; ++j) sums[j] = __int_as_float(0x7fffffff);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    unsigned left = __ballot_sync(0xffffffffu, row0 + j < args.n && !split_finite(sums[j]));
    while (left) {
      const int whose = __ffs(left) - 1;
      left &= left - 1;
      const float* w = args.w + static_cast<size_t>(__shfl_sync(0xffffffffu, row0, whose) + j) * k;
      float sum = 0.0f;
#pragma unroll 8
      for (int i = lane * 4; i < k; i += 128) {      // k is a multiple of four, w on a 16-byte boundary
        const float4 four = *reinterpret_cast<const float4*>(w + i);
        sum = fmaf(a[i + 3], four.w, fmaf(a[i + 2], four.z, fmaf(a[i + 1], four.y, fmaf(a[i], four.x, sum))));
      }
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      if (lane == whose) sums[j] = sum;
    }
  }
}

// The parts of A's rows, one part after the other: [3][m][kp], kp columns of which those behind k are zeros.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* a, int lda, int in_fours, __nv_bfloat16* parts, int m, int k, int kp) {
  const int col = (blockIdx.x * 256 + threadIdx.x) * 4, row = blockIdx.y;
  if (col >= kp) return;
  float v[4];
  const float* from = a + static_cast<size_t>(row) * lda + col;
  if (in_fours) {
    load_four_or_zeros(v, from, col < k);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = col < k ? from[j] : 0.0f;
  }
#pragma unroll
  for (int part = 0; part < 3; ++part)
    *reinterpret_cast<uint2*>(parts + (static_cast<size_t>(part) * m + row) * kp + col) = make_uint2(next_parts(v[0], v[1]), next_parts(v[2], v[3]));
}

// kCopied: the tokens' parts lie in memory (map_x: [3 m, kp] of them), else their rows do (map_x: [m, k] of float32).
template <int kTokens, bool kCopied>
__global__ void __launch_bounds__(SplitShape<kTokens, kCopied>::kThreads, SplitShape<kTokens, kCopied>::kPerMultiprocessor)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                      const __grid_constant__ SplitArgs args) {
  using Shape = SplitShape<kTokens, kCopied>;
  constexpr int kBuffers = Shape::kBuffers, kRaw = Shape::kRaw;
  constexpr int kAcc = (kTokens + 31) / 32 * 16;                    // outputs a thread
  extern __shared__ unsigned char split_raw[];
  __shared__ __align__(8) uint64_t full_bar[kBuffers], copied_bar[kBuffers], empty_bar[kBuffers], raw_full_bar[kRaw], raw_empty_bar[kRaw],
      acc_full_bar, acc_empty_bar, drain_bar;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int aborted_flag, fault_here;
  volatile int* aborted = &aborted_flag;
  int* fault = args.fault ? args.fault : &fault_here;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const uint32_t smem_base = (smem_addr(split_raw) + 1023u) & ~1023u;
  const int tokens = args.tile_tokens;
  const uint32_t part_x = static_cast<uint32_t>(tokens) * kSplitK * 2;
  auto buffer_x = [&](int b) { return smem_base + b * Shape::kBufferBytes; };
  auto raw_w = [&](int r) { return smem_base + kBuffers * Shape::kBufferBytes + r * Shape::kRawBytes; };
  auto raw_x = [&](int r) { return raw_w(r) + kSplitM * kSplitK * 4; };
  const int rank = blockIdx.x, segments = gridDim.x;                // a cluster is a row of the grid
  const int n0 = blockIdx.y * kSplitM, t0 = blockIdx.z * tokens;
  const int k_begin = rank * args.segment, k_end = min(args.k, k_begin + args.segment);
  const int steps = max(0, (k_end - k_begin + kSplitK - 1) / kSplitK);

  if (tid == 0) {
    for (int b = 0; b < kBuffers; ++b) {
      mbar_init(smem_addr(&full_bar[b]), kSplitWorkers / 64);
      mbar_init(smem_addr(&copied_bar[b]), 1);
      mbar_init(smem_addr(&empty_bar[b]), 1);
    }
    for (int r = 0; r < kRaw; ++r) {
      mbar_init(smem_addr(&raw_full_bar[r]), 1);
      mbar_init(smem_addr(&raw_empty_bar[r]), kSplitWorkers / 64);
    }
    mbar_init(smem_addr(&acc_full_bar), 1);
    mbar_init(smem_addr(&acc_empty_bar), kSplitWorkers / 32);
    mbar_init(smem_addr(&drain_bar), 1);
    aborted_flag = 0;
    fault_here = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    tmem_alloc(smem_addr(&tmem_base_slot), Shape::kColumns);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(tmem_base_slot);
  const uint32_t parts_w = tmem_base + 2 * kTokens;                 // [buffer][part][16 columns]
  const int live = min(tokens, args.m - t0);
  float* mine = reinterpret_cast<float*>(split_raw + (smem_base - smem_addr(split_raw)));      // [token][weight row]
  // a warp reads the 32 lanes of its number modulo four; the first four warps take the first columns, the others the rest
  const int first_half = (tokens + 31) / 32 * 16, my_col0 = warp < 4 ? 0 : first_half;
  const int my_cols = warp < 4 ? first_half : tokens - first_half;
  if (warp >= 8) {
    if (warp == 8) {
      const bool leader = elect_one();
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(tokens >> 3) << 17) |
                             (static_cast<uint32_t>(kSplitM >> 4) << 24);
      int b = 0;
      uint32_t phase = 0;
      for (int step = 0; step < steps; ++step) {
        bool ready = mbar_wait(smem_addr(&full_bar[b]), phase, aborted, fault);
        if (kCopied) ready = ready && mbar_wait(smem_addr(&copied_bar[b]), phase, aborted, fault);
        if (!__all_sync(0xffffffffu, ready)) break;
        tc_fence_after();
        const uint32_t w = parts_w + b * 3 * kSplitPartColumns, px = part_x >> 4;
        const uint64_t x = operand_desc_64(buffer_x(b));
        auto product = [&](uint32_t into, int wp, int xp, bool begin) {
#pragma unroll
          for (int h = 0; h < kSplitK / 16; ++h)
            umma_bf16_ts(into, w + wp * kSplitPartColumns + 8 * h, x + xp * px + 2 * h, idesc, (begin && h == 0) ? 0u : 1u);
        };
        if (leader) {
          product(tmem_base + kTokens, 0, 2, step == 0);
          product(tmem_base + kTokens, 2, 0, false);
          product(tmem_base + kTokens, 1, 1, false);
          product(tmem_base + kTokens, 0, 1, false);
          product(tmem_base + kTokens, 1, 0, false);
        }
        const bool begins = step % kSplitSum == 0;
        if (begins && step > 0) {
          if (!__all_sync(0xffffffffu, mbar_wait(smem_addr(&acc_empty_bar), (step / kSplitSum - 1) & 1, aborted, fault))) break;
          tc_fence_after();
        }
        if (leader) {
          product(tmem_base, 0, 0, begins);
          umma_commit(smem_addr(&empty_bar[b]));
          if (step % kSplitSum == kSplitSum - 1 || step == steps - 1) umma_commit(smem_addr(&acc_full_bar));
        }
        __syncwarp();
        if (++b == kBuffers) { b = 0; phase ^= 1u; }
      }
      // nothing of this CTA may still be running on the tensor core when its memory is freed
      if (leader) umma_commit(smem_addr(&drain_bar));
      __syncwarp();
      volatile int go_on = 0;
      mbar_wait(smem_addr(&drain_bar), 0, &go_on, fault);
    }
    // a ring's copies: `fill` starts those of one step.  They land before the shared memory goes, also when others have given up
    auto run_ring = [&](uint64_t* full, uint64_t* empty, int places, uint32_t bytes, auto fill) {
      int at = 0, filled = 0;
      uint32_t phase = 1;
      for (; filled < steps; ++filled) {
        if (!mbar_wait(smem_addr(&empty[at]), phase, aborted, fault) || *aborted) break;
        mbar_expect_tx(smem_addr(&full[at]), bytes);
        fill(filled, at, smem_addr(&full[at]));
        if (++at == places) { at = 0; phase ^= 1u; }
      }
      volatile int go_on = 0;
      for (int s = 0; s < places; ++s) {
        const int fills = (filled - s + places - 1) / places;
        if (fills > 0) mbar_wait(smem_addr(&full[s]), static_cast<uint32_t>((fills - 1) & 1), &go_on, fault);
      }
    };
    if (warp == 9 && lane == 0) {
      prefetch_tensormap(&map_w);
      run_ring(raw_full_bar, raw_empty_bar, kRaw, (kSplitM + (kCopied ? 0 : tokens)) * kSplitK * 4, [&](int step, int r, uint32_t bar) {
        tma_load_2d(raw_w(r), &map_w, bar, k_begin + step * kSplitK, n0);
        if constexpr (!kCopied) tma_load_2d(raw_x(r), &map_x, bar, k_begin + step * kSplitK, t0);
      });
    }
    if (kCopied && warp == 10 && lane == 0) {
      prefetch_tensormap(&map_x);
      run_ring(copied_bar, empty_bar, kBuffers, 3 * part_x, [&](int step, int b, uint32_t bar) {
        for (int part = 0; part < 3; ++part)      // (rows behind a part's last: the next part's, for outputs that are not stored)
          tma_load_2d(buffer_x(b) + part * part_x, &map_x, bar, k_begin + step * kSplitK, part * args.m + t0);
      });
    }
  } else {
    // four warps cut the even steps and four the odd ones, so that a step's chain of waits has two steps' time; a thread cuts
    // the weight row whose lane it may write
    const int group = warp >> 2, w_row = (warp & 3) * 32 + lane;
    const uint32_t to_w = parts_w + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    // of the tokens' rows, where they are cut here, eight columns; 16 bytes of a row of 64 change places by its bits 1 and 2
    const int eight = tid & 3, row = (tid & 127) >> 2;
    const uint32_t place = row * 64 + (((eight ^ (row >> 1)) & 3) << 4);
    float acc[kAcc];
    bool ok = true;
    auto add_sum = [&](uint32_t from) {
#pragma unroll
      for (int j = 0; j < kAcc; j += 16) {
        if (j < my_cols) {
          float v[16];
          tmem_load16(from + my_col0 + j + (static_cast<uint32_t>((warp & 3) * 32) << 16), v);
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[j + i] += v[i];
        }
      }
    };
    int taken = 0;
    auto take_sum = [&]() {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&acc_full_bar), taken & 1, aborted, fault));
      if (!ok) return;
      ++taken;
      tc_fence_after();
      add_sum(tmem_base);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_addr(&acc_empty_bar));
    };
#pragma unroll
    for (int j = 0; j < kAcc; ++j) acc[j] = 0.0f;
    int b = group, r = group;
    uint32_t phase = 1, raw_phase = 0;
    for (int step = group; step < steps; step += 2) {      // (a warp whose wait ran out hands nothing on)
      ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&raw_full_bar[r]), raw_phase, aborted, fault) &&
                                       mbar_wait(smem_addr(&empty_bar[b]), phase, aborted, fault));
      if (!ok) break;
      tc_fence_after();
      // few tokens, where the weights' stream is the bound: a place of the ring goes back as soon as its numbers are in registers, and
      // only the rows there are are cut.  One row by 24,576 x 4,096 87 -> 78 us (5.2 TB/s), 4,096 x 12,288 56 -> 40
      float early[kCopied ? 1 : 32];
      if constexpr (!kCopied) {
        float v[8];
        const bool cuts = row < live;           // (rows behind the last: anything, for outputs that are not stored)
        if (cuts) {
          load_raw(raw_x(r), row, 2 * eight, v);
          load_raw(raw_x(r), row, 2 * eight + 1, v + 4);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) load_raw(raw_w(r), w_row, j, early + 4 * j);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_addr(&raw_empty_bar[r]));
        if (cuts) {
          store_parts(buffer_x(b) + place, part_x, v);
          fence_async_smem();
        }
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float v[16];
        if constexpr (kCopied) {
#pragma unroll
          for (int j = 0; j < 4; ++j) load_raw(raw_w(r), w_row, half * 4 + j, v + 4 * j);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = early[half * 16 + j];
        }
#pragma unroll
        for (int part = 0; part < 3; ++part) {
          uint32_t packed[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) packed[j] = next_parts(v[2 * j], v[2 * j + 1]);
          tmem_store8(to_w + (b * 3 + part) * kSplitPartColumns + half * 8, packed);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_addr(&full_bar[b]));
        if (kCopied) mbar_arrive(smem_addr(&raw_empty_bar[r]));
      }
      if ((b += 2) >= kBuffers) { b -= kBuffers; phase ^= 1u; }
      if ((r += 2) >= kRaw) { r -= kRaw; raw_phase ^= 1u; }
      // the sum before this one, with every buffer handed on (no later: the first product of the next sum waits for it)
      if (step % kSplitSum - group == kBuffers - 2 && step >= kSplitSum) take_sum();
    }
    // the sums not taken yet: the last one, and the one before it where the last has a single buffer
    while (ok && taken * kSplitSum < steps) take_sum();
    if (ok && steps > 0) {
      tc_fence_after();
      add_sum(tmem_base + kTokens);
      tc_fence_before();
    }
    // a wait that ran out leaves no sum: such outputs are formed from the numbers themselves, and the fault word says so
    const float lost = *aborted ? __int_as_float(0x7fffffff) : 0.0f;
    const int at = (warp & 3) * 32 + lane;
#pragma unroll
    for (int j = 0; j < kAcc; ++j)
      if (j < my_cols) mine[(my_col0 + j) * kSplitM + at] = acc[j] + lost;      // every product has been formed: the buffers are free
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 8) tmem_dealloc(tmem_base, Shape::kColumns);
  cluster_sync();
  if (warp < 8) {
    for (int token = rank + warp * segments; token < live; token += 8 * segments) {
      const uint32_t at = smem_base + (token * kSplitM + lane * 4) * 4;
      float4 part[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < segments) part[s] = load_peer_f32x4(peer_smem(at, s));
      float4 sum = part[0];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < segments) { sum.x += part[s].x; sum.y += part[s].y; sum.z += part[s].z; sum.w += part[s].w; }
      float* to = args.c + static_cast<size_t>(t0 + token) * args.ldc;
      float sums[4] = {sum.x, sum.y, sum.z, sum.w};
      const int row0 = n0 + lane * 4;
      bool finite = true;
#pragma unroll
      for (int j = 0; j < 4; ++j) finite = finite && (row0 + j >= args.n || split_finite(sums[j]));
      if (!__all_sync(0xffffffffu, finite)) split_again(args, sums, t0 + token, row0);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (row0 + j < args.n) to[row0 + j] = sums[j] + (args.bias ? args.bias[row0 + j] : 0.0f);
    }
  }
  cluster_sync();      // the others may still be reading
}

// Segments of the columns, by n and k alone: the rounds of CTAs (two a multiprocessor) times a segment's steps and what a CTA
// costs beside them, about six, at their least.
static int split_segments(int n, int k) {
  const long long tiles = (n + kSplitM - 1) / kSplitM, slots = 2 * 148;
  int best = 1;
  long long least = 0;
  for (int segments = 1; segments <= 8 && (segments == 1 || k >= 512 * segments); segments *= 2) {
    const long long cost = (tiles * segments + slots - 1) / slots * (k / (kSplitK * segments) + 6);
    if (segments == 1 || cost < least) {
      best = segments;
      least = cost;
    }
  }
  return best;
}

static int split_map(CUtensorMap* map, const void* base, bool parts, long long rows, long long cols, long long pitch, int box_rows) {
  EncodeTiled encode = encode_tiled();
  if (encode == nullptr) return static_cast<int>(cudaErrorNotSupported);
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch) * (parts ? 2 : 4)};
  const cuuint32_t box[2] = {kSplitK, static_cast<cuuint32_t>(box_rows)}, elem[2] = {1, 1};
  const CUresult r = encode(map, parts ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base),
                            dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            parts ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(cudaErrorInvalidValue);
}

template <int kTokens, bool kCopied>
static int launch_split(SplitArgs args, __nv_bfloat16* parts, cudaStream_t stream) {
  using Shape = SplitShape<kTokens, kCopied>;
  auto kernel = gemm_f32_split_kernel<kTokens, kCopied>;
  static std::atomic<unsigned long long> configured;
  cudaError_t e = allow_shared(kernel, Shape::kSmem, configured);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int segments = split_segments(args.n, args.k);
  args.segment = ((args.k + segments - 1) / segments + 255) / 256 * 256;
  const int token_tiles = (args.m + args.tile_tokens - 1) / args.tile_tokens, row_tiles = (args.n + kSplitM - 1) / kSplitM;
  if (row_tiles > 65535) return static_cast<int>(cudaErrorInvalidValue);
  CUtensorMap map_w, map_x;
  int r = split_map(&map_w, args.w, false, args.n, args.k, args.k, kSplitM);
  if (r) return r;
  if constexpr (kCopied) {
    const int kp = (args.k + 7) / 8 * 8;
    split_rows_kernel<<<dim3((kp / 4 + 255) / 256, args.m), 256, 0, stream>>>(args.a, args.lda, args.a_in_fours, parts, args.m, args.k, kp);
    e = cudaGetLastError();
    if (e != cudaSuccess) return static_cast<int>(e);
    r = split_map(&map_x, parts, true, 3ll * args.m, kp, kp, args.tile_tokens);
  } else {
    r = split_map(&map_x, args.a, false, args.m, args.k, args.lda, args.tile_tokens);
  }
  if (r) return r;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(segments, row_tiles, token_tiles);
  config.blockDim = dim3(Shape::kThreads);
  config.dynamicSmemBytes = Shape::kSmem;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = segments;
  attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&config, kernel, map_w, map_x, args));
}

// Whether the product runs here: a rule on the weight alone, so that a row's bits do not depend on what it comes with.  The line
// lies where the weight's 32 MB are a few rounds of tiles; below it a product is its launches.  us at 1, 16, 64, 203 rows,
// sums down the columns / here: 4,096 x 4,096 23, 58, 167, 253 / 20, 21, 28, 74; 24,576 x 4,096 69, 167, 352, 1,076 / 77, 79,
// 99, 263; 4,096 x 12,288 62, 167, 490, 741 / 42, 42, 52, 176; 151,936 x 4,096 377, 790, 1,893, 5,828 / 395, 430, 617, 1,512
// (a single row of wide weights is the one that loses, by 5 to 11 %; a decode step of one row, four layers of the 8B sizes and the
// head, goes from 1,807 to 1,736).
bool gemm_f32_split_takes(const float* w, int n, int k) {
  return k % 4 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0 && n >= 1024 && k >= 1024 &&
         static_cast<long long>(n) * k >= 1 << 23 && n <= 65535 * kSplitM;
}
// 16-bit numbers of scratch that `gemm_f32_split` wants as `parts`: the parts of up to kSplitRows rows, where there are more than
// 32 or they cannot be fetched 16 bytes at a time.
constexpr int kSplitRows = 1024;
static bool split_rows_in_fours(const float* a, int lda) { return lda % 4 == 0 && reinterpret_cast<uintptr_t>(a) % 16 == 0; }
long long gemm_f32_split_scratch(const float* a, int m, int k, int lda) {
  if (m <= 32 && split_rows_in_fours(a, lda)) return 0;
  return 3ll * (m < kSplitRows ? m : kSplitRows) * ((k + 7) / 8 * 8);
}

int gemm_f32_split(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda, int ldc,
                   __nv_bfloat16* parts, int* fault, cudaStream_t stream) {
  for (int at = 0; at < m; at += kSplitRows) {
    const int rows = m - at < kSplitRows ? m - at : kSplitRows;
    SplitArgs args = {a + static_cast<size_t>(at) * lda, w, bias, c + static_cast<size_t>(at) * ldc, rows, n, k, lda, ldc, 0, 0, 0, fault};
    args.a_in_fours = split_rows_in_fours(a, lda);
    const int tiles = (rows + kSplitMaxTokens - 1) / kSplitMaxTokens;
    args.tile_tokens = ((rows + tiles - 1) / tiles + 15) / 16 * 16;
    const int tokens = args.tile_tokens;
    int e;
    if (rows <= 32 && args.a_in_fours) {
      e = tokens <= 16 ? launch_split<16, false>(args, parts, stream) : launch_split<32, false>(args, parts, stream);
    } else if (parts == nullptr || reinterpret_cast<uintptr_t>(parts) % 16) {
      return static_cast<int>(cudaErrorInvalidValue);
    } else {
      e = tokens <= 32    ? launch_split<32, true>(args, parts, stream)
          : tokens <= 64  ? launch_split<64, true>(args, parts, stream)
          : tokens <= 128 ? launch_split<128, true>(args, parts, stream)
                          : launch_split<kSplitMaxTokens, true>(args, parts, stream);
    }
    if (e) return e;
  }
  return 0;
}

}  // namespace rl
