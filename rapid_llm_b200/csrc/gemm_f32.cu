// 32-bit matrix product: C[M, N] = A[M, K] * W[N, K]^T (+ bias), float32 in, float32 out, no reduced-precision mode.
//
// Weights of a few million numbers and more run on the tensor cores, with every float32 cut into three exact parts
// (gemm_f32_split.cu); the others here, in float32 fused multiply-adds.  The weight alone decides, and either way an output's
// value does not depend on M, on the tile it falls in, or on what else is in the batch: here it is accumulated over
// k = 0 .. K-1 in that order by one thread.
// The reference has no 32-bit path (rapid_llm/models/config.py:134-146 downgrades float32
// checkpoints); its products go through a library call (rapid_llm/kernels/ops/gemm/linear.py:17-40).
#include "common.cuh"

namespace rl {

bool gemm_f32_split_takes(const float* w, int n, int k);
long long gemm_f32_split_scratch(const float* a, int m, int k, int lda);
int gemm_f32_split(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda, int ldc,
                   __nv_bfloat16* parts, int* fault, cudaStream_t stream);

__device__ __forceinline__ void f32_copy16(float* shared, const float* global, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(shared))),
               "l"(global), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void f32_copy4(float* shared, const float* global, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(shared))),
               "l"(global), "r"(ok ? 4 : 0) : "memory");
}

// ------------------------------------------------------------------ tiles
// What bounds them: shared memory hands a multiprocessor 128 bytes a cycle, broadcasts included, and a thread's kTm x kTn
// outputs take (kTm + kTn) * 4 bytes a column for kTm * kTn multiply-adds, so tiles of few outputs a thread starve the FMA
// pipe and tiles of many leave multiprocessors without a tile.  203 rows (us, before / now; K = 4,096): N = 6,144
// 477 / 353, N = 4,096 347 / 256, N = 24,576 1,627 / 1,087 (37 TFLOP/s); N = 4,096 with K = 12,288 1,021 / 749.  Before:
// 64 x 64 tiles, 4 x 4 outputs a thread, one buffer.  Tried and slower there: 8 x 8 and 8 x 16 outputs a thread
// on 128 x 128 tiles (393 at N = 4,096; ahead only from 512 rows on, 1,410 against 1,611 us at 2,048), operands
// transposed on their way into shared memory, and packed pairs of multiply-adds (the packing costs what they save).
constexpr int kF32TileK = 32, kF32Stages = 3;
constexpr int kF32Stride = kF32TileK + 4;      // floats between two rows in shared memory: eight neighbouring rows meet in no bank

template <int kTx, int kTy, int kTm, int kTn>
constexpr int f32_stage_floats() { return (kTy * kTm + kTx * kTn) * kF32Stride; }

// kTx x kTy threads with kTm x kTn outputs each.  Both operands lie in shared memory as they lie in memory, rows of 32
// columns, brought by asynchronous copies two steps ahead; a thread takes four columns of a row in one 16-byte fetch.
template <int kTx, int kTy, int kTm, int kTn, bool kAligned>
__global__ void __launch_bounds__(kTx * kTy)
gemm_f32_kernel(const float* __restrict__ a, const float* __restrict__ w,
                const float* __restrict__ bias, float* __restrict__ c, int m, int n, int k,
                int lda, int ldc) {
  constexpr int kThreads = kTx * kTy, kTileM = kTy * kTm, kTileN = kTx * kTn;
  extern __shared__ __align__(16) float f32_ring[];
  const int tid = threadIdx.x;
  const int tx = tid % kTx, ty = tid / kTx;
  const int m0 = blockIdx.y * kTileM, n0 = blockIdx.x * kTileN;
  const int steps = (k + kF32TileK - 1) / kF32TileK;

  auto fill = [&](int step) {
    float* sa = f32_ring + (step % kF32Stages) * f32_stage_floats<kTx, kTy, kTm, kTn>();
    const int k0 = step * kF32TileK;
    constexpr int kPiece = kAligned ? 4 : 1, kPieces = kF32TileK / kPiece;
    static_assert((kTileM + kTileN) * kPieces % kThreads == 0, "every thread copies as many pieces");
#pragma unroll
    for (int at = 0; at < (kTileM + kTileN) * kPieces; at += kThreads) {
      const int idx = at + tid, r = idx / kPieces, col = (idx % kPieces) * kPiece;
      const bool is_a = r < kTileM;
      const int row = is_a ? m0 + r : n0 + r - kTileM;
      const bool ok = row < (is_a ? m : n) && k0 + col < k;
      const float* from = is_a ? a + static_cast<size_t>(row) * lda : w + static_cast<size_t>(row) * k;
      from = ok ? from + k0 + col : w;
      if constexpr (kAligned) f32_copy16(sa + r * kF32Stride + col, from, ok);
      else f32_copy4(sa + r * kF32Stride + col, from, ok);
    }
  };
#pragma unroll
  for (int s = 0; s < kF32Stages - 1; ++s) {
    if (s < steps) fill(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[kTm][kTn];
#pragma unroll
  for (int i = 0; i < kTm; ++i)
#pragma unroll
    for (int j = 0; j < kTn; ++j) acc[i][j] = 0.0f;
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kF32Stages - 2) : "memory");
    __syncthreads();      // the step has landed for every thread, and the stage refilled below has been read
    if (step + kF32Stages - 1 < steps) fill(step + kF32Stages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* sa = f32_ring + (step % kF32Stages) * f32_stage_floats<kTx, kTy, kTm, kTn>() + ty * kF32Stride;
    const float* sw = f32_ring + (step % kF32Stages) * f32_stage_floats<kTx, kTy, kTm, kTn>() + (kTileM + tx) * kF32Stride;
#pragma unroll 1      // unrolled further it runs out of registers and slows down
    for (int kk = 0; kk < kF32TileK; kk += 4) {
      float4 ar[kTm], wr[kTn];
#pragma unroll
      for (int i = 0; i < kTm; ++i) ar[i] = *reinterpret_cast<const float4*>(sa + i * kTy * kF32Stride + kk);
#pragma unroll
      for (int j = 0; j < kTn; ++j) wr[j] = *reinterpret_cast<const float4*>(sw + j * kTx * kF32Stride + kk);
#pragma unroll
      for (int i = 0; i < kTm; ++i)
#pragma unroll
        for (int j = 0; j < kTn; ++j) acc[i][j] = fmaf(ar[i].x, wr[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < kTm; ++i)
#pragma unroll
        for (int j = 0; j < kTn; ++j) acc[i][j] = fmaf(ar[i].y, wr[j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < kTm; ++i)
#pragma unroll
        for (int j = 0; j < kTn; ++j) acc[i][j] = fmaf(ar[i].z, wr[j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < kTm; ++i)
#pragma unroll
        for (int j = 0; j < kTn; ++j) acc[i][j] = fmaf(ar[i].w, wr[j].w, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < kTm; ++i) {
    const int row = m0 + ty + kTy * i;
    if (row >= m) continue;
#pragma unroll
    for (int j = 0; j < kTn; ++j) {
      const int col = n0 + tx + kTx * j;
      if (col < n) c[static_cast<size_t>(row) * ldc + col] = acc[i][j] + (bias ? bias[col] : 0.0f);
    }
  }
}

// ------------------------------------------------------------------ few rows
// Up to kG * kPer rows of A (decoding, the head behind a step's prompts): bound by the weights' stream.  A block brings a
// band of W's rows kBk columns at a time through a ring in shared memory; a lane owns kR weight rows, a warp kPer rows
// of A, so an output's sum still runs down k in one thread.  kG of the four warps share the rows of A, the others take
// bands of their own.  Fetches of A are broadcasts but cost shared memory as much as any other, so with many weight rows
// (where blocks are plenty) a lane owns two of them.  Measured (us, 64 x 64 tiles before / now, K = 4,096): 1 row
// 292 / 26 at N = 4,096, 501 / 80 at N = 24,576 (5.0 TB/s); 5 rows of the head, N = 151,936, 2,321 / 484 (5.1 TB/s);
// 16 rows 292 / 60 and 505 / 176; 32 rows 293 / 78 and 505 / 212.
constexpr int kFewThreads = 128;

template <int kPer, int kG, int kR, int kBk, int kStages>
struct Few {
  static constexpr int kRows = 32 * kR * (4 / kG);
  static constexpr int kStride = kBk + 4;
  static constexpr int kStageFloats = kRows * kStride + kG * kPer * kBk;
  static constexpr int kSmem = kStages * kStageFloats * 4;
};

template <int kPer, int kG, int kR, int kBk, int kStages>
__global__ void __launch_bounds__(kFewThreads)
gemm_f32_few_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                    float* __restrict__ c, int m, int n, int k, int lda, int ldc) {
  using F = Few<kPer, kG, kR, kBk, kStages>;
  extern __shared__ __align__(16) float few_ring[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = warp % kG, band = warp / kG;
  const int n0 = blockIdx.x * F::kRows;
  const int steps = (k + kBk - 1) / kBk;
  auto fill = [&](int step) {
    float* sw = few_ring + (step % kStages) * F::kStageFloats;
    float* sa = sw + F::kRows * F::kStride;
    const int k0 = step * kBk;
    constexpr int kPieces = kBk / 4;
#pragma unroll
    for (int i = 0; i < F::kRows * kPieces / kFewThreads; ++i) {
      const int idx = tid + i * kFewThreads, r = idx / kPieces, col = (idx % kPieces) * 4;
      const bool ok = n0 + r < n && k0 + col < k;
      f32_copy16(sw + r * F::kStride + col, ok ? w + static_cast<size_t>(n0 + r) * k + k0 + col : w, ok);
    }
    for (int idx = tid; idx < kG * kPer * kPieces; idx += kFewThreads) {
      const int r = idx / kPieces, col = (idx % kPieces) * 4;
      const bool ok = r < m && k0 + col < k;
      f32_copy16(sa + r * kBk + col, ok ? a + static_cast<size_t>(r) * lda + k0 + col : a, ok);
    }
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < steps) fill(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[kR][kPer];
#pragma unroll
  for (int r = 0; r < kR; ++r)
#pragma unroll
    for (int i = 0; i < kPer; ++i) acc[r][i] = 0.0f;
  const bool works = group * kPer < m;      // a warp without rows of A only copies
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();      // the step has landed for every thread, and the stage refilled below has been read
    if (step + kStages - 1 < steps) fill(step + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (!works) continue;
    const float* sw = few_ring + (step % kStages) * F::kStageFloats;
    const float* mine = sw + (band * 32 * kR + lane) * F::kStride;
    const float* sa = sw + F::kRows * F::kStride + group * kPer * kBk;
#pragma unroll
    for (int kk = 0; kk < kBk; kk += 4) {
      float4 w4[kR];
#pragma unroll
      for (int r = 0; r < kR; ++r) w4[r] = *reinterpret_cast<const float4*>(mine + r * 32 * F::kStride + kk);
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const float4 a4 = *reinterpret_cast<const float4*>(sa + i * kBk + kk);
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          acc[r][i] = fmaf(a4.x, w4[r].x, acc[r][i]);
          acc[r][i] = fmaf(a4.y, w4[r].y, acc[r][i]);
          acc[r][i] = fmaf(a4.z, w4[r].z, acc[r][i]);
          acc[r][i] = fmaf(a4.w, w4[r].w, acc[r][i]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int col = n0 + (band * kR + r) * 32 + lane;
    if (col >= n) continue;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int row = group * kPer + i;
      if (row < m) c[static_cast<size_t>(row) * ldc + col] = acc[r][i] + (bias ? bias[col] : 0.0f);
    }
  }
}

template <int kTx, int kTy, int kTm, int kTn>
static int launch_f32_tiles(bool aligned, const float* a, const float* w, const float* bias, float* c, int m, int n, int k,
                            int lda, int ldc, cudaStream_t stream) {
  const dim3 grid((n + kTx * kTn - 1) / (kTx * kTn), (m + kTy * kTm - 1) / (kTy * kTm));
  if (grid.y > 65535) return static_cast<int>(cudaErrorInvalidValue);
  constexpr int smem = kF32Stages * f32_stage_floats<kTx, kTy, kTm, kTn>() * static_cast<int>(sizeof(float));
  auto kernel = aligned ? gemm_f32_kernel<kTx, kTy, kTm, kTn, true> : gemm_f32_kernel<kTx, kTy, kTm, kTn, false>;
  static std::atomic<unsigned long long> configured[2];
  const cudaError_t e = allow_shared(kernel, smem, configured[aligned]);
  if (e != cudaSuccess) return static_cast<int>(e);
  kernel<<<grid, kTx * kTy, smem, stream>>>(a, w, bias, c, m, n, k, lda, ldc);
  return launch_status();
}

template <int kPer, int kG, int kR, int kBk, int kStages>
static int launch_f32_few(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda, int ldc,
                          cudaStream_t stream) {
  using F = Few<kPer, kG, kR, kBk, kStages>;
  auto kernel = gemm_f32_few_kernel<kPer, kG, kR, kBk, kStages>;
  static std::atomic<unsigned long long> configured;
  const cudaError_t e = allow_shared(kernel, F::kSmem, configured);
  if (e != cudaSuccess) return static_cast<int>(e);
  kernel<<<(n + F::kRows - 1) / F::kRows, kFewThreads, F::kSmem, stream>>>(a, w, bias, c, m, n, k, lda, ldc);
  return launch_status();
}

}  // namespace rl

// The 16-bit numbers of scratch the product wants as `parts` (0: none), on a 16-byte boundary.
extern "C" long long rl_gemm_f32_scratch(const float* a, const float* w, int m, int n, int k, int lda) {
  return m > 0 && rl::gemm_f32_split_takes(w, n, k) ? rl::gemm_f32_split_scratch(a, m, k, lda) : 0;
}

// a: [m, k] with row stride lda; w: [n, k] contiguous; c: [m, n] with row stride ldc.  `fault` may be null.
extern "C" int rl_gemm_f32(const float* a, const float* w, const float* bias, float* c, int m,
                           int n, int k, int lda, int ldc, void* parts, int* fault, cudaStream_t stream) {
  if (m == 0 || n == 0) return 0;
  if (k <= 0 || lda < k || ldc < n) return static_cast<int>(cudaErrorInvalidValue);
  if (rl::gemm_f32_split_takes(w, n, k))
    return rl::gemm_f32_split(a, w, bias, c, m, n, k, lda, ldc, static_cast<__nv_bfloat16*>(parts), fault, stream);
  const bool aligned = (k % 4 == 0) && (lda % 4 == 0) &&
                       (reinterpret_cast<uintptr_t>(a) % 16 == 0) &&
                       (reinterpret_cast<uintptr_t>(w) % 16 == 0);
  if (aligned && m <= 32) {
    // a lane with two weight rows halves the blocks: from 16,384 rows on there are enough of them.  One weight row against
    // two, us at N = 4,096 and 24,576: 8 rows of A 35 and 150 against 125 and 132, 16 rows 60 and 215 against 107 and
    // 176, 32 rows 78 and 340 against 96 and 212; up to 4 rows one is ahead at both (26 and 80 against 80 and 99)
    const bool many = n >= 16384;
    if (m <= 4) return rl::launch_f32_few<1, 4, 1, 64, 6>(a, w, bias, c, m, n, k, lda, ldc, stream);
    if (m <= 8) return many ? rl::launch_f32_few<8, 1, 2, 32, 3>(a, w, bias, c, m, n, k, lda, ldc, stream)
                            : rl::launch_f32_few<2, 4, 1, 64, 6>(a, w, bias, c, m, n, k, lda, ldc, stream);
    if (m <= 16) return many ? rl::launch_f32_few<8, 2, 2, 32, 4>(a, w, bias, c, m, n, k, lda, ldc, stream)
                             : rl::launch_f32_few<4, 4, 1, 64, 6>(a, w, bias, c, m, n, k, lda, ldc, stream);
    return many ? rl::launch_f32_few<8, 4, 2, 64, 3>(a, w, bias, c, m, n, k, lda, ldc, stream)
                : rl::launch_f32_few<8, 4, 1, 64, 6>(a, w, bias, c, m, n, k, lda, ldc, stream);
  }
  // 64 x 64 tiles (4 x 8 outputs a thread) or 112 x 64 (7 x 8): a round of tiles on the B200's 148 multiprocessors takes about
  // 115 and 180 us at K = 4,096 (measured over 40 to 2,048 rows), both in proportion to K, so the rule compares the rounds
  const long long wide = (n + 63) / 64, sms = 148;
  const long long low = (((m + 63) / 64) * wide + sms - 1) / sms, high = (((m + 111) / 112) * wide + sms - 1) / sms;
  if (180 * high < 115 * low) return rl::launch_f32_tiles<8, 16, 7, 8>(aligned, a, w, bias, c, m, n, k, lda, ldc, stream);
  return rl::launch_f32_tiles<8, 16, 4, 8>(aligned, a, w, bias, c, m, n, k, lda, ldc, stream);
}
