// The routed feed-forward's products over many pairs on the tensor cores (see moe.cu for the plan they walk).
//
//   gated:  act[place, n] = unit(w_p (x_row . gate_n), w_p (x_row . up_n)), rows of x found by token or by place
//   plain:  y[pair, n] = a_row . w_n, float32
//
// A tile is 128 pairs of one expert by 256 weight rows (gated: 128 gate rows and the 128 up rows beside them, so that a
// thread finds both products of an output in its own lane).  The tile list is the plan's, known only on the device: every
// role reads it and walks the same tiles, one CTA per multiprocessor.  The pairs' rows lie anywhere in x, so four warps
// fetch them 16 bytes at a time into the 128-byte-swizzled layout that TMA gives the weights; a stage holds 64 columns of
// both operands, four stages.  One thread issues tcgen05.mma, the accumulators (256 columns) alternate between two buffers
// of tensor memory, and four warps write one tile out while the next is multiplied.  An output is one sum in the order of
// k, whatever else is in its tile.
//
// Bound by what a multiprocessor fetches per product: 48 KB for every 64 columns of a tile.  Before that the gated
// results' divisions held it up, one behind the other (a tile's 128 outputs a thread: 20 to 35 us more), so sixteen are
// formed together (moe_units).  Hidden 2,048, inter 512, 2 of 16 experts, 2,048 tokens: 50 + 43 us (mma.sync tiles of 64
// pairs: 80 + 59; a plain division: 82 + 43); hidden 4,096, inter 1,024: 119 + 82 (270 + 178; 137 + 80).
#include <cuda.h>

#include "common.cuh"
#include "moe_unit.cuh"
#include "tc_common.cuh"

namespace rl {

constexpr int kMoeTcM = 128;          // pairs per tile (lanes of the accumulator)
constexpr int kMoeTcN = 256;          // weight rows per tile
constexpr int kMoeTcK = 64;
constexpr int kMoeTcStages = 4;
constexpr int kMoeTcStageA = kMoeTcM * kMoeTcK * 2, kMoeTcStageB = kMoeTcN * kMoeTcK * 2;
constexpr int kMoeTcSmem = kMoeTcStages * (kMoeTcStageA + kMoeTcStageB) + 1024;
constexpr int kMoeTcThreads = 320;    // weights' copies, products, 4 x results, 4 x rows
constexpr int kMoeTcLag = 2;          // steps between asking for rows and handing them on

struct MoeTcArgs {
  const __nv_bfloat16* a;
  int a_stride;
  const int* sorted;
  const int* meta;
  const float* pair_weight;
  int top, by_token, n, k, w_rows;      // w_rows: weight rows per expert
  __nv_bfloat16* out_act;
  float* out_y;
  float glu_limit, glu_alpha;
  int* fault;
};

template <bool kGated>
__global__ void __launch_bounds__(kMoeTcThreads)
grouped_linear_tc_kernel(const __grid_constant__ CUtensorMap map_w, const MoeTcArgs args) {
  constexpr int kColumns = kGated ? kMoeTcN / 2 : kMoeTcN;      // output columns per tile
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kMoeTcN >> 3) << 17) |
                              (static_cast<uint32_t>(kMoeTcM >> 4) << 24);
  extern __shared__ unsigned char moe_tc_raw[];
  __shared__ __align__(8) uint64_t rows_bar[kMoeTcStages], weights_bar[kMoeTcStages], empty_bar[kMoeTcStages], acc_full_bar[2],
      acc_empty_bar[2], drain_bar;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int aborted_flag;
  volatile int* aborted = &aborted_flag;
  if (threadIdx.x == 0) pdl_trigger();
  const int warp = uniform(static_cast<int>(threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_addr(moe_tc_raw) + 1023u) & ~1023u;
  auto stage_a = [&](int s) { return smem_base + s * (kMoeTcStageA + kMoeTcStageB); };
  auto stage_b = [&](int s) { return stage_a(s) + kMoeTcStageA; };
  const int n_tiles = (args.n + kColumns - 1) / kColumns, steps = (args.k + kMoeTcK - 1) / kMoeTcK;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_w);
    for (int s = 0; s < kMoeTcStages; ++s) {
      mbar_init(smem_addr(&rows_bar[s]), 128);
      mbar_init(smem_addr(&weights_bar[s]), 1);
      mbar_init(smem_addr(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_addr(&acc_full_bar[b]), 1);
      mbar_init(smem_addr(&acc_empty_bar[b]), 4);
    }
    mbar_init(smem_addr(&drain_bar), 1);
    aborted_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_addr(&tmem_base_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(tmem_base_slot);
  pdl_wait();                                   // the plan, the rows and whoever still reads the results
  const int pair_tiles = args.meta[0];
  const int tiles = pair_tiles * n_tiles;       // neighbours share weights: the pairs' tiles run fastest

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0, filled = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int which = tile % pair_tiles, n0 = tile / pair_tiles * kColumns;
        const int row0 = args.meta[1 + 3 * which] * args.w_rows + n0;
        for (int step = 0; step < steps; ++step) {
          ok = mbar_wait(smem_addr(&empty_bar[stage]), phase ^ 1u, aborted, args.fault);
          if (!ok) break;
          const uint32_t bar = smem_addr(&weights_bar[stage]);
          mbar_expect_tx(bar, kMoeTcStageB);
          tma_load_2d(stage_b(stage), &map_w, bar, step * kMoeTcK, row0);
          tma_load_2d(stage_b(stage) + kMoeTcStageB / 2, &map_w, bar, step * kMoeTcK, row0 + (kGated ? args.n : kMoeTcN / 2));
          ++filled;
          if (++stage == kMoeTcStages) { stage = 0; phase ^= 1u; }
        }
      }
      // the copies land before the shared memory goes, also when the others have given up
      volatile int go_on = 0;
      for (int s = 0; s < kMoeTcStages; ++s) {
        const int fills = (filled - s + kMoeTcStages - 1) / kMoeTcStages;
        if (fills > 0) mbar_wait(smem_addr(&weights_bar[s]), static_cast<uint32_t>((fills - 1) & 1), &go_on, args.fault);
      }
    }
  } else if (warp == 1) {
    const bool issues = elect_one();
    const int last_tile = uniform(tiles);
    int stage = 0, buf = 0;
    uint32_t phase = 0, acc_phase = 0;                  // acc_phase: a bit for each buffer
    bool ok = true;
    for (int tile = blockIdx.x; tile < last_tile && ok; tile += gridDim.x) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&acc_empty_bar[buf]), ((acc_phase >> buf) & 1u) ^ 1u, aborted, args.fault));
      if (!ok) break;
      tc_fence_after();
      for (int step = 0; step < steps; ++step) {
        ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&weights_bar[stage]), phase, aborted, args.fault) &&
                                         mbar_wait(smem_addr(&rows_bar[stage]), phase, aborted, args.fault));
        if (!ok) break;
        tc_fence_after();
        const uint64_t a_desc = operand_desc(stage_a(stage)), b_desc = operand_desc(stage_b(stage));
        if (issues) {
#pragma unroll
          for (int k = 0; k < kMoeTcK / 16; ++k)
            umma_bf16(tmem_base + buf * kMoeTcN, a_desc + 2 * k, b_desc + 2 * k, kIdesc, (step > 0 || k > 0) ? 1u : 0u);
          umma_commit(smem_addr(&empty_bar[stage]));
        }
        __syncwarp();
        if (++stage == kMoeTcStages) { stage = 0; phase ^= 1u; }
      }
      if (!ok) break;
      if (issues) umma_commit(smem_addr(&acc_full_bar[buf]));
      __syncwarp();
      acc_phase ^= 1u << buf;
      buf ^= 1;
    }
    // nothing of this CTA may still be running on the tensor core when its memory is freed
    if (issues) umma_commit(smem_addr(&drain_bar));
    __syncwarp();
    mbar_wait(smem_addr(&drain_bar), 0, aborted, args.fault);
  } else if (warp < 6) {
    const int quarter = warp & 3;                       // the 32 tensor-memory lanes this warp may read
    const int row = quarter * 32 + lane;
    int buf = 0;
    uint32_t acc_phase[2] = {0, 0};
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int which = tile % pair_tiles, n0 = tile / pair_tiles * kColumns;
      const int place0 = args.meta[2 + 3 * which], rows = args.meta[3 + 3 * which];
      const bool live = row < rows;
      const int pair = live ? args.sorted[place0 + row] : 0;
      const float scale = kGated && live && args.pair_weight ? args.pair_weight[pair] : 1.0f;
      const bool full = mbar_wait(smem_addr(&acc_full_bar[buf]), acc_phase[buf], aborted, args.fault);
      if (!__all_sync(0xffffffffu, full)) break;        // the loads below are the whole warp's
      tc_fence_after();
      const uint32_t acc = tmem_base + buf * kMoeTcN + (static_cast<uint32_t>(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < kColumns; c += 16) {
        if (n0 + c >= args.n) break;                    // the same for the whole warp
        float v[16];
        tmem_load16(acc + c, v);
        if constexpr (kGated) {
          float u[16];
          tmem_load16(acc + kColumns + c, u);
          if (live) {
            float unit[16];
            __align__(16) __nv_bfloat16 packed[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              v[j] *= scale;
              u[j] *= scale;
            }
            moe_units(v, u, args.glu_limit, args.glu_alpha, unit);
#pragma unroll
            for (int j = 0; j < 16; ++j) packed[j] = __float2bfloat16_rn(unit[j]);
            __nv_bfloat16* o = args.out_act + static_cast<size_t>(place0 + row) * args.n + n0 + c;
#pragma unroll
            for (int j = 0; j < 16; j += 8)             // n is a multiple of 8 here
              if (n0 + c + j < args.n) *reinterpret_cast<uint4*>(o + j) = *reinterpret_cast<const uint4*>(packed + j);
          }
        } else if (live) {
          float* o = args.out_y + static_cast<size_t>(pair) * args.n + n0 + c;
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (n0 + c + j < args.n) *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_addr(&acc_empty_bar[buf]));
      acc_phase[buf] ^= 1u;
      buf ^= 1;
    }
  } else {
    // ------------------------------------------------------------------ the pairs' rows
    const int t = threadIdx.x - 192;                    // 0 .. 127
    const int col = (t & 7) * 8;                        // this thread's eight columns of every sixteenth row
    int stage = 0, pending = 0, ready = 0;              // steps asked for and not handed on yet; the stage handed on next
    uint32_t phase = 0;
    bool ok = true;
    auto hand_on = [&]() {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the tensor core reads what these copies wrote
      mbar_arrive(smem_addr(&rows_bar[ready]));
      ready = ready + 1 == kMoeTcStages ? 0 : ready + 1;
      --pending;
    };
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const int which = tile % pair_tiles;
      const int place0 = args.meta[2 + 3 * which], rows = args.meta[3 + 3 * which];
      const __nv_bfloat16* from[8];
      bool live[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * 16 + (t >> 3);
        live[i] = r < rows;
        size_t at = 0;
        if (live[i]) at = args.by_token ? static_cast<size_t>(args.sorted[place0 + r] / args.top) : static_cast<size_t>(place0 + r);
        from[i] = args.a + at * args.a_stride + col;
      }
      for (int step = 0; step < steps; ++step) {
        ok = mbar_wait(smem_addr(&empty_bar[stage]), phase ^ 1u, aborted, args.fault);
        if (!ok) break;
        const int k0 = step * kMoeTcK;
        const uint32_t base = stage_a(stage);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 16 + (t >> 3);
          const bool good = live[i] && k0 + col < args.k;
          const uint32_t to = base + r * 128 + (((t & 7) ^ (r & 7)) << 4);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(good ? from[i] + k0 : args.a), "r"(good ? 16 : 0)
                       : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++pending > kMoeTcLag) {
          asm volatile("cp.async.wait_group %0;" ::"n"(kMoeTcLag) : "memory");
          hand_on();
        }
        if (++stage == kMoeTcStages) { stage = 0; phase ^= 1u; }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    while (pending > 0) hand_on();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

template <bool kGated>
static int launch_grouped_tc(const CUtensorMap& map_w, const MoeTcArgs& args, int blocks, int pdl, cudaStream_t stream) {
  auto kernel = grouped_linear_tc_kernel<kGated>;
  static std::atomic<unsigned long long> configured;
  const cudaError_t e = allow_shared(kernel, kMoeTcSmem, configured);
  if (e != cudaSuccess) return static_cast<int>(e);
  return launch_kernel(kernel, dim3(blocks), dim3(kMoeTcThreads), kMoeTcSmem, stream, pdl != 0, map_w, args);
}

// `most_tiles`: a bound on the tiles of pairs; `experts`: of the weight [experts, gated ? 2 n : n, k].
int grouped_linear_tc(const void* a, int a_stride, const void* w, int experts, const int* sorted, const int* meta,
                      const float* pair_weight, int top, int by_token, int n, int k, int gated, void* out_act, float* out_y,
                      int most_tiles, float glu_limit, float glu_alpha, int* fault, int pdl, cudaStream_t stream) {
  if (k % 8 || n % 8 || a_stride % 8 || n < 1 || k < 1 || top < 1 || experts < 1 || fault == nullptr ||
      ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out_act) |
        reinterpret_cast<uintptr_t>(out_y)) & 15) != 0)
    return static_cast<int>(cudaErrorInvalidValue);
  MoeTcArgs args = {};
  args.a = static_cast<const __nv_bfloat16*>(a); args.a_stride = a_stride; args.sorted = sorted; args.meta = meta;
  args.pair_weight = pair_weight; args.top = top; args.by_token = by_token; args.n = n; args.k = k;
  args.w_rows = gated ? 2 * n : n;
  args.out_act = static_cast<__nv_bfloat16*>(out_act); args.out_y = out_y;
  args.glu_limit = glu_limit; args.glu_alpha = glu_alpha; args.fault = fault;
  CUtensorMap map_w;
  const int e = make_map(&map_w, w, static_cast<long long>(experts) * args.w_rows, k, kMoeTcN / 2);
  if (e) return e;
  const int columns = gated ? kMoeTcN / 2 : kMoeTcN;
  const long long tiles = static_cast<long long>(most_tiles) * ((n + columns - 1) / columns);
  int device = 0, sms = 148;
  if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const int blocks = static_cast<int>(tiles < sms ? tiles : sms);
  return gated ? launch_grouped_tc<true>(map_w, args, blocks, pdl, stream) : launch_grouped_tc<false>(map_w, args, blocks, pdl, stream);
}

}  // namespace rl
