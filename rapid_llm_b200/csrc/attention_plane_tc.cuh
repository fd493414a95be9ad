// Attention over rows that are keys and values at once, on the 5th-generation tensor cores.
//
// One CTA serves one work item: 128 packed query rows of one request (of a single token: its heads; softmax warps without
// rows sit out) against a range of its cached rows.  TMA brings
// the rows in page by page, 96 a block, and both products read the same tile: as it lies for the scores (K-major) and
// turned for the values (MN-major).
//
//     S[row, key]  = Q[row, :] . R[key, :]      tcgen05.mma  M = 128, N = 96 keys, K = D
//     O[row, d]   += P[row, key] . R[key, d]    A = P from tensor memory, M = 128, N = D, K = 96 keys, twice
//
// P enters as two bfloat16 terms, its rounding and what that left.  Rounded once, every weight is up to 2^-9 off, also the
// largest, which the mma.sync tiles take against itself and so without an error.  Root mean square error of the result
// against 64 bits: 2,048 tokens 1.63e-3 (the mma.sync tiles 1.90e-3, one term 1.96e-3), 64 single tokens behind 1,024
// 1.65e-3 (1.81e-3, 1.95e-3); rounding the result alone gives 1.6e-3.  One term against the running maximum itself: 1.91e-3
// and 1.87e-3.
//
// What bounds it is the chain from a block's scores through its softmax to its values (1.4 us; the three products alone
// take 1.2), so the scores of block j + 1 are issued before the values of block j, two threads share a row and the softmax of
// one block runs under the products of its neighbours: O takes D columns of tensor memory, two blocks of scores 2 x 128 (P
// lies over the scores it came from).  Blocks of 96: three tiles of 96 x 256 fit beside the queries, and a tile is held from its scores to its values, one block later; with two tiles
// of 128 the next scores would wait for a whole fetch, and blocks of 64 with the queries in tensor memory and six tiles
// pay the chain more often (with one term of P 60 us against 52 for the prompt below).  The softmax is that of the two-plane kernel: the
// reference point of the exponentials moves only when the maximum has grown by more than 2^8; scores, maxima, sums
// and O are float32.
//
// Rows behind the range come as zeros (whole boxes from outside the tensor, the rest of a box cleared here): what lies
// in memory that nothing wrote yet must not reach the product, where zero times it could be NaN.
//
// 16 heads, rows of 256: 2,048 tokens of a prompt 58 us (the mma.sync tiles 236; one term of P 52), 64 single tokens behind
// 1,024 34 (50; 32), behind 4,096 66 (101; 60); 32 heads, 2 prompts of 600 47 (105; 45).
//
// Takes rows of 64 to 256 numbers and pages of a multiple of 8 tokens; others run on the mma.sync tiles.
#pragma once

#include "tc_common.cuh"

namespace rl {
namespace RL_ATTENTION_NS {

constexpr bool kPlTakes = kD >= 64 && kD <= 256;
constexpr int kPlD = kPlTakes ? kD : 64;
constexpr int kPlKeys = 96;                     // rows per block
constexpr int kPlRows = 128;                    // packed query rows per work item
constexpr int kPlStages = 3;
constexpr int kPlAtoms = (kPlD + 63) / 64;      // 64-wide columns of swizzled 128-byte rows
constexpr int kPlThreads = 384;                 // warp 0: TMA, warp 1: MMA, warps 4..11: softmax, two threads a row
constexpr int kPlHalfKeys = kPlKeys / 2;        // scores per softmax thread and block
constexpr int kPlQAtomBytes = kPlRows * 128;
constexpr int kPlAtomBytes = kPlKeys * 128;
constexpr int kPlQBytes = kPlAtoms * kPlQAtomBytes;
constexpr int kPlTileBytes = kPlAtoms * kPlAtomBytes;
constexpr int kPlSmemBytes = kPlQBytes + kPlStages * kPlTileBytes + 1024;
constexpr int kPlStagedPages = 1024;
constexpr int kPlScoreColumn = 256;             // O: columns 0..D-1; scores: 256..351 and 384..479
constexpr uint32_t kPlIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
constexpr uint32_t kPlIdescScore = kPlIdesc | ((static_cast<uint32_t>(kPlKeys) >> 3) << 17);
constexpr uint32_t kPlIdescValue = kPlIdesc | ((static_cast<uint32_t>(kPlD) >> 3) << 17) | (1u << 16);   // B is MN-major
static_assert(kPlKeys % 32 == 0 && kPlD % 16 == 0 && kPlSmemBytes <= 226 * 1024, "tiles");

struct PlaneTcArgs {
  const bf16* q;
  bf16* out;
  float* part_out;
  float* part_lse;
  const int* items;
  const int* cu_seqlens;
  const int* entry_start;
  const int* entry_slot;
  const int* block_table;
  int hq, hkv, page_size, num_pages, max_pages, slots, window, chunk, splits;
  int box_rows;             // rows of a TMA box: divides a page and 32
  float scale_log2;
  int* fault;
  const float* sink;
  int out_stride;
  const bf16* gate;
  int gate_stride;
};

__global__ void __launch_bounds__(kPlThreads, 1)
attention_plane_tc_kernel(const __grid_constant__ CUtensorMap map_cache, const PlaneTcArgs args) {
  extern __shared__ unsigned char pl_smem_raw[];
  __shared__ __align__(8) uint64_t full[kPlStages], empty[kPlStages];
  __shared__ __align__(8) uint64_t score_ready[2], p_ready[2], value_done[2];
  __shared__ __align__(8) uint64_t q_ready, drained;
  __shared__ uint32_t tmem_slot;
  __shared__ int aborted_flag;
  __shared__ int staged_pages[kPlStagedPages];
  __shared__ float exchange[2][2][kPlRows];       // [block parity][half][row]
  volatile int* aborted = &aborted_flag;

  pdl_trigger();
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const uint32_t q_tile = (smem_addr(pl_smem_raw) + 1023u) & ~1023u;
  auto tile_at = [&](int s) { return q_tile + kPlQBytes + s * kPlTileBytes; };

  // ---- the item ------------------------------------------------------------------------
  const int* item = args.items + static_cast<size_t>(blockIdx.y) * 4;
  const int entry = item[0], row0 = item[1], split = item[2];
  const int kv_head = blockIdx.x;
  const int group = args.hq / args.hkv;
  const int tok_begin = args.cu_seqlens[entry];
  const int n_rows = min(kPlRows, (args.cu_seqlens[entry + 1] - tok_begin) * group - row0);
  const int start = args.entry_start[entry];
  const int slot = args.entry_slot[entry];
  const int min_pos = start + row0 / group, max_pos = start + (row0 + n_rows - 1) / group;
  const bool bad = slot < 0 || slot >= args.slots || start < 0 || n_rows <= 0 ||
                   max_pos >= args.max_pages * args.page_size;
  if (bad && tid == 0)
    atomicOr(args.fault, (slot < 0 || slot >= args.slots) ? kFaultSlot : kFaultPosition);
  // the keys the tile sees, from the start of a box on, in blocks; this split's share of them
  const int hi = bad ? 0 : max_pos + 1;
  const int seen = first_visible(min_pos, args.window, args.chunk) / args.box_rows * args.box_rows;
  const int all_blocks = hi > seen ? (hi - seen + kPlKeys - 1) / kPlKeys : 0;
  const int per_split = (all_blocks + args.splits - 1) / args.splits;
  const int first_block = min(split * per_split, all_blocks);
  const int n_blocks = min(per_split, all_blocks - first_block);
  const int k_begin = seen + first_block * kPlKeys;
  const int k_end = min(hi, k_begin + n_blocks * kPlKeys);
  const int* table = args.block_table + static_cast<size_t>(bad ? 0 : slot) * args.max_pages;

  const int live = max(1, min(4, (n_rows + 31) / 32));    // softmax warps that have rows; what the others' lanes hold is never read

  // ---- set-up --------------------------------------------------------------------------
  if (tid == 0) {
    for (int s = 0; s < kPlStages; ++s) {
      mbar_init(smem_addr(&full[s]), 1);
      mbar_init(smem_addr(&empty[s]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_addr(&score_ready[i]), 1);
      mbar_init(smem_addr(&p_ready[i]), 2 * live);
      mbar_init(smem_addr(&value_done[i]), 1);
    }
    mbar_init(smem_addr(&q_ready), 2 * live);
    mbar_init(smem_addr(&drained), 1);
    aborted_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_addr(&tmem_slot), 512);
    tmem_relinquish();
  }
  const int first_page = k_begin / args.page_size;
  const int page_count = n_blocks > 0 ? (k_end - 1) / args.page_size - first_page + 1 : 0;
  const bool staged = page_count <= kPlStagedPages;
  if (staged) {
    for (int i = tid; i < page_count; i += kPlThreads) {
      int page = table[first_page + i];
      if (page < 0 || page >= args.num_pages) {
        atomicOr(args.fault, kFaultPageId);
        page = -1;
      }
      staged_pages[i] = page;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_out = uniform(tmem_slot);
  auto tmem_score = [&](int b) { return tmem_out + kPlScoreColumn + (b & 1) * 128; };

  if (warp == 0) {
    // -------------------------------------------------------------------- TMA producer
    const int boxes = kPlKeys / args.box_rows;
    const int outside = args.num_pages * args.hkv * args.page_size;     // a row behind the last: the box is filled with zeros
    bool waited = false;
    int issued = 0;
    for (int b = 0; b < n_blocks; ++b) {
      const int stage = b % kPlStages;
      const int kb = k_begin + b * kPlKeys;
      if (b >= kPlStages) {
        if (!__all_sync(0xffffffffu, mbar_wait(smem_addr(&empty[stage]), ((b / kPlStages) - 1) & 1, aborted, args.fault, 1 << 8))) break;
      }
      // rows from `start` on are written by this step's earlier kernels
      if (!waited && kb + kPlKeys > start) {
        pdl_wait();
        waited = true;
      }
      if (lane == 0) mbar_expect_tx(smem_addr(&full[stage]), kPlTileBytes);
      __syncwarp();
      for (int i = lane; i < boxes * kPlAtoms; i += 32) {
        const int x = i / kPlAtoms, atom = i - x * kPlAtoms;
        const int j = kb + x * args.box_rows;              // first row of the box
        int row = outside;
        if (j < k_end) {
          const int page_index = j / args.page_size;
          int page;
          if (staged) {
            page = staged_pages[page_index - first_page];
          } else {
            page = table[page_index];
            if (page < 0 || page >= args.num_pages) {
              atomicOr(args.fault, kFaultPageId);
              page = -1;
            }
          }
          if (page >= 0) row = (page * args.hkv + kv_head) * args.page_size + (j - page_index * args.page_size);
        }
        tma_load_2d(tile_at(stage) + atom * kPlAtomBytes + x * args.box_rows * 128, &map_cache, smem_addr(&full[stage]), atom * 64, row);
      }
      __syncwarp();
      ++issued;
    }
    if (!waited) pdl_wait();
    // the copies land before the shared memory goes, also when the others have given up
    volatile int go_on = 0;
    for (int s = 0; s < kPlStages; ++s) {
      const int fills = (issued - s + kPlStages - 1) / kPlStages;
      if (fills > 0) mbar_wait(smem_addr(&full[s]), (fills - 1) & 1, &go_on, args.fault);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------- tensor-core issuer
    // Products run in the order they are issued: the scores of block j + 2 overwrite the columns that held P of
    // block j only after the values product that read them.
    const int blocks = uniform(n_blocks);
    const bool issues = elect_one();
    bool ok = blocks > 0;
    auto wait = [&](uint64_t* bar, int phase, int where) {
      return __all_sync(0xffffffffu, mbar_wait(smem_addr(bar), phase & 1, aborted, args.fault, where));
    };
    auto rows_here = [&](int b) {
      if (!wait(&full[b % kPlStages], b / kPlStages, 1 << 9)) return false;
      const int kept = k_end - (k_begin + b * kPlKeys);    // rows of this block inside the range
      if (kept < kPlKeys) {
        const int box_end = (kept + args.box_rows - 1) / args.box_rows * args.box_rows;
        for (int i = lane; i < (box_end - kept) * kPlAtoms * 8; i += 32) {
          const int r = kept + i / (kPlAtoms * 8), c = i % (kPlAtoms * 8);
          const uint32_t dst = tile_at(b % kPlStages) + (c >> 3) * kPlAtomBytes + r * 128 + (c & 7) * 16;
          asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(dst), "r"(0) : "memory");
        }
        fence_async_smem();
        __syncwarp();
      }
      tc_fence_after();
      return true;
    };
    auto issue_scores = [&](int b) {
      if (issues) {
        const uint64_t q_desc = operand_desc(q_tile), keys_desc = operand_desc(tile_at(b % kPlStages));
#pragma unroll
        for (int k = 0; k < kPlD / 16; ++k) {
          const uint32_t atom = (k >> 2), within = (k & 3) * 2;
          umma_bf16(tmem_score(b), q_desc + atom * (kPlQAtomBytes >> 4) + within,
                    keys_desc + atom * (kPlAtomBytes >> 4) + within, kPlIdescScore, k > 0 ? 1u : 0u);
        }
        umma_commit(smem_addr(&score_ready[b & 1]));
      }
      __syncwarp();
    };
    if (ok) ok = wait(&q_ready, 0, 1 << 10);
    if (ok) ok = rows_here(0);
    if (ok) issue_scores(0);
    for (int b = 0; b < blocks && ok; ++b) {
      if (b + 1 < blocks) {
        ok = rows_here(b + 1);
        if (!ok) break;
        issue_scores(b + 1);
      }
      ok = wait(&p_ready[b & 1], b >> 1, 1 << 11);
      if (!ok) break;
      tc_fence_after();
      if (issues) {
        const uint64_t values_desc = operand_desc_mn(tile_at(b % kPlStages), kPlAtomBytes);
#pragma unroll
        for (int part = 0; part < 2; ++part) {      // P as it rounds, then what the rounding left
#pragma unroll
          for (int k = 0; k < kPlKeys / 16; ++k)
            umma_bf16_ts(tmem_out, tmem_score(b) + part * (kPlKeys / 2) + k * 8, values_desc + k * (2048 >> 4), kPlIdescValue,
                         (b > 0 || part > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(smem_addr(&value_done[b & 1]));
        umma_commit(smem_addr(&empty[b % kPlStages]));
      }
      __syncwarp();
    }
    if (issues) umma_commit(smem_addr(&drained));
    __syncwarp();
    mbar_wait(smem_addr(&drained), 0, aborted, args.fault, 1 << 12);
    __syncwarp();
  } else if (warp >= 4 && (warp & 3) < live) {
    // -------------------------------------------------------------------- softmax and output
    // Warps 4 + i and 8 + i share the rows of lane quarter i, a half of the columns each.  What leads one of them past
    // a meeting point leads the other: they vote there.
    const int quarter = warp & 3;                      // tensor-memory lanes this warp may touch
    const int half = (warp - 4) >> 2;
    const int r = quarter * 32 + lane;                 // row of the tile = lane of S and O
    const uint32_t lane_bits = static_cast<uint32_t>(quarter * 32) << 16;
    const int p = row0 + r;                            // packed row of the request
    const bool exists = r < n_rows;
    const int token = p / group;
    const int pos = exists && !bad ? start + token : -1;        // -1: a row that sees no key
    const int lo_pos = first_visible(pos, args.window, args.chunk);
    pdl_wait();                                        // queries come from the kernel before
    if (n_blocks > 0) {
      // the 32 rows of Q into the K-major operand [row][64] per 64 columns, swizzled; each warp half of the pieces
      constexpr int kPieces = kPlD / 16;               // 16-byte pieces a lane fetches
      constexpr int kChunks = kPlD / 8;                // ... of a row
      const int shift = (group & (group - 1)) == 0 ? 31 - __clz(group) : -1;
      uint4 fetched[kPieces];
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int at = (half * kPieces + i) * 32 + lane;
        const int rr = quarter * 32 + at / kChunks, c = at % kChunks;
        const int pp = row0 + rr;
        const int tt = shift >= 0 ? pp >> shift : pp / group;
        fetched[i] = make_uint4(0, 0, 0, 0);
        if (rr < n_rows)
          fetched[i] = __ldcg(reinterpret_cast<const uint4*>(
              args.q + (static_cast<size_t>(tok_begin + tt) * args.hq + kv_head * group + (pp - tt * group)) * kPlD + c * 8));
      }
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int at = (half * kPieces + i) * 32 + lane;
        const int rr = quarter * 32 + at / kChunks, c = at % kChunks;
        const uint32_t dst = q_tile + (c >> 3) * kPlQAtomBytes + rr * 128 + (((c & 7) ^ (rr & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(fetched[i].x), "r"(fetched[i].y), "r"(fetched[i].z), "r"(fetched[i].w) : "memory");
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_addr(&q_ready));
    }

    float ref_max = -INFINITY;                         // exponentials are taken against ref_max, the same in both threads
    unsigned long long row_sum2 = pf_pack2(0.0f, 0.0f);   // of this thread's columns
    bool ok = true;
    for (int b = 0; b < n_blocks; ++b) {
      const int kb = k_begin + b * kPlKeys + half * kPlHalfKeys;     // this thread's first key
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&score_ready[b & 1]), (b >> 1) & 1, aborted, args.fault, 1 << 13));
      // (the values product two blocks back has ended: it was issued before these scores; the wait keeps the barrier's
      // phases in step with the blocks)
      if (ok && b >= 2)
        ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&value_done[b & 1]), ((b - 2) >> 1) & 1, aborted, args.fault, 1 << 14));
      float score[kPlHalfKeys];
      float half_max = -INFINITY;
      if (ok) {
        tc_fence_after();
        uint32_t low[32];
        float high[16];
        tmem_load32(tmem_score(b) + lane_bits + half * kPlHalfKeys, low);
        tmem_load16(tmem_score(b) + lane_bits + half * kPlHalfKeys + 32, high);      // waits for both
#pragma unroll
        for (int i = 0; i < 32; ++i) score[i] = __uint_as_float(low[i]);
#pragma unroll
        for (int i = 0; i < 16; ++i) score[32 + i] = high[i];
        if (kb + kPlHalfKeys - 1 > pos || kb < lo_pos) {
#pragma unroll
          for (int i = 0; i < kPlHalfKeys; ++i) {
            const int key = kb + i;
            if (!(key <= pos && key >= lo_pos)) score[i] = -INFINITY;
          }
        }
        float lane_max[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) lane_max[i] = fmaxf(score[i], score[i + 8]);
#pragma unroll
        for (int i = 16; i < kPlHalfKeys; i += 16) {
#pragma unroll
          for (int c = 0; c < 8; ++c) lane_max[c] = pf_max3(lane_max[c], score[i + c], score[i + c + 8]);
        }
        half_max = fmaxf(pf_max3(lane_max[0], lane_max[1], lane_max[2]),
                         fmaxf(pf_max3(lane_max[3], lane_max[4], lane_max[5]), fmaxf(lane_max[6], lane_max[7])));
        exchange[b & 1][half][r] = half_max;
      }
      // both have their scores in registers now, so that P may go over them
      tc_fence_before();
      ok = named_barrier_and(1 + quarter, 64, ok);
      if (!ok) break;
      tc_fence_after();
      const float block_max = fmaxf(half_max, exchange[b & 1][half ^ 1][r]) * args.scale_log2;     // the scale is positive
      const bool moves = block_max > ref_max + kPfRescaleStep || (ref_max == -INFINITY && block_max > -INFINITY);
      float alpha = 1.0f;
      if (moves) {
        alpha = ref_max == -INFINITY ? 0.0f : fast_exp2(ref_max - block_max);
        ref_max = block_max;
        float even, odd;
        pf_unpack2(row_sum2, even, odd);
        row_sum2 = pf_pack2(even * alpha, odd * alpha);
      }
      // warps one of whose rows moves rewrite their rows of O (the others times one), after the product of the block
      // before; the next one waits for this block's P.  A wait that ran out is told at the next meeting point.
      if (b > 0 && __any_sync(0xffffffffu, moves)) {
        ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&value_done[(b - 1) & 1]), ((b - 1) >> 1) & 1, aborted, args.fault, 1 << 15));
        if (!ok) continue;
        tc_fence_after();
#pragma unroll 2
        for (int c = half; c < kPlD / 16; c += 2) {
          float value[16];
          uint32_t raw[16];
          tmem_load16(tmem_out + lane_bits + c * 16, value);
#pragma unroll
          for (int i = 0; i < 16; ++i) raw[i] = __float_as_uint(value[i] * alpha);
          tmem_store16(tmem_out + lane_bits + c * 16, raw);
        }
      }
      const float shift = ref_max == -INFINITY ? 0.0f : ref_max;
      const unsigned long long scale2 = pf_pack2(args.scale_log2, args.scale_log2), shift2 = pf_pack2(-shift, -shift);
      uint32_t packed[kPlHalfKeys / 2], rest[kPlHalfKeys / 2];
#pragma unroll
      for (int i = 0; i < kPlHalfKeys / 2; ++i) {
        float x0, x1;
        pf_unpack2(pf_fma2(pf_pack2(score[2 * i], score[2 * i + 1]), scale2, shift2), x0, x1);
        const float e0 = fast_exp2(x0), e1 = fast_exp2(x1);
        row_sum2 = pf_add2(row_sum2, pf_pack2(e0, e1));
        const __nv_bfloat162 pair = __floats2bfloat162_rn(e0, e1);
        packed[i] = *reinterpret_cast<const uint32_t*>(&pair);
        const __nv_bfloat162 left = __floats2bfloat162_rn(e0 - __uint_as_float(packed[i] << 16), e1 - __uint_as_float(packed[i] & 0xffff0000u));
        rest[i] = *reinterpret_cast<const uint32_t*>(&left);
      }
      auto store = [&](uint32_t to, const uint32_t (&from)[kPlHalfKeys / 2]) {
        uint32_t first[16], second[8];
#pragma unroll
        for (int i = 0; i < 16; ++i) first[i] = from[i];
#pragma unroll
        for (int i = 0; i < 8; ++i) second[i] = from[16 + i];
        tmem_store16(to, first);
        tmem_store8(to + 16, second);
      };
      const uint32_t to = tmem_score(b) + lane_bits + half * (kPlHalfKeys / 2);
      store(to, packed);
      store(to + kPlKeys / 2, rest);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_addr(&p_ready[b & 1]));
    }
    if (ok && n_blocks > 0)
      ok = mbar_wait(smem_addr(&value_done[(n_blocks - 1) & 1]), ((n_blocks - 1) >> 1) & 1, aborted, args.fault, 1 << 16);
    float even, odd;
    pf_unpack2(row_sum2, even, odd);
    exchange[n_blocks & 1][half][r] = even + odd;
    if (named_barrier_and(1 + quarter, 64, ok)) {
      tc_fence_after();
      const int head = kv_head * group + (p - token * group);
      const size_t row = static_cast<size_t>(tok_begin + token) * args.hq + head;
      float row_sum = exchange[n_blocks & 1][0][r] + exchange[n_blocks & 1][1][r];
      const bool whole = args.splits == 1;
      if (!whole && exists && half == 0)
        args.part_lse[row * args.splits + split] = row_sum > 0.0f ? ref_max + log2f(row_sum) : -INFINITY;
      float inv = row_sum > 0.0f ? 1.0f / row_sum : 0.0f;
      if (whole && args.sink != nullptr && exists && ref_max > -INFINITY) {
        // the sink's term beside the keys', both against the larger of the two (an infinite one: it alone counts, the row is zero)
        const float sink2 = args.sink[head] * 1.4426950408889634f;
        const float top = fmaxf(ref_max, sink2), keys = exp2f(ref_max - top);
        inv = sink2 == INFINITY ? 0.0f : keys / (row_sum * keys + exp2f(sink2 - top));
      }
      if (whole && exists) inv *= head_gate(args.gate, args.gate_stride, tok_begin + token, head);
      bf16* dst = args.out + static_cast<size_t>(tok_begin + token) * args.out_stride + head * kPlD;
      float* part = args.part_out + (row * args.splits + split) * kPlD;
      if (whole || n_blocks > 0) {                     // (the merge does not read a part without keys)
#pragma unroll 4
        for (int c = half; c < kPlD / 16; c += 2) {
          float value[16];
          if (n_blocks > 0) {
            tmem_load16(tmem_out + lane_bits + c * 16, value);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) value[i] = 0.0f;
          }
          if (exists && whole) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint4 packed;
              __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
              for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(value[i * 8 + 2 * e] * inv, value[i * 8 + 2 * e + 1] * inv);
              *reinterpret_cast<uint4*>(dst + c * 16 + i * 8) = packed;
            }
          } else if (exists) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<float4*>(part + c * 16 + i * 4) =
                  make_float4(value[i * 4] * inv, value[i * 4 + 1] * inv, value[i * 4 + 2] * inv, value[i * 4 + 3] * inv);
          }
          __syncwarp();
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_out, 512);
  }
}

}  // namespace RL_ATTENTION_NS
}  // namespace rl
