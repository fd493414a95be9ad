// The recurrence over blocks of tokens (scan_blocks.cu): what one launch of it is given.
#pragma once

#include "common.cuh"

namespace rl {

constexpr int kScanBlock = 32;      // tokens per block

struct ScanBlockArgs {
  const float* q; int q_stride;
  const float* k; int k_stride;
  const float* v; int v_stride;
  const float* decay; int decay_mode;      // 0: [heads], 1: [T, heads], 2: [T, heads * dim]
  const float* beta;
  const float* v_scale;
  const float* skip;
  const float* bonus;
  float* out; int out_stride;
  float* state; long long state_stride;
  const int* cu_seqlens; const int* entry_slot; const int* entry_start;
  int heads, kv_heads, dim, vdim, slots, entries;
  int from;             // entries of so many tokens and more are taken here
  int wide_in;          // q, k, v and row decays can be fetched 16 bytes at a time
  float* records;       // [blocks, heads, scan_record_floats]
  int* fault;
};

// Floats a block of a head takes in `records`.
int scan_record_floats(int dim, bool corrected);
// `blocks`, `taken`: bounds on the blocks of the step's entries, and on the entries that have any.
int scan_blocks(const ScanBlockArgs& args, int blocks, int taken, cudaStream_t stream);

}  // namespace rl
