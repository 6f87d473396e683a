// recurrence.cuh — the arguments of a linear recurrence, shared by its two kernels (recurrence.cu, recurrence_chunked.cu).
#pragma once

#include "common.cuh"

namespace nvllm {

struct RecArgs {
  float* y; int64_t ldy;
  const float *q, *k, *v; int64_t ldq, ldk, ldv;
  int group_div;                 // head h reads q / k of group h / group_div
  const float* decay; int64_t decay_ld;   // [n, heads] (decay_ld = heads) or [heads] (decay_ld = 0); per channel: [n, heads * dk], rows decay_ld apart
  const float* step; int step_ld;     // same, or null (1)
  const float* skip;                  // [heads] or null (0)
  float* state;                       // [slots, heads, dk, dv]
  const int32_t *seq_slot, *cu_tokens; const int64_t* positions;
  int heads, dk, dv;
  float q_scale;                      // factor on the read-out (a constant scale of the queries)
};

// recurrence_chunked.cu: takes a recurrence with one decay per head if the sizes and the alignment suit it.
bool linear_recurrence_chunked_applies(const RecArgs& a, int n_seqs, int n_tokens);
int linear_recurrence_chunked(const RecArgs& a, int n_seqs, cudaStream_t st);

}  // namespace nvllm
