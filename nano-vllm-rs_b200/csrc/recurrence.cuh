// recurrence.cuh — the arguments of the recurrences, shared by their kernels (recurrence.cu; for prompts recurrence_chunked.cu, delta_chunked.cu), and
// what of their dispatch the models count launches by.
#pragma once

#include "common.cuh"

namespace nvllm {

__device__ __forceinline__ void cp_async_4(uint32_t smem_addr, const void* gptr) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_addr), "l"(gptr) : "memory");
}

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

struct DeltaArgs {
  float* y; int64_t ldy;
  const float *q, *k, *v; int64_t ldq, ldk, ldv;
  int group_div;                       // head h reads q / k of group h / group_div
  const float* decay; int64_t ldd;     // [n, heads * dk]: decay of every key channel; HEADG: [n, heads]
  const float* beta; int64_t ldb;      // [n, heads]
  float* state;                        // [slots, heads, dk, dv]
  const int32_t *seq_slot, *cu_tokens; const int64_t* positions;
  int heads, dk, dv;
};

// delta_chunked.cu: takes a gated delta rule (a decay per key channel, or one per head) if the sizes and the alignment suit it.
bool delta_chunked_applies(const DeltaArgs& a, bool head_decay, int n_seqs, int n_tokens);
int delta_chunked(const DeltaArgs& a, bool head_decay, int n_seqs, cudaStream_t st);

// recurrence_step.cu: take steps of single tokens (as many tokens as sequences; linear recurrences with a decay per head) if the sizes and the alignment suit them.
bool linear_recurrence_single_applies(const RecArgs& a, int n_seqs, int n_tokens);
int linear_recurrence_single(const RecArgs& a, int n_seqs, cudaStream_t st);
bool delta_single_applies(const DeltaArgs& a, int n_seqs, int n_tokens);
int delta_single(const DeltaArgs& a, bool head_decay, int n_seqs, cudaStream_t st);

// nvllm_causal_conv over a step of single tokens (as many tokens as sequences): one launch for the convolution and its state.
inline bool causal_conv_single(const float* out, int64_t ldo, const float* in, int64_t ldi, const float* state, int n, int n_seqs, int channels, int taps) {
  return n == n_seqs && taps >= 2 && taps <= 4 && channels % 4 == 0 && ldi % 4 == 0 && ldo % 4 == 0 && aligned16(in) && aligned16(out) && aligned16(state);
}
// Launches of nvllm_causal_conv over any step: its kernel and the state's, or one.
inline int causal_conv_launches(const float* out, int64_t ldo, const float* in, int64_t ldi, const float* state, int n, int n_seqs, int channels, int taps) {
  return taps == 1 || causal_conv_single(out, ldo, in, ldi, state, n, n_seqs, channels, taps) ? 1 : 2;
}

}  // namespace nvllm
