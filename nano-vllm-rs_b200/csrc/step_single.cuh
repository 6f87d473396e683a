// step_single.cuh — a decode step of one token in one launch (step_single.cu).
#pragma once

#include "common.cuh"

namespace nvllm {

constexpr int kStepLayers = 64, kStepRows = 128;       // at the most: layers, rows of h of a CTA
constexpr int kStepContext = 16384;                    // tokens of the context at the most
constexpr int kStepParts = 17, kStepPart = 130;         // parts of the keys at the most; words of one: 128 sums, maximum, sum of weights
constexpr unsigned kStepWait = 2000000;                // the usual limit of a wait: ~1 s of 1024 clocks

struct StepLayer {
  const bf16 *qkv, *o, *gate_up, *down, *input_ln, *post_ln, *q_norm, *k_norm;   // (q_norm, k_norm: may be NULL)
  bf16 *kc, *vc;
};
struct StepArgs {
  StepLayer layer[kStepLayers];
  bf16* h;                     // the stream
  uint64_t *ll_h, *ll_qkv, *ll_parts, *ll_attn, *ll_act;   // words of a value and its mark (step_single_words of them in one piece, zero at first)
  unsigned* sync;              // the last mark that was used, CTAs that are done, abort word (zero at first)
  int* error;                  // set where a word did not come
  const int64_t* pos;
  const int32_t *slots, *tables, *ctx;
  const float* cos_sin;
  int64_t blk_stride, tok_stride, head_stride, max_position;
  int layers, hidden, heads, kv_heads, inter, block_size, table_cap;
  float eps, scale_log2;
  unsigned wait;               // 1024 clocks that a CTA waits for a word at the most
  int silent;                  // a CTA that leaves its rows of the stream out (tests); -1: none
  int off_o, off_gu, off_down, off_x, max_splits;   // filled in by step_single
};

bool step_single_applies(int hidden, int heads, int kv_heads, int dim, int inter, int layers);
int64_t step_single_words(int hidden, int heads, int kv_heads, int inter);
int step_single(StepArgs& a, uint64_t* words, cudaStream_t st);

}  // namespace nvllm
