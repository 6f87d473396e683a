// prefill_attn.cuh — the prompt kernel of prefill_attn.cu for the registered models' attentions.
#pragma once

#include "common.cuh"

namespace nvllm {

// What these attentions add to a causal one: a row's position decides which keys it sees (the last `window` of them, if there is a window)
// and its temperature, 1 + temp_coef log(floor((position + 1) / temp_every) + 1); scores may be capped (softcap tanh(score / softcap)), a sink
// per head joins the denominator, a gate (sigmoid of f32 values, one per head or one per output) multiplies the output.
struct PromptAttn {
  const int64_t* positions;
  const float* gate; int64_t ldg; int gate_per_head;
  const float* sinks;
  float scale, softcap, temp_coef; int temp_every;
  int window;
  int n_seqs;
};

bool prompt_attention_applies(const PromptAttn& e, int n, int heads, int kv_heads, int dim, int vdim, int64_t ldq, int64_t k_row, int64_t v_row, int64_t ldo,
                              const void* out, const void* q, const void* k, const void* v, bool paged, int block_size);
// Heads of 128 values, bf16.  tables: nullptr, keys are the sequences' own rows; else block tables of a cache whose rows lie k_row / v_row apart.
int prompt_attention(const PromptAttn& e, void* out, int64_t ldo, const void* q, int64_t ldq, const void* k, const void* v, int64_t k_row, int64_t v_row,
                     const int32_t* cu_tokens, const int32_t* tables, int table_cap, int block_size, int n, int heads, int kv_heads, cudaStream_t st);

}  // namespace nvllm
