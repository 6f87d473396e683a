// capped_attn.cuh — what the kernels of the registered models' attentions share (capped_attn.cu, capped_decode.cu).
#pragma once

#include "common.cuh"

namespace nvllm {

struct CappedAttnArgs {
  void* out; int64_t ldo;
  const void* q; int64_t ldq;
  const float* gate; int64_t ldg;
  const void *kc, *vc; int64_t k_row, v_row;
  const int32_t* tok_seq; const int64_t* positions; const int32_t* tables;
  int table_cap, block_size, n, heads, kv_heads, dim, vdim;
  float scale, softcap, temp_coef; int temp_every;
  int window; const float* sinks; int gate_per_head;
  const int32_t* dense_cu;   // non-null (and tables null): keys are not paged, key j of sequence s is row dense_cu[s] + j
  // positional options of nvllm_biased_attention (all off when zero / null)
  int keep;                  // > 0: the keys 0 .. keep - 1 stay visible outside the window (or chunk), at their true positions
  int chunk;                 // > 0: position p sees only the keys of its own chunk, floor(p / chunk) * chunk .. p
  const float* head_scale;   // [heads]: a factor per head on the scaled score
  const float* dist_bias;    // [heads, dist_rows]: added to the score of key j: dist_bias[h, min(p - j, dist_rows - 1)]
  int dist_rows;
  const float2* out_rot;     // [max_pos, vdim / 2] (cos, sin): every head's output is turned by -p, value m paired with m + vdim / 2
  int max_pos;
  int bias_staged;           // tensor-core kernel: the CTA copies its heads' rows of dist_bias into shared memory first
  const float* slopes;       // [heads]: slopes[h] * (p - j) is taken off the score of key j, after the cap
  const void* ks; int64_t ks_row; int shared;   // shared > 0: the last `shared` values of every head's key are row `slot` of ks
};

// first key a row at position p sees
__device__ __forceinline__ int first_key(const CappedAttnArgs& a, int p) {
  int lo = a.window > 0 ? max(0, p - a.window + 1) : 0;
  if (a.chunk > 0) lo = max(lo, p / a.chunk * a.chunk);
  return lo;
}

constexpr float kLog2e = 1.4426950408889634f;

// tanh(x) = 1 - 2 / (2^(2 x log2 e) + 1): two MUFU operations (ex2, rcp), absolute error ~1e-6; exact at both saturations
// (2^inf -> 1, 2^-inf -> -1).  The one-instruction tanh.approx is 2^-11 relative: too coarse where two scores near the cap
// compete (cap x 5e-4 apart in the exponent).
__device__ __forceinline__ float fast_tanh(float x) { return 1.0f - __fdividef(2.0f, fast_exp2(x * (2.0f * kLog2e)) + 1.0f); }

// capped_decode.cu: takes steps of single tokens (as many tokens as sequences) if the options, the sizes and the alignment suit it.
bool capped_decode_applies(const CappedAttnArgs& a, int n_seqs);
int capped_decode(const CappedAttnArgs& a, cudaStream_t st);

}  // namespace nvllm
