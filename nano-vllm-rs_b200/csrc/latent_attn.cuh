// latent_attn.cuh — arguments of the latent attention kernels (latent_attn.cu, latent_attn_tc.cu).
#pragma once

#include "common.cuh"

namespace nvllm {

struct LatentAttnArgs {
  void* out; int64_t ldo;           // [n, heads, kv_rank]
  const float* q_abs; int64_t ldqa;  // [n, heads, kv_rank] f32
  const void* q; int64_t ldq;        // [n, heads, dim + rot_dim]: only the rotated part is read
  const int32_t* tok_seq; const int64_t* positions;
  const int32_t* tables; int table_cap, block_size;
  const void* cache; int64_t cache_row;
  int n, heads, dim, rot_dim, kv_rank;
  float scale;
  int window; const float* sinks; const float* gate; int64_t ldg;   // 0 / null: none
  int splits; float* part;   // splits > 1: CTAs along z share a token's key tiles; partial (acc[kv_rank], m, l) per (token, head, split)
  int cluster;               // cluster > 1: so does a cluster of that many CTAs along z, without partials in memory
  int skip_dense;            // the tcgen05 kernel takes the dense 8-token tiles of the batch (latent_tile_dense), this launch the others
};

constexpr int kLatentTileTokens = 8;

// A tile of 8 consecutive tokens of the batch is dense when the 8 tokens that end with its last one belong to at most two sequences:
// prompts and portions of prompts, not single decoded tokens.  (A short last tile is judged with the tokens in front of it: one or two
// tokens are always of two sequences at most, and 33 single tokens at 4001 keys took 290 us, 34 477, with the last ones walking their
// keys alone on the tcgen05 kernel, 32 took 98; the end of a prompt stays dense.)
__device__ __forceinline__ bool latent_tile_dense(const int32_t* __restrict__ tok_seq, int n, int tile) {
  const int t1 = min(n, (tile + 1) * kLatentTileTokens), t0 = max(0, t1 - kLatentTileTokens);
  int runs = 1;
  for (int t = t0 + 1; t < t1; ++t) runs += tok_seq[t] != tok_seq[t - 1];
  return runs <= 2;
}

bool latent_attn_tc_applies(const LatentAttnArgs& a);                 // latent_attn_tc.cu
int latent_attn_tc_launch(const LatentAttnArgs& a, cudaStream_t st);
bool latent_attn_decode_applies(const LatentAttnArgs& a);             // latent_attn_decode.cu
int latent_attn_decode_launch(const LatentAttnArgs& a, cudaStream_t st);

}  // namespace nvllm
