// capped_decode.cu — the attentions of capped_attn.cu over steps of single tokens (as many tokens as sequences): heads of 128 values, bf16.
//
// Such a step reads every key and value once and is bound by HBM.  The layout is that of paged_decode.cu: a CTA owns one (token, key / value
// head, up to 8 of its query heads) and a share of the keys; each of its 4 warps runs a cp.async pipeline of its own over sub-tiles of 16
// rows (8 KB of keys and values, 3 deep, no barrier of the CTA inside the loop), with the keys on the M side and the heads on the N side of
// mma.sync:  S^T = K Q^T, cap / mask / softmax in f32, O^T += V^T P^T.  Rows that the token does not see are not read (zeros).  The shares of a
// token's keys are the CTAs of a cluster: the host only knows how long contexts may get, the CTAs look at the token's own and agree how many
// of them take part.  The softmaxes meet in shared memory, then in distributed shared memory, in the order of the keys.
// (The kernel for prompts walks such a step with all its warps on the same 16 rows, one 64-key tile ahead, and a barrier around each.)
// Measured, 16 heads, 4 of keys, launched one by one (some 6 us of which are the launch), that kernel and this one: 64 tokens at 1024 keys (134 MB,
// 20 us at the copy rate) 64 and 31 us, 61 with a window of 512 43 and 19.5, 8 at 1500 60 and 15, one at 40 15 and 11; 16 heads of keys, 64 tokens
// at 1024 205 and 94.  More than 16 query heads a key head would read the keys more than twice: they stay there.
#include <algorithm>

#include "capped_attn.cuh"

namespace nvllm {
namespace {

constexpr int D = 128, kWarps = 4, kThreads = 32 * kWarps, kStages = 3, kHeads = 8;
constexpr int kRowBytes = 2 * D, kSubBytes = 16 * kRowBytes, kStageBytes = 2 * kSubBytes, kWarpBytes = kStages * kStageBytes;
constexpr int kTile = 16 * kWarps;
constexpr int kOPitch = D + 4;                                                   // floats of a head's parked values
constexpr int kMergeBytes = kWarps * kHeads * (kOPitch + 2) * 4;
constexpr int kSmem = kWarps * kWarpBytes;
constexpr int kPartBytes = kHeads * (D + 2) * 4;                                 // the CTA's own softmax, behind the warps'
static_assert(kMergeBytes + kPartBytes <= kSmem, "the parked values fit into the pipelines");
constexpr int kMaxCluster = 8, kShareTiles = 2;                                  // the portable size; tiles of a CTA of a cluster, at least

__global__ void __launch_bounds__(kThreads, 2) capped_decode_kernel(const CappedAttnArgs a, int ngrp, int cluster) {
  constexpr int KS = D / 16;
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x, kvh = blockIdx.y / ngrp, grp = blockIdx.y - kvh * ngrp;
  const int group = a.heads / a.kv_heads, heads = min(kHeads, group - grp * kHeads), h0 = kvh * group + grp * kHeads;
  pdl_wait();
  const int pos = static_cast<int>(a.positions[t]);
  const int32_t* table = a.tables + static_cast<int64_t>(a.tok_seq[t]) * a.table_cap;
  const int nkeys = pos + 1, lo = max(0, first_key(a, pos));
  const int base = lo & ~15, tiles_all = nkeys > base ? (nkeys - base + kTile - 1) / kTile : 0;
  int shares = 1, first = 0, tiles = tiles_all;
  if (cluster > 1) {
    const int most = max(1, min(cluster, tiles_all / kShareTiles)), per = (tiles_all + most - 1) / most, z = static_cast<int>(blockIdx.z);
    shares = per > 0 ? (tiles_all + per - 1) / per : 1;
    if (shares == 1 && z > 0) return;   // (the whole cluster agrees: nobody waits for this CTA)
    if (shares > 1) { first = min(z * per, tiles_all); tiles = min(per, tiles_all - first); }
  }
  const uint32_t pipe = smem_u32(smem) + warp * kWarpBytes;
  const bf16* kbase = static_cast<const bf16*>(a.kc) + static_cast<int64_t>(kvh) * D;
  const bf16* vbase = static_cast<const bf16*>(a.vc) + static_cast<int64_t>(kvh) * D;
  auto issue = [&](int i) {
    const int tok = base + ((first + i) * kWarps + warp) * 16;   // (a sub-tile lies in one block: blocks are multiples of 16 tokens)
    const int32_t blk = tok < nkeys ? __ldg(table + tok / a.block_size) : -1;
    const uint32_t sK = pipe + (i % kStages) * kStageBytes, sV = sK + kSubBytes;
    const int c = lane & 15, r0 = lane >> 4;
    const int64_t slot = blk < 0 ? 0 : static_cast<int64_t>(blk) * a.block_size + tok % a.block_size;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int r = r0 + 2 * j;
      const bool in = blk >= 0 && tok + r < nkeys && tok + r >= lo;
      const int64_t row = in ? slot + r : 0;
      const uint32_t dst = r * kRowBytes + ((c ^ (r & 7)) << 4);
      cp_async_16(sK + dst, kbase + row * a.k_row + c * 8, in ? 16 : 0);
      cp_async_16(sV + dst, vbase + row * a.v_row + c * 8, in ? 16 : 0);
    }
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < tiles) issue(s);
    cp_async_commit();
  }
  uint32_t qb[KS][2];   // Q^T: head lane / 4, values 16 ks + 2 (lane % 4) + {0, 1} (+ 8)
  {
    const int hn = lane >> 2;
    const bf16* qrow = static_cast<const bf16*>(a.q) + static_cast<int64_t>(t) * a.ldq + static_cast<int64_t>(h0 + (hn < heads ? hn : 0)) * D;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      qb[ks][0] = hn < heads ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + (lane & 3) * 2) : 0u;
      qb[ks][1] = hn < heads ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + (lane & 3) * 2 + 8) : 0u;
    }
  }
  const bool capped = a.softcap > 0.f;
  const float cap2 = a.softcap * kLog2e;   // scores are kept in log2 units
  const float qscale = a.scale * (1.0f + a.temp_coef * logf(floorf(static_cast<float>((pos + 1) / a.temp_every)) + 1.0f)) * (capped ? 1.0f / a.softcap : kLog2e);
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, acc[KS][4];
#pragma unroll
  for (int i = 0; i < KS; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  for (int i = 0; i < tiles; ++i) {
    cp_async_wait<kStages - 2>();
    __syncwarp();
    if (i + kStages - 1 < tiles) issue(i + kStages - 1);
    cp_async_commit();
    const int tok = base + ((first + i) * kWarps + warp) * 16;
    if (tok >= nkeys) continue;
    const uint32_t sK = pipe + (i % kStages) * kStageBytes, sV = sK + kSubBytes;
    const int mat = lane >> 3, sw = lane & 7;
    float s2[2][4] = {};   // two chains
    {
      const uint32_t row = sK + (sw + (mat & 1) * 8) * kRowBytes;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t k4[4];
        ldmatrix_x4(k4, row + (((2 * ks + (mat >> 1)) ^ sw) << 4));
        mma_bf16_16816(s2[ks & 1], k4, qb[ks][0], qb[ks][1]);
      }
    }
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float v = (s2[0][e] + s2[1][e]) * qscale;   // with a cap: the score over the cap
      const int j = tok + (lane >> 2) + 8 * (e >> 1);
      s[e] = j < nkeys && j >= lo ? (capped ? cap2 * fast_tanh(v) : v) : -INFINITY;
    }
    float corr[2], p[4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {   // lanes with the same lane % 4 hold the same heads
      float mx = fmaxf(s[e], s[e + 2]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[e], mx), off = mn == -INFINITY ? 0.f : mn;
      corr[e] = fast_exp2(m[e] - off);
      p[e] = fast_exp2(s[e] - off);
      p[e + 2] = fast_exp2(s[e + 2] - off);
      l[e] = l[e] * corr[e] + p[e] + p[e + 2];
      m[e] = mn;
    }
    const uint32_t p0 = movmatrix_trans(pack_bf16x2(p[0], p[1])), p1 = movmatrix_trans(pack_bf16x2(p[2], p[3]));
    const bool rescale = __any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f);
    const uint32_t row = sV + (sw + (mat >> 1) * 8) * kRowBytes;
#pragma unroll
    for (int mt = 0; mt < KS; ++mt) {
      if (rescale) { acc[mt][0] *= corr[0]; acc[mt][1] *= corr[1]; acc[mt][2] *= corr[0]; acc[mt][3] *= corr[1]; }
      uint32_t v4[4];
      ldmatrix_x4_trans(v4, row + (((2 * mt + (mat & 1)) ^ sw) << 4));
      mma_bf16_16816(acc[mt], v4, p0, p1);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    l[0] += __shfl_xor_sync(0xffffffffu, l[0], o);
    l[1] += __shfl_xor_sync(0xffffffffu, l[1], o);
  }
  __syncthreads();   // every warp is done with its pipeline
  float* so = reinterpret_cast<float*>(smem);                     // [warp][8][pitch]
  float* sml = so + kWarps * kHeads * kOPitch;                    // [warp][8][2]
  {
    const int hn = (lane & 3) * 2;
    float* w = so + warp * kHeads * kOPitch;
#pragma unroll
    for (int mt = 0; mt < KS; ++mt) {
      const int d = mt * 16 + (lane >> 2);
      w[hn * kOPitch + d] = acc[mt][0];
      w[(hn + 1) * kOPitch + d] = acc[mt][1];
      w[hn * kOPitch + d + 8] = acc[mt][2];
      w[(hn + 1) * kOPitch + d + 8] = acc[mt][3];
    }
    if (lane < 4) {
#pragma unroll
      for (int e = 0; e < 2; ++e) { sml[(warp * kHeads + hn + e) * 2] = m[e]; sml[(warp * kHeads + hn + e) * 2 + 1] = l[e]; }
    }
  }
  __syncthreads();
  // An unnormalised softmax joins another with its factor; one without a key (no maximum, no sum) has nothing to add.
  auto factor = [](float ms, float ls, float mx) { return ms == -INFINITY && ls == 0.f ? 0.f : fast_exp2(ms - mx); };
  auto store = [&](int hn, int d, float o, float den) {
    float v = den != 0.f ? o / den : 0.f;
    const int h = h0 + hn;
    if (a.gate) v *= 1.0f / (1.0f + __expf(-a.gate[static_cast<int64_t>(t) * a.ldg + (a.gate_per_head ? h : static_cast<int64_t>(h) * D + d)]));
    static_cast<bf16*>(a.out)[static_cast<int64_t>(t) * a.ldo + static_cast<int64_t>(h) * D + d] = __float2bfloat16_rn(v);
  };
  float* part = reinterpret_cast<float*>(smem + kMergeBytes);     // [8][D], then [8][2]
  for (int e = threadIdx.x; e < heads * D; e += kThreads) {
    const int hn = e / D, d = e % D;
    const float sk = a.sinks && shares == 1 ? a.sinks[h0 + hn] * kLog2e : -INFINITY;   // joins the denominator only, once
    float mx = sk;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, sml[(w * kHeads + hn) * 2]);
    float o = 0.f, den = sk == -INFINITY ? 0.f : fast_exp2(sk - mx);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float ls = sml[(w * kHeads + hn) * 2 + 1], f = factor(sml[(w * kHeads + hn) * 2], ls, mx);
      if (f == 0.f && ls == 0.f) continue;
      o = fmaf(f, so[(w * kHeads + hn) * kOPitch + d], o);
      den = fmaf(f, ls, den);
    }
    if (shares == 1) {
      store(hn, d, o, den);
    } else {
      part[e] = o;
      if (d == 0) { part[kHeads * D + 2 * hn] = mx; part[kHeads * D + 2 * hn + 1] = den; }
    }
  }
  if (shares == 1) return;
  cluster_sync();
  const uint32_t at = smem_u32(part);
  for (int e = static_cast<int>(blockIdx.z) * kThreads + threadIdx.x; e < heads * D; e += cluster * kThreads) {
    const int hn = e / D, d = e % D;
    const float sk = a.sinks ? a.sinks[h0 + hn] * kLog2e : -INFINITY;
    float mx = sk, ms[kMaxCluster], ls[kMaxCluster], os[kMaxCluster];
#pragma unroll
    for (int s = 0; s < kMaxCluster; ++s)
      if (s < shares) {
        ms[s] = ld_peer_f32(at + (kHeads * D + 2 * hn) * 4, s);
        ls[s] = ld_peer_f32(at + (kHeads * D + 2 * hn + 1) * 4, s);
        os[s] = ld_peer_f32(at + e * 4, s);
      }
#pragma unroll
    for (int s = 0; s < kMaxCluster; ++s)
      if (s < shares) mx = fmaxf(mx, ms[s]);
    float o = 0.f, den = sk == -INFINITY ? 0.f : fast_exp2(sk - mx);
#pragma unroll
    for (int s = 0; s < kMaxCluster; ++s) {
      if (s >= shares) continue;
      const float f = factor(ms[s], ls[s], mx);
      if (f == 0.f && ls[s] == 0.f) continue;
      o = fmaf(f, os[s], o);
      den = fmaf(f, ls[s], den);
    }
    store(hn, d, o, den);
  }
  cluster_sync();   // nobody leaves while a peer still reads
}

// The largest cluster of which `clusters` run at once (two CTAs an SM).
int cluster_that_fits(int64_t clusters) {
  static std::once_flag once;
  static int room[kMaxCluster + 1];
  std::call_once(once, [] {
    for (int s = 2; s <= kMaxCluster; ++s) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(1, 1, s);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = kSmem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = s;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&room[s], capped_decode_kernel, &cfg) != cudaSuccess) { (void)cudaGetLastError(); room[s] = 0; }
    }
  });
  int s = kMaxCluster;
  while (s > 1 && room[s] < clusters) --s;
  return s;
}

}  // namespace

// The options that the prompt kernel takes too: a window, a cap, a temperature, sinks and a gate; and the alignment with which a step goes to the tensor
// cores at all (the kernel needs less of q and out): other calls have their probabilities in f32.
bool capped_decode_applies(const CappedAttnArgs& a, int n_seqs) {
  return n_seqs > 0 && a.n == n_seqs && a.heads / a.kv_heads <= 2 * kHeads && a.dim == D && a.vdim == D && a.tables != nullptr && a.block_size % 16 == 0 && a.keep == 0 && a.chunk == 0 &&
         a.head_scale == nullptr && a.dist_bias == nullptr && a.out_rot == nullptr && a.slopes == nullptr && a.shared == 0 && a.ldq % 8 == 0 &&
         aligned16(a.q) && a.ldo % 2 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 3u) == 0 && a.k_row % 8 == 0 && a.v_row % 8 == 0 && aligned16(a.kc) && aligned16(a.vc) &&
         a.kv_heads * ((a.heads / a.kv_heads + kHeads - 1) / kHeads) <= 65535;
}

int capped_decode(const CappedAttnArgs& a, cudaStream_t st) {
  NVLLM_SMEM_ATTR_ONCE(capped_decode_kernel, kSmem);
  const int ngrp = (a.heads / a.kv_heads + kHeads - 1) / kHeads;
  int64_t keys = static_cast<int64_t>(a.table_cap) * a.block_size;
  if (a.window > 0) keys = std::min<int64_t>(keys, a.window);
  const int cluster = static_cast<int>(std::min<int64_t>(cluster_that_fits(static_cast<int64_t>(a.n) * a.kv_heads * ngrp), std::max<int64_t>(1, keys / kTile / kShareTiles)));
  const dim3 grid(a.n, a.kv_heads * ngrp, cluster);
  if (cluster > 1) NVLLM_CUDA(launch_pdl_cluster_z(capped_decode_kernel, grid, dim3(kThreads), kSmem, st, a, ngrp, cluster));
  else NVLLM_CUDA(launch_pdl(capped_decode_kernel, grid, dim3(kThreads), kSmem, st, a, ngrp, cluster));
  NVLLM_LAUNCH_CHECK("capped_decode_kernel");
  return 0;
}

}  // namespace nvllm
