// latent_attn_decode.cu — latent attention of single tokens (decode steps) with kv_rank 512 and bf16 caches.
//
// The folded form of latent_attn.cu: the 16 heads of a CTA are the M side of mma.sync m16n8k16 and share every cached row.  What bounds it is
// reading a token's keys once; everything else has to hide behind that:
//   warps 8-11 copy key tiles of 32 rows into a ring (cp.async in 16-byte steps: rows may lie anywhere, keys start at the first one that the
//              token sees), as far ahead as the ring allows: 5 or 6 tiles, 190 KB in flight on an SM
//   warps 0-7  two groups of four take the tiles in turn, so that one group's chain (scores -> exchange -> softmax -> values) runs under
//              the other's.  In a group a warp scores 16 keys over one half of the reduction (its part of Q stays in registers); the halves meet
//              in shared memory behind ONE barrier of the group, from where every warp reads all scores in the layout of the value
//              product's A operand, does the softmax of the 16 heads for itself, and multiplies its 128 of the 512 value columns.
// A group's next scores are multiplied under the softmax of its present tile (their buffers' mbarriers are what a warp waits for).
// The groups' softmaxes, and those of the CTAs of a cluster that share a token's keys, meet at the end in (distributed) shared memory.
// Rows behind the last key repeat that key: what the unused columns of a tile multiply by zero is no other token's row.
// Measured, 16 heads, back to back, before (one 64-key tile ahead, three barriers a tile) and so: 32 tokens at 4001 keys (147 MB, 23 us at the
// copy rate) 66.3 and 38.3 us; with a launch's overhead in both, 1 at 4001 41 and 29, 150 at 500 72 and 45, 64 with a window of 512 41 and 20,
// 40 at 33 14 and 14.  Of the 38 us 33 are there without any product (queries, tables, the copies on 128 SMs, the merge).
// Copied by cp.async.bulk, a row each lane, a tile takes as long (1.1 us on an SM).
#include <algorithm>

#include "latent_attn.cuh"
#include "tc.cuh"

namespace nvllm {
namespace {

constexpr int kRank = 512, kHeads = 16, kTile = 32, kGroups = 2, kMathWarps = 8, kCopyWarps = 4, kThreads = 32 * (kMathWarps + kCopyWarps);
// Registers a thread: 168 at launch; the copying warps give up 128 of theirs, the others take 64 each (2 x 64 = 128: the sum stays).
constexpr int kLaunchRegs = 168, kCopyRegs = 40, kMathRegs = 232;
static_assert(kMathWarps * kMathRegs + kCopyWarps * kCopyRegs <= (kMathWarps + kCopyWarps) * kLaunchRegs, "registers of the launch");
constexpr int kMaxCluster = 8;      // the portable size
constexpr int kShareTiles = 4;      // key tiles of a CTA of a cluster, at least
constexpr int kSsPitch = 40;        // floats of a row of scores: 8-byte accesses of four neighbouring rows fall into different banks
constexpr int kPartPitch = kRank + 8;

template <int KSTEPS>   // 16-wide steps of the reduction: 32 (no rotated part) or 36
struct Cfg {
  static constexpr int kPitch = KSTEPS * 32 + 16;   // bytes of a key row: an odd number of 16-byte pieces, ldmatrix without conflicts
  static constexpr int kStages = KSTEPS == 32 ? 6 : 5;
  static constexpr int kTileBytes = kTile * kPitch;
  static constexpr int kRing = kStages * kTileBytes;
  static constexpr int kScores = kGroups * 2 * 2 * kHeads * kSsPitch * 4;   // [group][buffer][half of the reduction][16][pitch]
  static constexpr int kSmem = kRing + kScores + (2 * kStages + 1 + 2 * kGroups) * 8;
  static_assert(kGroups * kHeads * kPartPitch * 4 <= kRing, "the parked values fit into the ring");
};

// Arrives on `bar` (one of its counted arrivals) once this thread's copies up to here have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory"); }

template <int KSTEPS>
__global__ void __launch_bounds__(kThreads, 1) latent_attn_decode_kernel(const LatentAttnArgs a) {
  using C = Cfg<KSTEPS>;
  constexpr int KH = KSTEPS / 2;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float m_s[kGroups * kHeads], l_s[kGroups * kHeads], f_s[kMaxCluster * kGroups * kHeads], inv_s[kHeads];
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const uint32_t ring = smem_u32(smem), bars = ring + C::kRing + C::kScores;
  auto full = [&](int s) { return bars + s * 8; };
  auto empty = [&](int s) { return bars + (C::kStages + s) * 8; };
  const uint32_t q_empty = bars + 2 * C::kStages * 8, s_full = q_empty + 8;   // the queries pass through the ring's last tile
  if (tid == 0) {
    for (int s = 0; s < C::kStages; ++s) { mbar_init(full(s), 32 * kCopyWarps); mbar_init(empty(s), kMathWarps / kGroups); }
    mbar_init(q_empty, kMathWarps);
    for (int b = 0; b < 2 * kGroups; ++b) mbar_init(s_full + 8 * b, kMathWarps / kGroups);
    fence_barrier_init();
  }
  const int row_elems = (kRank + a.rot_dim + 7) & ~7;   // copied of a cached row
  pdl_wait();
  pdl_launch_dependents();
  if (a.skip_dense && latent_tile_dense(a.tok_seq, a.n, static_cast<int>(blockIdx.x) / kLatentTileTokens)) return;   // (no cluster then)
  const int t = blockIdx.x, hbase = blockIdx.y * kHeads, heads_here = min(kHeads, a.heads - hbase);
  // The queries set out first: a math thread takes 4 neighbouring values of 8 rows and, of one row, 4 values of the rotated part.
  constexpr int kRotPieces = (KSTEPS * 16 - kRank) / 4;
  float4 qv[kHeads / 2];
  uint32_t qrot[2] = {0u, 0u};
  if (warp < kMathWarps) {
    const float* qa = a.q_abs + static_cast<int64_t>(t) * a.ldqa + static_cast<int64_t>(hbase) * kRank + 4 * (tid & 127);
#pragma unroll
    for (int i = 0; i < kHeads / 2; ++i) {
      const int r = 2 * i + (tid >> 7);
      qv[i] = r < heads_here ? *reinterpret_cast<const float4*>(qa + static_cast<int64_t>(r) * kRank) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (kRotPieces > 0 && tid < kHeads * kRotPieces && tid / max(kRotPieces, 1) < heads_here) {
      const int r = tid / max(kRotPieces, 1), c = 4 * (tid % max(kRotPieces, 1));
      const uint16_t* x = static_cast<const uint16_t*>(a.q) + static_cast<int64_t>(t) * a.ldq + static_cast<int64_t>(hbase + r) * (a.dim + a.rot_dim) + a.dim + c;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + e < a.rot_dim) qrot[e >> 1] |= static_cast<uint32_t>(x[e]) << (16 * (e & 1));
    }
  }
  const int32_t* table = a.tables + static_cast<int64_t>(a.tok_seq[t]) * a.table_cap;
  int nkeys = static_cast<int>(a.positions[t]) + 1;
  int jstart = a.window > 0 && nkeys > a.window ? nkeys - a.window : 0;   // (from the position alone)
  const int blocks = nkeys > 0 ? (nkeys + a.block_size - 1) / a.block_size : 0;
  for (int b = 0; b < blocks; b += 32) {   // a missing block ends the sequence's keys (padding rows of a graph: none)
    const unsigned miss = __ballot_sync(0xffffffffu, b + lane < blocks && table[b + lane] < 0);
    if (miss != 0) { nkeys = (b + __ffs(miss) - 1) * a.block_size; break; }
  }
  nkeys = max(nkeys, 0);
  jstart = min(jstart, nkeys);
  int shares = 1;   // CTAs of the cluster that have tiles of this token: the host only knows how long contexts may get
  if (a.cluster > 1) {
    const int tiles = (nkeys - jstart + kTile - 1) / kTile, most = max(1, min(a.cluster, tiles / kShareTiles));
    const int per = (tiles + most - 1) / most, z = static_cast<int>(blockIdx.z);
    shares = per > 0 ? (tiles + per - 1) / per : 1;
    if (shares == 1 && z > 0) return;   // (the whole cluster agrees: nobody waits for this CTA)
    if (shares > 1) {
      jstart = min(jstart + z * per * kTile, nkeys);
      nkeys = min(nkeys, jstart + per * kTile);
    }
  }
  const int tiles = (nkeys - jstart + kTile - 1) / kTile;
  auto math_sync = [] { asm volatile("bar.sync 3, 256;\n" ::: "memory"); };
  __syncthreads();   // barriers

  if (warp >= kMathWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kCopyRegs));
    const int p = tid - 32 * kMathWarps;
    // 8 threads take 128 neighbouring bytes of a row, a thread 2 rows
    const int piece = p & 7, row0 = p >> 3, pieces = row_elems / 8;
    for (int it = 0; it < tiles; ++it) {
      const int s = it % C::kStages;
      const bf16* src[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = min(jstart + it * kTile + row0 + 16 * i, nkeys - 1);
        src[i] = static_cast<const bf16*>(a.cache) + (static_cast<int64_t>(table[j / a.block_size]) * a.block_size + j % a.block_size) * a.cache_row + piece * 8;
      }
      if (it >= C::kStages) mbar_wait(empty(s), (it / C::kStages - 1) & 1);
      else if (s == C::kStages - 1) mbar_wait(q_empty, 0);
      const uint32_t dst = ring + s * C::kTileBytes + row0 * C::kPitch + piece * 16;
#pragma unroll
      for (int c = 0; c < (KSTEPS + 3) / 4; ++c) {
        if (c * 8 + piece < 2 * KSTEPS) {   // zeros behind the row
          const bool in = c * 8 + piece < pieces;
          cp_async_16(dst + c * 128, in ? src[0] + c * 64 : src[0], in ? 16 : 0);
          cp_async_16(dst + 16 * C::kPitch + c * 128, in ? src[1] + c * 64 : src[1], in ? 16 : 0);
        }
      }
      cp_async_arrive(full(s));
    }
    cp_async_wait<0>();
    return;   // (behind its copies; the rest, cluster barriers too, is for the threads that stay)
  }
  {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kMathRegs));
    const int grp = warp >> 2, w = warp & 3, kh = w & 1, kq = w >> 1;   // of the group: half of the reduction, half of the tile's keys
    // Q: bf16 rows through the ring's last tile; a warp keeps its half of the reduction as A operands
    uint32_t qf[KH][4];
    {
      uint8_t* qs = smem + (C::kStages - 1) * C::kTileBytes;
#pragma unroll
      for (int i = 0; i < kHeads / 2; ++i)
        *reinterpret_cast<uint2*>(qs + (2 * i + (tid >> 7)) * C::kPitch + 8 * (tid & 127)) = make_uint2(pack_bf16x2(qv[i].x, qv[i].y), pack_bf16x2(qv[i].z, qv[i].w));
      if (kRotPieces > 0 && tid < kHeads * kRotPieces)
        *reinterpret_cast<uint2*>(qs + tid / max(kRotPieces, 1) * C::kPitch + kRank * 2 + 8 * (tid % max(kRotPieces, 1))) = make_uint2(qrot[0], qrot[1]);
      math_sync();
      const uint32_t at = smem_u32(qs) + (lane & 15) * C::kPitch + (lane >> 4) * 16 + kh * KH * 32;
#pragma unroll
      for (int i = 0; i < KH; ++i) ldmatrix_x4(qf[i], at + i * 32);
      __syncwarp();
      if (lane == 0) mbar_arrive(q_empty);
    }
    const float scale2 = a.scale * 1.4426950408889634f;   // scores in log2 units
    float acc[kRank / 4 / 8][4];
#pragma unroll
    for (int i = 0; i < kRank / 4 / 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};   // rows g and g + 8; l: this lane's columns only
    float* scores = reinterpret_cast<float*>(smem + C::kRing) + grp * (2 * 2 * kHeads * kSsPitch);
    const uint32_t k_lane = (kq * 16 + (lane & 7) + 8 * (lane >> 4)) * C::kPitch + ((lane >> 3) & 1) * 16 + kh * KH * 32;
    const uint32_t v_lane = ((lane & 7) + 8 * ((lane >> 3) & 1)) * C::kPitch + w * (kRank / 4) * 2 + (lane >> 4) * 16;
    // This warp's share of a tile's scores: two chains of products for each 8 keys, then into the group's buffer of that tile.
    auto score = [&](int it, float (&sp)[2][2][4]) {
      const uint32_t at = ring + (it % C::kStages) * C::kTileBytes + k_lane;
      mbar_wait(full(it % C::kStages), (it / C::kStages) & 1);
#pragma unroll
      for (int i = 0; i < 4; ++i) sp[i >> 1][i & 1][0] = sp[i >> 1][i & 1][1] = sp[i >> 1][i & 1][2] = sp[i >> 1][i & 1][3] = 0.f;
#pragma unroll
      for (int i = 0; i < KH; ++i) {
        uint32_t b[4];
        ldmatrix_x4(b, at + i * 32);
        mma_bf16_16816(sp[0][i & 1], qf[i], b[0], b[1]);
        mma_bf16_16816(sp[1][i & 1], qf[i], b[2], b[3]);
      }
    };
    auto hand_over = [&](int buf, const float (&sp)[2][2][4]) {
      float* sb = scores + buf * (2 * kHeads * kSsPitch);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<float2*>(sb + (kh * kHeads + g + 8 * i) * kSsPitch + kq * 16 + nt * 8 + 2 * t4) =
              make_float2(sp[nt][0][2 * i] + sp[nt][1][2 * i], sp[nt][0][2 * i + 1] + sp[nt][1][2 * i + 1]);
      __syncwarp();
      if (lane == 0) mbar_arrive(s_full + 8 * (2 * grp + buf));
    };
    if (grp < tiles) {
      float sp[2][2][4];
      score(grp, sp);
      hand_over(0, sp);
    }
    for (int it = grp, n = 0; it < tiles; it += kGroups, ++n) {
      const int s = it % C::kStages;
      const uint32_t tile = ring + s * C::kTileBytes;
      // the products of the group's next tile run under this one's softmax
      const bool more = it + kGroups < tiles;
      float sp[2][2][4];
      if (more) score(it + kGroups, sp);
      const float* sb = scores + (n & 1) * (2 * kHeads * kSsPitch);
      mbar_wait(s_full + 8 * (2 * grp + (n & 1)), (n >> 1) & 1);
      float p[4][4];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 x = *reinterpret_cast<const float2*>(sb + (g + 8 * i) * kSsPitch + nt * 8 + 2 * t4);
          const float2 y = *reinterpret_cast<const float2*>(sb + (kHeads + g + 8 * i) * kSsPitch + nt * 8 + 2 * t4);
          p[nt][2 * i] = x.x + y.x;
          p[nt][2 * i + 1] = x.y + y.y;
        }
      const int left = nkeys - jstart - it * kTile;   // columns from here on repeat the last key
      if (left < kTile) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (nt * 8 + 2 * t4 + (e & 1) >= left) p[nt][e] = -INFINITY;
      }
      float corr[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float mx = -INFINITY;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) mx = fmaxf(mx, fmaxf(p[nt][2 * i], p[nt][2 * i + 1]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mn = fmaxf(m[i], mx * scale2), off = mn == -INFINITY ? 0.f : mn;
        corr[i] = fast_exp2(m[i] - off);
        m[i] = mn;
        float sum = 0.f;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          p[nt][2 * i] = fast_exp2(fmaf(p[nt][2 * i], scale2, -off));
          p[nt][2 * i + 1] = fast_exp2(fmaf(p[nt][2 * i + 1], scale2, -off));
          sum += p[nt][2 * i] + p[nt][2 * i + 1];
        }
        l[i] = l[i] * corr[i] + sum;
      }
      if (!__all_sync(0xffffffffu, corr[0] == 1.0f && corr[1] == 1.0f)) {
#pragma unroll
        for (int i = 0; i < kRank / 4 / 8; ++i) { acc[i][0] *= corr[0]; acc[i][1] *= corr[0]; acc[i][2] *= corr[1]; acc[i][3] *= corr[1]; }
      }
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        const uint32_t pf[4] = {pack_bf16x2(p[2 * kk][0], p[2 * kk][1]), pack_bf16x2(p[2 * kk][2], p[2 * kk][3]),
                                pack_bf16x2(p[2 * kk + 1][0], p[2 * kk + 1][1]), pack_bf16x2(p[2 * kk + 1][2], p[2 * kk + 1][3])};
#pragma unroll
        for (int c = 0; c < kRank / 4 / 16; ++c) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, tile + v_lane + kk * 16 * C::kPitch + c * 32);
          mma_bf16_16816(acc[2 * c], pf, b[0], b[1]);
          mma_bf16_16816(acc[2 * c + 1], pf, b[2], b[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(s));
      if (more) hand_over((n + 1) & 1, sp);   // (every warp of the group has read that buffer's last scores: it has handed over this tile's since)
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
      l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    }
    math_sync();   // both groups are through: the ring is free (its last copies were waited for)
    float* part = reinterpret_cast<float*>(smem) + grp * (kHeads * kPartPitch);
#pragma unroll
    for (int i = 0; i < kRank / 4 / 8; ++i) {
      const int col = w * (kRank / 4) + i * 8 + 2 * t4;
      *reinterpret_cast<float2*>(part + g * kPartPitch + col) = make_float2(acc[i][0], acc[i][1]);
      *reinterpret_cast<float2*>(part + (g + 8) * kPartPitch + col) = make_float2(acc[i][2], acc[i][3]);
    }
    if (w == 0 && t4 == 0) {
      m_s[grp * kHeads + g] = m[0]; m_s[grp * kHeads + g + 8] = m[1];
      l_s[grp * kHeads + g] = l[0]; l_s[grp * kHeads + g + 8] = l[1];
    }
  }

  // the softmaxes of all groups of all CTAs with keys of this token, in the order of the keys' owners
  const bool cluster = shares > 1;
  if (cluster) cluster_sync(); else math_sync();
  if (tid < kHeads) {
    const int h = hbase + tid;
    const float sk = a.sinks && h < a.heads ? a.sinks[h] * 1.4426950408889634f : -INFINITY;   // joins the denominator only
    float mx = sk, ms[kMaxCluster * kGroups], ls[kMaxCluster * kGroups];
#pragma unroll
    for (int s = 0; s < kMaxCluster * kGroups; ++s) {
      if (s >= shares * kGroups) continue;
      const float *mp = m_s + (s % kGroups) * kHeads + tid, *lp = l_s + (s % kGroups) * kHeads + tid;
      ms[s] = cluster ? ld_peer_f32(smem_u32(mp), s / kGroups) : *mp;
      ls[s] = cluster ? ld_peer_f32(smem_u32(lp), s / kGroups) : *lp;
      mx = fmaxf(mx, ms[s]);
    }
    float den = a.sinks ? fast_exp2(sk - mx) : 0.f;
#pragma unroll
    for (int s = 0; s < kMaxCluster * kGroups; ++s) {
      if (s >= shares * kGroups) continue;
      // -1: no key there (scores that are no number have no maximum either, but a sum)
      const float f = ms[s] == -INFINITY && ls[s] == 0.f ? -1.f : fast_exp2(ms[s] - mx);
      if (!(f < 0.f)) den = fmaf(f, ls[s], den);
      f_s[s * kHeads + tid] = f;
    }
    float inv = den > 0.f ? 1.0f / den : 0.f;
    if (a.gate && h < a.heads) inv *= 1.0f / (1.0f + expf(-a.gate[static_cast<int64_t>(t) * a.ldg + h]));
    inv_s[tid] = inv;
  }
  math_sync();
  const int owners = cluster ? a.cluster : 1, rank = cluster ? static_cast<int>(blockIdx.z) : 0;
  for (int e = rank * 32 * kMathWarps + tid; e < heads_here * (kRank / 4); e += owners * 32 * kMathWarps) {
    const int r = e / (kRank / 4), c = 4 * (e % (kRank / 4));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < shares; s0 += 4) {   // four CTAs' values requested at once
      float4 x[4 * kGroups];
#pragma unroll
      for (int i = 0; i < 4 * kGroups; ++i) {
        const int s = s0 + i / kGroups;
        if (s >= shares) continue;
        const float* at = reinterpret_cast<float*>(smem) + ((i % kGroups) * kHeads + r) * kPartPitch + c;
        x[i] = cluster ? ld_peer_f32x4(smem_u32(at), s) : *reinterpret_cast<const float4*>(at);
      }
#pragma unroll
      for (int i = 0; i < 4 * kGroups; ++i) {
        if (s0 + i / kGroups >= shares) continue;
        const float f = f_s[(s0 * kGroups + i) * kHeads + r];
        if (!(f < 0.f)) v = make_float4(fmaf(f, x[i].x, v.x), fmaf(f, x[i].y, v.y), fmaf(f, x[i].z, v.z), fmaf(f, x[i].w, v.w));
      }
    }
    const float inv = inv_s[r];
    bf16* dst = static_cast<bf16*>(a.out) + static_cast<int64_t>(t) * a.ldo + static_cast<int64_t>(hbase + r) * kRank + c;
    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v.x * inv, v.y * inv), pack_bf16x2(v.z * inv, v.w * inv));
  }
  if (cluster) cluster_sync();   // nobody leaves while a peer still reads
}

// The largest cluster of which `clusters` run at once, one CTA an SM (see latent_attn.cu).
template <int KSTEPS>
int cluster_that_fits(int64_t clusters) {
  static std::once_flag once;
  static int room[kMaxCluster + 1];
  std::call_once(once, [] {
    for (int s = 2; s <= kMaxCluster; ++s) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(1, 1, s);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = Cfg<KSTEPS>::kSmem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = s;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&room[s], latent_attn_decode_kernel<KSTEPS>, &cfg) != cudaSuccess) { (void)cudaGetLastError(); room[s] = 0; }
    }
  });
  int s = kMaxCluster;
  while (s > 1 && room[s] < clusters) --s;
  return s;
}

template <int KSTEPS>
int launch(LatentAttnArgs a, cudaStream_t st) {
  auto kern = latent_attn_decode_kernel<KSTEPS>;
  NVLLM_SMEM_ATTR_ONCE(kern, Cfg<KSTEPS>::kSmem);
  static const int regs = [] {   // (a launch with fewer could not hand out what the math warps ask for, and they would wait for it)
    cudaFuncAttributes f;
    return cudaFuncGetAttributes(&f, latent_attn_decode_kernel<KSTEPS>) == cudaSuccess ? f.numRegs : 0;
  }();
  NVLLM_CHECK_ARG(regs >= kLaunchRegs, NVLLM_ERR_STATE, "latent_attention: the kernel was built with %d registers a thread, not %d", regs, kLaunchRegs);
  const int groups = (a.heads + kHeads - 1) / kHeads;
  int64_t keys = static_cast<int64_t>(a.table_cap) * a.block_size;
  if (a.window > 0) keys = std::min<int64_t>(keys, a.window);
  const int64_t tiles = (keys + kTile - 1) / kTile;
  a.cluster = a.skip_dense ? 1 : static_cast<int>(std::min<int64_t>(cluster_that_fits<KSTEPS>(static_cast<int64_t>(a.n) * groups), std::max<int64_t>(1, tiles / kShareTiles)));
  const dim3 grid(a.n, groups, a.cluster);
  if (a.cluster > 1) NVLLM_CUDA(launch_pdl_cluster_z(kern, grid, dim3(kThreads), Cfg<KSTEPS>::kSmem, st, a));
  else NVLLM_CUDA(launch_pdl(kern, grid, dim3(kThreads), Cfg<KSTEPS>::kSmem, st, a));
  NVLLM_LAUNCH_CHECK("latent_attn_decode_kernel");
  return 0;
}

}  // namespace

// kv_rank 512, a rotated part of up to 64 values, 16-byte rows and vector accesses everywhere else
bool latent_attn_decode_applies(const LatentAttnArgs& a) {
  return a.scale > 0.f && a.kv_rank == kRank && a.rot_dim <= 64 && a.cache_row % 8 == 0 && a.cache_row >= kRank + a.rot_dim && aligned16(a.cache) && a.ldqa % 4 == 0 &&
         aligned16(a.q_abs) && a.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 7u) == 0 &&
         (reinterpret_cast<uintptr_t>(a.q) & 1u) == 0;
}

int latent_attn_decode_launch(const LatentAttnArgs& a, cudaStream_t st) {
  return a.rot_dim > 0 ? launch<36>(a, st) : launch<32>(a, st);
}

}  // namespace nvllm
