// latent_attn_tc.cu — latent attention of prompts and portions of prompts on tcgen05 / TMEM.
//
// The folded form of latent_attn.cu (heads score against the cached latents themselves), for kv_rank 512 and bf16 caches.  With
// `dense` tiles (8 consecutive tokens of one or two sequences) 8 tokens x 16 heads fill the 128 rows of an MMA:
//   S[128 x 64]  = [q_abs | q_rot][128 x 576] . K^T[576 x 64]     36 k-steps of M128 N64
//   O[128 x 256] += P[128 x 64] . C[64 x 256]                      4 k-steps of M128 N256, once per half of the 512 latent values
// What bounds it: the tensor pipe and, in S, shared memory (an M128 N64 step with both operands there reads 6 KB for 32 cycles of
// math).  512 TMEM columns cannot hold a 512-wide O beside S, so a CTA walks the keys once per half of the latent values and
// recomputes S (1664 instead of 1088 multiply-adds a score; a second CTA for the half would read the queries again instead).  The
// columns that a 256-wide O and two S tiles leave hold the first 256 query values as the A operand (read from TMEM, not from
// shared memory); the other 320 sit in shared memory beside two 64-key tiles (80 + 2 x 72 KB).
// Roles: warps 0-3 own a row each thread (softmax, P back into the S columns, output), warps 4-7 copy key tiles (cp.async in 16-byte
// steps through the block table, zeros past the sequence's keys), warp 8 issues the MMAs (converged, one elected lane).  S of the next
// tile runs while a tile's softmax does.
// Measured, 8 x 1024 tokens x 16 heads, back to back: 380 us (411 before the queries were asked into L2 first and the output left in 32-byte
// pieces; mma.sync kernel: 1526).  An N64 step of S costs what an N128 one does.  The copies bind: 74 KB a tile and half come in at 47 GB/s an
// SM (7 TB/s from L2 over all), 1.6 of the 1.8 us of a tile.  CTAs that stay (clusterlaunchcontrol) with TMA copies, the chunks that only S
// reads released early and a warp each for S and P . C took 394 us here, 6 to 10 % more than these for long portions.
#include "latent_attn.cuh"
#include "tc.cuh"

namespace nvllm {
namespace {

constexpr int kRank = 512, kHalf = 256, kKeys = 64, kRows = 128, kHeads = 16;
constexpr int kQTmem = 256;                                   // query values in TMEM: two bf16 per column
constexpr int kQChunks = (kRank - kQTmem) / 64 + 1;           // 64-value chunks of the query in shared memory (the last: the rotated part)
constexpr int kChunks = kRank / 64 + 1;                       // of a cached row
constexpr int kQChunkBytes = kRows * 128, kKChunkBytes = kKeys * 128;
constexpr int kTileBytes = kChunks * kKChunkBytes;
constexpr int kSmemK = kQChunks * kQChunkBytes, kSmemBar = kSmemK + 2 * kTileBytes;
constexpr int kSmemBytes = kSmemBar + 9 * 8 + 8 + 1024;
constexpr int kThreads = 288;
constexpr int kColO = 0, kColQ = kHalf, kColS = kColQ + kQTmem / 2;   // TMEM columns: O 256 | Q 128 | S 2 x 64

struct Span { int seq, t0, t1, jstart, nkeys; };   // tokens [t0, t1) of one sequence; keys [jstart, nkeys), jstart a multiple of 64

// What a CTA asks about its tile's tokens, requested at once (8 x 1024 tokens 383 -> 380 us).
struct Tokens { int seq[kLatentTileTokens], nkeys[kLatentTileTokens]; };
__device__ __forceinline__ Tokens tokens_of(const LatentAttnArgs& a, int tile0, int tend) {
  Tokens t;
#pragma unroll
  for (int i = 0; i < kLatentTileTokens; ++i) t.seq[i] = tile0 + i < tend ? a.tok_seq[tile0 + i] : -1;
#pragma unroll
  for (int i = 0; i < kLatentTileTokens; ++i) t.nkeys[i] = tile0 + i < tend ? static_cast<int>(a.positions[tile0 + i]) + 1 : 0;
  return t;
}

// The tile's one or two runs of tokens, from token t0 on (a whole warp; every lane computes the same).
__device__ __forceinline__ Span span_of(const LatentAttnArgs& a, const Tokens& tok, int tile0, int t0, int tend) {
  Span s;
  s.t0 = s.t1 = t0;
  s.seq = -1;
  int nkeys = 0, first = 1 << 30;
#pragma unroll
  for (int i = 0; i < kLatentTileTokens; ++i) {
    const int t = tile0 + i;
    if (t == t0) s.seq = tok.seq[i];
    if (t == s.t1 && t < tend && tok.seq[i] == s.seq) {
      const int nk = tok.nkeys[i];
      nkeys = max(nkeys, nk);
      first = min(first, a.window > 0 && nk > a.window ? nk - a.window : 0);
      s.t1 = t + 1;
    }
  }
  const int32_t* table = a.tables + static_cast<int64_t>(s.seq) * a.table_cap;
  const int lane = threadIdx.x & 31, blocks = (nkeys + a.block_size - 1) / a.block_size;
  for (int b = 0; b < blocks; b += 32) {   // a missing block ends the sequence's keys
    const unsigned miss = __ballot_sync(0xffffffffu, b + lane < blocks && table[b + lane] < 0);
    if (miss != 0) { nkeys = (b + __ffs(miss) - 1) * a.block_size; break; }
  }
  s.nkeys = nkeys;
  s.jstart = min(first, nkeys) & ~(kKeys - 1);
  return s;
}

// The factor on a row's accumulated values, from its running maximum (log2 units) and sum.
__device__ __forceinline__ float row_factor(const LatentAttnArgs& a, int tok, int head, float m, float l) {
  float oc = 1.0f, den = l;
  if (a.sinks) {   // the sink joins the denominator only
    const float sk = a.sinks[head] * 1.4426950408889634f, mn = fmaxf(m, sk);
    oc = fast_exp2(m - mn);
    den = l * oc + fast_exp2(sk - mn);
  }
  float inv = den > 0.f ? oc / den : 0.f;
  if (a.gate) inv *= 1.0f / (1.0f + expf(-a.gate[static_cast<int64_t>(tok) * a.ldg + head]));
  return inv;
}

// One row by one warp, over the keys [lo, hi) that it sees and no others: a NaN or an infinity in a cached row that a query of the tile
// does not see would reach it through P = 0 (0 x Inf) in the tile's products.  Such rows are computed again here, for one half of the
// values (8 neighbouring ones a lane); caches that hold numbers never get here.
__device__ __noinline__ void row_alone(const LatentAttnArgs& a, int tok, int head, int lo, int hi, int half, int lane) {
  const float* qa = a.q_abs + static_cast<int64_t>(tok) * a.ldqa + static_cast<int64_t>(head) * kRank + 8 * lane;
  const bf16* qr = static_cast<const bf16*>(a.q) + static_cast<int64_t>(tok) * a.ldq + static_cast<int64_t>(head) * (a.dim + a.rot_dim) + a.dim + 2 * lane;
  const bool rot = 2 * lane < a.rot_dim;
  float q[2][8], acc[8] = {};
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 8; ++e) q[i][e] = __bfloat162float(__float2bfloat16_rn(qa[i * kHalf + e]));
  const float r0 = rot ? __bfloat162float(qr[0]) : 0.f, r1 = rot ? __bfloat162float(qr[1]) : 0.f;
  const int32_t* table = a.tables + static_cast<int64_t>(a.tok_seq[tok]) * a.table_cap;
  float m = -INFINITY, l = 0.f;
#pragma unroll 4
  for (int j = lo; j < hi; ++j) {
    const bf16* row = static_cast<const bf16*>(a.cache) + (static_cast<int64_t>(table[j / a.block_size]) * a.block_size + j % a.block_size) * a.cache_row;
    float v[2][8], s = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint4 x = *reinterpret_cast<const uint4*>(row + i * kHalf + 8 * lane);
      const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) { v[i][2 * e] = bf16_lo(u[e]); v[i][2 * e + 1] = bf16_hi(u[e]); }
#pragma unroll
      for (int e = 0; e < 8; ++e) s = fmaf(q[i][e], v[i][e], s);
    }
    if (rot) s = fmaf(r0, __bfloat162float(row[kRank + 2 * lane]), fmaf(r1, __bfloat162float(row[kRank + 2 * lane + 1]), s));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s *= a.scale * 1.4426950408889634f;
    const float mn = fmaxf(m, s), corr = m == -INFINITY ? 0.f : fast_exp2(m - mn), p = fast_exp2(s - (mn == -INFINITY ? 0.f : mn));
    m = mn;
    l = l * corr + p;
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = fmaf(p, half ? v[1][e] : v[0][e], j == lo ? 0.f : acc[e] * corr);
  }
  const float inv = row_factor(a, tok, head, m, l);
  uint4 w;
  w.x = pack_bf16x2(acc[0] * inv, acc[1] * inv);
  w.y = pack_bf16x2(acc[2] * inv, acc[3] * inv);
  w.z = pack_bf16x2(acc[4] * inv, acc[5] * inv);
  w.w = pack_bf16x2(acc[6] * inv, acc[7] * inv);
  *reinterpret_cast<uint4*>(static_cast<bf16*>(a.out) + static_cast<int64_t>(tok) * a.ldo + static_cast<int64_t>(head) * kRank + half * kHalf + 8 * lane) = w;
}

__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}

// wide: rows of the output lie on 32 bytes
__global__ void __launch_bounds__(kThreads, 1) latent_attn_tc_kernel(const __grid_constant__ LatentAttnArgs a, int halves, bool wide) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int tile = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x);   // late tokens of the batch (most keys) first
  // all of the queries set out for L2 while the CTA finds its way (8 tokens x 32 KB; they are read a quarter at a time)
  if (threadIdx.x < kLatentTileTokens && tile * kLatentTileTokens + static_cast<int>(threadIdx.x) < a.n)
    prefetch_l2(a.q_abs + static_cast<int64_t>(tile * kLatentTileTokens + threadIdx.x) * a.ldqa + static_cast<int64_t>(blockIdx.y) * kHeads * kRank, kHeads * kRank * 4);
  const int tile0 = tile * kLatentTileTokens, tend = min(a.n, tile0 + kLatentTileTokens);
  const Tokens tok = tokens_of(a, tile0, tend);
  if (tend - tile0 < kLatentTileTokens) {
    if (!latent_tile_dense(a.tok_seq, a.n, tile)) return;
  } else {   // (the same)
    int runs = 1;
#pragma unroll
    for (int i = 1; i < kLatentTileTokens; ++i) runs += tok.seq[i] != tok.seq[i - 1];
    if (runs > 2) return;
  }
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t sQ = base, sK = base + kSmemK, bars = base + kSmemBar;
  auto k_full = [&](int b) { return bars + b * 8; };          // 64 arrivals: the producers' copies of tile buffer b have landed
  auto k_empty = [&](int b) { return bars + (2 + b) * 8; };   // the MMAs that read buffer b have retired
  auto s_full = [&](int b) { return bars + (4 + b) * 8; };
  auto p_ready = [&](int b) { return bars + (6 + b) * 8; };   // 128 arrivals: P is in TMEM (and O rescaled where it had to be)
  const uint32_t o_done = bars + 8 * 8;
  const uint32_t tmem_slot = bars + 9 * 8;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // (warp: uniform)
  const int hbase = blockIdx.y * kHeads;
  const int half0 = halves == 2 ? 0 : static_cast<int>(blockIdx.z);   // this CTA's halves of the latent values: half0 .. half0 + halves - 1

  if (tid == 0) {
    for (int b = 0; b < 2; ++b) { mbar_init(k_full(b), 64); mbar_init(k_empty(b), 1); mbar_init(s_full(b), 1); mbar_init(p_ready(b), 128); }
    mbar_init(o_done, 1);
    fence_barrier_init();
  }
  if (warp == 8) tmem_alloc<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  pdl_launch_dependents();   // (behind the allocation)
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<uint32_t*>(gen + kSmemBar + 9 * 8);
  const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const int my_tok = tile0 + (tid & 127) / kHeads, my_head = hbase + (tid & 127) % kHeads;   // of a row owner

  // The queries, read along the rows (a lane packs 8 neighbouring values): warps 4-7 put the values 256 .. 511 and the rotated part
  // into shared memory; warps 0-3 stage the first 256 in the second key buffer, from where every row owner moves its own into TMEM.
  auto q_row = [&](int r) { return a.q_abs + static_cast<int64_t>(tile0 + r / kHeads) * a.ldqa + static_cast<int64_t>(hbase + r % kHeads) * kRank; };
  const int q_rows = (tend - tile0) * kHeads;   // rows of tokens that exist
  if (warp < 8) {
    const int r0 = (warp & 3) * 32, first = warp < 4 ? 0 : kQTmem;
    constexpr int kStagePitch = kQTmem * 2 + 16;
    static_assert(kRows * kStagePitch <= kTileBytes, "the staged queries fit the second key buffer");
    uint8_t* stage = gen + kSmemK + kTileBytes;
#pragma unroll 1
    for (int i = 0; i < 32; i += 8) {
      float4 v[8][2];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = r0 + i + u;
        const float4* src = reinterpret_cast<const float4*>(q_row(r < q_rows ? r : 0) + first) + 2 * lane;
        v[u][0] = r < q_rows ? src[0] : make_float4(0.f, 0.f, 0.f, 0.f);
        v[u][1] = r < q_rows ? src[1] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = r0 + i + u;
        const uint4 w = make_uint4(pack_bf16x2(v[u][0].x, v[u][0].y), pack_bf16x2(v[u][0].z, v[u][0].w), pack_bf16x2(v[u][1].x, v[u][1].y),
                                   pack_bf16x2(v[u][1].z, v[u][1].w));
        uint8_t* dst = warp < 4 ? stage + r * kStagePitch + lane * 16 : gen + (lane >> 3) * kQChunkBytes + r * 128 + (((lane & 7) ^ (r & 7)) * 16);
        *reinterpret_cast<uint4*>(dst) = w;
      }
    }
    if (warp < 4) {
      __syncwarp();
#pragma unroll 1
      for (int c = 0; c < kQTmem / 64; ++c) {
        uint32_t w[32];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const uint4 x = *reinterpret_cast<const uint4*>(stage + tid * kStagePitch + c * 128 + p * 16);
          w[4 * p] = x.x; w[4 * p + 1] = x.y; w[4 * p + 2] = x.z; w[4 * p + 3] = x.w;
        }
        tmem_st_32x32b_x32(tmem + lane_off + kColQ + c * 32, w);
      }
      tmem_st_wait();
    } else {
      const int piece = lane & 7;
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const int r = r0 + i + (lane >> 3);
        const bf16* src = static_cast<const bf16*>(a.q) + static_cast<int64_t>(tile0 + r / kHeads) * a.ldq + static_cast<int64_t>(hbase + r % kHeads) * (a.dim + a.rot_dim) + a.dim;
        const uint4 x = r < q_rows && piece * 8 < a.rot_dim ? *reinterpret_cast<const uint4*>(src + piece * 8) : make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(gen + (kQChunks - 1) * kQChunkBytes + r * 128 + ((piece ^ (r & 7)) * 16)) = x;
      }
    }
    fence_proxy_async();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();

  // Every role walks the same sequence: runs of tokens, halves of the latent values, key tiles; `it` counts the tiles.
  if (warp >= 4 && warp < 8) {
    // warps 4, 5 copy the even tiles (buffer 0), warps 6, 7 the odd ones: a tile's copies do not wait for the landing of the other's.
    // 8 threads take a row's 128 bytes of every 64-value chunk, a thread 8 rows.
    const int p = (tid - 128) & 63, mine = (tid - 128) >> 6, piece = p & 7, row0 = p >> 3;
    const int pieces = (kRank + a.rot_dim) / 8;                                // 16-byte pieces of a cached row
    const int chunks = a.rot_dim > 0 ? kChunks : kChunks - 1;                  // chunks the MMAs read: zeros behind the row
    const bf16* cache = static_cast<const bf16*>(a.cache);
    int it = 0;
    for (int t = tile0; t < tend;) {
      const Span s = span_of(a, tok, tile0, t, tend);
      const int32_t* table = a.tables + static_cast<int64_t>(s.seq) * a.table_cap;
      for (int h = 0; h < halves; ++h)
        for (int j0 = s.jstart; j0 < s.nkeys; j0 += kKeys, ++it) {
          const int b = it & 1;
          if (b != mine) continue;
          const bf16* src[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int j = j0 + row0 + 8 * i;
            src[i] = j < s.nkeys ? cache + (static_cast<int64_t>(table[j / a.block_size]) * a.block_size + j % a.block_size) * a.cache_row + piece * 8 : nullptr;
          }
          mbar_wait(k_empty(b), ((it >> 1) & 1) ^ 1);
          const uint32_t dst = sK + b * kTileBytes + row0 * 128 + ((piece ^ (row0 & 7)) * 16);
          for (int c = 0; c < chunks; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const bool in = src[i] != nullptr && c * 8 + piece < pieces;
              cp_async_16(dst + c * kKChunkBytes + i * 1024, in ? src[i] + c * 64 : cache, in ? 16 : 0);
            }
          cp_async_commit();
          cp_async_wait<0>();
          fence_proxy_async();
          mbar_arrive(k_full(b));
        }
      t = s.t1;
    }
  } else if (warp == 8) {
    {   // the whole warp walks the tiles, one lane issues
      const uint32_t el = elect_one() ? 1u : 0u;
      auto uni = [](uint32_t v) { return __reduce_max_sync(0xffffffffu, v); };   // a value that is uniform for the compiler too
      auto test = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)) != 0; };
      const uint32_t tm = uni(tmem);
      constexpr uint32_t idesc_s = umma_idesc_bf16(kRows, kKeys, 0, 0), idesc_o = umma_idesc_bf16(kRows, kHalf, 0, 1);
      const int rot_steps = (a.rot_dim + 15) / 16;
      auto issue_s = [&](int it) {   // S_it = Q . K_it^T
        const int b = it & 1;
        const uint32_t k0 = sK + b * kTileBytes, d = tm + kColS + b * kKeys;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < kQTmem / 16; ++ks)
          umma_bf16_ts_warp(d, tm + kColQ + ks * 8, umma_desc_lo(k0, 16) + (((ks >> 2) * kKChunkBytes + (ks & 3) * 32) >> 4), idesc_s, ks != 0, el);
#pragma unroll
        for (int ks = 0; ks < (kRank - kQTmem) / 16; ++ks)
          umma_bf16_ss_warp(d, umma_desc_lo(sQ, 16) + (((ks >> 2) * kQChunkBytes + (ks & 3) * 32) >> 4),
                       umma_desc_lo(k0, 16) + (((kQTmem / 64 + (ks >> 2)) * kKChunkBytes + (ks & 3) * 32) >> 4), idesc_s, 1, el);
        for (int ks = 0; ks < rot_steps; ++ks)
          umma_bf16_ss_warp(d, umma_desc_lo(sQ, 16) + (((kQChunks - 1) * kQChunkBytes + ks * 32) >> 4),
                       umma_desc_lo(k0, 16) + (((kChunks - 1) * kKChunkBytes + ks * 32) >> 4), idesc_s, 1, el);
        umma_commit_warp(s_full(b), el);
      };
      auto issue_pv = [&](int it, int half, bool first) {   // O (+)= P_it . C_it
        const int b = it & 1;
        const uint32_t v0 = sK + b * kTileBytes + half * (kHalf / 64) * kKChunkBytes;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < kKeys / 16; ++ks)
          umma_bf16_ts_warp(tm + kColO, tm + kColS + b * kKeys + ks * 8, umma_desc_lo(v0, kKChunkBytes) + ((ks * 2048) >> 4), idesc_o, !first || ks != 0, el);
        umma_commit_warp(o_done, el);
        umma_commit_warp(k_empty(b), el);
      };
      // The key tiles of the two spans (the second may be empty), each walked once per half of the values.
      int tiles[2] = {0, 0}, ns = 0;
      for (int t = tile0; t < tend; ++ns) {
        const Span s = span_of(a, tok, tile0, t, tend);
        tiles[ns] = static_cast<int>(uni((s.nkeys - s.jstart + kKeys - 1) / kKeys));
        t = static_cast<int>(uni(s.t1));
      }
      const int total = halves * (tiles[0] + tiles[1]);
      // S of the next tile goes first when its keys are there (it runs while this tile's softmax does), PV of this tile otherwise.
      // S of tile j overwrites P of tile j - 2: PV of that one has been issued before (one thread's MMAs run in order).
      int js = 0, jp = 0;
      long long t0 = clock64();
      while (jp < total) {
        if (js < total && js <= jp + 1 && test(k_full(js & 1), (js >> 1) & 1)) {
          issue_s(js++);
        } else if (jp < js && test(p_ready(jp & 1), (jp >> 1) & 1)) {
          const int in1 = jp - halves * tiles[0], span_tiles = in1 < 0 ? tiles[0] : tiles[1], in = in1 < 0 ? jp : in1;
          issue_pv(jp, half0 + in / span_tiles, in % span_tiles == 0);
          ++jp;
        } else {
          if (clock64() - t0 > 4000000000ll) __trap();   // as mbar_wait: a pipeline fault ends the launch
          continue;
        }
        t0 = clock64();
      }
    }
  } else if (warp < 4) {
    const float scale2 = a.scale * 1.4426950408889634f;
    const uint32_t tO = tmem + lane_off + kColO;
    constexpr float kRescale = 8.0f;   // log2 units: O is rescaled only when a row's maximum grows by more
    int it = 0, again_lo = 0, again_hi = 0;
    bool again = false;
    for (int t = tile0; t < tend;) {
      const Span s = span_of(a, tok, tile0, t, tend);
      const bool mine = my_tok >= s.t0 && my_tok < s.t1;
      const int pos = mine ? static_cast<int>(a.positions[my_tok]) : -1;
      const int hi = min(pos + 1, s.nkeys), lo = a.window > 0 && pos + 1 > a.window ? pos + 1 - a.window : 0;   // the row sees the keys [lo, hi)
      for (int h = 0; h < halves; ++h) {
        float m = -INFINITY, l = 0.f;
        bool odd = false;   // some score of a tile with keys that the row does not see is no number: nor is that cached row
        const int it0 = it;
        for (int j0 = s.jstart; j0 < s.nkeys; j0 += kKeys, ++it) {
          const int b = it & 1;
          const uint32_t tS = tmem + lane_off + kColS + b * kKeys;
          mbar_wait(s_full(b), (it >> 1) & 1);
          // PV of the tile before: O is quiet from here on (the phases are consumed in order; S of this tile was issued before it
          // and the next S runs meanwhile)
          if (it > it0) mbar_wait(o_done, (it - 1) & 1);
          tc_fence_after();
          uint32_t sr[2][32];
          tmem_ld_32x32b_x32(tS, sr[0]);
          tmem_ld_32x32b_x32(tS + 32, sr[1]);
          tmem_ld_wait();
          if (j0 + kKeys > hi || j0 < lo) {   // (a sum shows any score that is no number; a test of each one cost 3 % of the kernel)
            float z8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < kKeys; ++c) z8[c & 7] += __uint_as_float(sr[c >> 5][c & 31]);
            odd |= !(fabsf(((z8[0] + z8[1]) + (z8[2] + z8[3])) + ((z8[4] + z8[5]) + (z8[6] + z8[7]))) < INFINITY);
#pragma unroll
            for (int c = 0; c < kKeys; ++c)
              if (j0 + c >= hi || j0 + c < lo) sr[c >> 5][c & 31] = 0xff800000u;
          }
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c = 0; c < kKeys; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], __uint_as_float(sr[c >> 5][c & 31]));
          const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale2;
          const bool refresh = mx - m > kRescale || (m == -INFINITY && mx > -INFINITY);
          float corr = 1.f;
          if (refresh) {
            corr = m == -INFINITY ? 0.f : fast_exp2(m - mx);
            m = mx;
            l *= corr;
          }
          if (it > it0 && __any_sync(0xffffffffu, refresh)) {
#pragma unroll 1
            for (int c = 0; c < kHalf / 32; ++c) {
              uint32_t o[32];
              tmem_ld_32x32b_x32(tO + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
              tmem_st_32x32b_x32(tO + c * 32, o);
            }
          }
          const float off = m == -INFINITY ? 0.f : m;
          float l4[4] = {0.f, 0.f, 0.f, 0.f};
          uint32_t pk[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float p0 = fast_exp2(fmaf(__uint_as_float(sr[(2 * e) >> 5][(2 * e) & 31]), scale2, -off));
            const float p1 = fast_exp2(fmaf(__uint_as_float(sr[(2 * e + 1) >> 5][(2 * e + 1) & 31]), scale2, -off));
            l4[e & 3] += p0 + p1;
            pk[e] = pack_bf16x2(p0, p1);
          }
          tmem_st_32x32b_x32(tS, pk);   // P over this thread's own S values
          l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(p_ready(b));
        }
        const float inv = mine ? row_factor(a, my_tok, my_head, m, l) : 0.f;
        bf16* out = static_cast<bf16*>(a.out) + static_cast<int64_t>(mine ? my_tok : tile0) * a.ldo + static_cast<int64_t>(my_head) * kRank + (half0 + h) * kHalf;
        if (it > it0) {
          mbar_wait(o_done, (it - 1) & 1);
          tc_fence_after();
        }
#pragma unroll 1
        for (int c = 0; c < kHalf / 32; ++c) {
          uint32_t o[32];
          if (it > it0) {
            tmem_ld_32x32b_x32(tO + c * 32, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = 0u;   // no key at all
          }
          if (mine) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              uint32_t v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = pack_bf16x2(__uint_as_float(o[16 * e + 2 * i]) * inv, __uint_as_float(o[16 * e + 2 * i + 1]) * inv);
              if (wide) {
                st_global_32(out + c * 32 + e * 16, v);
              } else {
                *reinterpret_cast<uint4*>(out + c * 32 + e * 16) = make_uint4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<uint4*>(out + c * 32 + e * 16 + 8) = make_uint4(v[4], v[5], v[6], v[7]);
              }
            }
          }
        }
        // (l is no number where a key that the row does see is none: the row's values are none, whatever the others hold)
        if (mine && odd && fabsf(l) < INFINITY) { again = true; again_lo = lo; again_hi = hi; }
        tc_fence_before();   // the next half's first PV overwrites O: it waits for this group's next p_ready
      }
      t = s.t1;
    }
    __syncwarp();   // other lanes write a row that its owner has written
    for (unsigned rows = __ballot_sync(0xffffffffu, again); rows != 0; rows &= rows - 1) {   // (no other role waits for this one any more)
      const int src = __ffs(rows) - 1, tok = __shfl_sync(0xffffffffu, my_tok, src), head = __shfl_sync(0xffffffffu, my_head, src);
      const int lo = __shfl_sync(0xffffffffu, again_lo, src), hi = __shfl_sync(0xffffffffu, again_hi, src);
      for (int h = 0; h < halves; ++h) row_alone(a, tok, head, lo, hi, half0 + h, lane);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc<512>(tmem);
  }
}

}  // namespace

// kv_rank 512, whole groups of 16 heads, a rotated part of up to 64 values, 16-byte rows everywhere, and enough tokens that a
// dense tile is likely (the others go to the mma.sync kernel).
bool latent_attn_tc_applies(const LatentAttnArgs& a) {
  return a.n >= 32 && a.kv_rank == kRank && a.heads % kHeads == 0 && a.rot_dim <= 64 && a.rot_dim % 8 == 0 && a.dim % 8 == 0 && a.cache_row % 8 == 0 &&
         a.cache_row >= kRank + a.rot_dim && a.ldqa % 4 == 0 && a.ldo % 8 == 0 && (a.rot_dim == 0 || a.ldq % 8 == 0) && aligned16(a.q_abs) &&
         aligned16(a.q) && a.scale > 0.f && aligned16(a.out) && aligned16(a.cache);
}

int latent_attn_tc_launch(const LatentAttnArgs& a, cudaStream_t st) {
  NVLLM_SMEM_ATTR_ONCE(latent_attn_tc_kernel, kSmemBytes);
  const int tiles = (a.n + kLatentTileTokens - 1) / kLatentTileTokens, groups = a.heads / kHeads;
  // One CTA per (tile, head group) walks both halves of the latent values on one copy of the queries; where that leaves SMs without
  // a CTA the halves are CTAs of their own.
  const bool split = static_cast<int64_t>(tiles) * groups * 2 <= sm_count();
  NVLLM_CUDA(launch_pdl(latent_attn_tc_kernel, dim3(tiles, groups, split ? 2 : 1), dim3(kThreads), kSmemBytes, st, a, split ? 1 : 2,
                        a.ldo % 16 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 31u) == 0));
  NVLLM_LAUNCH_CHECK("latent_attn_tc_kernel");
  return 0;
}

}  // namespace nvllm
