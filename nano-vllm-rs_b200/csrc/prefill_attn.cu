// prefill_attn.cu — K3 / K4: varlen causal flash-attention forward on tcgen05 / TMEM (tensor-bound).
//
// Replaces Attention::flash_attention_varlen + create_causal_mask (reference src/layers/attention.rs:177-208,
// 321-339: per-sequence loop, O(L^2) host-built mask, dense matmul) and flash_attention_varlen_with_cache
// (:211-222, prefill of the uncached suffix against the paged prefix).
//
// One work item = two row groups (RG) of 128 threads, one query row per thread (== one TMEM lane), that share the K/V tiles
// (64 keys) of a KV head: the same 128 rows of two of its query heads where the heads pair up (both groups then end at the
// same tile and a block of rows reads half the keys of its diagonal), else 256 rows of one head.
// CTAs stay: each starts with its own block index and takes further ones from the grid's not yet started CTAs
// (clusterlaunchcontrol), so that the loads and the first S of the next item run under the last softmax and the output of
// this one, and barriers, TMEM and the launch are paid once.
//   warp 8              TMA producer: per item K_0, Q (2 x 128 x 128), V_0, K_1, V_1, ... through a ring of NSLOT 16 KiB slots.  Maps see a
//                       head's 128 values as two halves of 64 (128 bytes each): one copy brings a tile, [half][row][64] in shared memory;
//                       dense K/V (64, token, half), paged K/V (64, token, half, head, block) + block_tables
//   warps 9, 11         MMAs of group 0, 1: S = Q . K^T (8 x tcgen05.mma M128 N64 K16, both operands K-major in shared memory) and
//                       O += P . V (4 x M128 N128 K16 with A = P read from TENSOR MEMORY, V MN-major).  Warps 8, 9 and 11 stay converged, one
//                       elected lane issues: a diverged one takes over 100 clocks for every copy or MMA, and a converged one 50 to 76
//                       where the pipe takes 48, hence a warp for each group.
//   warp 10             claims the next item while this one is worked on
//   RG threads          tcgen05.ld S row -> row max -> exp2 (MUFU) -> P as packed bf16 written BACK INTO TMEM over the S columns
//                       (tcgen05.st; each thread only touches its own lane, so no cross-thread hazard) -> mbarrier arrive -> row sum.
//                       O accumulates in TMEM across tiles; the reference maximum is refreshed lazily (only when a tile exceeds it
//                       by 2^8), and only then is O read, scaled and written back.
// Each group has two S buffers: S of tile j + 2 follows P.V of tile j, so a group's softmax finds its next S ready and waits for no MMA;
// with one buffer of 128 keys every tile waited 850 of 3870 clocks for P.V and S of its own.
// TMEM: 512 columns = 2 RG x (2 x S/P 64 + O 128).  Causal mask is bottom-right aligned (row r of Lq sees keys <= Lk - Lq + r)
// so the same kernel serves Lq == Lk and suffix-over-prefix.  Items are ordered by their distance from the last rows of their
// sequence: longest first within a sequence, and the empty ones of short sequences at the end.
// Bound by the exponentials and the MMAs' issue side by side.  Measured, against one CTA per 256 rows with 128-key tiles and diverged issuing
// lanes (us): 24 prompts of up to 1021 tokens, 16/8 heads 128 and 80; 64 x 512 213 and 131; 2 x 4096, 32/8 heads 354 and 246; 16384 tokens 1140
// and 877 (1.25 PFLOP/s); 32 suffixes behind 2048 shared keys, paged 184 and 132; 64 x 5 47 and 20; 1 x 300 15 and 15.
#include <type_traits>

#include "prefill_attn.cuh"
#include "tc.cuh"

namespace nvllm {

int check_layout(const nvllm_kv_layout* L);  // store_kvcache.cu

namespace pf {
constexpr int D = 128, BM = 128, BN = 64, NSLOT = 8;
constexpr int kQBytes = BM * D * 2;          // one RG's Q tile: 2 halves of [128 x 64]
constexpr int kTileBytes = BN * D * 2;       // one K (or V) tile: 2 halves of [64 x 64]
constexpr int kSmemQ = 0;
constexpr int kSmemKV = kSmemQ + 2 * kQBytes;
constexpr int kSmemBar = kSmemKV + NSLOT * kTileBytes;
constexpr int kNumBars = 2 + 2 * NSLOT + 12 + 4;        // even: what follows lies on 16 bytes
constexpr int kSmemClaim = kSmemBar + kNumBars * 8;   // 16-byte answer to a claim
constexpr int kSmemItem = kSmemClaim + 16;            // the next item and whether there is one
constexpr int kSmemTmem = kSmemItem + 64;
constexpr int kSmemGate = kSmemTmem + 16;             // EXT: 4 KiB for each softmax warp
constexpr int kSmemBytes = kSmemTmem + 16 + 1024;
constexpr int kSmemBytesExt = kSmemBytes + 8 * 4096;
constexpr int kThreads = 384;   // 2 softmax warpgroups + 1 warpgroup holding the TMA, claim and two MMA warps
constexpr int kReaders = 3 + 8; // of the next item: one lane of the TMA warp, the MMA warps and the softmax warps
static_assert(kSmemClaim % 16 == 0, "the claim's answer is written as 16 bytes");
}  // namespace pf

struct PrefillParams {
  bf16* out;
  const bf16 *q, *k, *v;   // what the maps cover, for rows that are computed alone (row_alone)
  int64_t ldq, k_tok, k_head, k_blk, v_tok, v_head, v_blk, rows_k;   // strides in elements; rows_k: rows of dense K/V
  const int32_t* cu_q;
  const int32_t* cu_k;
  const int32_t* tables;  // NULL: dense K/V
  int H, Hkv, max_blocks, block_size;
  int box_tok;   // tokens of a K / V copy: 0 dense, else min(64, block size)
  int pair;      // 1: row group g = query head 2u + g of the same 128 rows; 0: rows [128 g, 128 g + 128) of 256 rows of head u
  int units;     // grid.x = units * (row blocks per grid.z step)
  int z_blocks;
  int64_t out_stride;
  float scale_log2;
  PromptAttn e;  // EXT only
};

namespace pf {

struct Item {
  int seq, head[2], first[2], n[2];  // per row group: query head, first row within the sequence's queries, KV tiles
  int kvh, q0, k0, Lq, Lk, n_cta;
  int kt0;  // EXT: the key tile that tile 0 of the item is
};

// The item of a block index; false if the sequence has no such rows.
__device__ __forceinline__ bool decode_item(const PrefillParams& p, int bx, int by, int bz, Item& it) {
  const int unit = bx % p.units, zz = bz * p.z_blocks + bx / p.units;
  it.seq = by;
  it.q0 = __ldg(p.cu_q + by);
  it.Lq = __ldg(p.cu_q + by + 1) - it.q0;
  it.k0 = __ldg(p.cu_k + by);
  it.Lk = __ldg(p.cu_k + by + 1) - it.k0;
  const int rows = p.pair ? BM : 2 * BM;
  const int qblk = (it.Lq + rows - 1) / rows - 1 - zz;  // zz counts from the sequence's last rows
  it.n_cta = 0;
  if (qblk < 0) return false;
  it.kvh = (p.pair ? 2 * unit : unit) / (p.H / p.Hkv);
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    it.head[g] = p.pair ? 2 * unit + g : unit;
    it.first[g] = qblk * rows + (p.pair ? 0 : g * BM);
    // KV tiles the row group needs (0 when it has no valid row); bottom-right aligned
    const int last = min(it.first[g] + BM, it.Lq) - 1;
    const int visible = max(1, min(it.Lk, it.Lk - it.Lq + last + 1));
    it.n[g] = it.first[g] >= it.Lq ? 0 : (visible + BN - 1) / BN;
    it.n_cta = max(it.n_cta, it.n[g]);
  }
  return true;
}

// EXT: grid.x = units * blocks of all sequences, the last block of the last sequence first.  A whole converged warp; lane i looks at sequence i of 32.
__device__ __forceinline__ bool decode_prompt_item(const PrefillParams& p, int index, Item& it) {
  const int by = index / p.units, bx = index - by * p.units, lane = threadIdx.x & 31, rows = p.pair ? BM : 2 * BM;
  auto blocks_of = [&](int s) { return s < p.e.n_seqs ? (__ldg(p.cu_q + s + 1) - __ldg(p.cu_q + s) + rows - 1) / rows : 0; };
  int total = 0;
  for (int s = lane; s < p.e.n_seqs; s += 32) total += blocks_of(s);
  int tile = static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(total))) - 1 - by, qblk = 0;
  it.n_cta = 0;
  if (tile < 0) return false;
  it.seq = -1;
  for (int s0 = 0; s0 < p.e.n_seqs; s0 += 32) {
    int end = blocks_of(s0 + lane);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, end, o); end += lane >= o ? v : 0; }
    const unsigned behind = __ballot_sync(0xffffffffu, tile < end);
    if (behind != 0u) {
      const int l = __ffs(behind) - 1, before = __shfl_sync(0xffffffffu, end, l > 0 ? l - 1 : 0);
      it.seq = s0 + l;
      qblk = tile - (l > 0 ? before : 0);
      break;
    }
    tile -= __shfl_sync(0xffffffffu, end, 31);
  }
  if (it.seq < 0) return false;
  it.q0 = __ldg(p.cu_q + it.seq);
  it.Lq = __ldg(p.cu_q + it.seq + 1) - it.q0;
  it.k0 = it.q0;                              // keys that are not paged are the sequence's own rows
  it.kvh = (p.pair ? 2 * bx : bx) / (p.H / p.Hkv);
  const int p0 = static_cast<int>(__ldg(p.e.positions + it.q0 + qblk * rows));
  it.kt0 = p.e.window > 0 ? max(0, p0 - p.e.window + 1) / BN : 0;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    it.head[g] = p.pair ? 2 * bx + g : bx;
    it.first[g] = qblk * rows + (p.pair ? 0 : g * BM);
    const int last = min(it.first[g] + BM, it.Lq) - 1;
    it.n[g] = it.first[g] >= it.Lq ? 0 : max(1, static_cast<int>(__ldg(p.e.positions + it.q0 + last)) / BN + 1 - it.kt0);
    it.n_cta = max(it.n_cta, it.n[g]);
  }
  it.Lk = 0;
  return true;
}

// Asks for the block index of a CTA of this grid that has not started (it then never will); 16 bytes arrive at `dst`.
__device__ __forceinline__ void claim_next(uint32_t dst, uint32_t bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n" ::"r"(dst), "r"(bar) : "memory");
}
__device__ __forceinline__ bool claim_read(uint32_t src, int& bx, int& by, int& bz) {
  uint32_t ok, x = 0, y = 0, z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\t"
      "ld.shared.b128 h, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.u32 %3, 1, 0, p;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, h;\n\t}\n"
      : "=&r"(x), "=&r"(y), "=&r"(z), "=&r"(ok)
      : "r"(src)
      : "memory");
  bx = static_cast<int>(x); by = static_cast<int>(y); bz = static_cast<int>(z);
  return ok != 0;
}

// pairs of f32 in one 64-bit register: one instruction slot for two values
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Exponentials of 32 scores (in place, f32) and the packed bf16 of them.
__device__ __forceinline__ void exp_chunk(uint32_t (&s)[32], uint32_t (&pk)[16], uint64_t scale2, uint64_t off2) {
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    float p0, p1;
    unpack2(fma2(pack2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), scale2, off2), p0, p1);
    p0 = fast_exp2(p0);
    p1 = fast_exp2(p1);
    s[2 * e] = __float_as_uint(p0);
    s[2 * e + 1] = __float_as_uint(p1);
    pk[e] = pack_bf16x2(p0, p1);      // low half = even key: consecutive K elements share a 32-bit column
  }
}
// tanh(x) = 1 - 2 / (2^(2 x log2 e) + 1): absolute error ~1e-6, exact at both saturations (as in the kernels of capped_attn.cu)
__device__ __forceinline__ float ratio_tanh(float x) { return 1.0f - __fdividef(2.0f, fast_exp2(x * 2.8853900817779268f) + 1.0f); }

// EXT: the factor on a row's accumulated values, from its maximum (log2 units) and sum: 1 / sum, with the sink and the head's gate.
__device__ __forceinline__ float row_factor(const PrefillParams& p, int64_t tok, int head, float m, float l) {
  float inv = l > 0.f ? 1.0f / l : 0.f;
  if (p.e.sinks != nullptr) {   // the sink joins the denominator only
    const float sk = __ldg(p.e.sinks + head) * 1.4426950408889634f, mn = fmaxf(m, sk), oc = fast_exp2(m - mn);
    const float ll = l * oc + fast_exp2(sk - mn);
    inv = ll > 0.f ? oc / ll : 0.f;
  }
  if (p.e.gate != nullptr && p.e.gate_per_head) inv *= 1.0f / (1.0f + __expf(-__ldg(p.e.gate + tok * p.e.ldg + head)));
  return inv;
}

// One row by one warp, over the keys [from, vis) that it sees and no others.  P is 0 for the keys of a tile that a row does not see (later
// tokens, keys before its window, rows of the next sequence, the unwritten rest of a block), but 0 x NaN and 0 x Inf are NaN: a value there
// that is no number would reach the row through the tile's P.V.  So rows whose O is not finite are computed again here; inputs
// that are numbers never get here.  The test is 64 instructions a row beside the 192 and more of every tile (two prompts of 4096 tokens at the
// 8B widths, whole steps without and with it: 27.79 and 27.83 ms, runs of one side 1.4 % apart).  qscale: factor on the score before the cap, or to
// log2 units.
template <bool EXT>
__device__ __noinline__ void row_alone(const PrefillParams& p, int seq, int64_t tok, int head, int kvh, int k0, int from, int vis, float qscale) {
  const int lane = threadIdx.x & 31;
  auto load4 = [&](const bf16* at, float (&x)[4]) {
    const uint2 u = *reinterpret_cast<const uint2*>(at + 4 * lane);
    x[0] = bf16_lo(u.x); x[1] = bf16_hi(u.x); x[2] = bf16_lo(u.y); x[3] = bf16_hi(u.y);
  };
  const int32_t* table = p.tables ? p.tables + static_cast<int64_t>(seq) * p.max_blocks : nullptr;
  float q[4], acc[4] = {}, m = -INFINITY, l = 0.f;
  load4(p.q + tok * p.ldq + static_cast<int64_t>(head) * D, q);
#pragma unroll 4
  for (int j = from; j < vis; ++j) {
    int64_t blk = 0, at = static_cast<int64_t>(k0) + j;
    bool there = at < p.rows_k;
    if (table != nullptr) {
      const int b = j / p.block_size;
      blk = b < p.max_blocks ? table[b] : -1;
      at = j - b * p.block_size;
      there = blk >= 0;
    }
    float k[4] = {}, v[4] = {};   // (a block that is not there: zeros, as in the tiles)
    if (there) {
      load4(p.k + blk * p.k_blk + at * p.k_tok + kvh * p.k_head, k);
      load4(p.v + blk * p.v_blk + at * p.v_tok + kvh * p.v_head, v);
    }
    float s = fmaf(q[0], k[0], fmaf(q[1], k[1], fmaf(q[2], k[2], q[3] * k[3])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s *= qscale;
    if constexpr (EXT) {
      if (p.e.softcap > 0.f) s = p.e.softcap * 1.4426950408889634f * ratio_tanh(s);
    }
    const float mn = fmaxf(m, s), corr = m == -INFINITY ? 0.f : fast_exp2(m - mn), w = fast_exp2(s - (mn == -INFINITY ? 0.f : mn));
    m = mn;
    l = l * corr + w;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = fmaf(w, v[e], j == from ? 0.f : acc[e] * corr);
  }
  float inv = l > 0.f ? 1.0f / l : 0.f;
  if constexpr (EXT) {
    inv = row_factor(p, tok, head, m, l);
    if (p.e.gate != nullptr && !p.e.gate_per_head) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(p.e.gate + tok * p.e.ldg + head * D) + lane);
      const float x[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] *= 1.0f / (1.0f + __expf(-x[e]));
    }
  }
  *reinterpret_cast<uint2*>(p.out + tok * p.out_stride + static_cast<int64_t>(head) * D + 4 * lane) =
      make_uint2(pack_bf16x2(acc[0] * inv, acc[1] * inv), pack_bf16x2(acc[2] * inv, acc[3] * inv));
}

__device__ __forceinline__ float max3(uint32_t a, uint32_t b, float m) {
  float r;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(r) : "f"(__uint_as_float(a)), "f"(__uint_as_float(b)), "f"(m));
  return r;
}
__device__ __forceinline__ float max32(const uint32_t (&s)[32]) {
  float a[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int e = 0; e < 16; ++e) a[e & 3] = max3(s[2 * e], s[2 * e + 1], a[e & 3]);
  return fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3]));
}
__device__ __forceinline__ uint64_t sum32(const uint32_t (&s)[32], uint64_t acc) {
  uint64_t b = pack2(0.f, 0.f);
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    acc = add2(acc, pack2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])));
    b = add2(b, pack2(__uint_as_float(s[2 * e + 2]), __uint_as_float(s[2 * e + 3])));
  }
  return add2(acc, b);
}
}  // namespace pf

// EXT: what PromptAttn adds.
template <bool EXT>
__global__ void __launch_bounds__(pf::kThreads, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ PrefillParams p) {
  using namespace pf;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bars = smem_base + kSmemBar;
  const uint32_t q_full = bars, q_empty = bars + 8;
  auto slot_full = [&](int s) { return bars + (2 + s) * 8; };
  auto slot_empty = [&](int s) { return bars + (2 + NSLOT + s) * 8; };
  auto s_full = [&](int g, int b) { return bars + (2 + 2 * NSLOT + 2 * g + b) * 8; };       // S is in buffer b of group g
  auto p_ready = [&](int g, int b) { return bars + (2 + 2 * NSLOT + 4 + 2 * g + b) * 8; };  // P is in buffer b of group g (128 arrivals)
  auto o_done = [&](int g, int b) { return bars + (2 + 2 * NSLOT + 8 + 2 * g + b) * 8; };   // P.V with buffer b of group g has retired
  const uint32_t item_full = bars + (2 + 2 * NSLOT + 12) * 8, item_empty = item_full + 8, answered = item_full + 16;
  const uint32_t claim = smem_base + kSmemClaim, tmem_slot = smem_base + kSmemTmem;
  Item* const item_smem = reinterpret_cast<Item*>(smem_gen + kSmemItem);
  static_assert(sizeof(Item) + 4 <= 64 && kSmemItem % 4 == 0, "an item and a word beside it fit their 64 bytes");
  int* const item_ok = reinterpret_cast<int*>(item_smem + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform: the roles below stay converged)
  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
    mbar_init(q_full, 1); mbar_init(q_empty, 2);
    for (int s = 0; s < NSLOT; ++s) { mbar_init(slot_full(s), 1); mbar_init(slot_empty(s), 2); }
    for (int g = 0; g < 2; ++g)
      for (int b = 0; b < 2; ++b) { mbar_init(s_full(g, b), 1); mbar_init(p_ready(g, b), BM); mbar_init(o_done(g, b), 1); }
    mbar_init(item_full, 1); mbar_init(item_empty, kReaders); mbar_init(answered, 1);
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();   // (behind the allocation)
  const uint32_t tmem_base = *reinterpret_cast<uint32_t*>(smem_gen + kSmemTmem);
  pdl_wait();  // q / k / v (and the cache) come from the previous kernel

  auto item_of = [&](int x, int y, int z, Item& it) {
    if constexpr (EXT) return decode_prompt_item(p, x, it);
    else return decode_item(p, x, y, z, it);
  };
  // Every role walks the same list of items: its own block index, then what warp 10 publishes.
  uint32_t item_phase = 0;
  auto take_item = [&](Item& it) {       // the item behind a completed item_full
    item_phase ^= 1;
    it = *item_smem;
    return *reinterpret_cast<volatile int*>(item_ok) != 0;
  };
  auto next_item = [&](Item& it) {       // a whole warp
    mbar_wait(item_full, item_phase);
    const bool ok = take_item(it);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(item_empty);
    return ok;
  };
  // what the control flow and the addresses of a converged warp depend on, as values that are uniform for the compiler too
  auto uni = [](int v) { return static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<uint32_t>(v))); };
  Item it;
  const bool own = item_of(blockIdx.x, blockIdx.y, blockIdx.z, it);

  // Register reallocation (setmaxnreg, per warpgroup): the producer / MMA warpgroup keeps 120 registers per thread and
  // donates the rest: 192 for a softmax thread.
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 120;\n");  // must dominate the role code below (and only it)
  }
  if (warp == 10) {
    // ===== claims: one item ahead of the softmax; empty items end here, the others go out decoded =====
    // The next claim goes out once every role has read the last item, which no role puts off until another item is done.
    uint32_t ph = 0, answer_phase = 0;
    int x, y, z;
    bool ok = true;
    while (true) {
      do {
        if (lane == 0) {
          mbar_expect_tx(answered, 16);
          claim_next(claim, answered);
        }
        mbar_wait(answered, answer_phase);
        answer_phase ^= 1;
        ok = claim_read(claim, x, y, z);
        fence_proxy_async();             // the next answer is written by the async proxy
        __syncwarp();
      } while (ok && !item_of(x, y, z, it));
      if (lane == 0) {
        *item_smem = it;
        *item_ok = ok;
        mbar_arrive(item_full);
      }
      if (!ok) break;
      mbar_wait(item_empty, ph);
      ph ^= 1;
    }
  } else if (warp == 8) {
    // ===== TMA producer =====
    const uint32_t el = elect_one() ? 1u : 0u;
    int t = 0;            // tiles through the ring so far
    uint32_t q_phase = 1; // the first item finds Q's buffer empty
    for (bool more = uni(own) != 0 || uni(next_item(it)) != 0; more; more = uni(next_item(it)) != 0) {
      const int n_cta = uni(it.n_cta), kvh = uni(it.kvh), kt0 = EXT ? uni(it.kt0) : 0, k0 = uni(it.k0) + kt0 * BN;
      const int32_t* table = p.tables ? p.tables + static_cast<int64_t>(it.seq) * p.max_blocks : nullptr;
      // whole-tile boxes: a lane holds one of 32 consecutive entries of the table, entry `bi` is the present tile's
      int bi = kt0 * BN / p.block_size, in_block = kt0 * BN % p.block_size, entry = -1;
      for (int j = 0; j < n_cta; ++j) {
        int blk = 0;
        if (p.box_tok == BN) {
          if (j == 0 || ((bi & 31) == 0 && in_block == 0)) entry = (bi & ~31) + lane < p.max_blocks ? __ldg(table + (bi & ~31) + lane) : -1;
          blk = __shfl_sync(0xffffffffu, entry, bi & 31);
          blk = uni(blk < 0 ? 0x3fffff : blk);  // past the sequence end: far out of bounds -> TMA zero-fills
        }
        for (int kv = 0; kv < 2; ++kv, ++t) {  // K_j, V_j
          const int slot = t & (NSLOT - 1);
          const CUtensorMap* map = kv ? &tmap_v : &tmap_k;
          mbar_wait(slot_empty(slot), ((t / NSLOT) & 1) ^ 1);
          mbar_expect_tx_warp(slot_full(slot), kTileBytes, el);
          const uint32_t dst = smem_base + kSmemKV + slot * kTileBytes;
          if (p.box_tok == 0) {                 // dense
            tma_load_3d_warp(dst, map, slot_full(slot), 0, k0 + j * BN, kvh * 2, el);
          } else if (p.box_tok == BN) {
            tma_load_5d_warp(dst, map, slot_full(slot), 0, in_block, 0, kvh, blk, el);
          } else {                              // blocks smaller than a tile: a copy for each block and half
            for (int c = 0; c < BN / p.box_tok; ++c) {
              const int tok = (kt0 + j) * BN + c * p.box_tok, b = tok / p.block_size;
              const int e = b < p.max_blocks ? __ldg(table + b) : -1;
              for (int hf = 0; hf < 2; ++hf)
                tma_load_5d_warp(dst + hf * (BN * 128) + c * p.box_tok * 128, map, slot_full(slot), 0, tok - b * p.block_size, hf, kvh, uni(e < 0 ? 0x3fffff : e), el);
            }
          }
          if (j == 0 && kv == 0) {
            mbar_wait(q_empty, q_phase);
            q_phase ^= 1;
            mbar_expect_tx_warp(q_full, 2 * kQBytes, el);
            for (int g = 0; g < 2; ++g)
              tma_load_3d_warp(smem_base + kSmemQ + g * kQBytes, &tmap_q, q_full, 0, uni(it.q0 + it.first[g]), uni(it.head[g]) * 2, el);
          }
        }
        in_block += BN;
        if (in_block >= p.block_size) { in_block = 0; ++bi; }
      }
    }
  } else if (warp == 9 || warp == 11) {
    // ===== MMA issuers, a warp for each row group =====
    constexpr uint32_t idesc_s = umma_idesc_bf16(BM, BN, 0, 0);  // Q K-major, K K-major
    constexpr uint32_t idesc_o = umma_idesc_bf16(BM, D, 0, 1);   // P K-major (TMEM), V MN-major
    const uint32_t el = elect_one() ? 1u : 0u;
    auto test = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)) != 0; };
    auto slot_of = [&](int t) { return t & (NSLOT - 1); };
    auto tile_full = [&](int t) { mbar_wait(slot_full(slot_of(t)), (t / NSLOT) & 1); tc_fence_after(); };
    auto run = [&](auto group) {
      constexpr int g = decltype(group)::value;
      const uint32_t tm = __reduce_max_sync(0xffffffffu, tmem_base) + g * 256;
      struct Tiles { int n, n_cta; };  // of this group, of the item
      auto tiles_of = [&](const Item& it) { return Tiles{uni(it.n[g]), uni(it.n_cta)}; };
      auto next = [&](Tiles& nt) {
        const bool ok = uni(next_item(it)) != 0;
        nt = tiles_of(it);
        return ok;
      };
      uint32_t q_phase = 0, s_cnt = 0, p_cnt = 0;   // S and P.V issued so far: tile n of the group uses buffer n & 1
      // S = Q . K^T of tile `tile` of an item whose K_0 is number `base` of the ring; a group that does not need the tile lets it go
      auto s_of = [&](const Tiles& ti, int base, int tile) {
        const int t = base + 2 * tile;
        if (tile == 0) { mbar_wait(q_full, q_phase); q_phase ^= 1; }
        tile_full(t);
        if (tile < ti.n) {
          const uint32_t ad = umma_desc_lo(smem_base + kSmemQ + g * kQBytes, 16), bd = umma_desc_lo(smem_base + kSmemKV, 16) + slot_of(t) * (kTileBytes >> 4);
          const uint32_t b = s_cnt++ & 1;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            umma_bf16_ss_warp(tm + b * BN, ad + (((ks >> 2) * (BM * 128) + (ks & 3) * 32) >> 4), bd + (((ks >> 2) * (BN * 128) + (ks & 3) * 32) >> 4), idesc_s,
                              ks != 0, el);   // executes after P.V of the buffer's last tile, which has been issued
          umma_commit_warp(s_full(g, b), el);
        }
        umma_commit_warp(slot_empty(slot_of(t)), el);
        if (tile + 1 == ti.n_cta) umma_commit_warp(q_empty, el);   // that was the last S of its item
      };
      auto pv_of = [&](const Tiles& ti, int base, int j) {   // O (+)= P_j . V_j
        const int t = base + 2 * j + 1;
        if (j < ti.n) {
          const uint32_t b = p_cnt & 1;
          mbar_wait(p_ready(g, b), (p_cnt >> 1) & 1);  // the softmax wrote P_j (and rescaled O if it had to)
          ++p_cnt;
          tile_full(t);
          // P: 16 keys = 8 packed columns per step.  V tile: rows = keys, 64 contiguous d per row; the two d halves
          // (MN groups) are 8 KiB apart, 8 keys per 1 KiB.
          const uint32_t vd = umma_desc_lo(smem_base + kSmemKV, BN * 128) + slot_of(t) * (kTileBytes >> 4);
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            umma_bf16_ts_warp(tm + 2 * BN, tm + b * BN + ks * 8, vd + ((ks * 2048) >> 4), idesc_o, ks != 0 ? 1u : (j == 0 ? 0u : 1u), el);
          umma_commit_warp(o_done(g, b), el);
        } else {
          tile_full(t);
        }
        umma_commit_warp(slot_empty(slot_of(t)), el);
      };
      int base = 0;                    // ring number of the present item's K_0; its V_j is base + 2 j + 1, K_j base + 2 j
      int s_now = 0;                   // tiles of the present item whose S has been issued
      Tiles cur{}, nxt{};
      bool more = uni(own) != 0;
      if (more) cur = tiles_of(it); else more = next(cur);
      while (more) {
        for (; s_now < min(2, cur.n_cta); ++s_now) s_of(cur, base, s_now);
        bool known = false;
        int s_next = 0;                // tiles of the next item whose S has been issued
        const int base_next = base + 2 * cur.n_cta;
        for (int j = 0; j < cur.n_cta; ++j) {
          pv_of(cur, base, j);
          // the S behind this tile's P.V: of the tile after next, or of the next item's first ones if nothing of it has to be waited for
          if (s_now < cur.n_cta) {
            s_of(cur, base, s_now++);
          } else {
            if (!known && test(item_full, item_phase)) { more = next(nxt); known = true; }
            const int kt = base_next + 2 * s_next;
            if (known && more && s_next < min(2, nxt.n_cta) && (s_next > 0 || test(q_full, q_phase)) && test(slot_full(slot_of(kt)), (kt / NSLOT) & 1))
              s_of(nxt, base_next, s_next++);
          }
        }
        if (!known) more = next(nxt);
        base = base_next;
        cur = nxt;
        s_now = s_next;
      }
    };
    if (warp == 9) run(std::integral_constant<int, 0>{}); else run(std::integral_constant<int, 1>{});
  } else {
    // ===== row groups: softmax + output =====
    asm volatile("setmaxnreg.inc.sync.aligned.u32 192;\n");
    const int g = warp >> 2;               // row group 0 / 1
    const int t = threadIdx.x & 127;       // row within the group's tile == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS0 = tmem_base + g * 256 + lane_off;  // two buffers of S (fp32, 64 columns) / P (packed bf16, first 32 columns)
    const uint32_t tO = tS0 + 2 * BN;
    constexpr float kRescaleThreshold = 8.0f;  // log2 units: P stays <= 2^8 between refreshes
    const uint64_t scale2 = EXT ? pack2(1.f, 1.f) : pack2(p.scale_log2, p.scale_log2);
    uint32_t tile = 0;                         // tiles of this group so far
    bool more = own;
    while (true) {
      if (!more) {
        mbar_wait(item_full, item_phase);
        const bool ok = take_item(it);
        __syncwarp();
        if (lane == 0) mbar_arrive(item_empty);
        if (!ok) break;
      }
      more = false;
      const int n_my = g ? it.n[1] : it.n[0], Lk = it.Lk;
      const int row = (g ? it.first[1] : it.first[0]) + t;             // row within the sequence's queries
      int vis, vis_lo, from = 0, from_hi = 0;       // keys [from, vis) are visible; vis_lo, from_hi: to all rows of the warp
      float qscale = 0.f;                           // EXT: factor on the score: over the cap, or to log2 units
      if constexpr (EXT) {
        const int pos = static_cast<int>(__ldg(p.e.positions + it.q0 + min(row, it.Lq - 1)));
        vis = pos + 1;
        from = p.e.window > 0 ? max(0, pos - p.e.window + 1) : 0;
        vis_lo = __reduce_min_sync(0xffffffffu, vis);
        from_hi = __reduce_max_sync(0xffffffffu, from);
        qscale = p.e.scale * (1.0f + p.e.temp_coef * logf(floorf(static_cast<float>((pos + 1) / p.e.temp_every)) + 1.0f)) *
                 (p.e.softcap > 0.f ? 1.0f / p.e.softcap : 1.4426950408889634f);
      } else {
        vis = min(Lk, Lk - it.Lq + row + 1);
        vis_lo = min(Lk, Lk - it.Lq + row - lane + 1);
      }
      const float to_log2 = EXT ? 1.f : p.scale_log2;   // EXT scores are in log2 units before the maximum
      float m_ref = -INFINITY, l_run = 0.f;  // m_ref: the (stale-by-design) maximum the exponentials are taken against
      for (int j = 0; j < n_my; ++j, ++tile) {
        const int kbase = EXT ? (it.kt0 + j) * BN : j * BN;
        const int b = tile & 1;
        const uint32_t tS = tS0 + b * BN;
        mbar_wait(s_full(g, b), (tile >> 1) & 1);
        tc_fence_after();
        uint32_t sr[2][32], pk[16];
        tmem_ld_32x32b_x32(tS, sr[0]);
        tmem_ld_32x32b_x32(tS + 32, sr[1]);
        tmem_ld_wait(sr[0]);
        tmem_ld_wait(sr[1]);
        if constexpr (EXT) {
          if (p.e.softcap > 0.f) {
            const float cap2 = p.e.softcap * 1.4426950408889634f;
#pragma unroll
            for (int c = 0; c < BN; ++c) sr[c >> 5][c & 31] = __float_as_uint(cap2 * ratio_tanh(__uint_as_float(sr[c >> 5][c & 31]) * qscale));
          } else {
#pragma unroll
            for (int c = 0; c < BN; ++c) sr[c >> 5][c & 31] = __float_as_uint(__uint_as_float(sr[c >> 5][c & 31]) * qscale);
          }
          if (from_hi > kbase) {
#pragma unroll
            for (int c = 0; c < BN; ++c)
              if (kbase + c < from) sr[c >> 5][c & 31] = 0xff800000u;  // -inf
          }
        }
        if (vis_lo < kbase + BN) {     // some row of the warp has a hidden key in this tile
#pragma unroll
          for (int c = 0; c < BN; ++c)
            if (kbase + c >= vis) sr[c >> 5][c & 31] = 0xff800000u;  // -inf
        }
        const float mx = fmaxf(max32(sr[0]), max32(sr[1]));
        // lazy rescale: refresh the reference maximum only when this tile exceeds it by more than the threshold
        const bool refresh = (mx - m_ref) * to_log2 > kRescaleThreshold;  // also true for the first finite tile
        float corr = 1.f;
        if (refresh) {
          corr = (m_ref == -INFINITY) ? 0.f : fast_exp2((m_ref - mx) * to_log2);
          m_ref = mx;
          l_run *= corr;
        }
        if (j > 0 && __any_sync(0xffffffffu, refresh)) {  // tcgen05.ld/st are warp-collective: the whole warp takes part
          // O rests once P.V of the tile before has retired.  (That of two tiles before has: S of this tile was issued after it.  So the
          // barrier is at most one phase ahead of what is waited for here.)
          mbar_wait(o_done(g, b ^ 1), ((tile - 1) >> 1) & 1);
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t orr[16];
            tmem_ld_32x32b_x16(tO + c * 16, orr);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) orr[e] = __float_as_uint(__uint_as_float(orr[e]) * corr);
            tmem_st_32x32b_x16(tO + c * 16, orr);
          }
        }
        const float moff = (m_ref == -INFINITY) ? 0.f : -m_ref * to_log2;
        const uint64_t off2 = pack2(moff, moff);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          exp_chunk(sr[c], pk, scale2, off2);
          tmem_st_32x32b_x16(tS + c * 16, pk);  // P over this thread's own S lane
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(p_ready(g, b));
        uint64_t ls = sum32(sr[1], sum32(sr[0], pack2(0.f, 0.f)));
        float l0, l1;
        unpack2(ls, l0, l1);
        l_run += l0 + l1;
      }
      // ---- output -----------------------------------------------------------------------------------
      if (n_my > 0) {
        mbar_wait(o_done(g, (tile - 1) & 1), ((tile - 1) >> 1) & 1);
        tc_fence_after();
        float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
        const int head = g ? it.head[1] : it.head[0];
        // EXT: the gate of one head and 32 columns of the warp's rows, read along the rows (8 lanes a row) and passed through shared memory
        // (the 16-byte piece c of row r lies at c ^ (r & 7))
        [[maybe_unused]] float4 gate4[8];
        [[maybe_unused]] uint8_t* const stage = smem_gen + kSmemGate + warp * 4096;
        [[maybe_unused]] auto load_gate = [&](int c) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = row - lane + i * 4 + (lane >> 3);
            gate4[i] = r < it.Lq ? __ldg(reinterpret_cast<const float4*>(p.e.gate + static_cast<int64_t>(it.q0 + r) * p.e.ldg + head * D + c * 32) + (lane & 7))
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        };
        const bool gated = EXT && p.e.gate != nullptr && !p.e.gate_per_head;
        if constexpr (EXT) {
          inv = row_factor(p, it.q0 + min(row, it.Lq - 1), head, m_ref, l_run);
          if (gated) load_gate(0);
        }
        bf16* orow = p.out + static_cast<int64_t>(it.q0 + row) * p.out_stride + head * D;
        const bool wide = rows_on_32(p.out, p.out_stride);
        float most = 0.f;   // largest |O| of the row, no number if one of them is none
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t orr[32];
          tmem_ld_32x32b_x32(tO + c * 32, orr);
          tmem_ld_wait(orr);
#pragma unroll
          for (int e = 0; e < 32; e += 2) most = abs_max(__uint_as_float(orr[e]), __uint_as_float(orr[e + 1]), most);
          if constexpr (EXT) {
            if (gated) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int r = i * 4 + (lane >> 3);
                *reinterpret_cast<float4*>(stage + r * 128 + (((lane & 7) ^ (r & 7)) * 16)) = gate4[i];
              }
              __syncwarp();
              if (c + 1 < D / 32) load_gate(c + 1);
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const float4 v = *reinterpret_cast<const float4*>(stage + lane * 128 + ((e ^ (lane & 7)) * 16));
                const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) orr[4 * e + k] = __float_as_uint(__uint_as_float(orr[4 * e + k]) * (1.0f / (1.0f + __expf(-x[k]))));
              }
              __syncwarp();
            }
          }
          if (row < it.Lq) {
#pragma unroll
            for (int e = 0; e < 32; e += 16) {
              uint32_t v[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) v[k] = pack_bf16x2(__uint_as_float(orr[e + 2 * k]) * inv, __uint_as_float(orr[e + 2 * k + 1]) * inv);
              if (wide) st_global_32(orow + c * 32 + e, v);
              else {
                *reinterpret_cast<uint4*>(orow + c * 32 + e) = make_uint4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<uint4*>(orow + c * 32 + e + 8) = make_uint4(v[4], v[5], v[6], v[7]);
              }
            }
          }
        }
        tc_fence_before();   // ordered before the first P of the next item, whose P.V overwrites O
        for (uint32_t odd = __ballot_sync(0xffffffffu, row < it.Lq && !(most < INFINITY)); odd != 0u; odd &= odd - 1) {   // (stored above: stored again)
          const int src = __ffs(odd) - 1;
          __syncwarp();
          row_alone<EXT>(p, it.seq, it.q0 + row - lane + src, head, it.kvh, it.k0, __shfl_sync(0xffffffffu, from, src), __shfl_sync(0xffffffffu, vis, src),
                         EXT ? __shfl_sync(0xffffffffu, qscale, src) : p.scale_log2);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc<512>(tmem_base);
  }
}

// (64 values, row, half of a head): a head's two halves come in one copy
static int head_rows_map(CUtensorMap* map, const void* base, int64_t rows, int heads, int64_t ld, int box_rows) {
  NVLLM_CHECK_ARG(ld % 8 == 0, NVLLM_ERR_ALIGN, "TMA: base must be 16-byte aligned and the row pitch a multiple of 16 bytes");
  const uint64_t dims[3] = {64, (uint64_t)rows, 2 * (uint64_t)heads}, strides[2] = {(uint64_t)ld * 2, 128};
  const uint32_t box[3] = {64, (uint32_t)box_rows, 2};
  return make_tmap_bf16_nd(map, base, 3, dims, strides, box);
}
// (64 values, token, half, head, block) of a paged cache
static int head_blocks_map(CUtensorMap* map, const void* base, int block_size, int kv_heads, int64_t token_stride, int64_t head_stride, int64_t block_stride,
                           int box_tok) {
  const uint64_t dims[5] = {64, (uint64_t)block_size, 2, (uint64_t)kv_heads, 0x3fffffull};
  const uint64_t strides[4] = {(uint64_t)token_stride * 2, 128, (uint64_t)head_stride * 2, (uint64_t)block_stride * 2};
  const uint32_t box[5] = {64, (uint32_t)box_tok, box_tok == pf::BN ? 2u : 1u, 1, 1};
  return make_tmap_bf16_nd(map, base, 5, dims, strides, box);
}
static bool heads_pair(int heads, int kv_heads) { return (heads / kv_heads) % 2 == 0; }

// From 96 tokens a sequence on: shorter ones leave the 128 rows of a block half empty (16/4 heads, us on mma.sync and here: 32 x 64 capped 37 and
// 41, windowed 25 and 23; 24 x 130 69 and 67, 43 and 31; 8 x 1024 capped, gate per value 302 and 167, window of 512 180 and 71, dense keys of
// 16 heads 198 and 76; 8192 tokens capped 1354 and 569).
bool prompt_attention_applies(const PromptAttn& e, int n, int heads, int kv_heads, int dim, int vdim, int64_t ldq, int64_t k_row, int64_t v_row, int64_t ldo,
                              const void* out, const void* q, const void* k, const void* v, bool paged, int block_size) {
  const int64_t blocks = n / pf::BM + 1 + e.n_seqs;   // at the most; a grid's first dimension holds 2^31 - 1 CTAs
  return dim == pf::D && vdim == pf::D && e.n_seqs <= 4096 && blocks * heads <= INT32_MAX && n >= 96 * static_cast<int64_t>(e.n_seqs) && ldq % 8 == 0 && k_row % 8 == 0 && v_row % 8 == 0 &&
         ldo % 8 == 0 && aligned16(out) && aligned16(q) && aligned16(k) && aligned16(v) && heads <= 65535 &&
         (!paged || (block_size % 16 == 0 && (block_size >= pf::BN ? block_size % pf::BN == 0 : pf::BN % block_size == 0))) &&
         (e.gate == nullptr || e.gate_per_head || (aligned16(e.gate) && e.ldg % 4 == 0)) && k_row >= static_cast<int64_t>(kv_heads) * dim &&
         v_row >= static_cast<int64_t>(kv_heads) * vdim;
}

int prompt_attention(const PromptAttn& e, void* out, int64_t ldo, const void* q, int64_t ldq, const void* k, const void* v, int64_t k_row, int64_t v_row,
                     const int32_t* cu_tokens, const int32_t* tables, int table_cap, int block_size, int n, int heads, int kv_heads, cudaStream_t st) {
  CUtensorMap tq, tk, tv;
  PrefillParams p{};
  if (int rc = head_rows_map(&tq, q, n, heads, ldq, pf::BM)) return rc;
  if (tables == nullptr) {
    if (int rc = head_rows_map(&tk, k, n, kv_heads, k_row, pf::BN)) return rc;
    if (int rc = head_rows_map(&tv, v, n, kv_heads, v_row, pf::BN)) return rc;
    p.block_size = 1;
  } else {
    p.box_tok = block_size < pf::BN ? block_size : pf::BN;
    if (int rc = head_blocks_map(&tk, k, block_size, kv_heads, k_row, pf::D, k_row * block_size, p.box_tok)) return rc;
    if (int rc = head_blocks_map(&tv, v, block_size, kv_heads, v_row, pf::D, v_row * block_size, p.box_tok)) return rc;
    p.block_size = block_size;
    p.max_blocks = table_cap;
  }
  p.out = static_cast<bf16*>(out);
  p.q = static_cast<const bf16*>(q);
  p.k = static_cast<const bf16*>(k);
  p.v = static_cast<const bf16*>(v);
  p.ldq = ldq;
  p.k_tok = k_row;
  p.v_tok = v_row;
  p.k_head = p.v_head = pf::D;
  p.k_blk = k_row * block_size;
  p.v_blk = v_row * block_size;
  p.rows_k = n;
  p.cu_q = p.cu_k = cu_tokens;
  p.tables = tables;
  p.H = heads;
  p.Hkv = kv_heads;
  p.out_stride = ldo;
  p.e = e;
  p.pair = heads_pair(heads, kv_heads) ? 1 : 0;
  p.units = p.pair ? heads / 2 : heads;
  p.z_blocks = 1;
  const int rows = p.pair ? pf::BM : 2 * pf::BM;
  const int64_t blocks = (static_cast<int64_t>(n) + rows - 1) / rows + e.n_seqs;
  NVLLM_SMEM_ATTR_ONCE(prefill_attn_kernel<true>, pf::kSmemBytesExt);
  NVLLM_CUDA(launch_plain(prefill_attn_kernel<true>, dim3(static_cast<unsigned>(p.units * blocks)), dim3(pf::kThreads), pf::kSmemBytesExt, st, tq, tk, tv, p));
  NVLLM_LAUNCH_CHECK("prefill_attn_kernel");
  return 0;
}

}  // namespace nvllm

extern "C" int nvllm_varlen_prefill_attention(void* out, const void* q, const void* k, const void* v,
                                              const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k,
                                              int32_t batch, int32_t total_q, int32_t total_k,
                                              int32_t max_seqlen_q, int32_t max_seqlen_k, int32_t num_heads,
                                              int32_t num_kv_heads, int32_t head_dim, int64_t q_token_stride,
                                              int64_t kv_token_stride, int64_t out_token_stride,
                                              const void* k_cache, const void* v_cache,
                                              const int32_t* block_tables, int32_t max_blocks_per_seq,
                                              const nvllm_kv_layout* layout, float scale, int32_t dtype,
                                              void* stream) {
  using namespace nvllm;
  NVLLM_CHECK_ARG(dtype == NVLLM_BF16, NVLLM_ERR_DTYPE, "prefill_attention: dtype %d (bf16 only)", dtype);
  NVLLM_CHECK_ARG(head_dim == pf::D, NVLLM_ERR_ARG, "prefill_attention: head_dim %d (128 only)", head_dim);
  NVLLM_CHECK_ARG(batch >= 0 && batch <= 65535 && total_q >= 0 && max_seqlen_q >= 0, NVLLM_ERR_ARG,
                  "prefill_attention: batch %d total_q %d", batch, total_q);
  if (batch == 0 || total_q == 0 || max_seqlen_q == 0) return 0;
  NVLLM_CHECK_ARG(num_heads > 0 && num_kv_heads > 0 && num_heads % num_kv_heads == 0 && num_heads <= 65535,
                  NVLLM_ERR_ARG, "prefill_attention: heads %d / kv heads %d", num_heads, num_kv_heads);
  NVLLM_CHECK_ARG(out && q && cu_seqlens_q && cu_seqlens_k, NVLLM_ERR_ARG, "prefill_attention: NULL pointer");
  NVLLM_CHECK_ARG(aligned16(out) && out_token_stride % 8 == 0 && out_token_stride >= (int64_t)num_heads * head_dim,
                  NVLLM_ERR_ALIGN, "prefill_attention: out alignment / stride");
  const bool paged = block_tables != nullptr;
  CUtensorMap tq, tk, tv;
  if (int rc = head_rows_map(&tq, q, total_q, num_heads, q_token_stride, pf::BM)) return rc;
  PrefillParams p{};
  p.box_tok = 0;
  if (!paged) {
    NVLLM_CHECK_ARG(k && v && total_k > 0, NVLLM_ERR_ARG, "prefill_attention: dense k/v missing");
    if (int rc = head_rows_map(&tk, k, total_k, num_kv_heads, kv_token_stride, pf::BN)) return rc;
    if (int rc = head_rows_map(&tv, v, total_k, num_kv_heads, kv_token_stride, pf::BN)) return rc;
    p.block_size = 1;
    p.max_blocks = 0;
  } else {
    if (int rc = check_layout(layout)) return rc;
    NVLLM_CHECK_ARG(k_cache && v_cache && max_blocks_per_seq > 0, NVLLM_ERR_ARG, "prefill_attention: paged cache missing");
    NVLLM_CHECK_ARG(layout->num_kv_heads == num_kv_heads && layout->head_dim == head_dim, NVLLM_ERR_ARG,
                    "prefill_attention: layout heads/dim mismatch");
    const int bs = layout->block_size;
    constexpr int kUnit = 128;
    NVLLM_CHECK_ARG(bs % 16 == 0 && (bs >= kUnit ? bs % kUnit == 0 : kUnit % bs == 0), NVLLM_ERR_ARG,
                    "prefill_attention: block_size %d must divide or be a multiple of %d", bs, kUnit);
    p.box_tok = bs < pf::BN ? bs : pf::BN;
    if (int rc = head_blocks_map(&tk, k_cache, bs, num_kv_heads, layout->token_stride, layout->head_stride, layout->block_stride, p.box_tok)) return rc;
    if (int rc = head_blocks_map(&tv, v_cache, bs, num_kv_heads, layout->token_stride, layout->head_stride, layout->block_stride, p.box_tok)) return rc;
    p.block_size = bs;
    p.max_blocks = max_blocks_per_seq;
  }
  p.out = static_cast<bf16*>(out);
  p.q = static_cast<const bf16*>(q);
  p.k = static_cast<const bf16*>(paged ? k_cache : k);
  p.v = static_cast<const bf16*>(paged ? v_cache : v);
  p.ldq = q_token_stride;
  p.k_tok = p.v_tok = paged ? layout->token_stride : kv_token_stride;
  p.k_head = p.v_head = paged ? layout->head_stride : pf::D;
  p.k_blk = p.v_blk = paged ? layout->block_stride : 0;
  p.rows_k = total_k;
  p.cu_q = cu_seqlens_q;
  p.cu_k = cu_seqlens_k;
  p.tables = block_tables;
  p.H = num_heads;
  p.Hkv = num_kv_heads;
  p.out_stride = out_token_stride;
  p.scale_log2 = scale * 1.4426950408889634f;
  const bool pair = heads_pair(num_heads, num_kv_heads);
  p.pair = pair ? 1 : 0;
  p.units = pair ? num_heads / 2 : num_heads;
  const int rows = pair ? pf::BM : 2 * pf::BM;
  const int blocks = (max_seqlen_q + rows - 1) / rows;
  p.z_blocks = (blocks + 65534) / 65535;
  (void)max_seqlen_k;
  const dim3 grid(p.units * p.z_blocks, batch, (blocks + p.z_blocks - 1) / p.z_blocks);
  NVLLM_SMEM_ATTR_ONCE(prefill_attn_kernel<false>, pf::kSmemBytes);
  NVLLM_CUDA(launch_pdl(prefill_attn_kernel<false>, grid, dim3(pf::kThreads), pf::kSmemBytes, static_cast<cudaStream_t>(stream), tq, tk, tv, p));
  return 0;
}
