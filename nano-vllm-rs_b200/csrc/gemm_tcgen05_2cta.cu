// gemm_tcgen05_2cta.cu — K5 for M > 128: the same contract as gemm_tcgen05.cu on CTA PAIRS (tcgen05 cta_group::2).
//
// GEMM throughput on B200 is bound by the L2 -> SM operand feed (a 128 x 256 single-CTA tile moves 1 byte per
// ~43 MACs; the measured 1.35 PFLOP/s of gemm_tcgen05.cu matches that bound).  A CTA pair computes a 256 x BN tile:
// each CTA stages its own 128 rows of x and only HALF of the w tile, the leader CTA issues one
// tcgen05.mma.cta_group::2 (M = 256) that reads both CTAs' shared memory and writes 128 accumulator rows into each
// CTA's TMEM -> 64 MACs per byte fetched, i.e. 1.5x less L2 traffic per FLOP.
//   both CTAs, warp 0 lane 0   TMA producer (cp.async.bulk.tensor ... cta_group::2: bytes complete on the LEADER's barrier)
//   leader,    warp 1 lane 0   MMA issuer; tcgen05.commit ... multicast releases the smem stage / publishes the tile in BOTH CTAs
//   both CTAs, warp 2          TMEM allocator (cta_group::2)
//   both CTAs, warps 4-7       epilogue on the CTA's own 128 TMEM lanes; drained-signal goes to the leader (remote mbarrier arrive).
//                              Gated outputs and those that are added to y have warps 8-11 besides, on the upper half of the columns: with
//                              four warps their epilogue outlasts a tile's k-blocks (added, 12.4 K x 1024 x 2048 and 3072 in a prefill 63 us
//                              in the mean, with eight 54).  A plain epilogue only
//                              stores; eight warps are no faster at it (8192 x 10304 x 2048 f32 256 us with either).
#include <algorithm>
#include "tc.cuh"

namespace nvllm {

template <int GATE, bool ROPE = false, bool ADD = false>
constexpr int gemm2_epilogue_warps() { return GATE != kGateNone || ROPE || ADD ? 8 : 4; }
template <int GATE, bool ROPE = false, bool ADD = false>
constexpr int gemm2_threads() { return 128 + 32 * gemm2_epilogue_warps<GATE, ROPE, ADD>(); }

constexpr int kRopeStage = 2 * 16 * 256;   // bytes of shared memory of an epilogue warp of the qkv form

template <int BN>
struct Gemm2Cfg {
  static constexpr int BM = 256, BM_CTA = 128, BK = 64;
  static constexpr int kABytes = BM_CTA * BK * 2;
  static constexpr int kBBytes = (BN / 2) * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;  // per CTA
  static constexpr int kStagesRaw = (200 * 1024) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
  static constexpr int kTmemCols = (2 * BN <= 64) ? 64 : (2 * BN <= 128) ? 128 : (2 * BN <= 256) ? 256 : 512;
  static constexpr int kSmemBytes = kStages * kStageBytes + (2 * kStages + 4) * 8 + 16 + 1024;
};

// The qkv epilogue of a warp: 16 tokens (from row0 on) of the tile's two heads.  In the accumulator's layout (a lane per token) it is bound
// by the LSU: angles and rows are then 16-byte accesses to 32 different lines each (13.4 K tokens x 4096 x 1024: 168 us, against 96 + 67 for
// the projection and a pass of its own; as here 113; 8192 x 6144 x 4096: 315 against 315 + 69).  So the tokens go through shared memory (per head 16 rows of 256 bytes; the 16-byte piece c of row r
// lies at c ^ (r & 7)) and come back with 8 lanes a token, 8 neighbouring values of each half of the head a lane: a rotation
// then needs no other lane, and every access covers whole lines.  The angles serve both heads (the table does not fit the L1 that the
// operand ring leaves, and L2 -> SM is what binds the GEMM) and are requested before the accumulator is ready.
struct RopeAngles { float4 c[4][2], s[4][2]; int slot; };

__device__ __forceinline__ void rope_angles(RopeAngles& an, const RopeEpi& re, int row0, int M, bool rotate) {
  const int lane = threadIdx.x & 31, row = row0 + (lane & 15);
  int64_t pos = row < M ? re.positions[row] : 0;
  pos = pos < 0 ? 0 : (pos >= re.max_position ? re.max_position - 1 : pos);
  an.slot = row < M && re.k_cache != nullptr ? __ldg(re.slot_mapping + row) : -1;
  if (!rotate) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t p = __shfl_sync(0xffffffffu, static_cast<int>(pos), 4 * i + (lane >> 3));
    const float4* cs = reinterpret_cast<const float4*>(re.cos_sin + p * 128) + 2 * (lane & 7);
    an.c[i][0] = __ldg(cs); an.c[i][1] = __ldg(cs + 1); an.s[i][0] = __ldg(cs + 16); an.s[i][1] = __ldg(cs + 17);
  }
}
__device__ __forceinline__ void rope_rows(bf16* __restrict__ y, int64_t ldy, const RopeEpi& re, const RopeAngles& an, uint32_t taddr, uint8_t* stage,
                                          int row0, int M, int head0, int half) {
  const int lane = threadIdx.x & 31, l = lane & 15, j = lane & 7;
#pragma unroll 1
  for (int c = 0; c < 8; ++c) {      // 32 columns at a time; the warp's tokens are the lanes of its half
    uint32_t r[32];
    tmem_ld_32x32b_x32(taddr + c * 32, r);
    tmem_ld_wait();
    if ((lane >> 4) == half) {
#pragma unroll
      for (int e = 0; e < 4; ++e)    // bf16 qkv
        *reinterpret_cast<uint4*>(stage + (c >> 2) * 4096 + l * 256 + ((((c & 3) * 4 + e) ^ (l & 7)) * 16)) =
            make_uint4(pack_bf16x2(__uint_as_float(r[8 * e]), __uint_as_float(r[8 * e + 1])), pack_bf16x2(__uint_as_float(r[8 * e + 2]), __uint_as_float(r[8 * e + 3])),
                       pack_bf16x2(__uint_as_float(r[8 * e + 4]), __uint_as_float(r[8 * e + 5])), pack_bf16x2(__uint_as_float(r[8 * e + 6]), __uint_as_float(r[8 * e + 7])));
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const int head = head0 + h;                                               // packed row: H q heads, Hkv k heads, Hkv v heads
    const int kind = head < re.H ? 0 : (head < re.H + re.Hkv ? 1 : 2);
    const bf16* w = kind == 0 ? re.q_norm_w : (kind == 1 ? re.k_norm_w : nullptr);
    bf16* const cache = kind == 1 ? re.k_cache + (head - re.H) * re.head_stride : re.v_cache + (head - re.H - re.Hkv) * re.head_stride;
    uint4 wa = make_uint4(0, 0, 0, 0), wb = wa;
    if (w != nullptr) { wa = __ldg(reinterpret_cast<const uint4*>(w) + j); wb = __ldg(reinterpret_cast<const uint4*>(w) + 8 + j); }
    const uint32_t w1[4] = {wa.x, wa.y, wa.z, wa.w}, w2[4] = {wb.x, wb.y, wb.z, wb.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = 4 * i + (lane >> 3), row = row0 + rr;
      const uint8_t* src = stage + h * 4096 + rr * 256;
      const uint4 a4 = *reinterpret_cast<const uint4*>(src + ((j ^ (rr & 7)) * 16)), b4 = *reinterpret_cast<const uint4*>(src + (((8 + j) ^ (rr & 7)) * 16));
      uint32_t a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
      const int slot = __shfl_sync(0xffffffffu, an.slot, rr);
      if (kind < 2) {
        if (w != nullptr) {
          float ss[2] = {0.f, 0.f};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ss[0] = fmaf(bf16_lo(a[e]), bf16_lo(a[e]), fmaf(bf16_hi(a[e]), bf16_hi(a[e]), ss[0]));
            ss[1] = fmaf(bf16_lo(b[e]), bf16_lo(b[e]), fmaf(bf16_hi(b[e]), bf16_hi(b[e]), ss[1]));
          }
          float t = ss[0] + ss[1];
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          const float inv = 1.0f / sqrtf(t * (1.0f / 128.0f) + re.eps);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            a[e] = pack_bf16x2(bf16_lo(a[e]) * inv * bf16_lo(w1[e]), bf16_hi(a[e]) * inv * bf16_hi(w1[e]));
            b[e] = pack_bf16x2(bf16_lo(b[e]) * inv * bf16_lo(w2[e]), bf16_hi(b[e]) * inv * bf16_hi(w2[e]));
          }
        }
        const float c[8] = {an.c[i][0].x, an.c[i][0].y, an.c[i][0].z, an.c[i][0].w, an.c[i][1].x, an.c[i][1].y, an.c[i][1].z, an.c[i][1].w};
        const float s[8] = {an.s[i][0].x, an.s[i][0].y, an.s[i][0].z, an.s[i][0].w, an.s[i][1].x, an.s[i][1].y, an.s[i][1].z, an.s[i][1].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x0 = bf16_lo(a[e]), x1 = bf16_hi(a[e]), z0 = bf16_lo(b[e]), z1 = bf16_hi(b[e]);
          a[e] = pack_bf16x2(x0 * c[2 * e] - z0 * s[2 * e], x1 * c[2 * e + 1] - z1 * s[2 * e + 1]);
          b[e] = pack_bf16x2(z0 * c[2 * e] + x0 * s[2 * e], z1 * c[2 * e + 1] + x1 * s[2 * e + 1]);
        }
      }
      if (row < M) {
        auto store = [&](bf16* dst) {
          reinterpret_cast<uint4*>(dst)[j] = make_uint4(a[0], a[1], a[2], a[3]);
          reinterpret_cast<uint4*>(dst)[8 + j] = make_uint4(b[0], b[1], b[2], b[3]);
        };
        store(y + row * ldy + head * 128);
        if (kind >= 1 && slot >= 0) {
          const int blk = slot / re.block_size;
          store(cache + blk * re.blk_stride + (slot - blk * re.block_size) * re.tok_stride);
        }
      }
    }
  }
  __syncwarp();
}

// GATE != kGateNone: w is the packed [gate (N rows) | up (N rows)] matrix of MergedColumnParallelLinear (linear.rs:421-433);
// the leader CTA stages BN/2 gate rows, its peer the matching BN/2 up rows, so accumulator columns [0, BN/2) are gate and
// [BN/2, BN) are up for the same BN/2 output features, and the epilogue writes y[:, n_tile*BN/2 + c] = silu(gate)*up
// (SiluAndMul::forward, activation.rs:46-63; or another gate of gated_pair) without the [M, 2N] intermediate ever reaching HBM.  N = output features.
// ROPE: the qkv epilogue that RopeEpi describes, on the two heads of a tile; see rope_rows.
// GROUPED: the experts' product.  tile_group names the weight block (group_rows rows of w) of each 128-row tile, in device memory; a pair
// takes two neighbouring tiles of one group, the last of an odd run alone (its second half multiplies the next group's rows and stores
// nothing).  Every CTA makes the list of pairs itself.  n-tiles run fastest: the pairs at work then share a dozen groups' weights and x
// comes from HBM once, where the other order reads it again for every n-tile (8192 tokens x 6 of 64 experts, 2048 -> 1408: single CTAs 356 us
// with m-tiles fastest, 297 with n-tiles, pairs 259; 1408 -> 2048: 341, 286, 245).  Bound by the L2 -> SM feed like the plain product, and by
// the rows that fill up tiles and pairs.
template <int BN, typename OutT, int GATE, bool ROPE, bool GROUPED, bool ADD>
__global__ void __launch_bounds__(gemm2_threads<GATE, ROPE, ADD>(), 1)
gemm_tcgen05_2cta_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                         OutT* __restrict__ y, int M, int N, int K, int64_t ldy, int num_m_tiles, int num_tiles, float glu_limit,
                         const RopeEpi re, const int32_t* __restrict__ tile_group, int group_rows, bool relu2, int panel) {
  using C = Gemm2Cfg<BN>;
  constexpr int STAGES = C::kStages - (ROPE ? 1 : 0);   // (the qkv epilogue takes a stage's room)
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sA = smem_base;
  const uint32_t sB = smem_base + STAGES * C::kABytes;
  const uint32_t bars = smem_base + STAGES * C::kStageBytes + (ROPE ? 8 * kRopeStage : 0);
  auto full_bar = [&](int s) { return bars + s * 8; };
  auto empty_bar = [&](int s) { return bars + (STAGES + s) * 8; };
  auto tfull_bar = [&](int a) { return bars + (2 * STAGES + a) * 8; };
  auto tempty_bar = [&](int a) { return bars + (2 * STAGES + 2 + a) * 8; };
  const uint32_t tmem_slot = bars + (2 * STAGES + 4) * 8;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform)
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int num_kb = K / C::BK;
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_w);
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);   // leader: its producer's arrive.expect_tx (+ both CTAs' TMA bytes)
      mbar_init(empty_bar(s), 1);  // each CTA: multicast tcgen05.commit from the leader
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);     // each CTA: multicast commit
      mbar_init(tempty_bar(a), 64 * gemm2_epilogue_warps<GATE, ROPE, ADD>());  // leader: the epilogue threads of both CTAs
    }
    fence_barrier_init();
  }
  if (warp == 2) tmem_alloc_cg2<C::kTmemCols>(tmem_slot);
  tc_fence_before();
  cluster_sync_all();  // barriers of BOTH CTAs are initialised before any remote signal can arrive
  pdl_launch_dependents();   // (behind the allocation)
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  [[maybe_unused]] uint32_t* const pairs = tmem_slot_ptr + 4;   // GROUPED: m-tile | second half live << 12 | group << 13
  if constexpr (GROUPED) {
    // num_m_tiles: 128-row tiles (at most kMaxGroupedTiles); num_tiles: n-tiles
    pdl_wait();
    for (int i = threadIdx.x; i < num_m_tiles; i += blockDim.x) pairs[i] = static_cast<uint32_t>(tile_group[i]);
    __syncthreads();
    if (warp == 3) {
      int count = 0, start = 0, prev = -1;                      // (in place: a pair's entry never lies behind the tile that it starts at)
      for (int i0 = 0; i0 < num_m_tiles; i0 += 32) {
        const int i = i0 + lane;
        const int g = i < num_m_tiles ? static_cast<int>(pairs[i]) : -1, next = i + 1 < num_m_tiles ? static_cast<int>(pairs[i + 1]) : -1;
        const int up = __shfl_up_sync(0xffffffffu, g, 1);
        const uint32_t breaks = __ballot_sync(0xffffffffu, g != (lane == 0 ? prev : up)) & (0xffffffffu >> (31 - lane));
        const int run = breaks ? i0 + 31 - __clz(breaks) : start;
        const bool first = g >= 0 && ((i - run) & 1) == 0;
        const uint32_t firsts = __ballot_sync(0xffffffffu, first);
        if (first) pairs[count + __popc(firsts & ((1u << lane) - 1))] = static_cast<uint32_t>(i) | (next == g ? 1u << 12 : 0u) | static_cast<uint32_t>(g) << 13;
        count += __popc(firsts);
        start = __shfl_sync(0xffffffffu, run, 31);
        prev = __shfl_sync(0xffffffffu, g, 31);
        __syncwarp();
      }
      if (lane == 0) tmem_slot_ptr[1] = static_cast<uint32_t>(count);
    }
    __syncthreads();
    num_m_tiles = num_tiles;                                    // (now the divisor of a tile's number)
    num_tiles = __reduce_max_sync(0xffffffffu, static_cast<int>(tmem_slot_ptr[1])) * num_m_tiles;
  }
  // a tile's first row for this CTA, its n-tile, the first row that holds nothing of it, and its weight block's first row
  struct Where { int row0, n_tile, m_end, w0; };
  auto where = [&](int tile) {
    if constexpr (GROUPED) {
      const uint32_t p = pairs[tile / num_m_tiles];
      const int row0 = static_cast<int>(p & 0xfffu) * C::BM_CTA;
      return Where{row0 + static_cast<int>(rank) * C::BM_CTA, tile % num_m_tiles, row0 + (p & 0x1000u ? C::BM : C::BM_CTA), static_cast<int>(p >> 13) * group_rows};
    } else {
      if (panel == 1) return Where{tile % num_m_tiles * C::BM + static_cast<int>(rank) * C::BM_CTA, tile / num_m_tiles, M, 0};
      const int p = tile / (panel * num_m_tiles), n0 = p * panel, in = tile - n0 * num_m_tiles, wide = min(panel, num_tiles / num_m_tiles - n0);
      return Where{in / wide * C::BM + static_cast<int>(rank) * C::BM_CTA, n0 + in % wide, M, 0};
    }
  };

  if (warp == 0 && lane == 0) {
    // ===== TMA producer (both CTAs) =====
    pdl_wait();
    int stage = 0;
    uint32_t phase = 0;
    for (int tile = cluster_id; tile < num_tiles; tile += num_clusters) {
      const Where at = where(tile);
      for (int kb = 0; kb < num_kb; ++kb) {
        mbar_wait(empty_bar(stage), phase ^ 1);
        if (leader) mbar_expect_tx(full_bar(stage), 2 * C::kStageBytes);
        tma_load_2d_cg2(sA + stage * C::kABytes, &tmap_x, full_bar(stage), kb * C::BK, at.row0);
        tma_load_2d_cg2(sB + stage * C::kBBytes, &tmap_w, full_bar(stage), kb * C::BK,
                        at.w0 + (GATE != kGateNone ? static_cast<int>(rank) * N + at.n_tile * (BN / 2) : at.n_tile * BN + static_cast<int>(rank) * (BN / 2)));
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1 && leader) {
    // ===== MMA issuer (leader CTA): the whole warp walks the tiles, one lane issues =====
    const uint32_t el = elect_one() ? 1u : 0u, tm = __reduce_max_sync(0xffffffffu, tmem_base);   // (read from shared memory: uniform from here on)
    constexpr uint32_t idesc = umma_idesc_bf16(C::BM, BN, 0, 0);
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    pdl_wait();  // keep the wait for the predecessor out of the bounded mbarrier waits
    for (int tile = cluster_id; tile < num_tiles; tile += num_clusters) {
      mbar_wait(tempty_bar(acc), acc_phase ^ 1);
      tc_fence_after();
      const uint32_t tmem_d = tm + acc * BN;
      for (int kb = 0; kb < num_kb; ++kb) {
        mbar_wait(full_bar(stage), phase);
        tc_fence_after();
        const uint32_t a0 = sA + stage * C::kABytes, b0 = sB + stage * C::kBBytes;
#pragma unroll
        for (int k = 0; k < C::BK / 16; ++k) {
          const uint32_t adesc = umma_desc_lo(a0, 16) + k * 2;
          const uint32_t bdesc = umma_desc_lo(b0, 16) + k * 2;
          umma_bf16_ss_cg2_warp(tmem_d, adesc, bdesc, idesc, (kb | k) != 0 ? 1u : 0u, el);
        }
        umma_commit_cg2_warp(empty_bar(stage), 0b11, el);
        if (kb == num_kb - 1) umma_commit_cg2_warp(tfull_bar(acc), 0b11, el);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  } else if (warp >= 4) {
    // ===== epilogue (both CTAs): own 128 TMEM lanes -> global =====
    pdl_wait();
    const int q = warp & 3;
    [[maybe_unused]] const bool wide = rows_on_32(y, ldy);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = cluster_id; tile < num_tiles; tile += num_clusters) {
      const Where at = where(tile);
      const int n_tile = at.n_tile;
      [[maybe_unused]] RopeAngles angles;
      [[maybe_unused]] const int rope_row0 = at.row0 + q * 32 + (warp < 8 ? 0 : 16);
      if constexpr (ROPE) {
        static_assert(!ROPE || BN == 256, "two heads a tile");
        rope_angles(angles, re, rope_row0, M, n_tile * 2 < re.H + re.Hkv);
      }
      mbar_wait(tfull_bar(acc), acc_phase);
      tc_fence_after();
      const int row = at.row0 + q * 32 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
      if constexpr (ROPE) {
        rope_rows(y, ldy, re, angles, taddr, smem_raw + (smem_base - smem_u32(smem_raw)) + STAGES * C::kStageBytes + (warp - 4) * kRopeStage, rope_row0, M,
                  n_tile * 2, warp < 8 ? 0 : 1);
      } else if constexpr (GATE != kGateNone) {
#pragma unroll 1
        for (int c = warp < 8 ? 0 : BN / 128; c < (warp < 8 ? BN / 128 : BN / 64); ++c) {
          uint32_t g[32], u[32];
          tmem_ld_32x32b_x32(taddr + c * 32, g);
          tmem_ld_32x32b_x32(taddr + BN / 2 + c * 32, u);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            // same rounding points as the unfused path: gate_up is a bf16 tensor, silu(gate) is a bf16 tensor
            const uint32_t gb = pack_bf16x2(__uint_as_float(g[e]), __uint_as_float(g[e + 1]));
            const uint32_t ub = pack_bf16x2(__uint_as_float(u[e]), __uint_as_float(u[e + 1]));
            const float2 p = gated_pair<GATE>(gb, ub, glu_limit);
            g[e] = __float_as_uint(p.x);
            g[e + 1] = __float_as_uint(p.y);
          }
          const int col0 = n_tile * (BN / 2) + c * 32;
          if (row < at.m_end && col0 < N) store_row32<OutT>(y + row * ldy + col0, g, col0, N, wide);
        }
      } else {
        // add: y holds the residual stream, and the product's bf16 values are added to it in place.  A chunk's old values are requested
        // while the chunk before it is on its way.
        [[maybe_unused]] uint4 old[4];
        auto request = [&](int c) {
          const int col0 = n_tile * BN + c * 32;
          const bf16* src = reinterpret_cast<const bf16*>(y) + row * ldy + col0;
#pragma unroll
          for (int j = 0; j < 4; ++j) old[j] = row < at.m_end && col0 + j * 8 < N ? *reinterpret_cast<const uint4*>(src + j * 8) : make_uint4(0, 0, 0, 0);
        };
        const int c0 = ADD && warp >= 8 ? BN / 64 : 0, c1 = ADD && warp < 8 ? BN / 64 : BN / 32;
        if constexpr (ADD) request(c0);
#pragma unroll 1
        for (int c = c0; c < c1; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + c * 32, r);
          tmem_ld_wait();
          if constexpr (GROUPED) {
            if (relu2) relu2_row32(r);
          }
          if constexpr (ADD) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t o[4] = {old[j].x, old[j].y, old[j].z, old[j].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const uint32_t b = pack_bf16x2(__uint_as_float(r[8 * j + 2 * e]), __uint_as_float(r[8 * j + 2 * e + 1]));
                r[8 * j + 2 * e] = __float_as_uint(bf16_lo(b) + bf16_lo(o[e]));
                r[8 * j + 2 * e + 1] = __float_as_uint(bf16_hi(b) + bf16_hi(o[e]));
              }
            }
            if (c + 1 < c1) request(c + 1);
          }
          const int col0 = n_tile * BN + c * 32;
          if (row < at.m_end && col0 < N) store_row32<OutT>(y + row * ldy + col0, r, col0, N, wide);
        }
      }
      tc_fence_before();
      mbar_arrive_cluster(tempty_bar(acc), 0);  // tell the leader this CTA's half of the accumulator is drained
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  tc_fence_before();
  cluster_sync_all();  // neither CTA may exit (or free TMEM) while its peer can still touch its smem / barriers
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_cg2<C::kTmemCols>(tmem_base);
  }
}

// The order of the tiles: panels of this many n-tiles, n fastest within a panel.  Up to K = 2048 one n-tile after the other (a w tile is read
// once, x stays in L2): 8192 x 8192 x 2048 (gated) 401 us, 407 in panels of 12.  Longer rows of x leave L2 again before the next n-tile reads
// them; in panels of 12 a wave of 74 tiles reads 12 tiles of w and 6 of x.  Measured (us, one n-tile after the other -> in panels of 12):
// 8192 x 4096 x 12288 568 -> 527, 8192 x 6144 x 4096 281 -> 262, 8192 x 2048 x 8192 202 -> 184, 12400 x 1024 x 3072 59 -> 55.
// Where a few m-tiles are no more than a wave anyway, panels of 2 do best: 3000 x 24576 x 4096 497 -> 461 (12: 470),
// 1500 x 24576 x 4096 (gated) 247 -> 230 (237), 1500 x 4096 x 12288 161 -> 160 (161).  From 16 to 23 m-tiles it depends on the length of the rows (one n-tile
// after the other, panels of 2, of 12): 4400 x 6144 x 4096 142, 140, 144, 4400 x 12288 x 4096 (gated) 570, 560, 577; 4400 x 2048 x 8192 101.5, 100.5, 97.9, 5000 x 4096 x 12288
// 357, 351, 349.
static int panel_tiles(int num_m_tiles, int k) { return k < 3072 ? 1 : (num_m_tiles >= 24 || (num_m_tiles >= 16 && k >= 8192) ? 12 : 2); }

constexpr int kMaxGroupedTiles = 4096;   // (the list's entries hold 12 bits of tile and 19 of group)

template <int BN, typename OutT, int GATE = kGateNone, bool ROPE = false, bool GROUPED = false, bool ADD = false>
static int launch_gemm2(const CUtensorMap& tx, const CUtensorMap& tw, void* y, int M, int N, int K, int64_t ldy,
                        cudaStream_t st, float glu_limit = 0.f, const RopeEpi& re = RopeEpi{}, const int32_t* tile_group = nullptr, int group_rows = 0, bool relu2 = false) {
  using C = Gemm2Cfg<BN>;
  auto kern = gemm_tcgen05_2cta_kernel<BN, OutT, GATE, ROPE, GROUPED, ADD>;
  constexpr int smem_max = C::kSmemBytes + (ROPE ? 8 * kRopeStage - C::kStageBytes : 0) + (GROUPED ? 4 * kMaxGroupedTiles : 0);
  static_assert(smem_max <= 227 * 1024, "");
  NVLLM_SMEM_ATTR_ONCE(kern, smem_max);
  const int num_m_tiles = GROUPED ? M / C::BM_CTA : (M + C::BM - 1) / C::BM;
  const int smem = smem_max - (GROUPED ? 4 * (kMaxGroupedTiles - num_m_tiles) : 0);
  const int num_n_tiles = GATE != kGateNone ? (N + BN / 2 - 1) / (BN / 2) : (N + BN - 1) / BN;
  const int num_tiles = num_m_tiles * num_n_tiles;
  const int max_clusters = sm_count() / 2;
  const int clusters = num_tiles < max_clusters ? num_tiles : max_clusters;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(gemm2_threads<GATE, ROPE, ADD>());
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  NVLLM_CUDA(cudaLaunchKernelEx(&cfg, kern, tx, tw, static_cast<OutT*>(y), M, N, K, ldy, num_m_tiles, GROUPED ? num_n_tiles : num_tiles, glu_limit, re, tile_group,
                                group_rows, relu2, std::min(num_n_tiles, panel_tiles(num_m_tiles, K))));
  return 0;
}

// Tile width for the CTA-pair kernel: small problems take the narrowest tile that still fits in one wave of 74
// clusters; otherwise the widest tile whose last wave is reasonably full.
static int pick_bn_2cta(int M, int N) {
  const int clusters = sm_count() / 2;
  const long mt = (M + 255) / 256;
  const int small[3] = {64, 128, 256};
  for (int i = 0; i < 3; ++i)
    if (mt * ((N + small[i] - 1) / small[i]) <= clusters) return small[i];
  const int wide[3] = {256, 128, 64};
  int best = 256;
  double best_score = -1.0;
  for (int i = 0; i < 3; ++i) {
    const long tiles = mt * ((N + wide[i] - 1) / wide[i]);
    const long waves = (tiles + clusters - 1) / clusters;
    const double eff = static_cast<double>(tiles) / static_cast<double>(waves * clusters);
    const double reuse = wide[i] == 256 ? 1.0 : (wide[i] == 128 ? 0.8 : 0.6);  // MACs per byte fetched
    if (eff * reuse > best_score) { best_score = eff * reuse; best = wide[i]; }
  }
  return best;
}

int gemm_2cta_dispatch(void* y, const void* x, const void* w, int m, int n, int k, int64_t ldx, int64_t ldw,
                       int64_t ldy, int out_dtype, cudaStream_t st, bool add) {
  const int forced = knobs().gemm_bn;
  const int bn = (forced == 64 || forced == 128 || forced == 256) ? forced : pick_bn_2cta(m, n);
  CUtensorMap tx, tw;
  if (int rc = make_tmap_bf16_2d(&tx, x, m, k, ldx, 128)) return rc;
  if (int rc = make_tmap_bf16_2d(&tw, w, n, k, ldw, bn / 2)) return rc;
#define NVLLM_G2(BNV)                                                                            \
  case BNV:                                                                                      \
    if (add) return launch_gemm2<BNV, bf16, kGateNone, false, false, true>(tx, tw, y, m, n, k, ldy, st); \
    return out_dtype == NVLLM_BF16 ? launch_gemm2<BNV, bf16>(tx, tw, y, m, n, k, ldy, st)        \
                                   : launch_gemm2<BNV, float>(tx, tw, y, m, n, k, ldy, st)
  switch (bn) {
    NVLLM_G2(256);
    NVLLM_G2(128);
    default:
      NVLLM_G2(64);
  }
#undef NVLLM_G2
}

// qkv = x . Wqkv^T with the qkv epilogue; n = 128 x heads, a multiple of 256.
int gemm_qkv_2cta_dispatch(void* qkv, const void* x, const void* w, int m, int n, int k, int64_t ldx, int64_t ldw, const RopeEpi& re, cudaStream_t st) {
  CUtensorMap tx, tw;
  if (int rc = make_tmap_bf16_2d(&tx, x, m, k, ldx, 128)) return rc;
  if (int rc = make_tmap_bf16_2d(&tw, w, n, k, ldw, 128)) return rc;
  return launch_gemm2<256, bf16, kGateNone, true>(tx, tw, qkv, m, n, k, n, st, 0.f, re);
}

// The experts' product of nvllm_gemm_bf16_grouped on CTA pairs.  A group of one tile wastes half a pair, but a tile that no group uses costs
// nothing: 64 experts' tiles of 2048 -> 1408 take, on single CTAs and on pairs, 76 and 89 us at 67 tiles' room, 86 and 88 at 76, 103 and 88 at
// 112; 8 experts, 2048 -> 2048, 18.5 and 18.3 at 10, 20 and 18 at 16.  Hence a quarter more tiles than groups.
bool grouped_2cta(int max_rows, int n, int groups) {
  const int tiles = max_rows / 128;
  return knobs().gemm_2cta != 0 && n >= 256 && groups <= (1 << 19) && tiles <= kMaxGroupedTiles && 4 * static_cast<int64_t>(tiles) >= 5 * static_cast<int64_t>(groups);
}
int gemm_grouped_2cta_dispatch(void* y, const void* x, const void* w, int max_rows, int n, int k, int groups, int64_t ldx, int64_t ldw, int64_t ldy,
                               const int32_t* tile_group, bool relu2, cudaStream_t st) {
  CUtensorMap tx, tw;
  if (int rc = make_tmap_bf16_2d(&tx, x, max_rows, k, ldx, 128)) return rc;
  if (int rc = make_tmap_bf16_2d(&tw, w, static_cast<int64_t>(groups) * n, k, ldw, 128)) return rc;
  return launch_gemm2<256, bf16, kGateNone, false, true>(tx, tw, y, max_rows, n, k, ldy, st, 0.f, RopeEpi{}, tile_group, n, relu2);
}

// y[M, inter] = silu(x . Wgate^T) * (x . Wup^T) (or another gate) with w = [Wgate | Wup] packed row-wise ([2*inter, K]).
int gemm_silu_2cta_dispatch(void* y, const void* x, const void* w, int m, int inter, int k, int64_t ldx, int64_t ldw,
                            int64_t ldy, int gate, float glu_limit, cudaStream_t st) {
  // accumulator tile BN covers BN/2 output features; reuse the tile heuristic on the 2*inter accumulator columns
  const int bn = pick_bn_2cta(m, 2 * inter);
  NVLLM_CHECK_ARG(inter % (bn / 2) == 0 || true, NVLLM_ERR_ARG, "gemm_silu: inter");
  CUtensorMap tx, tw;
  if (int rc = make_tmap_bf16_2d(&tx, x, m, k, ldx, 128)) return rc;
  if (int rc = make_tmap_bf16_2d(&tw, w, 2 * static_cast<int64_t>(inter), k, ldw, bn / 2)) return rc;
#define NVLLM_G2G(BNV)                                                                                                    \
  case BNV:                                                                                                               \
    return gate == kGateClamped ? launch_gemm2<BNV, bf16, kGateClamped>(tx, tw, y, m, inter, k, ldy, st, glu_limit)       \
           : gate == kGateGelu  ? launch_gemm2<BNV, bf16, kGateGelu>(tx, tw, y, m, inter, k, ldy, st)                     \
                                : launch_gemm2<BNV, bf16, kGateSilu>(tx, tw, y, m, inter, k, ldy, st)
  switch (bn) {
    NVLLM_G2G(256);
    NVLLM_G2G(128);
    default:
      NVLLM_G2G(64);
  }
#undef NVLLM_G2G
}

}  // namespace nvllm
