// tc.cuh — Blackwell tensor-core plumbing used by the GEMM and prefill-attention kernels:
// mbarrier, TMA (cp.async.bulk.tensor), tcgen05 (alloc / mma / commit / ld / fences) and the UMMA
// shared-memory + instruction descriptors.  Hand-written inline PTX for sm_100a; bit layouts follow
// the PTX ISA "tcgen05 matrix descriptors" (same fields CUTLASS' cute/arch/mma_sm100_desc.hpp names).
#pragma once

#include <cuda.h>  // CUtensorMap

#include "common.cuh"

namespace nvllm {

// ---- host: TMA descriptor for a row-major bf16 matrix [rows, cols] with leading dimension ld -------
// box = box_rows x 64 columns (128 bytes), SWIZZLE_128B, out-of-bounds elements read as zero.
int make_tmap_bf16_2d(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld,
                      int box_rows, int box_cols = 64);  // tc_host.cu
int make_tmap_bf16_nd(CUtensorMap* map, const void* base, int rank, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box);  // tc_host.cu

// relu(v)^2 of 32 accumulator values, v rounded to bf16 first (the product as a tensor of its own would be).
__device__ __forceinline__ void relu2_row32(uint32_t (&r)[32]) {
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    const float v = fmaxf(__bfloat162float(__float2bfloat16_rn(__uint_as_float(r[e]))), 0.f);
    r[e] = __float_as_uint(v * v);
  }
}

// ---- qkv epilogue of the GEMMs ---------------------------------------------------------------------
// What Qwen3Attention::forward does between qkv_proj and Attention::forward (qwen3.rs:219-229) plus Attention::store_kv_cache
// (attention.rs:150-174), on the accumulators of x . Wqkv^T: round to bf16 (the qkv tensor), per-head RMSNorm (q/k), bf16, half-split
// RoPE from the f32 table, bf16; q/k/v rows go to the qkv buffer and k/v additionally into the paged cache at slot_mapping[token] —
// same rounding points as the stand-alone kernel.
struct RopeEpi {
  const int64_t* positions;
  const float* cos_sin;     // [max_position, 128]
  const bf16* q_norm_w;     // may be NULL (no qk-norm)
  const bf16* k_norm_w;
  bf16* k_cache;
  bf16* v_cache;
  const int32_t* slot_mapping;
  int H, Hkv, max_position, block_size;
  int64_t blk_stride, tok_stride, head_stride;
  float eps;
};


#ifdef __CUDACC__

// ---- mbarrier ------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same without suspending the thread (try_wait may hold it for microseconds): for a thread that polls several barriers.
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: a pipeline bug must surface as a trap (clean CUDA error), never as a hung GPU.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > 4000000000ll) {  // ~2 s at 2 GHz
      printf("nvllm: mbarrier timeout (block %d,%d thread %d bar 0x%x parity %u)\n", blockIdx.x,
             blockIdx.y, threadIdx.x, bar, parity);
      __trap();
    }
  }
}

// ---- TMA -----------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];\n" ::"l"(m) : "memory");
}
// 2-D tile load: coordinates are (c0 = innermost/column index, c1 = row index), in elements.
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::"r"(smem_dst),
      "l"(m), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
// Loads (tiles of 3 and 5 dimensions) and the bytes to expect, as predicated instructions of a whole converged warp (see umma_bf16_ss_warp).
__device__ __forceinline__ void mbar_expect_tx_warp(uint32_t bar, uint32_t bytes, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}\n" ::"r"(bar), "r"(bytes), "r"(elected)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_warp(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}\n" ::"r"(smem_dst),
      "l"(m), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(elected)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d_warp(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2, int c3, int c4,
                                                 uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %8, 0;\n\t"
      "@q cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];\n\t}\n" ::"r"(smem_dst),
      "l"(m), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(elected)
      : "memory");
}

// ---- tcgen05 ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Whole warp; writes the TMEM base address to *smem_out.  ncols: power of two in [32, 512].
template <int NCOLS>
__device__ __forceinline__ void tmem_alloc(uint32_t smem_out) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_out), "n"(NCOLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
template <int NCOLS>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "n"(NCOLS) : "memory");
}

// D[tmem] (+)= A[smem desc] . B[smem desc], accumulate == 0 overwrites D; _ts: A (M = 128 lanes x K, 16-bit elements packed two per 32-bit
// column, K-major) is read straight from tensor memory, for P of the attention kernels; commit: arrives (count 1) on `bar` once every
// MMA that this thread issued before has completed.
// These are predicated instructions of a whole converged warp: `elected` is 1 in the one lane that issues (elect_one(), always the same
// lane).  Addresses and descriptors are then computed once per warp in uniform registers, where the instruction takes them; under an
// `if (lane == 0)` every MMA first moves its own, and a thread issues one in about 130 clocks, twice what an M128 N128 K16 one runs for.
// Descriptors come as their lower words (umma_desc_lo); the upper one is the same for all SWIZZLE_128B tiles here.  Before and after, in
// turn on one GPU: 8192 x 4096 x 12288 672 and 583 us, 8192 x 6144 x 4096 322 and 286, 13420 x 1024 x 2048 42.3 and 39.9, 256 x 4096 x 1024
// 10.6 and 8.1, 64 x 2048 x 8192 15.2 and 11.2; latent attention of 8 x 1024 tokens, 16 heads 472 and 390.
// Shared-memory matrix descriptor (64-bit): start address [0,14) >>4, LBO [16,30) >>4, SBO [32,46) >>4,
// version [46,48) = 1 on sm_100, base offset [49,52) = 0 (tiles are 1024-byte aligned), layout [61,64):
// 2 = SWIZZLE_128B.
//   K-major, SW128 (rows of 64 bf16 = 128 B, as TMA writes them): SBO = 8 rows * 128 B = 1024, LBO unused.
//   MN-major, SW128 (rows = k index, 64 contiguous MN elements per row): SBO = 1024 (next 8 k),
//   LBO = byte distance between consecutive 64-element MN groups.
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO 1024, version 1, SWIZZLE_128B
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3FFFFu) >> 4) | (lbo_bytes >> 4) << 16;
}
__device__ __forceinline__ void umma_bf16_ss_warp(uint32_t tmem_d, uint32_t adesc_lo, uint32_t bdesc_lo, uint32_t idesc, uint32_t accumulate,
                                                  uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "mov.b64 a, {%1, %6};\n\t"
      "mov.b64 b, {%2, %6};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}\n" ::"r"(tmem_d),
      "r"(adesc_lo), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"(elected), "r"(kDescHi)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_ts_warp(uint32_t tmem_d, uint32_t tmem_a, uint32_t bdesc_lo, uint32_t idesc, uint32_t accumulate,
                                                  uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "mov.b64 b, {%2, %6};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n\t}\n" ::"r"(tmem_d),
      "r"(tmem_a), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"(elected), "r"(kDescHi)
      : "memory");
}
__device__ __forceinline__ void umma_commit_warp(uint32_t bar, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(bar), "r"(elected)
      : "memory");
}
// TMEM -> registers: this warp's 32 lanes x 32 consecutive fp32 columns (thread i <- lane base+i).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// The same wait, tied to the registers of one load: no use of them can be moved ahead of it while a later load is in flight.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                 "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
}
// registers -> TMEM (same shape as the load above).
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
      "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// ---- CTA-pair (cta_group::2) variants ----------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Arrive (count 1) on the mbarrier at the same offset in CTA `target_cta` of the cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t local_bar, uint32_t target_cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local_bar), "r"(target_cta));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(remote) : "memory");
}
// 2-D tile load issued by either CTA of a pair into ITS OWN shared memory; the transaction bytes complete on the
// barrier at the same offset in the pair's even (leader) CTA (peer bit of the shared::cluster address cleared).
__device__ __forceinline__ void tma_load_2d_cg2(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::"r"(smem_dst),
      "l"(m), "r"(bar & 0xFEFFFFFFu), "r"(c0), "r"(c1)
      : "memory");
}
template <int NCOLS>
__device__ __forceinline__ void tmem_alloc_cg2(uint32_t smem_out) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_out), "n"(NCOLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
}
template <int NCOLS>
__device__ __forceinline__ void tmem_dealloc_cg2(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "n"(NCOLS) : "memory");
}
// D[tmem of both CTAs, 256 rows] (+)= A[128 rows from each CTA] . B[N/2 rows from each CTA]; leader CTA only.
__device__ __forceinline__ void umma_bf16_ss_cg2_warp(uint32_t tmem_d, uint32_t adesc_lo, uint32_t bdesc_lo, uint32_t idesc,
                                                      uint32_t accumulate, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "mov.b64 a, {%1, %6};\n\t"
      "mov.b64 b, {%2, %6};\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}\n" ::"r"(tmem_d),
      "r"(adesc_lo), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"(elected), "r"(kDescHi)
      : "memory");
}
// Arrives on the barrier at this offset in every CTA of `cta_mask` once the issued cta_group::2 MMAs have completed.
__device__ __forceinline__ void umma_commit_cg2_warp(uint32_t bar, uint16_t cta_mask, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}\n" ::"r"(bar),
      "h"(cta_mask), "r"(elected)
      : "memory");
}
// ---- descriptors -----------------------------------------------------------------------------------
// Instruction descriptor for kind::f16, bf16 x bf16 -> f32: c_format[4,6)=1, a_format[7,10)=1,
// b_format[10,13)=1, a_major[15], b_major[16] (0 = K-major, 1 = MN-major), N>>3 [17,23), M>>4 [24,29).
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, int a_mn_major, int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a_mn_major) << 15) |
         (static_cast<uint32_t>(b_mn_major) << 16) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(pred));
  return pred != 0;
}

// 32 accumulator columns of a lane's row; wide: rows_on_32.  Products of CTA pairs by 16 and by 32 bytes (us): 8192 x 10304 x 2048 f32 297 and
// 256, 8192 x 8192 x 2048 f32 236 and 210, 8192 x 2048 x 2048 f32 67 and 63, 12400 x 4096 x 1024 bf16 97 and 84, gated 12400 x 3072 x 1024 125 and
// 120; from 4096 k-values or below a wave of tiles on the same.  Other rows have a branch of their own: as the second half of one per 32 bytes, and with the panels'
// divisions where there are none, products of 1500 to 6000 x 2056 x 2048 took 1 to 1.5 % longer.
template <typename OutT>
__device__ __forceinline__ void store_row32(OutT* dst, const uint32_t (&r)[32], int col0, int n, bool wide) {
  constexpr int kPer = 32 / sizeof(OutT);
  if (!wide) {
#pragma unroll
    for (int j = 0; j < 64 / kPer; ++j) {
      if (col0 + j * kPer / 2 < n) {
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if constexpr (sizeof(OutT) == 2) v[e] = pack_bf16x2(__uint_as_float(r[8 * j + 2 * e]), __uint_as_float(r[8 * j + 2 * e + 1]));
          else v[e] = r[4 * j + e];
        }
        *reinterpret_cast<uint4*>(dst + j * kPer / 2) = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 32 / kPer; ++j) {
    uint32_t v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if constexpr (sizeof(OutT) == 2) v[e] = pack_bf16x2(__uint_as_float(r[16 * j + 2 * e]), __uint_as_float(r[16 * j + 2 * e + 1]));
      else v[e] = r[8 * j + e];
    }
    if (col0 + (j + 1) * kPer <= n) st_global_32(dst + j * kPer, v);
    else {
      if (col0 + j * kPer < n) *reinterpret_cast<uint4*>(dst + j * kPer) = make_uint4(v[0], v[1], v[2], v[3]);
      if (col0 + j * kPer + kPer / 2 < n) *reinterpret_cast<uint4*>(dst + j * kPer + kPer / 2) = make_uint4(v[4], v[5], v[6], v[7]);
    }
  }
}

#endif  // __CUDACC__

}  // namespace nvllm
