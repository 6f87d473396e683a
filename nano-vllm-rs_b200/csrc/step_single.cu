// step_single.cu — all layers of a decode step of one token in one launch.
//
// Kernel by kernel (gemm_skinny.cu, paged_decode.cu) such a step is a chain of five launches a layer of 5 us each, of which reading the weights takes one:
// a kernel starts when the whole one before it has ended.  Here one CTA per SM stays for all layers, owns some rows of every matrix, and where
// its share of a layer fits its shared memory the share of layer l + 1 is copied there, one bulk copy a matrix, as soon as layer l has left
// the room, so that the weights stream whatever the CTAs wait for.  What they hand to one another, the stream, q / k / v, parts of the attention and the gated
// values, travels as 8-byte words of a value and a mark that tells layer and launch: the reader asks for the word itself until it carries
// the mark.  (With a barrier between the stages, a step took 601 us instead of 532: the release behind the stores, the wait for the counter and the read of the
// data are three trips to L2 instead of one.)
//   1  norm + q, k, v projection         every CTA norms its own copy of the token's row
//   2  attention                         item = (kv head, part of the keys): q/k norm and rotation in the CTA, a half warp per key, the first keys
//                                        asked for a stage ahead; part 0 stores the step's own key, and merges the parts
//   3  o projection + residual
//   4  norm + gate / up projection + SiLU gate
//   5  down projection + residual
// A word is written anew only behind a stage that every CTA takes part in and that needs what was read from it, so no reader can miss its mark; every CTA has
// rows of every matrix for that reason.  Rounded to bf16 in the same places as by the separate kernels, but probabilities stay f32 (logits of
// Qwen3-0.6B against 64 bits, mean of 24 steps: 0.0128 kernel by kernel, 0.0127 here).
// Bound by the chain of stages, 2 to 4 K clocks each: the trip of the words through L2, then the products' and sums' latency.
// Measured, Qwen3-0.6B (28 layers, 151936 rows of the head, us, kernel by kernel and here): behind 300 tokens 798 and 532, 1000 900 and 603, 3900 937 and 759,
// 10000 1118 and 982, 20000 1285 and 1335: contexts of more than 16384 stay with the separate kernels (the runner decides).
#include <type_traits>

#include "step_single.cuh"
#include "tc.cuh"

namespace nvllm {
namespace {

// Parts of 64 keys and more: up to 9, of which one collects the other 8 in one go, and from 2880 keys on 17 (a step behind 1000, 2500, 3900, 7000 tokens, us: 9 parts
// 605, 702, 795, 1019; 17 parts 629, 713, 759, 882).
constexpr int kFewKeys = 2880, kFewParts = 9;
constexpr int kThreads = 512, kWarps = 16, kD = 128, kParts = kStepParts, kSplitKeys = 64, kAhead = 4, kMine = 4;

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) { f[2 * e] = bf16_lo(u[e]); f[2 * e + 1] = bf16_hi(u[e]); }
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void put(uint64_t* p, uint32_t value, uint32_t mark) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(static_cast<uint64_t>(mark) << 32 | value) : "memory");
}
// N words of which the first n of the thread count, `stride` apart, once they carry the mark.  Bounded: where one does not come, the step ends with an
// error; the abort word then ends the waits of all CTAs.
struct Waiting { unsigned* abort; unsigned aborted; int* error; long long limit; };   // aborted: what the abort word is set to by this launch

__device__ __forceinline__ uint64_t look(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// true: give up
__device__ __forceinline__ bool in_vain(int& tries, long long& t0, const Waiting& wt) {
  if ((++tries & 255) != 0) return false;
  if (t0 == 0) t0 = clock64();
  if (*reinterpret_cast<volatile unsigned*>(wt.abort) == wt.aborted) return true;
  if (((clock64() - t0) >> 10) < wt.limit) return false;   // (a 64-bit argument, or a word in memory, takes registers and 3 us a step)
  *reinterpret_cast<volatile unsigned*>(wt.abort) = wt.aborted;
  *wt.error = 1;
  return true;
}
// (whole warps come here)
template <int N, bool FIRST = true>
__device__ __forceinline__ void take(uint32_t (&out)[N], const uint64_t* p, int stride, int n, uint32_t mark, const Waiting& wt) {
  long long t0 = 0;
  int tries = 0;
  // FIRST: a warp asks for its first word alone until that is there (see first_word)
  if (FIRST) {
    if ((threadIdx.x & 31) == 0 && n > 0)
      while (static_cast<uint32_t>(look(p) >> 32) != mark && !in_vain(tries, t0, wt)) {}
    __syncwarp();
  }
  bool all;
  do {
    all = true;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint64_t v = i < n ? look(p + static_cast<int64_t>(i) * stride) : static_cast<uint64_t>(mark) << 32;
      out[i] = static_cast<uint32_t>(v);
      all &= static_cast<uint32_t>(v >> 32) == mark;
    }
  } while (!all && !in_vain(tries, t0, wt));
}

// Dot products of R rows (in shared memory) with x over the 16-byte pieces [c0, c1), summed over the warp.
template <int R>
__device__ __forceinline__ void dots(float (&sum)[R], const uint4* const (&w)[R], const uint4* xs, int c0, int c1) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < R; ++r) sum[r] = 0.f;
#pragma unroll 4
  for (int c = c0 + lane; c < c1; c += 32) {
    float x[8];
    unpack8(xs[c], x);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float f[8];
      unpack8(w[r][c], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) sum[r] = fmaf(f[e], x[e], sum[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) sum[r] = warp_sum(sum[r]);
}

struct Half {   // of the attention: what a half warp has of G heads, 8 of the 128 values a lane
  float m, l, o[8];
};

template <int G>
__global__ void __launch_bounds__(kThreads, 1) step_single_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t bar_mem[4];
  __shared__ float part_sum[2 * kStepRows];
  __shared__ bf16 own[kStepRows];              // the CTA's rows of the stream
  __shared__ float ssq[kWarps];
  __shared__ uint4 head_rows[(G + 2) * 16];    // q (G heads), k and v of the step
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x, grid = gridDim.x;
  const int HD = a.heads * kD, qkv_dim = HD + 2 * a.kv_heads * kD;
  auto share = [&](int n, int& r0, int& cnt) {
    r0 = static_cast<int>(static_cast<int64_t>(cta) * n / grid);
    cnt = static_cast<int>(static_cast<int64_t>(cta + 1) * n / grid) - r0;
  };
  int q0, qn, h0, hn, f0, fn;   // first row and rows of the CTA: q/k/v and gate (and up) in pairs, o and down
  share(qkv_dim / 2, q0, qn);
  share(a.hidden, h0, hn);
  share(a.inter / 2, f0, fn);
  q0 *= 2; qn *= 2; f0 *= 2; fn *= 2;
  if (cta == a.silent) hn = 0;   // (asked once: at the rows themselves it takes 4 us a step)
  uint8_t* const w_qkv = smem;
  uint8_t* const w_o = w_qkv + a.off_o;
  uint8_t* const w_gu = w_qkv + a.off_gu;
  uint8_t* const w_down = w_qkv + a.off_down;
  uint4* const xs = reinterpret_cast<uint4*>(smem + a.off_x);
  uint32_t* const xw = reinterpret_cast<uint32_t*>(xs);
  bf16* const xb = reinterpret_cast<bf16*>(xs);
  const uint32_t bars = smem_u32(bar_mem);
  const int hp = a.hidden / 8;
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(bars + 8 * i, 1);
    fence_barrier_init();
  }
  __syncthreads();
  auto fetch = [&](int which, int layer) {
    if (layer >= a.layers) return;
    fence_proxy_async();
    const StepLayer& w = a.layer[layer];
    const uint32_t bar = bars + 8 * which, row = 2u * (which == 0 || which == 2 ? a.hidden : (which == 1 ? HD : a.inter));
    const uint32_t rows = which == 0 ? qn : (which == 2 ? fn : hn), bytes = rows * row;
    mbar_expect_tx(bar, which == 2 ? 2 * bytes : bytes);
    if (which == 0) bulk_load(smem_u32(w_qkv), w.qkv + static_cast<int64_t>(q0) * a.hidden, bytes, bar);
    if (which == 1 && rows > 0) bulk_load(smem_u32(w_o), w.o + static_cast<int64_t>(h0) * HD, bytes, bar);
    if (which == 2) {
      bulk_load(smem_u32(w_gu), w.gate_up + static_cast<int64_t>(f0) * a.hidden, bytes, bar);
      bulk_load(smem_u32(w_gu) + bytes, w.gate_up + static_cast<int64_t>(a.inter + f0) * a.hidden, bytes, bar);
    }
    if (which == 3 && rows > 0) bulk_load(smem_u32(w_down), w.down + static_cast<int64_t>(h0) * a.inter, bytes, bar);
  };
  if (tid == 0)
    for (int i = 0; i < 4; ++i) fetch(i, 0);
  const uint32_t base = *reinterpret_cast<volatile unsigned*>(a.sync);   // the marks of this launch: base + 1 .. base + 2 layers
  const Waiting wt{a.sync + 2, base + 1, a.error, a.wait};
  // One thread asks for one word, then all ask for theirs: asked for again and again by many, the words are written later (a step behind 300 tokens: 640 us
  // with all threads asking from the start, 582 with a lane of every warp, 549 with four, 532 so; copies of the words, or pauses, give nothing).
  auto first_word = [&](const uint64_t* p, uint32_t mark) {
    if (tid == 0) {
      long long t0 = 0;
      int tries = 0;
      while (static_cast<uint32_t>(look(p) >> 32) != mark && !in_vain(tries, t0, wt)) {}
    }
    __syncthreads();
  };
  // x = bf16(rms(h) * w) into shared memory; nw: the thread's values of w
  const int mine = (a.hidden - tid + kThreads - 1) / kThreads;           // values of h that the thread takes
  auto norm = [&](const bf16 (&nw)[kMine], uint32_t mark) {
    uint32_t v[kMine];
    if (mark == base) {   // before the first layer: as the embedding left it
#pragma unroll
      for (int i = 0; i < kMine; ++i) v[i] = i < mine ? __ldcg(reinterpret_cast<const unsigned short*>(a.h) + tid + i * kThreads) : 0u;
    } else {
      first_word(a.ll_h + (cta * 7) % a.hidden, mark);
      take<kMine, false>(v, a.ll_h + tid, kThreads, mine, mark, wt);
    }
    float f[kMine], s = 0.f;
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      f[i] = bf16_lo(v[i]);
      s = fmaf(f[i], f[i], s);
    }
    s = warp_sum(s);
    if (lane == 0) ssq[warp] = s;
    __syncthreads();
    s = 0.f;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) s += ssq[i];
    const float inv = 1.0f / sqrtf(s / static_cast<float>(a.hidden) + a.eps);
#pragma unroll
    for (int i = 0; i < kMine; ++i)
      if (i < mine) xb[tid + i * kThreads] = __float2bfloat16_rn(f[i] * inv * __bfloat162float(nw[i]));
    __syncthreads();
  };
  auto norm_weights = [&](bf16 (&nw)[kMine], const bf16* w) {
#pragma unroll
    for (int i = 0; i < kMine; ++i) nw[i] = i < mine ? w[tid + i * kThreads] : __float2bfloat16_rn(0.f);
  };
  // x = the 2 n values of n words
  auto gather = [&](const uint64_t* words, int n, uint32_t mark) {
    first_word(words + (cta * 7) % n, mark);
    for (int i0 = 0; i0 < n; i0 += kMine * kThreads) {
      uint32_t v[kMine];
      const int cnt = (n - i0 - tid + kThreads - 1) / kThreads;
      take<kMine, false>(v, words + i0 + tid, kThreads, cnt, mark, wt);
#pragma unroll
      for (int i = 0; i < kMine; ++i)
        if (i < cnt) xw[i0 + tid + i * kThreads] = v[i];
    }
    __syncthreads();
  };
  // h += rows of w times x: two warps a row
  auto add_rows = [&](const uint8_t* w, int k, uint32_t mark, bool last) {
    const int pieces = k / 8, cut = (pieces / 2 + 31) / 32 * 32;
    for (int it = warp; it < 2 * hn; it += kWarps) {
      const uint4* const row[1] = {reinterpret_cast<const uint4*>(w) + static_cast<int64_t>(it >> 1) * pieces};
      float s[1];
      dots<1>(s, row, xs, it & 1 ? cut : 0, it & 1 ? pieces : min(cut, pieces));
      if (lane == 0) part_sum[it] = s[0];
    }
    __syncthreads();
    if (tid < hn) {
      const bf16 v = __float2bfloat16_rn(__bfloat162float(own[tid]) + __bfloat162float(__float2bfloat16_rn(part_sum[2 * tid] + part_sum[2 * tid + 1])));
      own[tid] = v;
      put(a.ll_h + h0 + tid, __bfloat16_as_ushort(v), mark);
      if (last) a.h[h0 + tid] = v;
    }
  };
  if (tid < hn) own[tid] = a.h[h0 + tid];

  // attention: this CTA's item
  const int ctx_all = __ldg(a.ctx), ctx = max(ctx_all - 1, 0), splits = min(max((ctx_all + kSplitKeys - 1) / kSplitKeys, 1), ctx_all <= kFewKeys ? min(kFewParts, a.max_splits) : a.max_splits);
  const int kvh = cta % a.kv_heads, split = cta / a.kv_heads;
  const bool item = split < splits;
  const int per = (ctx_all + splits - 1) / splits, key0 = min(split * per, ctx_all), key1 = min(key0 + per, ctx_all);   // (key ctx: the step's own)
  const int hw = tid >> 4, hl = tid & 15;
  const int slot = __ldg(a.slots);
  float cs[8], sn[8];
  if (item) {
    int64_t pos = __ldg(a.pos);
    pos = pos < 0 ? 0 : (pos >= a.max_position ? a.max_position - 1 : pos);
    const float4* c = reinterpret_cast<const float4*>(a.cos_sin + pos * kD) + 2 * (hl & 7);
    const float4 c0 = __ldg(c), c1 = __ldg(c + 1), s0 = __ldg(c + 16), s1 = __ldg(c + 17);
    cs[0] = c0.x; cs[1] = c0.y; cs[2] = c0.z; cs[3] = c0.w; cs[4] = c1.x; cs[5] = c1.y; cs[6] = c1.z; cs[7] = c1.w;
    sn[0] = s0.x; sn[1] = s0.y; sn[2] = s0.z; sn[3] = s0.w; sn[4] = s1.x; sn[5] = s1.y; sn[6] = s1.z; sn[7] = s1.w;
  }
  // q/k norm and rotation of 8 of a head's values a lane; the pair of value d is in lane hl ^ 8
  auto rotate = [&](uint4 raw, bool norm, const uint4& nw) {
    float x[8], w[8];
    unpack8(raw, x);
    float s = 0.f;   // (norm differs between the halves of a warp, and the shuffles take whole warps)
#pragma unroll
    for (int e = 0; e < 8; ++e) s = fmaf(x[e], x[e], s);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float inv = 1.0f / sqrtf(s * (1.0f / kD) + a.eps);
    unpack8(nw, w);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = norm ? __bfloat162float(__float2bfloat16_rn(x[e] * inv * w[e])) : x[e];
    uint32_t out[4];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float other = __shfl_xor_sync(0xffffffffu, x[e], 8);
      w[e] = hl < 8 ? x[e] * cs[e] - other * sn[e] : x[e] * cs[e] + other * sn[e];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) out[e] = pack_bf16x2(w[2 * e], w[2 * e + 1]);
    return make_uint4(out[0], out[1], out[2], out[3]);
  };
  // where the keys of this half warp lie, from `first` on, one for each of the first kAhead rounds; -1: none, or the step's own
  auto key_at = [&](int first, int i) -> int64_t {
    const int key = first + hw + i * 2 * kWarps, bi = key / a.block_size;
    const int blk = key < min(key1, ctx) && bi < a.table_cap ? __ldg(a.tables + bi) : -1;
    return blk < 0 ? -1 : blk * a.blk_stride + (key - bi * a.block_size) * a.tok_stride + kvh * a.head_stride + 8 * hl;
  };
  int64_t first_at[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) first_at[i] = item ? key_at(key0, i) : -1;

  for (int l = 0; l < a.layers; ++l) {
    const StepLayer& w = a.layer[l];
    const uint32_t parity = l & 1;
    uint4 kf[kAhead], vf[kAhead];
    auto load_key = [&](int i, int64_t at) {
      kf[i] = at >= 0 ? *reinterpret_cast<const uint4*>(w.kc + at) : make_uint4(0, 0, 0, 0);
      vf[i] = at >= 0 ? *reinterpret_cast<const uint4*>(w.vc + at) : make_uint4(0, 0, 0, 0);
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i) load_key(i, first_at[i]);
    // the half warps 0 .. G + 1 work out the G rotated rows of q, the step's key, and take its value
    const bf16* const my_norm = hw < G ? w.q_norm : (hw == G ? w.k_norm : nullptr);
    const uint4 head_norm = item && my_norm != nullptr ? __ldg(reinterpret_cast<const uint4*>(my_norm) + hl) : make_uint4(0, 0, 0, 0);
    const uint32_t mark1 = base + 2 * l + 1, mark2 = mark1 + 1;
    // ---- 1: q, k, v --------------------------------------------------------------------------------------------------------
    {
      bf16 nw[kMine];
      norm_weights(nw, w.input_ln);
      norm(nw, base + 2 * l);
      mbar_wait(bars, parity);
      for (int r = 2 * warp; r < qn; r += 2 * kWarps) {
        const uint4* const row = reinterpret_cast<const uint4*>(w_qkv) + static_cast<int64_t>(r) * hp;
        const uint4* const rows[2] = {row, row + hp};
        float s[2];
        dots<2>(s, rows, xs, 0, hp);
        if (lane == 0) put(a.ll_qkv + (q0 + r) / 2, pack_bf16x2(s[0], s[1]), mark1);
      }
    }
    __syncthreads();
    // ---- 2: attention ------------------------------------------------------------------------------------------------------
    if (item) {
      if (warp < (G + 3) / 2) {   // (whole warps: the shuffles span them)
        const int row = hw < G ? kvh * G + hw : (hw == G ? a.heads : a.heads + a.kv_heads) + kvh;
        uint32_t raw[4];
        take<4>(raw, a.ll_qkv + row * (kD / 2) + 4 * hl, 1, hw < G + 2 ? 4 : 0, mark1, wt);
        const uint4 plain = make_uint4(raw[0], raw[1], raw[2], raw[3]), rot = rotate(plain, my_norm != nullptr, head_norm), mine_row = hw <= G ? rot : plain;
        if (hw < G + 2) head_rows[hw * 16 + hl] = mine_row;
        if ((hw == G || hw == G + 1) && split == 0 && slot >= 0) {
          const int blk = slot / a.block_size;
          const int64_t at = blk * a.blk_stride + (slot - blk * a.block_size) * a.tok_stride + kvh * a.head_stride + 8 * hl;
          *reinterpret_cast<uint4*>((hw == G ? w.kc : w.vc) + at) = mine_row;
        }
      }
      __syncthreads();
      float q[G][8];
#pragma unroll
      for (int g = 0; g < G; ++g) unpack8(head_rows[g * 16 + hl], q[g]);
      const uint4 knew = head_rows[G * 16 + hl], vnew = head_rows[(G + 1) * 16 + hl];
      Half st[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        st[g].m = -INFINITY; st[g].l = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) st[g].o[e] = 0.f;
      }
      // N rounds of a key a half warp
      auto rounds = [&](auto N_, int first) {
        constexpr int N = decltype(N_)::value;
        float s[N][G];
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int key = first + hw + i * 2 * kWarps;
          if (key == ctx) { kf[i] = knew; vf[i] = vnew; }
          float k[8];
          unpack8(kf[i], k);
#pragma unroll
          for (int g = 0; g < G; ++g) {
            s[i][g] = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) s[i][g] = fmaf(q[g][e], k[e], s[i][g]);
          }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < N; ++i)
#pragma unroll
            for (int g = 0; g < G; ++g) s[i][g] += __shfl_xor_sync(0xffffffffu, s[i][g], o);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          float mn = st[g].m;
#pragma unroll
          for (int i = 0; i < N; ++i) {
            s[i][g] = first + hw + i * 2 * kWarps < key1 ? s[i][g] * a.scale_log2 : -INFINITY;
            mn = fmaxf(mn, s[i][g]);
          }
          const float ms = mn == -INFINITY ? 0.f : mn, c = fast_exp2(st[g].m - ms);
          st[g].m = mn;
          st[g].l *= c;
#pragma unroll
          for (int e = 0; e < 8; ++e) st[g].o[e] *= c;
#pragma unroll
          for (int i = 0; i < N; ++i) {
            s[i][g] = fast_exp2(s[i][g] - ms);
            st[g].l += s[i][g];
          }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
          float v[8];
          unpack8(vf[i], v);
#pragma unroll
          for (int g = 0; g < G; ++g)
#pragma unroll
            for (int e = 0; e < 8; ++e) st[g].o[e] = fmaf(s[i][g], v[e], st[g].o[e]);
        }
      };
      for (int first = key0; first < key1; first += kAhead * 2 * kWarps) {
        if (first != key0) {
#pragma unroll
          for (int i = 0; i < kAhead; ++i) load_key(i, key_at(first, i));
        }
        if (key1 - first <= 2 * 2 * kWarps) rounds(std::integral_constant<int, 2>{}, first);
        else rounds(std::integral_constant<int, kAhead>{}, first);
      }
      // the halves of a warp, then the warps (through the room of the q/k/v rows, which the next layer's fill only after this)
      float* const so = reinterpret_cast<float*>(w_qkv);            // [warp][G][128]
      float* const sml = so + kWarps * G * kD;                      // [warp][G][2]
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float m2 = __shfl_xor_sync(0xffffffffu, st[g].m, 16), mn = fmaxf(st[g].m, m2), ms = mn == -INFINITY ? 0.f : mn;
        const float c = fast_exp2(st[g].m - ms);
        float ll = st[g].l * c;
        ll += __shfl_xor_sync(0xffffffffu, ll, 16);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          st[g].o[e] *= c;
          st[g].o[e] += __shfl_xor_sync(0xffffffffu, st[g].o[e], 16);
        }
        if (lane < 16) {
          float4* dst = reinterpret_cast<float4*>(so + (warp * G + g) * kD + 8 * hl);
          dst[0] = make_float4(st[g].o[0], st[g].o[1], st[g].o[2], st[g].o[3]);
          dst[1] = make_float4(st[g].o[4], st[g].o[5], st[g].o[6], st[g].o[7]);
          if (hl == 0) { sml[(warp * G + g) * 2] = mn; sml[(warp * G + g) * 2 + 1] = ll; }
        }
      }
      __syncthreads();
      for (int i = tid; i < G * kD; i += kThreads) {
        const int g = i / kD, d = i - g * kD;
        float m = -INFINITY, ll = 0.f, o = 0.f;
#pragma unroll
        for (int ww = 0; ww < kWarps; ++ww) m = fmaxf(m, sml[(ww * G + g) * 2]);
        const float ms = m == -INFINITY ? 0.f : m;
#pragma unroll
        for (int ww = 0; ww < kWarps; ++ww) {
          const float c = fast_exp2(sml[(ww * G + g) * 2] - ms);
          ll = fmaf(sml[(ww * G + g) * 2 + 1], c, ll);
          o = fmaf(so[(ww * G + g) * kD + d], c, o);
        }
        uint64_t* const part = a.ll_parts + static_cast<int64_t>(kvh * kParts) * G * kStepPart + g * kStepPart;   // [part][G][128 sums, maximum, sum of weights]
        if (split > 0) {
          uint64_t* const mine_part = part + static_cast<int64_t>(split) * G * kStepPart;
          put(mine_part + d, __float_as_uint(o), mark1);
          if (d == 0) {
            put(mine_part + kD, __float_as_uint(m), mark1);
            put(mine_part + kD + 1, __float_as_uint(ll), mark1);
          }
        } else {   // part 0 merges
          for (int s0 = 1; s0 < splits; s0 += 8) {
            uint32_t po[8], pm[8], pl[8];
            const uint64_t* const src = part + static_cast<int64_t>(s0) * G * kStepPart;
            const int n = min(splits - s0, 8);
            take<8>(po, src + d, G * kStepPart, n, mark1, wt);
            take<8, false>(pm, src + kD, G * kStepPart, n, mark1, wt);
            take<8, false>(pl, src + kD + 1, G * kStepPart, n, mark1, wt);
            float mn = m;
#pragma unroll
            for (int i = 0; i < 8; ++i) mn = i < n ? fmaxf(mn, __uint_as_float(pm[i])) : mn;
            const float ms2 = mn == -INFINITY ? 0.f : mn, c0 = fast_exp2(m - ms2);
            ll *= c0;
            o *= c0;
            m = mn;
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (i < n) {
                const float c = fast_exp2(__uint_as_float(pm[i]) - ms2);
                ll = fmaf(__uint_as_float(pl[i]), c, ll);
                o = fmaf(__uint_as_float(po[i]), c, o);
              }
          }
          const float v = ll == 0.f ? 0.f : o / ll, next = __shfl_xor_sync(0xffffffffu, v, 1);
          if ((d & 1) == 0) put(a.ll_attn + ((kvh * G + g) * kD + d) / 2, pack_bf16x2(v, next), mark1);
        }
      }
    }
    // ---- 3: o projection ---------------------------------------------------------------------------------------------------
    gather(a.ll_attn, HD / 2, mark1);
    if (tid == 0) fetch(0, l + 1);
    mbar_wait(bars + 8, parity);
    add_rows(w_o, HD, mark1, false);
    if (tid == 0) fetch(1, l + 1);
    // ---- 4: gate, up -------------------------------------------------------------------------------------------------------
    {
      bf16 nw[kMine];
      norm_weights(nw, w.post_ln);
      norm(nw, mark1);
      mbar_wait(bars + 16, parity);
      for (int r = 2 * warp; r < fn; r += 2 * kWarps) {
        const uint4* const gate = reinterpret_cast<const uint4*>(w_gu) + static_cast<int64_t>(r) * hp;
        const uint4* const up = gate + static_cast<int64_t>(fn) * hp;
        const uint4* const rows[4] = {gate, up, gate + hp, up + hp};
        float s[4];
        dots<4>(s, rows, xs, 0, hp);
        const float2 p = gated_pair<kGateSilu>(pack_bf16x2(s[0], s[2]), pack_bf16x2(s[1], s[3]), 0.f);
        if (lane == 0) put(a.ll_act + (f0 + r) / 2, pack_bf16x2(p.x, p.y), mark1);
      }
    }
    __syncthreads();
    if (tid == 0) fetch(2, l + 1);
    // ---- 5: down -----------------------------------------------------------------------------------------------------------
    gather(a.ll_act, a.inter / 2, mark1);
    mbar_wait(bars + 24, parity);
    add_rows(w_down, a.inter, mark2, l + 1 == a.layers);
    if (tid == 0) fetch(3, l + 1);
  }
  // the last CTA to come here moves the marks on: all have read them
  if (tid == 0 && atomicAdd(a.sync + 1, 1u) == static_cast<unsigned>(grid) - 1) {
    a.sync[0] = base + 2 * a.layers;
    a.sync[1] = 0;
  }
}

template <int G>
int launch_step(const StepArgs& a, int smem, cudaStream_t st) {
  NVLLM_SMEM_ATTR_ONCE(step_single_kernel<G>, 224 * 1024);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(sm_count());
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];   // cooperative: the CTAs wait for one another
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  NVLLM_CUDA(cudaLaunchKernelEx(&cfg, step_single_kernel<G>, a));
  NVLLM_LAUNCH_CHECK("step_single_kernel");
  return 0;
}

int up128(int64_t x) { return static_cast<int>((x + 127) / 128 * 128); }

}  // namespace

// Where it takes over: one token, and layers whose weights fit the SMs' shared memory (33 MB, with the room for x): with less the weights would wait
// for the stages, and the chain is then no shorter than that of the separate kernels.  The other limits are those of the code above.
int step_single_smem(StepArgs* a, int group) {
  const int grid = sm_count(), HD = a->heads * kD, qkv = HD + 2 * a->kv_heads * kD;
  const auto rows = [&](int n) { return static_cast<int64_t>((n + grid - 1) / grid); };
  const int64_t scratch = static_cast<int64_t>(kWarps) * group * (kD + 2) * 4;
  a->off_o = up128(std::max(2 * rows(qkv / 2) * a->hidden * 2, scratch));
  a->off_gu = a->off_o + up128(rows(a->hidden) * HD * 2);
  a->off_down = a->off_gu + up128(4 * rows(a->inter / 2) * a->hidden * 2);
  a->off_x = a->off_down + up128(rows(a->hidden) * a->inter * 2);
  const int64_t total = a->off_x + 2ll * std::max(a->hidden, std::max(HD, a->inter));
  return total <= 224 * 1024 ? static_cast<int>(total) : 0;
}

bool step_single_applies(int hidden, int heads, int kv_heads, int dim, int inter, int layers) {
  if (!knobs().gemm_skinny || dim != kD || kv_heads < 1 || heads % kv_heads != 0 || layers < 1 || layers > kStepLayers || hidden % 64 != 0 || inter % 64 != 0) return false;
  const int g = heads / kv_heads, grid = sm_count(), qkv_heads = heads + 2 * kv_heads;
  if ((g != 1 && g != 2 && g != 4) || hidden > kMine * kThreads || kv_heads > grid || (hidden + grid - 1) / grid > kStepRows || hidden < grid || inter < 2 * grid || qkv_heads * kD < 2 * grid) return false;
  if (static_cast<int64_t>(hidden) * (heads + 2 * kv_heads) * kD > (64 << 20) || static_cast<int64_t>(hidden) * inter > (64 << 20)) return false;
  StepArgs a{};
  a.heads = heads; a.kv_heads = kv_heads; a.hidden = hidden; a.inter = inter;
  return step_single_smem(&a, g) > 0;
}

int64_t step_single_words(int hidden, int heads, int kv_heads, int inter) {
  return hidden + (heads + 2 * kv_heads) * kD / 2 + static_cast<int64_t>(heads) * kParts * kStepPart + heads * kD / 2 + inter / 2;
}

int step_single(StepArgs& a, uint64_t* words, cudaStream_t st) {
  a.ll_h = words;
  a.ll_qkv = a.ll_h + a.hidden;
  a.ll_parts = a.ll_qkv + (a.heads + 2 * a.kv_heads) * kD / 2;
  a.ll_attn = a.ll_parts + static_cast<int64_t>(a.heads) * kParts * kStepPart;
  a.ll_act = a.ll_attn + a.heads * kD / 2;
  const int g = a.heads / a.kv_heads, smem = step_single_smem(&a, g);
  a.max_splits = std::min(kParts, sm_count() / a.kv_heads);
  return g == 1 ? launch_step<1>(a, smem, st) : (g == 2 ? launch_step<2>(a, smem, st) : launch_step<4>(a, smem, st));
}

}  // namespace nvllm
