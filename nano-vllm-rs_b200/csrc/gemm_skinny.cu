// gemm_skinny.cu — projections of a few tokens (M <= 16): decode steps of small batches, bound by reading the weights once.
//
// The tcgen05 kernels stage 128-row tiles of x for one token and are bound by their fixed steps (operand ring, TMEM, split-K
// exchange: 6-20 us a launch however small M is).  Here the weight rows are the M side of mma.sync m16n8k16 and the tokens the N side:
// a warp loads its weight fragments straight from global memory into registers (a lane owns 8 neighbouring values of a row, one
// 16-byte load; the product does not care in which order k is visited, so both operands use that order), all of a CTA's loads are in
// flight at once, and they start BEFORE the wait for the predecessor kernel.  8 warps share a CTA's 16 (or, for narrow outputs, 8)
// rows and split K; their f32 partial sums meet in shared memory in fixed order.
// Fused around it, with the roundings of the separate kernels:
//   norm_w    x is the residual stream and every CTA normalises its own copy of the few rows (rms(x) * w rounded to bf16)
//   GATE      w = [gate | up]; the CTA computes the matching rows of both and writes silu(gate) * up
//   residual  y = bf16(y + bf16(x . w^T)): the projection's output goes into the stream in place
// Measured, a decode step of one token (Qwen3-0.6B, 28 layers, graph replay): 1408 us on the tcgen05 kernels, 760 with these; 28 layers of
// weights and the head take 180 us at the copy rate, the rest is latency: 143 dependent launches of 5 us (all layers of one token in one
// launch, where their weights fit the SMs: step_single.cu).
#include "tc.cuh"

namespace nvllm {
namespace {

constexpr int kSkThreads = 256, kSkWarps = 8;

struct SkinnyArgs {
  void* y; const bf16* x; const bf16* w; const bf16* norm_w;
  int64_t ldx, ldw, ldy;
  int m, n, k;
  float eps;
  int residual;
};

// NT: tokens / 8; ROWS: weight rows of a CTA (16, or 8 with the upper half of the MMA rows unused); PRE: 32-wide k-blocks a warp
// loads ahead.
template <int NT, int ROWS, int PRE, bool GATE, bool NORM, typename OutT>
__global__ void __launch_bounds__(kSkThreads, sizeof(OutT) == 4 && NT == 1 ? 4 : 1) gemm_skinny_kernel(const SkinnyArgs a) {
  constexpr int MATS = GATE ? 2 : 1, HV = ROWS / 8;   // 8-row halves
  __shared__ float red[kSkWarps][MATS][NT * 8][ROWS + 1];
  __shared__ float ssq[kSkWarps][NT * 8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int n0 = blockIdx.x * ROWS, nkb = a.k / 32;
  const bf16* wrow[MATS][HV];
#pragma unroll
  for (int i = 0; i < MATS; ++i)
#pragma unroll
    for (int h = 0; h < HV; ++h) {
      const int r = n0 + 8 * h + g;
      wrow[i][h] = r < a.n ? a.w + (static_cast<int64_t>(i) * a.n + r) * a.ldw + 8 * t4 : nullptr;
    }
  uint4 wf[PRE][MATS][HV];
  auto load_w = [&](int kb, uint4 (&f)[MATS][HV]) {
#pragma unroll
    for (int i = 0; i < MATS; ++i)
#pragma unroll
      for (int h = 0; h < HV; ++h)
        f[i][h] = (kb < nkb && wrow[i][h] != nullptr) ? ld_nc_stream(wrow[i][h] + kb * 32) : make_uint4(0, 0, 0, 0);
  };
#pragma unroll
  for (int p = 0; p < PRE; ++p) load_w(warp + p * kSkWarps, wf[p]);
  uint4 nk[PRE];
  if (NORM) {
#pragma unroll
    for (int p = 0; p < PRE; ++p)
      nk[p] = warp + p * kSkWarps < nkb ? __ldg(reinterpret_cast<const uint4*>(a.norm_w + (warp + p * kSkWarps) * 32 + 8 * t4)) : make_uint4(0, 0, 0, 0);
  }
  pdl_wait();   // the weights are in flight; x (and a residual y) come from the predecessor
  // Only now may the successor start: launched any earlier, several kernels of the chain sit on the SMs at once and a step of one
  // token is slower than without the overlap (28 layers: 925 us, 914 without, 836 so).
  pdl_launch_dependents();
  const bf16* xrow[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) xrow[j] = 8 * j + g < a.m ? a.x + (8 * j + g) * a.ldx + 8 * t4 : nullptr;
  // the first PRE blocks of x stay in registers between the norm's sum and the products
  uint4 xk[PRE][NT];
#pragma unroll
  for (int p = 0; p < PRE; ++p)
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int kb = warp + p * kSkWarps;
      xk[p][j] = (xrow[j] != nullptr && kb < nkb) ? *reinterpret_cast<const uint4*>(xrow[j] + kb * 32) : make_uint4(0, 0, 0, 0);
    }
  float inv[NT];
  if (NORM) {
    auto squares = [](const uint4& v) {
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
      float s = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) s += bf16_lo(u[e]) * bf16_lo(u[e]) + bf16_hi(u[e]) * bf16_hi(u[e]);
      return s;
    };
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      inv[j] = 0.f;
#pragma unroll
      for (int p = 0; p < PRE; ++p) inv[j] += squares(xk[p][j]);
      if (xrow[j] != nullptr)
        for (int kb = warp + PRE * kSkWarps; kb < nkb; kb += kSkWarps) inv[j] += squares(*reinterpret_cast<const uint4*>(xrow[j] + kb * 32));
      inv[j] += __shfl_xor_sync(0xffffffffu, inv[j], 1);
      inv[j] += __shfl_xor_sync(0xffffffffu, inv[j], 2);
      if (t4 == 0) ssq[warp][8 * j + g] = inv[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < kSkWarps; ++i) s += ssq[i][8 * j + g];
      inv[j] = 1.0f / sqrtf(s / static_cast<float>(a.k) + a.eps);
    }
  }
  float acc[MATS][NT][4];
#pragma unroll
  for (int i = 0; i < MATS; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  for (int kb0 = warp; kb0 < nkb; kb0 += kSkWarps * PRE) {
#pragma unroll
    for (int p = 0; p < PRE; ++p) {
      const int kb = kb0 + p * kSkWarps;
      if (kb >= nkb) break;
      uint4 xf[NT];
#pragma unroll
      for (int j = 0; j < NT; ++j)
        xf[j] = kb0 == warp ? xk[p][j] : (xrow[j] != nullptr ? *reinterpret_cast<const uint4*>(xrow[j] + kb * 32) : make_uint4(0, 0, 0, 0));
      if (NORM) {
        const uint4 nv = kb0 == warp ? nk[p] : __ldg(reinterpret_cast<const uint4*>(a.norm_w + kb * 32 + 8 * t4));
        const uint32_t nw[4] = {nv.x, nv.y, nv.z, nv.w};
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          uint32_t u[4] = {xf[j].x, xf[j].y, xf[j].z, xf[j].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) u[e] = pack_bf16x2(bf16_lo(u[e]) * inv[j] * bf16_lo(nw[e]), bf16_hi(u[e]) * inv[j] * bf16_hi(nw[e]));
          xf[j] = make_uint4(u[0], u[1], u[2], u[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < MATS; ++i) {
        const uint4 lo = wf[p][i][0], hi = HV == 2 ? wf[p][i][HV - 1] : make_uint4(0, 0, 0, 0);
        const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          mma_bf16_16816(acc[i][j], a0, xf[j].x, xf[j].y);
          mma_bf16_16816(acc[i][j], a1, xf[j].z, xf[j].w);
        }
      }
      load_w(kb + kSkWarps * PRE, wf[p]);   // (nothing beyond the last block)
    }
  }
#pragma unroll
  for (int i = 0; i < MATS; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < 2 || HV == 2) red[warp][i][8 * j + 2 * t4 + (e & 1)][g + 8 * (e >> 1)] = acc[i][j][e];
  __syncthreads();
  for (int e = threadIdx.x; e < ROWS * NT * 8; e += kSkThreads) {
    const int t = e / ROWS, r = e - t * ROWS;
    if (t >= a.m || n0 + r >= a.n) continue;
    float s[MATS];
#pragma unroll
    for (int i = 0; i < MATS; ++i) {
      s[i] = 0.f;
#pragma unroll
      for (int wv = 0; wv < kSkWarps; ++wv) s[i] += red[wv][i][t][r];
    }
    OutT* dst = static_cast<OutT*>(a.y) + t * a.ldy + n0 + r;
    if constexpr (GATE) {
      const float2 p = gated_pair<kGateSilu>(pack_bf16x2(s[0], 0.f), pack_bf16x2(s[MATS - 1], 0.f), 0.f);
      *dst = __float2bfloat16_rn(p.x);
    } else if constexpr (sizeof(OutT) == 4) {
      *dst = s[0];
    } else {
      float v = s[0];
      if (a.residual) v = __bfloat162float(*dst) + __bfloat162float(__float2bfloat16_rn(v));
      *dst = __float2bfloat16_rn(v);
    }
  }
}

// Heads (f32 out, many rows): the same products by CTAs that stay.  x is normed once per CTA and kept in shared memory, and a warp's
// weight loads run kHeadPre blocks ahead across the edges of its 16-row tiles, so that HBM never waits for a tile's prologue or its sum.
// Bound by HBM.  Measured, 1 x 1024 by 151936 rows (311 MB, 47 us at the copy rate): 81 us with a CTA per tile, 54 so.  Launched
// plainly: CTAs that stay and start early share SMs unevenly (a decode step of one token 838 us early, 797 plainly, 824 before).
constexpr int kHeadPre = 4, kHeadCtas = 3, kHeadSmem = 72 * 1024;
template <int NT>
constexpr int head_red_bytes() { return 2 * kSkWarps * NT * 8 * 17 * 4; }

template <int NT>
__global__ void __launch_bounds__(kSkThreads, kHeadCtas) gemm_skinny_head_kernel(const SkinnyArgs a) {
  extern __shared__ __align__(16) uint8_t head_smem[];
  __shared__ float ssq[kSkWarps][NT * 8];
  float* red = reinterpret_cast<float*>(head_smem);   // [2][warp][token][17]: one barrier a tile
  bf16* xs = reinterpret_cast<bf16*>(head_smem + head_red_bytes<NT>());
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int nkb = a.k / 32, nb = (nkb + kSkWarps - 1) / kSkWarps, tiles = (a.n + 15) / 16, step = static_cast<int>(gridDim.x);
  const int pitch = a.k + 32;   // rows 64 bytes apart in the banks
  int lt = blockIdx.x, lb = 0;  // the next block to load
  auto load = [&](uint4 (&f)[2]) {
    const int kb = warp + lb * kSkWarps;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 16 * lt + 8 * h + g;
      f[h] = (lt < tiles && r < a.n && kb < nkb) ? ld_nc_stream(a.w + static_cast<int64_t>(r) * a.ldw + kb * 32 + 8 * t4) : make_uint4(0, 0, 0, 0);
    }
    if (++lb == nb) { lb = 0; lt += step; }
  };
  uint4 wf[kHeadPre][2];
#pragma unroll
  for (int p = 0; p < kHeadPre; ++p) load(wf[p]);
  pdl_launch_dependents();
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    float ss = 0.f;
    if (8 * j + g < a.m)
      for (int kb = warp; kb < nkb; kb += kSkWarps) {
        const uint4 v = *reinterpret_cast<const uint4*>(a.x + (8 * j + g) * a.ldx + kb * 32 + 8 * t4);
        *reinterpret_cast<uint4*>(xs + (8 * j + g) * pitch + kb * 32 + 8 * t4) = v;
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) s += bf16_lo(u[e]) * bf16_lo(u[e]) + bf16_hi(u[e]) * bf16_hi(u[e]);
        ss += s;
      }
    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
    ss += __shfl_xor_sync(0xffffffffu, ss, 2);
    if (t4 == 0) ssq[warp][8 * j + g] = ss;
  }
  __syncthreads();
  if (a.norm_w != nullptr) {   // every thread norms the values that it stored
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      if (8 * j + g >= a.m) continue;
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < kSkWarps; ++i) s += ssq[i][8 * j + g];
      const float inv = 1.0f / sqrtf(s / static_cast<float>(a.k) + a.eps);
      for (int kb = warp; kb < nkb; kb += kSkWarps) {
        uint4* at = reinterpret_cast<uint4*>(xs + (8 * j + g) * pitch + kb * 32 + 8 * t4);
        const uint4 v = *at, nv = __ldg(reinterpret_cast<const uint4*>(a.norm_w + kb * 32 + 8 * t4));
        uint32_t u[4] = {v.x, v.y, v.z, v.w};
        const uint32_t nw[4] = {nv.x, nv.y, nv.z, nv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) u[e] = pack_bf16x2(bf16_lo(u[e]) * inv * bf16_lo(nw[e]), bf16_hi(u[e]) * inv * bf16_hi(nw[e]));
        *at = make_uint4(u[0], u[1], u[2], u[3]);
      }
    }
  }
  // (a lane reads back, below, only blocks that it stored itself)
  float acc[NT][4] = {};
  int tile = blockIdx.x, b = 0, buf = 0;
  while (tile < tiles) {
#pragma unroll
    for (int p = 0; p < kHeadPre; ++p) {
      if (tile >= tiles) break;   // (the same for all threads of the CTA)
      const int kb = warp + b * kSkWarps;
      if (kb < nkb) {
        const uint32_t a0[4] = {wf[p][0].x, wf[p][1].x, wf[p][0].y, wf[p][1].y}, a1[4] = {wf[p][0].z, wf[p][1].z, wf[p][0].w, wf[p][1].w};
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const uint4 xf = 8 * j + g < a.m ? *reinterpret_cast<const uint4*>(xs + (8 * j + g) * pitch + kb * 32 + 8 * t4) : make_uint4(0, 0, 0, 0);
          mma_bf16_16816(acc[j], a0, xf.x, xf.y);
          mma_bf16_16816(acc[j], a1, xf.z, xf.w);
        }
      }
      load(wf[p]);   // (nothing beyond the last tile)
      if (++b < nb) continue;
      float* rb = red + buf * kSkWarps * NT * 8 * 17;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          rb[(warp * NT * 8 + 8 * j + 2 * t4 + (e & 1)) * 17 + g + 8 * (e >> 1)] = acc[j][e];
          acc[j][e] = 0.f;
        }
      __syncthreads();
      for (int e = threadIdx.x; e < 16 * a.m; e += kSkThreads) {
        const int t = e / 16, r = e - t * 16;
        if (16 * tile + r >= a.n) continue;
        float s = 0.f;
#pragma unroll
        for (int wv = 0; wv < kSkWarps; ++wv) s += rb[(wv * NT * 8 + t) * 17 + r];
        static_cast<float*>(a.y)[t * a.ldy + 16 * tile + r] = s;
      }
      b = 0;
      buf ^= 1;
      tile += step;
    }
  }
}

template <int NT>
int skinny_head(const SkinnyArgs& a, cudaStream_t st) {
  NVLLM_SMEM_ATTR_ONCE(gemm_skinny_head_kernel<NT>, kHeadSmem);
  NVLLM_CUDA(launch_plain(gemm_skinny_head_kernel<NT>, dim3(kHeadCtas * sm_count()), dim3(kSkThreads), head_red_bytes<NT>() + a.m * (a.k + 32) * 2, st, a));
  return 0;
}

template <int NT, int ROWS, int PRE, bool GATE, typename OutT>
int skinny_run(const SkinnyArgs& a, cudaStream_t st) {
  const dim3 grid((a.n + ROWS - 1) / ROWS);
  NVLLM_CUDA(launch_pdl(a.norm_w != nullptr ? gemm_skinny_kernel<NT, ROWS, PRE, GATE, true, OutT> : gemm_skinny_kernel<NT, ROWS, PRE, GATE, false, OutT>,
                        grid, dim3(kSkThreads), 0, st, a));
  return 0;
}

template <int NT>
int skinny_rows(const SkinnyArgs& a, bool gate, int out_dtype, cudaStream_t st) {
  // 8-row CTAs while all of them run at once (two rounds of them lose to one of 16-row ones); k-blocks ahead: all of a warp's up to
  // K = 1024 (narrow outputs: 3072)
  if (gate) return skinny_run<NT, 16, 4, true, bf16>(a, st);
  if constexpr (NT == 1)   // heads: CTAs that stay where each has two tiles or more (gemm_skinny_applies lets no more than 8 rows of 2560 come here)
    if (out_dtype == NVLLM_F32 && a.n >= 2 * 16 * kHeadCtas * sm_count()) return skinny_head<NT>(a, st);
  if (out_dtype == NVLLM_F32) return skinny_run<NT, 16, 2, false, float>(a, st);   // heads: many CTAs, bound by bytes in flight: four on an SM
  if ((a.n + 7) / 8 <= sm_count()) return skinny_run<NT, 8, 12, false, bf16>(a, st);
  return skinny_run<NT, 16, 4, false, bf16>(a, st);
}

}  // namespace

// Where these kernels take over: up to 16 rows of x, and matrices small enough that the fixed steps of the general kernels decide their
// time.  A warp asks for x block by block behind the first ones, so long rows lose, and CTAs that end and start anew do not keep HBM busy
// over a large matrix.  Measured beside the general path with weights from HBM (us, general -> here, 1 and 16 rows):
//   bf16   4096 x 1024  7.2 -> 3.3, 4.1    1024 x 3072  6.5 -> 3.4, 5.2    4096 x 2048  9.2 -> 6.7, 7.7    | 8192 x 2048 0.95, 1.11 of it
//          2560 x 4096 10.7 -> 12.0, 13.1  6144 x 4096 13.7 -> 22.8, 25.4  2048 x 8192 14.3 -> 35, 40
//   gate   3072 x 1024 16.0 -> 5.0, 6.5    8192 x 2048 31.9 -> 25.5, 28.8  | 16384 x 2304 1.00, 1.10 of it  12288 x 4096 61 -> 76, 83
//   f32    4096 x 2048  9.2 -> 6.8, 7.8    151936 x 2560 139 -> 119, 215   1024 x 3072 7.3 -> 8.2, 8.7
bool gemm_skinny_applies(int m, int n, int k, int64_t ldx, int64_t ldw, bool f32_out, bool gate) {
  if (!knobs().gemm_skinny || m < 1 || m > 16 || k % 32 != 0 || ldx % 8 != 0 || ldw % 8 != 0 || n < 1) return false;
  if (gate) return k <= 2048;
  if (f32_out)
    return m <= 8 ? k <= (n <= 1024 ? 2048 : 2560) && (n <= 8192 || k >= 1024) : (n <= 4096 && k <= (n <= 1024 ? 1536 : 2048)) || (n <= 8192 && k <= 1024);
  // (8-row CTAs up to 8 rows an SM; then 16-row ones, first too few of them to fill the SMs)
  const int most = n <= 8 * sm_count() ? 3072 : (n <= 16 * sm_count() ? (m <= 8 ? 2048 : 1536) : (m <= 8 ? 3072 : 2304));
  return (n <= 4096 && k <= most) || (n <= 8192 && k <= 1024);
}

int gemm_skinny(void* y, const void* x, const void* w, int m, int n, int k, int64_t ldx, int64_t ldw, int64_t ldy, int out_dtype, bool silu_gate,
                const void* norm_w, float eps, bool residual, cudaStream_t st) {
  const SkinnyArgs a{y, static_cast<const bf16*>(x), static_cast<const bf16*>(w), static_cast<const bf16*>(norm_w), ldx, ldw, ldy, m, n, k, eps, residual ? 1 : 0};
  return m <= 8 ? skinny_rows<1>(a, silu_gate, out_dtype, st) : skinny_rows<2>(a, silu_gate, out_dtype, st);
}

}  // namespace nvllm
