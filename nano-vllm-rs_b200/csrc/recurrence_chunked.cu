// recurrence_chunked.cu — the linear recurrence  S_t = a_t S_(t-1) + b_t k_t v_t^T,  y_t = S_t^T q_t + d v_t  (one decay per head) for
// prompts: 32 tokens at a time as matrix products.  With D_ij = a_(j+1) ... a_i (i >= j) a chunk is
//   y_i = (a_1 ... a_i) S^T q_i + sum_(j <= i) (q_i . k_j) D_ij b_j v_j + d v_i,     S <- (a_1 ... a_32) S + sum_j k_j (D_(32)j b_j v_j)^T.
//
// Precision: inputs, state and results are f32, and the products lose nothing that the token-by-token form (recurrence.cu) keeps.
// Every operand is split into three bf16 values (8 bits each, f32's range), and six products on mma.sync keep what is above 2^-24:
// hi.hi, hi.mid, mid.hi, mid.mid, hi.lo, lo.hi.  mma.sync cuts off: it aligns its addends to 2^-26 of the largest and its sum to 24 bits.  So hi.hi
// of one or two steps is added up in f32 outside (four in a row lose more than the additions do), and the rest, 2^-8 and smaller, is summed apart.
// Accumulators start from zero in every chunk and are added to the state in f32, so that the state is rounded once per 32 tokens instead of 32
// times; D_(32)j b_j v_j is split from a value in two parts.  A state that keeps less than 2^-8 of the chunk's start is made of this one rounding,
// so there the products of hi.hi run once more on top of the negated sum and give what was cut off (for every chunk 7 % more time; without
// it the state's error reaches 1.04 times the other form's).  (Two fp16 values
// and three products would need half the instructions, but their 22-bit products meet the cut: 4.5e-7 from 64 bits.)  Relative
// error of y and of the state against 64 bits, token by token and here, 1e-7: retention 1.99, 1.89 and 0.83, 0.60; state-space duality as the models
// have it 0.81, 0.68 and 0.67, 0.51; decays of 0.3 a token 0.79, 0.46 and 0.74, 0.45; any decay from 0 to 1 1.22, 0.47 and 0.82, 0.46.
// A chunk with a value that is no number, infinite, or far from the others' range (rows of q and k outside 2^-60 .. 2^40, d beyond 2^40) is stepped
// through token by token in f32 instead, by the warps that it concerns: what such a value reaches is then the same as there.
//
// CTA = (head, sequence, 64 columns of v), 4 warps; a warp keeps 16 columns of the state, transposed, in the accumulator layout of
// m16n8k16 (64 registers), which is also that of the B operand of S^T q, so the state never leaves its registers.  v comes from
// global memory straight into the layout that serves as A (v^T of the update) and as B (of the middle product).  q and k of the
// next chunk fly (cp.async) under the products of this one.  Bound by mma.sync issue (about 540 of them per warp and chunk) and the conversions
// around it; two CTAs an SM (91 KB each) hide each other's barriers.
// Token by token and here (us, back to back on one GPU): 16 heads of 128 x 128, 8 x 1024 tokens 542 and 270, 500 tokens 205 and 100; 64 heads of 128 x 64,
// 8 x 1024 868 and 531, 2 x 40 25 and 17.
#include <type_traits>

#include "split_mma.cuh"

namespace nvllm {
namespace {

using namespace split;

constexpr int kC = 32, kDk = 128, kCols = 64, kWarps = 4;
constexpr int kRow = kDk * 2 + 16;               // bytes of a row of pieces: 16 more, so that ldmatrix rows fall into different banks
constexpr int kPiece = kC * kRow;
constexpr int kPs = 40;                          // floats of a row of the middle factor (8 r + 2 c: no conflicts for 8-byte reads)
constexpr int kSmRaw = 0;                        // q, then k of a chunk as they come: [32][128] f32 each
constexpr int kSmQ = kSmRaw + 2 * kC * kDk * 4;  // hi, mid, lo
constexpr int kSmK = kSmQ + 3 * kPiece;
constexpr int kSmP = kSmK + 3 * kPiece;          // D_ij, overwritten in place by the middle factor
constexpr int kSmVec = kSmP + kC * kPs * 4;      // floats: pre, w [32 each], a [2][32], b [2][32], second part of w [32], flag, that of the product of all decays
constexpr int kSmBytes = kSmVec + 7 * kC * 4 + 16;

template <bool TOGETHER>
__global__ void __launch_bounds__(kWarps * 32, 2) linear_recurrence_chunked_kernel(const RecArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  float* raw = reinterpret_cast<float*>(smem + kSmRaw);
  float* mid = reinterpret_cast<float*>(smem + kSmP);
  float* vec = reinterpret_cast<float*>(smem + kSmVec);
  float *pre = vec, *wgt = vec + kC, *wgt_lo = vec + 6 * kC;
  volatile uint32_t* flag = reinterpret_cast<volatile uint32_t*>(vec + 7 * kC);
  const int h = blockIdx.x, s = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col0 = blockIdx.z * kCols + warp * 16;       // the warp's first column of the head
  const int r = lane >> 2, c2 = (lane & 3) * 2;          // row and first column of the lane in an accumulator tile
  const int t0 = a.cu_tokens[s], t1 = a.cu_tokens[s + 1];
  const int slot = a.seq_slot[s];
  if (t1 <= t0) return;
  float* const yh = a.y + static_cast<int64_t>(h) * a.dv + col0;
  if (slot < 0) {  // padding sequence of a captured batch: defined output, no state
    for (int64_t t = t0; t < t1; ++t)
      if (lane < 16) yh[t * a.ldy + lane] = 0.f;
    return;
  }
  const int g = h / a.group_div;
  const float* const qg = a.q + static_cast<int64_t>(g) * kDk;
  const float* const kg = a.k + static_cast<int64_t>(g) * kDk;
  const float* const vh = a.v + static_cast<int64_t>(h) * a.dv + col0;

  // q, k, decays and steps of the chunk that starts at token tb; tokens past the end are neutral.  A thread copies one 16-byte piece of every
  // fourth row.
  const float *qp = qg + (t0 + warp) * a.ldq + lane * 4, *kp = kg + (t0 + warp) * a.ldk + lane * 4;
  auto issue = [&](int tb, int buf) {
    const uint32_t dst = smem_u32(raw + warp * kDk + lane * 4);
#pragma unroll
    for (int i = 0; i < kC / kWarps; ++i) {
      const bool in = tb + warp + i * kWarps < t1;
      cp_async_16(dst + i * kWarps * kDk * 4, in ? qp + i * kWarps * a.ldq : qg, in ? 16 : 0);
      cp_async_16(dst + (kC + i * kWarps) * kDk * 4, in ? kp + i * kWarps * a.ldk : kg, in ? 16 : 0);
    }
    qp += kC * a.ldq;
    kp += kC * a.ldk;
    if (tid < kC) {
      const int64_t t = tb + tid;
      float *as = vec + 2 * kC + buf * kC + tid, *bs = vec + 4 * kC + buf * kC + tid;
      if (t < t1) cp_async_4(smem_u32(as), a.decay + (a.decay_ld ? t * a.decay_ld + h : h)); else *as = 1.f;
      if (t < t1 && a.step) cp_async_4(smem_u32(bs), a.step + (a.step_ld ? t * a.step_ld + h : h)); else *bs = t < t1 ? 1.f : 0.f;
    }
    cp_async_commit();
  };
  // v of a chunk in the order of the A operand of v^T (16 columns x 32 tokens): [token step of 16][register][token of the pair]
  float vr[2][4][2];
  auto load_v = [&](int tb) {
    const float* vp = vh + (tb + c2) * a.ldv + r;
    const bool all = tb + kC <= t1;
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int o = ks * 16 + hh * 8 + e;
          const bool in = all || tb + c2 + o < t1;
          vr[ks][2 * hh][e] = in ? vp[o * a.ldv] : 0.f;
          vr[ks][2 * hh + 1][e] = in ? vp[o * a.ldv + 8] : 0.f;
        }
  };

  if (tid == 0) *flag = 0u;
  issue(t0, 0);
  load_v(t0);
  // state, transposed: tile n holds keys 8n + c2 + {0, 1} of columns r (registers 0, 1) and r + 8 (registers 2, 3)
  float S[16][4];
  float* const sp = a.state + (static_cast<int64_t>(slot) * a.heads + h) * kDk * a.dv + col0;
  const bool fresh = a.positions[t0] == 0;
#pragma unroll
  for (int n = 0; n < 16; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      S[n][i] = fresh ? 0.f : sp[static_cast<int64_t>(8 * n + c2 + (i & 1)) * a.dv + r + (i >> 1) * 8];
  const float d = a.skip ? a.skip[h] : 0.f;

  int buf = 0;
  for (int tb = t0; tb < t1; tb += kC, buf ^= 1) {
    const int cnt = min(kC, t1 - tb);
    const float* as = vec + 2 * kC + buf * kC;
    const float* bs = vec + 4 * kC + buf * kC;
    cp_async_wait<0>();
    __syncthreads();
    // ---- q and k: a warp per row, split; D and the factors it makes ------------------------------------------------------
    bool bad = false;
#pragma unroll
    for (int op = 0; op < 2; ++op) {            // q, k
      float4 x[kC / kWarps];
#pragma unroll
      for (int i = 0; i < kC / kWarps; ++i) x[i] = *reinterpret_cast<const float4*>(raw + (op * kC + i * kWarps + warp) * kDk + lane * 4);
      uint32_t most = 0u;
#pragma unroll
      for (int i = 0; i < kC / kWarps; ++i) {
        most = max(max(most, max(abs_bits(x[i].x), abs_bits(x[i].y))), max(abs_bits(x[i].z), abs_bits(x[i].w)));
        uint2 p[3];
        split3(x[i].x, x[i].y, p[0].x, p[1].x, p[2].x);
        split3(x[i].z, x[i].w, p[0].y, p[1].y, p[2].y);
        uint8_t* dst = smem + (op ? kSmK : kSmQ) + (i * kWarps + warp) * kRow + lane * 8;
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(dst + j * kPiece) = p[j];
      }
      bad |= far_off(__reduce_max_sync(0xffffffffu, most), -60, 40);
    }
    {
      // Lane 0 takes the products a_1 ... a_i, lane j + 1 the column D_ij, in two f32 parts each: a decay's powers come back chunk after
      // chunk, so their rounding would not average out as that of single steps does.
      float x[kC];
#pragma unroll
      for (int i = 0; i < kC / 4; ++i) {
        const float4 v4 = reinterpret_cast<const float4*>(as)[i];
        x[4 * i] = v4.x; x[4 * i + 1] = v4.y; x[4 * i + 2] = v4.z; x[4 * i + 3] = v4.w;
      }
      const float av = as[lane], bv = bs[lane], b_prev = __shfl_up_sync(0xffffffffu, bv, 1);
      float* const col = lane == 0 ? pre : mid + lane - 1;
      const int step_f = lane == 0 ? 1 : kPs;
      float hi = 1.f, lo = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        float row[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (8 * w + i >= lane) {
            const float p = hi * x[8 * w + i];
            lo = fmaf(lo, x[8 * w + i], fmaf(hi, x[8 * w + i], -p));
            hi = p;
          }
          row[i] = 8 * w + i >= lane - 1 ? hi + lo : 0.f;
        }
        if (warp == w) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            col[(8 * w + i) * step_f] = row[i];
            if (lane == 31) mid[(8 * w + i) * kPs + 31] = 8 * w + i == 31 ? 1.f : 0.f;
          }
        }
      }
      if (warp == kWarps - 1) {
        const float all = hi + lo;
        if (lane == 0) {
          vec[7 * kC + 1] = (hi - all) + lo;
        } else {
          const float p = __fmul_rn(b_prev, hi);
          wgt[lane - 1] = p;
          wgt_lo[lane - 1] = fmaf(b_prev, lo, fmaf(b_prev, hi, -p));
        }
        if (lane == 31) { wgt[31] = bv; wgt_lo[31] = 0.f; }
      }
      // decays above 1 are rare enough to step through: D then stays in [0, 1]
      bad |= !(av >= 0.f && av <= 1.f) || far_off(abs_bits(bv), -60, 40) || !(fabsf(d) < 1.1e12f);
    }
    if (bad) *flag = 1u;
    __syncthreads();
    const bool slow = *flag != 0u;
    if (tb + kC < t1) issue(tb + kC, buf ^ 1);
    const uint32_t q_addr = sbase + kSmQ + (lane & 15) * kRow + (lane >> 4) * 16;
    // ---- middle factor (q_i . k_j) D_ij b_j (+ d on the diagonal): warp w computes tokens 16 (w / 2) .. + 15, keys 16 (w % 2) .. + 15 (warp 1's keys lie
    // behind all of its tokens: it keeps nothing); and S^T q of the chunk's start.  Each alone is a chain of dependent products, the first of two at a time.
    // TOGETHER, step by step beside each other, 8 x 1024 tokens take 270 and 531 us (16 and 64 heads, see above), and one after the other, the first left out by
    // warp 1, 292 and 576.  With one CTA an SM at the most it is the longest warp that counts, and one after the other is shorter: 500 tokens, 16 heads,
    // 102.1 us together and 99.9 so, 4 x 300 72.7 and 72.2.
    const int mt = warp >> 1, nt = warp & 1;
    // B of 16 keys x 16 dims: lanes 0-7 keys 0-7 dims 0-7, 8-15 the same keys dims 8-15, 16-31 keys 8-15
    const uint32_t mk_addr = sbase + kSmK + (nt * 16 + (lane & 7) + (lane >> 4) * 8) * kRow + ((lane >> 3) & 1) * 16;
    float yi[2][2][4] = {};           // S^T q: [16 tokens][8 columns]
    auto products = [&](auto which) {   // 1: the middle factor, 2: S^T q, 3: both
      constexpr bool kMiddle = (decltype(which)::value & 1) != 0, kState = (decltype(which)::value & 2) != 0;
      float sum[2][4] = {}, ah[1][2][4], al[2][1][2][4] = {};   // (al: even and odd steps)
      float yl[2][2][4] = {}, hh[2][2][4];
#pragma unroll
      for (int kk = 0; kk < kDk / 16; ++kk) {
        uint32_t qm[1][3][4], kf[3][2][2], qf[2][3][4], sf[3][2][2];          // sf: [piece][8 columns][half of the 16 keys]
        if (kk % 2 == 0) { zero(ah); zero(hh); }
        if constexpr (kMiddle) {
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            ldmatrix_x4(qm[0][j], q_addr + mt * 16 * kRow + kk * 32 + j * kPiece);
            ldmatrix_x4(reinterpret_cast<uint32_t(&)[4]>(kf[j]), mk_addr + kk * 32 + j * kPiece);
          }
        }
        if constexpr (kState) {
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) split3(S[2 * kk + e][2 * n], S[2 * kk + e][2 * n + 1], sf[0][n][e], sf[1][n][e], sf[2][n][e]);
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int j = 0; j < 3; ++j) ldmatrix_x4(qf[m][j], q_addr + m * 16 * kRow + kk * 32 + j * kPiece);
        }
        if constexpr (kMiddle) mma6<1, 2>(ah, al[kk & 1], qm, kf);
        if constexpr (kState) mma6<2, 2>(hh, yl, qf, sf);
        if (kk % 2 == 1) {
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if constexpr (kMiddle) sum[n][i] += ah[0][n][i];
              if constexpr (kState) {
                yi[0][n][i] += hh[0][n][i];
                yi[1][n][i] += hh[1][n][i];
              }
            }
        }
      }
      if constexpr (kMiddle) {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = mt * 16 + r + (i >> 1) * 8, key = nt * 16 + n * 8 + c2 + (i & 1);
            float* m = mid + row * kPs + key;
            if (warp != 1) *m = fmaf(join(sum[n][i], al[0][0][n][i] + al[1][0][n][i]) * bs[key], *m, row == key ? d : 0.f);      // D is zero above the diagonal
          }
      }
      if constexpr (kState) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) yi[m][n][i] = join(yi[m][n][i], yl[m][n][i]);
      }
    };
    if constexpr (!TOGETHER) {
      if (!slow && warp != 1) products(std::integral_constant<int, 1>{});
    }
    // v and the state: their largest magnitude decides whether the warp takes the products
    float vmax = 0.f;
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int i = 0; i < 4; ++i) vmax = abs_max(vr[ks][i][0], vr[ks][i][1], vmax);
    float smax[2] = {vmax, 0.f};
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      smax[0] = abs_max(S[n][0], S[n][1], smax[0]);
      smax[1] = abs_max(S[n][2], S[n][3], smax[1]);
    }
    const bool step = __any_sync(0xffffffffu, slow || !(smax[0] < 1.2e24f && smax[1] < 1.2e24f));      // 2^80
    if constexpr (TOGETHER) {
      if (!slow) products(std::integral_constant<int, 3>{});   // (also where this warp steps: the middle factor is for all)
    } else {
      if (!step) products(std::integral_constant<int, 2>{});
    }
    uint32_t vf[2][3][2][2];           // v as B: [token step][piece][8 columns][half of the 16 tokens]
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int i = 0; i < 4; ++i) split3(vr[ks][i][0], vr[ks][i][1], vf[ks][0][i & 1][i >> 1], vf[ks][1][i & 1][i >> 1], vf[ks][2][i & 1][i >> 1]);
    __syncthreads();                   // the middle factor is complete
    if (!step) {
      // ---- middle factor . v -------------------------------------------------------------------------------------------
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        float ah[1][2][4] = {}, al[1][2][4] = {};
#pragma unroll
        for (int ks = 0; ks <= m; ++ks) {   // the first 16 tokens see no key of the second 16
          uint32_t pf[1][3][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 x = *reinterpret_cast<const float2*>(mid + (m * 16 + r + (i & 1) * 8) * kPs + ks * 16 + (i >> 1) * 8 + c2);
            split3(x.x, x.y, pf[0][0][i], pf[0][1][i], pf[0][2][i]);
          }
          mma6<1, 2>(ah, al, pf, vf[ks]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {   // token rows r, r + 8
          const int tt = m * 16 + r + e * 8;
          if (tt < cnt) {
            const float fi = pre[tt];
            const int64_t t = tb + tt;
#pragma unroll
            for (int n = 0; n < 2; ++n)
              *reinterpret_cast<float2*>(yh + t * a.ldy + n * 8 + c2) =
                  make_float2(fmaf(yi[m][n][2 * e], fi, join(ah[0][n][2 * e], al[0][n][2 * e])), fmaf(yi[m][n][2 * e + 1], fi, join(ah[0][n][2 * e + 1], al[0][n][2 * e + 1])));
          }
        }
      }
      // ---- state: S <- (a_1 ... a_32) S + sum_j k_j (D_(32)j b_j v_j)^T ---------------------------------------------------
      uint32_t wf[2][1][3][4];
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 w = *reinterpret_cast<const float2*>(wgt + ks * 16 + (i >> 1) * 8 + c2), wl = *reinterpret_cast<const float2*>(wgt_lo + ks * 16 + (i >> 1) * 8 + c2);
          const float p0 = __fmul_rn(vr[ks][i][0], w.x), p1 = __fmul_rn(vr[ks][i][1], w.y);   // (not to be fused with what follows: the second parts are p0's and p1's)
          split3(p0, p1, fmaf(vr[ks][i][0], wl.x, fmaf(vr[ks][i][0], w.x, -p0)), fmaf(vr[ks][i][1], wl.y, fmaf(vr[ks][i][1], w.y, -p1)), wf[ks][0][0][i],
                 wf[ks][0][1][i], wf[ks][0][2][i]);
        }
      if (tb + kC < t1) load_v(tb + kC);
      const float at = pre[kC - 1], at_lo = vec[7 * kC + 1];   // the product of the decays in two parts
      // the state is nearly all of this chunk's making: the mean that small_part() puts back is not enough
      const bool forgets = at < 0.00390625f;
      // B of 16 tokens x 16 dims, transposed on the way: lanes 0-15 tokens 0-15 of dims 0-7, lanes 16-31 of dims 8-15
      const uint32_t k_addr = sbase + kSmK + (lane & 15) * kRow + (lane >> 4) * 16;
#pragma unroll
      for (int np = 0; np < kDk / 32; ++np) {
        float ah[2][1][4][4] = {}, al[1][4][4] = {};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          uint32_t kf[3][4][2];
#pragma unroll
          for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int u = 0; u < 2; ++u)
              ldmatrix_x4_trans(reinterpret_cast<uint32_t(&)[4]>(kf[j][2 * u]), k_addr + ks * 16 * kRow + np * 64 + u * 32 + j * kPiece);
          mma6<1, 4>(ah[ks], al, wf[ks], kf);
          if (forgets) {   // what mma.sync cut off of hi.hi: the same products once more, on top of the negated sum
#pragma unroll
            for (int n = 0; n < 4; ++n) {
              float cut[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) cut[i] = -ah[ks][0][n][i];
              mma(cut, wf[ks][0][0], kf[0][n][0], kf[0][n][1]);
#pragma unroll
              for (int i = 0; i < 4; ++i) al[0][n][i] += cut[i];
            }
          } else
          {
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
              for (int i = 0; i < 4; ++i) al[0][n][i] = small_part(ah[ks][0][n][i], al[0][n][i]);
          }
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float s = S[4 * np + n][i];
            S[4 * np + n][i] = fmaf(s, at, (ah[0][0][n][i] + ah[1][0][n][i]) + fmaf(s, at_lo, al[0][n][i]));
          }
      }
    } else {
      // ---- token by token, as the general kernel does it ---------------------------------------------------------------
      for (int tt = 0; tt < cnt; ++tt) {
        const int64_t t = tb + tt;
        const float av = as[tt], bt = bs[tt];
        const float x0 = vh[t * a.ldv + r], x1 = vh[t * a.ldv + r + 8], b0 = bt * x0, b1 = bt * x1;
        const float* kr = kg + t * a.ldk + c2;
        const float* qr = qg + t * a.ldq + c2;
        float y0 = 0.f, y1 = 0.f;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          const float2 k2 = *reinterpret_cast<const float2*>(kr + 8 * n), q2 = *reinterpret_cast<const float2*>(qr + 8 * n);
          S[n][0] = fmaf(av, S[n][0], b0 * k2.x); y0 = fmaf(S[n][0], q2.x, y0);
          S[n][1] = fmaf(av, S[n][1], b0 * k2.y); y0 = fmaf(S[n][1], q2.y, y0);
          S[n][2] = fmaf(av, S[n][2], b1 * k2.x); y1 = fmaf(S[n][2], q2.x, y1);
          S[n][3] = fmaf(av, S[n][3], b1 * k2.y); y1 = fmaf(S[n][3], q2.y, y1);
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          y0 += __shfl_xor_sync(0xffffffffu, y0, o);
          y1 += __shfl_xor_sync(0xffffffffu, y1, o);
        }
        if (c2 == 0) {
          yh[t * a.ldy + r] = fmaf(d, x0, y0);
          yh[t * a.ldy + r + 8] = fmaf(d, x1, y1);
        }
      }
      if (tb + kC < t1) load_v(tb + kC);
    }
    __syncthreads();        // pieces, factors and the flag are free again
    if (tid == 0) *flag = 0u;
  }
#pragma unroll
  for (int n = 0; n < 16; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) sp[static_cast<int64_t>(8 * n + c2 + (i & 1)) * a.dv + r + (i >> 1) * 8] = S[n][i];
}

}  // namespace

// a CTA an SM at the most
static bool at_once(const RecArgs& a, int n_seqs) { return static_cast<int64_t>(a.heads) * n_seqs * (a.dv / kCols) <= sm_count(); }

// From 40 tokens a sequence on; from 16 on where all CTAs run at once and the steps' latency is what counts.  (32 x 33 tokens, two chunks
// each: 16 heads of 128 columns 78 us here, 77 token by token; 32 x 16 tokens, 64 heads of 64: 85 and 83; 2 x 40 tokens 21 and 30.)  One decoded
// token costs a chunk, 10 times a step.
bool linear_recurrence_chunked_applies(const RecArgs& a, int n_seqs, int n_tokens) {
  return a.dk == kDk && a.dv % kCols == 0 && static_cast<int64_t>(n_tokens) >= (at_once(a, n_seqs) ? 16 : 40) * static_cast<int64_t>(n_seqs) && n_seqs <= 65535 &&
         a.ldq % 4 == 0 && a.ldk % 4 == 0 && a.ldy % 2 == 0 && aligned16(a.q) && aligned16(a.k) && aligned16(a.y);
}

int linear_recurrence_chunked(const RecArgs& a, int n_seqs, cudaStream_t st) {
  NVLLM_SMEM_ATTR_ONCE(linear_recurrence_chunked_kernel<true>, kSmBytes);
  NVLLM_SMEM_ATTR_ONCE(linear_recurrence_chunked_kernel<false>, kSmBytes);
  const auto kern = at_once(a, n_seqs) ? linear_recurrence_chunked_kernel<false> : linear_recurrence_chunked_kernel<true>;   // (see the kernel)
  NVLLM_CUDA(launch_plain(kern, dim3(a.heads, n_seqs, a.dv / kCols), dim3(kWarps * 32), kSmBytes, st, a));
  NVLLM_LAUNCH_CHECK("linear_recurrence_chunked_kernel");
  return 0;
}

}  // namespace nvllm
