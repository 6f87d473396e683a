// delta_chunked.cu — the gated delta rule with a decay per key channel,  S <- diag(g_t) S,  u_t = beta_t (v_t - S^T k_t),  S <- S + k_t u_t^T,
// y_t = S^T q_t,  for prompts: 16 tokens at a time as matrix products and one triangular inverse.  With G_t = g_1 ... g_t (per channel, from
// the chunk's start; * and / per channel) and S the state before the chunk,
//   A_ij = beta_i (G_i * k_i) . (k_j / G_j)  (j < i),   X = V - (G * K) S,   U = beta X + ((I + A)^-1 - I) beta X,
//   y_i = (G_i * q_i)^T S + sum_(j <= i) ((G_i * q_i) . (k_j / G_j)) u_j,   S <- G_16 * S + sum_j (R_j * k_j) u_j^T,  R_j = g_(j+1) ... g_16.
// The quotients pair with products of the same channel, so every term carries G_i / G_j <= 1 whatever the decays are; only the range of f32
// limits them.  (R_j and not G_16 / G_j for the state: two roundings fewer in what stays.)
//
// Precision: as in recurrence_chunked.cu, three bf16 pieces and six products of every f32 operand, hi.hi summed apart.  What the state keeps is rounded
// as rarely as token by token: the inverse without its diagonal is small, so u is beta X with a small correction (solving for u
// column by column rounds every u fifteen times), and u, R * k and k / G are split from values in two parts.  Relative error of y and the
// state against 64 bits, token by token and here, 1e-7: decays per channel as the models make them 0.84, 0.95 and 0.67, 0.60; per head 0.81,
// 0.84 and 0.70, 0.61; near one 2.01, 3.09 and 0.83, 0.89; 0.6 a token 0.78, 0.66 and 0.72, 0.60; inputs of one sign 0.57, 1.01 and 0.55, 0.60.
// (With the solve per column and operands of one part: 0.93, 0.97; 0.97, 0.99; 1.10, 1.21; 1.00, 0.96; 0.73, 0.84; 10 % less time.)
// A chunk with a decay outside [0, 1] or a product of decays below 2^-90, or with a value that is no number, infinite or far from the
// others' range (q outside 2^-30 .. 2^30, k outside 2^-30 .. 2^8, beta, v or the state beyond 2^4, 2^20), or where U grows beyond 2^64 (keys
// far from unit vectors), is stepped through token by token in f32 by the warps that it concerns: what such a value reaches is then the same as
// in the general kernel.  (P is 0 where a token does not see a later one's u, but 0 x Inf is NaN.)
//
// CTA = (head, sequence, 64 columns of v), 4 warps; a warp keeps 16 columns of the state, transposed, in the accumulator layout of m16n8k16
// (64 registers), which is also that of the B operand of (G * K) S and (G * q) S.  q, k and the decays of the next chunk fly (cp.async) under the
// products of this one.  Bound by mma.sync issue (360 a warp and chunk) and the conversions around it; two CTAs an SM (94 KB each).
// Token by token and here, 16 heads of 128 x 128 (us): 8 x 1024 tokens 784 and 520, with a decay per head 692 and 525; 32 x 256 642 and 510, 32 x 16
// 60 and 46, 8 x 40 44 and 33.
#include "split_mma.cuh"

namespace nvllm {
namespace {

using namespace split;

constexpr int kC = 16, kDk = 128, kCols = 64, kWarps = 4;
constexpr int kRow = kDk * 2 + 16;               // bytes of a row of pieces: 16 more, so that ldmatrix rows fall into different banks
constexpr int kPiece = kC * kRow;
constexpr int kPs = 24;                          // floats of a row of A and P (8-byte reads of 4 rows of a quarter warp: 24 r + 2 c, no conflicts)
constexpr int kUs = 17;                          // floats of a row of a warp's X / U
constexpr int kSmRaw = 0;                        // q, k, g of a chunk as they come: [16][128] f32 each
constexpr int kSmQ = kSmRaw + 3 * kC * kDk * 4;  // G * q, G * k, k / G, R * k: three pieces each
constexpr int kSmKu = kSmQ + 3 * kPiece;
constexpr int kSmKd = kSmKu + 3 * kPiece;
constexpr int kSmKr = kSmKd + 3 * kPiece;
constexpr int kSmA = kSmKr + 3 * kPiece;         // A transposed: row j holds A_ij over i
constexpr int kSmP = kSmA + kC * kPs * 4;
constexpr int kSmU = kSmP + kC * kPs * 4;        // per warp [two parts][16 tokens][16 columns]
constexpr int kSmT = kSmU + kWarps * 2 * kC * kUs * 4;   // per warp: T beta below the diagonal
constexpr int kSmVec = kSmT + kWarps * kC * kPs * 4;   // floats: G_16 in two parts [2][128], beta [2][16], flag
constexpr int kSmBytes = kSmVec + (2 * kDk + 2 * kC) * 4 + 16;

template <bool HEADG>
__global__ void __launch_bounds__(kWarps * 32, 2) delta_chunked_kernel(const DeltaArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  float* raw = reinterpret_cast<float*>(smem + kSmRaw);
  float* At = reinterpret_cast<float*>(smem + kSmA);
  float* Pm = reinterpret_cast<float*>(smem + kSmP);
  float* gam = reinterpret_cast<float*>(smem + kSmVec);
  float* beta = gam + 2 * kDk;
  volatile uint32_t* flag = reinterpret_cast<volatile uint32_t*>(beta + 2 * kC);
  const int h = blockIdx.x, s = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col0 = blockIdx.z * kCols + warp * 16;       // the warp's first column of the head
  const int r = lane >> 2, c2 = (lane & 3) * 2;          // row and first column of the lane in an accumulator tile
  float* const U = reinterpret_cast<float*>(smem + kSmU) + warp * 2 * kC * kUs;
  float* const Ul = U + kC * kUs;
  float* const T = reinterpret_cast<float*>(smem + kSmT) + warp * kC * kPs;
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
  const float* const gh = a.decay + (HEADG ? h : static_cast<int64_t>(h) * kDk);

  // q, k, decays and beta of the chunk that starts at token tb; tokens past the end: zeros, decays of 1.  A thread copies one 16-byte piece of every
  // fourth row.
  auto issue = [&](int tb, int buf) {
    const uint32_t dst = smem_u32(raw + warp * kDk + lane * 4);
#pragma unroll
    for (int i = 0; i < kC / kWarps; ++i) {
      const bool in = tb + warp + i * kWarps < t1;
      const int64_t t = in ? tb + warp + i * kWarps : t0;
      cp_async_16(dst + i * kWarps * kDk * 4, qg + t * a.ldq + lane * 4, in ? 16 : 0);
      cp_async_16(dst + (kC + i * kWarps) * kDk * 4, kg + t * a.ldk + lane * 4, in ? 16 : 0);
      float4* const gd = reinterpret_cast<float4*>(raw + (2 * kC + warp + i * kWarps) * kDk + lane * 4);
      if (!in) *gd = make_float4(1.f, 1.f, 1.f, 1.f);
      else if (HEADG) { const float x = gh[t * a.ldd]; *gd = make_float4(x, x, x, x); }
      else cp_async_16(dst + (2 * kC + i * kWarps) * kDk * 4, gh + t * a.ldd + lane * 4, 16);
    }
    if (tid < kC) {
      float* b = beta + buf * kC + tid;
      if (tb + tid < t1) cp_async_4(smem_u32(b), a.beta + (tb + tid) * a.ldb + h); else *b = 0.f;
    }
    cp_async_commit();
  };
  // v of a chunk in accumulator order: tokens r, r + 8 (second index), columns 8 n + c2, + 1
  float2 vr[2][2];
  auto load_v = [&](int tb) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int n = 0; n < 2; ++n)
        vr[n][e] = tb + r + 8 * e < t1 ? *reinterpret_cast<const float2*>(vh + static_cast<int64_t>(tb + r + 8 * e) * a.ldv + 8 * n + c2) : make_float2(0.f, 0.f);
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

  int buf = 0;
  for (int tb = t0; tb < t1; tb += kC, buf ^= 1) {
    const int cnt = min(kC, t1 - tb);
    const float* bs = beta + buf * kC;
    cp_async_wait<0>();
    __syncthreads();
    // ---- operands: a thread takes two channels of 8 tokens ----------------------------------------------------------------
    bool bad = false;
    {
      const int ch = 2 * (tid & 63), first = (tid >> 6) * 8;
      // products of decays in two parts each
      float2 x[3][8], y[8], G = make_float2(1.f, 1.f), Gl = make_float2(0.f, 0.f), R = G, Rl = Gl;
      auto times = [](float2& hi, float2& lo, float2 g) {
        const float px = hi.x * g.x, py = hi.y * g.y;
        lo.x = fmaf(lo.x, g.x, fmaf(hi.x, g.x, -px));
        lo.y = fmaf(lo.y, g.y, fmaf(hi.y, g.y, -py));
        hi.x = px; hi.y = py;
      };
#pragma unroll
      for (int op = 0; op < 3; ++op)
#pragma unroll
        for (int i = 0; i < 8; ++i) x[op][i] = *reinterpret_cast<const float2*>(raw + (op * kC + first + i) * kDk + ch);
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] = *reinterpret_cast<const float2*>(raw + (2 * kC + 8 - first + i) * kDk + ch);   // the other half's decays
      if (first != 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) times(G, Gl, y[i]);
      } else {
#pragma unroll
        for (int i = 7; i >= 0; --i) times(R, Rl, y[i]);
      }
      auto put = [&](int operand, int i, const uint32_t (&p)[3]) {
        uint8_t* dst = smem + kSmQ + (first + i) * kRow + ch * 2;
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<uint32_t*>(dst + (3 * operand + j) * kPiece) = p[j];
      };
      uint32_t p[3];
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        const float2 k = x[1][i];      // R * k, the pieces of the unrounded value
        const float px = __fmul_rn(k.x, R.x), py = __fmul_rn(k.y, R.y);
        split3(px, py, fmaf(k.x, Rl.x, fmaf(k.x, R.x, -px)), fmaf(k.y, Rl.y, fmaf(k.y, R.y, -py)), p[0], p[1], p[2]);
        put(3, i, p);
        times(R, Rl, x[2][i]);
      }
      uint32_t most[2] = {0u, 0u};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        times(G, Gl, x[2][i]);
        bad |= !(x[2][i].x >= 0.f && x[2][i].x <= 1.f && x[2][i].y >= 0.f && x[2][i].y <= 1.f);
        const float2 P = make_float2(G.x + Gl.x, G.y + Gl.y);
#pragma unroll
        for (int op = 0; op < 2; ++op) {
          most[op] = max(most[op], max(abs_bits(x[op][i].x), abs_bits(x[op][i].y)));
          split3(x[op][i].x * P.x, x[op][i].y * P.y, p[0], p[1], p[2]);
          put(op, i, p);
        }
        // k / G: a quotient and, divided again, what it leaves over (the quotient of two-part numbers, Dekker 1971)
        const float2 k = x[1][i];
        const float qx = __fdividef(k.x, G.x), qy = __fdividef(k.y, G.y);
        split3(qx, qy, __fdividef(fmaf(-qx, Gl.x, fmaf(-qx, G.x, k.x)), G.x), __fdividef(fmaf(-qy, Gl.y, fmaf(-qy, G.y, k.y)), G.y), p[0], p[1], p[2]);
        put(2, i, p);
      }
      if (first != 0) {
        const float2 P = make_float2(G.x + Gl.x, G.y + Gl.y);
        *reinterpret_cast<float2*>(gam + ch) = P;
        *reinterpret_cast<float2*>(gam + kDk + ch) = make_float2((G.x - P.x) + Gl.x, (G.y - P.y) + Gl.y);
      }
      bad |= !(G.x >= 8.1e-28f && G.y >= 8.1e-28f);      // 2^-90
#pragma unroll
      for (int op = 0; op < 2; ++op) bad |= far_off(__reduce_max_sync(0xffffffffu, most[op]), -30, op == 0 ? 30 : 8);
      if (tid < kC) bad |= !(fabsf(bs[tid]) < 16.f);
    }
    if (bad) *flag = 1u;
    __syncthreads();
    const bool slow = *flag != 0u;
    if (tb + kC < t1) issue(tb + kC, buf ^ 1);
    const uint32_t a_addr = sbase + (lane & 15) * kRow + (lane >> 4) * 16;
    // ---- A (warps 0, 1) and P (warps 2, 3), 8 keys a warp --------------------------------------------------------------------
    if (!slow) {
      const int nt = warp & 1;
      float sum[4] = {}, hh[1][1][4], al[4][1][1][4] = {};
      // B of 8 keys x 16 dims: lanes 0-7 keys 0-7 dims 0-7, 8-15 the same keys dims 8-15 (the others repeat)
      const uint32_t k_addr = sbase + kSmKd + (nt * 8 + (lane & 7)) * kRow + ((lane >> 3) & 1) * 16;
#pragma unroll
      for (int kk = 0; kk < kDk / 16; ++kk) {
        uint32_t af[1][3][4], kf[3][1][2];
        if (kk % 2 == 0) zero(hh);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          ldmatrix_x4(af[0][j], a_addr + (warp < 2 ? kSmKu : kSmQ) + kk * 32 + j * kPiece);
          ldmatrix_x2(kf[j][0], k_addr + kk * 32 + j * kPiece);
        }
        mma6<1, 1>(hh, al[kk & 3], af, kf);
        if (kk % 2 == 1) {
#pragma unroll
          for (int i = 0; i < 4; ++i) sum[i] += hh[0][0][i];
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = r + (i >> 1) * 8, key = nt * 8 + c2 + (i & 1);
        const float x = join(sum[i], (al[0][0][0][i] + al[1][0][0][i]) + (al[2][0][0][i] + al[3][0][0][i]));
        if (warp < 2) At[key * kPs + row] = key < row ? bs[row] * x : 0.f;
        else Pm[row * kPs + key] = key <= row ? x : 0.f;
      }
    }
    // v and the state: their largest magnitude decides whether the warp takes the products
    float vmax = 0.f, smax[2];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) vmax = abs_max(vr[n][e].x, vr[n][e].y, vmax);
    smax[0] = vmax;
    smax[1] = 0.f;
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      smax[0] = abs_max(S[n][0], S[n][1], smax[0]);
      smax[1] = abs_max(S[n][2], S[n][3], smax[1]);
    }
    bool step = __any_sync(0xffffffffu, slow || !(smax[0] < 1.0e6f && smax[1] < 1.0e6f));      // 2^20: k / G reaches 2^98
    float sy[2][2][4] = {}, lo[2][2][4] = {};            // [G * k, G * q] . S in two parts: [16 tokens][8 columns]
    if (!step) {
      float hh[2][2][4];
#pragma unroll
      for (int kk = 0; kk < kDk / 16; ++kk) {
        if (kk % 2 == 0) zero(hh);
        uint32_t sf[3][2][2], af[2][3][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) split3(S[2 * kk + e][2 * n], S[2 * kk + e][2 * n + 1], sf[0][n][e], sf[1][n][e], sf[2][n][e]);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          ldmatrix_x4(af[0][j], a_addr + kSmKu + kk * 32 + j * kPiece);
          ldmatrix_x4(af[1][j], a_addr + kSmQ + kk * 32 + j * kPiece);
        }
        mma6<2, 2>(hh, lo, af, sf);
        if (kk % 2 == 1) {
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
              for (int i = 0; i < 4; ++i) sy[m][n][i] += hh[m][n][i];
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) lo[m][n][i] = small_part(sy[m][n][i], lo[m][n][i]);
      // X = V - (G * K) S, token by column
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 v = vr[n][i >> 1];
          U[(r + 8 * (i >> 1)) * kUs + 8 * n + c2 + (i & 1)] = ((i & 1 ? v.y : v.x) - sy[0][n][i]) - lo[0][n][i];
        }
    }
    __syncthreads();                   // A and P are complete
    if (!step) {
      // ---- T = (I + A)^-1, a lane per column; U = beta X + (T - I) beta X -----------------------------------------------------------
      {
        float u[kC];
        const int col = lane & 15;
#pragma unroll
        for (int i = 0; i < kC; ++i) u[i] = i == col ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < kC - 1; ++j) {
#pragma unroll
          for (int q4 = (j + 1) / 4; q4 < kC / 4; ++q4) {
            const float4 c = *reinterpret_cast<const float4*>(At + j * kPs + 4 * q4);
            if (4 * q4 > j) u[4 * q4] = fmaf(-c.x, u[j], u[4 * q4]);
            if (4 * q4 + 1 > j) u[4 * q4 + 1] = fmaf(-c.y, u[j], u[4 * q4 + 1]);
            if (4 * q4 + 2 > j) u[4 * q4 + 2] = fmaf(-c.z, u[j], u[4 * q4 + 2]);
            if (4 * q4 + 3 > j) u[4 * q4 + 3] = fmaf(-c.w, u[j], u[4 * q4 + 3]);
          }
        }
        const int half = (lane >> 4) * 8;      // the lower half of the lanes stores the first eight rows, the upper the others
        const float b = bs[col];
#pragma unroll
        for (int i = 0; i < 8; ++i) T[(half + i) * kPs + col] = half + i > col ? (half ? u[8 + i] : u[i]) * b : 0.f;
        __syncwarp();
      }
      {
        float hh[1][2][4] = {}, rest[1][2][4] = {};
        uint32_t tf[1][3][4], xf[3][2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 x = *reinterpret_cast<const float2*>(T + (r + (i & 1) * 8) * kPs + (i >> 1) * 8 + c2);
          split3(x.x, x.y, tf[0][0][i], tf[0][1][i], tf[0][2][i]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int at = (c2 + 8 * e) * kUs + r + 8 * n;
            split3(U[at], U[at + kUs], xf[0][n][e], xf[1][n][e], xf[2][n][e]);
          }
        mma6<1, 2>(hh, rest, tf, xf);
        __syncwarp();
        float umax = 0.f;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = r + 8 * (i >> 1), at = row * kUs + 8 * n + c2 + (i & 1);
            const float b = bs[row], x = U[at], p = __fmul_rn(b, x), e = fmaf(b, x, -p);
            float err;
            float u = two_sum(p, hh[0][n][i], err);
            u = two_sum(u, (err + e) + small_part(hh[0][n][i], rest[0][n][i]), err);
            U[at] = u;
            Ul[at] = err;
            umax = abs_max(u, u, umax);
          }
        step = __any_sync(0xffffffffu, !(umax < 1.8e19f));     // 2^64: P reaches 2^45
        __syncwarp();
      }
    }
    if (!step) {
      uint32_t uf[3][2][2], ua[1][3][4];   // U as B (16 tokens x 8 columns) and, the same values, U^T as A
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int at = (c2 + 8 * e) * kUs + r + 8 * n;
          split3(U[at], U[at + kUs], Ul[at], Ul[at + kUs], uf[0][n][e], uf[1][n][e], uf[2][n][e]);
#pragma unroll
          for (int j = 0; j < 3; ++j) ua[0][j][2 * e + n] = uf[j][n][e];
        }
      // ---- y ---------------------------------------------------------------------------------------------------------------
      {
        float hh[1][2][4] = {}, rest[1][2][4] = {};
        uint32_t pf[1][3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 x = *reinterpret_cast<const float2*>(Pm + (r + (i & 1) * 8) * kPs + (i >> 1) * 8 + c2);
          split3(x.x, x.y, pf[0][0][i], pf[0][1][i], pf[0][2][i]);
        }
        mma6<1, 2>(hh, rest, pf, uf);
        auto sum = [&](int n, int i) {
          float err;
          const float s1 = two_sum(sy[1][n][i], hh[0][n][i], err);
          return s1 + (err + (lo[1][n][i] + small_part(hh[0][n][i], rest[0][n][i])));
        };
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (r + 8 * e < cnt) {
#pragma unroll
            for (int n = 0; n < 2; ++n)
              *reinterpret_cast<float2*>(yh + static_cast<int64_t>(tb + r + 8 * e) * a.ldy + n * 8 + c2) = make_float2(sum(n, 2 * e), sum(n, 2 * e + 1));
          }
      }
      if (tb + kC < t1) load_v(tb + kC);
      // ---- state: S <- G_16 * S + sum_j (R_j * k_j) u_j^T ----------------------------------------------------------------------
      // B of 16 tokens x 16 dims, transposed on the way: lanes 0-15 tokens 0-15 of dims 0-7, lanes 16-31 of dims 8-15
#pragma unroll
      for (int np = 0; np < kDk / 32; ++np) {
        float hh[1][4][4] = {}, rest[1][4][4] = {};
        uint32_t kf[3][4][2];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int u = 0; u < 2; ++u)
            ldmatrix_x4_trans(reinterpret_cast<uint32_t(&)[4]>(kf[j][2 * u]), a_addr + kSmKr + np * 64 + u * 32 + j * kPiece);
        mma6<1, 4>(hh, rest, ua, kf);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const float2 G = *reinterpret_cast<const float2*>(gam + 8 * (4 * np + n) + c2), Gl = *reinterpret_cast<const float2*>(gam + kDk + 8 * (4 * np + n) + c2);
#pragma unroll
          for (int i = 0; i < 4; ++i) S[4 * np + n][i] = fmaf(S[4 * np + n][i], i & 1 ? G.y : G.x, fmaf(S[4 * np + n][i], i & 1 ? Gl.y : Gl.x, join(hh[0][n][i], rest[0][n][i])));
        }
      }
    } else {
      // ---- token by token, as the general kernel does it ---------------------------------------------------------------
      for (int tt = 0; tt < cnt; ++tt) {
        const int64_t t = tb + tt;
        const float bt = bs[tt], x0 = vh[t * a.ldv + r], x1 = vh[t * a.ldv + r + 8];
        const float* kr = kg + t * a.ldk + c2;
        const float* qr = qg + t * a.ldq + c2;
        const float* gr = HEADG ? gh + t * a.ldd : gh + t * a.ldd + c2;
        float rk0 = 0.f, rk1 = 0.f, rq0 = 0.f, rq1 = 0.f, kq = 0.f;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          const float2 k2 = *reinterpret_cast<const float2*>(kr + 8 * n), q2 = *reinterpret_cast<const float2*>(qr + 8 * n);
          const float2 g2 = HEADG ? make_float2(gr[0], gr[0]) : *reinterpret_cast<const float2*>(gr + 8 * n);
          kq = fmaf(k2.x, q2.x, fmaf(k2.y, q2.y, kq));
          S[n][0] *= g2.x; rk0 = fmaf(S[n][0], k2.x, rk0); rq0 = fmaf(S[n][0], q2.x, rq0);
          S[n][1] *= g2.y; rk0 = fmaf(S[n][1], k2.y, rk0); rq0 = fmaf(S[n][1], q2.y, rq0);
          S[n][2] *= g2.x; rk1 = fmaf(S[n][2], k2.x, rk1); rq1 = fmaf(S[n][2], q2.x, rq1);
          S[n][3] *= g2.y; rk1 = fmaf(S[n][3], k2.y, rk1); rq1 = fmaf(S[n][3], q2.y, rq1);
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          kq += __shfl_xor_sync(0xffffffffu, kq, o);
          rk0 += __shfl_xor_sync(0xffffffffu, rk0, o);
          rk1 += __shfl_xor_sync(0xffffffffu, rk1, o);
          rq0 += __shfl_xor_sync(0xffffffffu, rq0, o);
          rq1 += __shfl_xor_sync(0xffffffffu, rq1, o);
        }
        const float u0 = bt * (x0 - rk0), u1 = bt * (x1 - rk1);
        if (c2 == 0) {
          yh[t * a.ldy + r] = fmaf(u0, kq, rq0);
          yh[t * a.ldy + r + 8] = fmaf(u1, kq, rq1);
        }
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          const float2 k2 = *reinterpret_cast<const float2*>(kr + 8 * n);
          S[n][0] = fmaf(k2.x, u0, S[n][0]);
          S[n][1] = fmaf(k2.y, u0, S[n][1]);
          S[n][2] = fmaf(k2.x, u1, S[n][2]);
          S[n][3] = fmaf(k2.y, u1, S[n][3]);
        }
      }
      if (tb + kC < t1) load_v(tb + kC);
    }
    __syncthreads();        // pieces, A, P and the flag are free again
    if (tid == 0) *flag = 0u;
  }
#pragma unroll
  for (int n = 0; n < 16; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) sp[static_cast<int64_t>(8 * n + c2 + (i & 1)) * a.dv + r + (i >> 1) * 8] = S[n][i];
}

template <bool HEADG>
int launch(const DeltaArgs& a, int n_seqs, cudaStream_t st) {
  NVLLM_SMEM_ATTR_ONCE(delta_chunked_kernel<HEADG>, kSmBytes);
  NVLLM_CUDA(launch_plain(delta_chunked_kernel<HEADG>, dim3(a.heads, n_seqs, a.dv / kCols), dim3(kWarps * 32), kSmBytes, st, a));
  NVLLM_LAUNCH_CHECK("delta_chunked_kernel");
  return 0;
}

}  // namespace

// Where the CTAs take half the SMs at the least: fewer wait for a chunk's chain of phases as long as for its 16 steps (one prompt of 8192 tokens
// 2.68 and 2.69 ms, 2 x 40 tokens 25 and 24 us).  From 16 tokens a sequence on, if they fill three quarters of their chunks (five sixths with a decay
// per head, where the steps load less): a chunk takes its time however few its tokens are.  Token by token and here (us), 16 heads of 128 x 128, 32
// sequences, a decay per channel: 16 tokens 58 and 43, 17 62 and 75, 23 76 and 75, 24 79 and 75, 33 101 and 106, 36 108 and 106, 49 141 and 138;
// per head: 17 57 and 75, 24 71 and 76, 28 81 and 76, 33 92 and 108, 40 108 and 108, 49 128 and 138, 56 143 and 139, 65 163 and 171, 80 196 and 171;
// 5 and 16 sequences have the same crossings.  (Of a batch of mixed lengths only the mean is known here.)  One decoded token costs a chunk.
bool delta_chunked_applies(const DeltaArgs& a, bool head_decay, int n_seqs, int n_tokens) {
  const int64_t per_chunk = kC * static_cast<int64_t>(n_seqs), chunks = (n_tokens + per_chunk - 1) / per_chunk;   // of a sequence of the mean length
  const bool full = head_decay ? 6 * static_cast<int64_t>(n_tokens) >= 5 * chunks * per_chunk : 4 * static_cast<int64_t>(n_tokens) >= 3 * chunks * per_chunk;
  return a.dk == kDk && a.dv % kCols == 0 && 2 * static_cast<int64_t>(a.heads) * n_seqs * (a.dv / kCols) >= sm_count() && n_tokens >= per_chunk && full &&
         n_seqs <= 65535 && a.ldq % 4 == 0 && a.ldk % 4 == 0 && a.ldv % 2 == 0 && a.ldy % 2 == 0 && aligned16(a.q) && aligned16(a.k) && aligned16(a.v) &&
         aligned16(a.y) && (head_decay || (a.ldd % 4 == 0 && aligned16(a.decay)));
}

int delta_chunked(const DeltaArgs& a, bool head_decay, int n_seqs, cudaStream_t st) {
  return head_decay ? launch<true>(a, n_seqs, st) : launch<false>(a, n_seqs, st);
}

}  // namespace nvllm
