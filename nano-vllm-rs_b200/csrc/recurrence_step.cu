// recurrence_step.cu — the recurrences of recurrence.cu over steps of single tokens (as many tokens as sequences), keys of 128 values.
//
// Such a step reads and writes every state once and does next to nothing with it: it is bound by HBM, and by how soon the state is asked for.
// CTA = (head, sequence, slice of COLS value columns), 256 threads; a thread holds 4 neighbouring columns of every (1024 / COLS)-th row, so
// that a warp reads whole 128- to 512-byte pieces of rows in 16-byte accesses, all of them in flight before anything else is waited for (the
// kernel for prompts reads 4 bytes a lane and stages 16 tokens' rows in shared memory first).  The rows' sums meet by shuffles and, over
// the 8 warps, in shared memory in fixed order.  A sequence that does have several tokens is walked through with its state in registers.
// Measured (us, launched one by one, some 6 us of which are the launch), the kernel for prompts and this one: 64 sequences x 64 heads of 128 x 64
// (268 MB, 41 at the copy rate) 79 and 52, 64 x 16 heads of 128 x 128 44 and 31, the delta rule there 47 and 29; one sequence, 64 heads of
// 128 x 64 15 and 8, the delta rule with 16 heads of 128 x 128 12 and 8.
#include "recurrence.cuh"

namespace nvllm {
namespace {

constexpr int kDk = 128, kThreads = 256, kWarps = 8;

// What the linear recurrences and the delta rules have in common; linear: step and skip; delta: beta in the place of step.
struct StepArgs {
  float* y; int64_t ldy;
  const float *q, *k, *v; int64_t ldq, ldk, ldv;
  int group_div;
  const float* decay; int64_t decay_ld;   // a value per head (row decay_ld apart, or one row for all), or per head and key channel
  const float* step; int64_t step_ld;
  const float* skip;
  float* state;
  const int32_t *seq_slot, *cu_tokens; const int64_t* positions;
  int heads, dv;
  float q_scale;
};

// (128 columns: two CTAs an SM; left to itself the compiler may take a few registers too many for that, and 256 sequences of the delta rule with 16 heads
// of 128 x 128 take 141 us instead of 100)
template <bool DELTA, bool CHANNEL, int COLS>
__global__ void __launch_bounds__(kThreads, COLS == 128 ? 2 : 0) recurrence_step_kernel(const StepArgs a) {
  constexpr int CT = COLS / 4, RG = kThreads / CT, R = kDk / RG;   // threads of a row, row groups, rows of a thread
  __shared__ float ks[kDk], qs[kDk], gs[CHANNEL ? kDk : 1];
  __shared__ __align__(16) float vs[COLS];
  __shared__ float4 red[DELTA ? 2 : 1][kWarps][CT];
  __shared__ float kq_s[kWarps];
  pdl_wait();
  pdl_launch_dependents();
  const int h = blockIdx.x, s = blockIdx.y, p0 = blockIdx.z * COLS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = tid % CT, rg = tid / CT;
  const int t0 = a.cu_tokens[s], t1 = a.cu_tokens[s + 1], slot = a.seq_slot[s];
  if (t1 <= t0) return;
  if (slot < 0) {  // padding sequence of a captured batch: defined output, no state
    for (int t = t0; t < t1; ++t)
      if (tid < COLS) a.y[t * a.ldy + static_cast<int64_t>(h) * a.dv + p0 + tid] = 0.f;
    return;
  }
  float4* sp = reinterpret_cast<float4*>(a.state + (static_cast<int64_t>(slot) * a.heads + h) * kDk * a.dv + p0) + c;
  const int64_t pitch = a.dv / 4;   // of a state's row
  float4 S[R];
  if (a.positions[t0] != 0) {
#pragma unroll
    for (int i = 0; i < R; ++i) S[i] = sp[(rg + i * RG) * pitch];
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i) S[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int64_t g = h / a.group_div;
  const float d = !DELTA && a.skip ? a.skip[h] : 0.f;
  for (int t = t0; t < t1; ++t) {
    if (t > t0) __syncthreads();   // the token before is done with the shared rows
    if (tid < kDk) {
      ks[tid] = a.k[t * a.ldk + g * kDk + tid];
      if (CHANNEL) gs[tid] = a.decay[t * a.decay_ld + static_cast<int64_t>(h) * kDk + tid];
    } else {
      qs[tid - kDk] = a.q[t * a.ldq + g * kDk + tid - kDk];
    }
    if (tid < COLS) vs[tid] = a.v[t * a.ldv + static_cast<int64_t>(h) * a.dv + p0 + tid];
    const float gh = CHANNEL ? 0.f : a.decay[t * a.decay_ld + h], bt = a.step ? a.step[t * a.step_ld + h] : 1.f;
    __syncthreads();
    const float4 v = *reinterpret_cast<const float4*>(vs + 4 * c);
    float4 rk = make_float4(0.f, 0.f, 0.f, 0.f), rq = rk;   // S^T k (delta rule) and S^T q over this thread's rows
    float kq = 0.f;
    const float4 bv = make_float4(bt * v.x, bt * v.y, bt * v.z, bt * v.w);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int n = rg + i * RG;
      const float kn = ks[n], qn = qs[n], gn = CHANNEL ? gs[n] : gh;
      if (DELTA) {
        S[i] = make_float4(S[i].x * gn, S[i].y * gn, S[i].z * gn, S[i].w * gn);
        rk = make_float4(fmaf(S[i].x, kn, rk.x), fmaf(S[i].y, kn, rk.y), fmaf(S[i].z, kn, rk.z), fmaf(S[i].w, kn, rk.w));
        kq = fmaf(kn, qn, kq);
      } else {
        S[i] = make_float4(fmaf(gn, S[i].x, bv.x * kn), fmaf(gn, S[i].y, bv.y * kn), fmaf(gn, S[i].z, bv.z * kn), fmaf(gn, S[i].w, bv.w * kn));
      }
      rq = make_float4(fmaf(S[i].x, qn, rq.x), fmaf(S[i].y, qn, rq.y), fmaf(S[i].z, qn, rq.z), fmaf(S[i].w, qn, rq.w));
    }
    auto rows = [](float x) {   // over the row groups of a warp
#pragma unroll
      for (int o = CT; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      return x;
    };
    rq = make_float4(rows(rq.x), rows(rq.y), rows(rq.z), rows(rq.w));
    if (DELTA) {
      rk = make_float4(rows(rk.x), rows(rk.y), rows(rk.z), rows(rk.w));
      kq = rows(kq);
      if (lane == 0) kq_s[warp] = kq;
    }
    if (lane < CT) {
      red[0][warp][lane] = rq;
      if (DELTA) red[DELTA ? 1 : 0][warp][lane] = rk;
    }
    __syncthreads();
    auto warps = [&](int which, int at) {
      float4 x = red[which][0][at];
#pragma unroll
      for (int w = 1; w < kWarps; ++w) {
        const float4 o = red[which][w][at];
        x = make_float4(x.x + o.x, x.y + o.y, x.z + o.z, x.w + o.w);
      }
      return x;
    };
    float* y = a.y + t * a.ldy + static_cast<int64_t>(h) * a.dv + p0 + 4 * c;
    if (DELTA) {
      const float4 sk = warps(DELTA ? 1 : 0, c);
      const float4 u = make_float4(bt * (v.x - sk.x), bt * (v.y - sk.y), bt * (v.z - sk.z), bt * (v.w - sk.w));
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float kn = ks[rg + i * RG];
        S[i] = make_float4(fmaf(kn, u.x, S[i].x), fmaf(kn, u.y, S[i].y), fmaf(kn, u.z, S[i].z), fmaf(kn, u.w, S[i].w));
      }
      if (rg == 0) {   // the read-out of the updated state: S^T q + u (k . q)
        float all = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) all += kq_s[w];
        const float4 sq = warps(0, c);
        y[0] = fmaf(u.x, all, sq.x); y[1] = fmaf(u.y, all, sq.y); y[2] = fmaf(u.z, all, sq.z); y[3] = fmaf(u.w, all, sq.w);
      }
    } else if (rg == 0) {
      const float4 sq = warps(0, c);
      y[0] = fmaf(d, v.x, sq.x * a.q_scale); y[1] = fmaf(d, v.y, sq.y * a.q_scale);
      y[2] = fmaf(d, v.z, sq.z * a.q_scale); y[3] = fmaf(d, v.w, sq.w * a.q_scale);
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) sp[(rg + i * RG) * pitch] = S[i];
}

template <bool DELTA, bool CHANNEL>
int launch(const StepArgs& a, int n_seqs, cudaStream_t st) {
  // slices as wide as the columns divide and two CTAs an SM allow: whole rows are the longest reads
  int cols = a.dv % 128 == 0 ? 128 : (a.dv % 64 == 0 ? 64 : 32);
  while (cols > 32 && static_cast<int64_t>(a.heads) * n_seqs * (a.dv / cols) < 2 * sm_count()) cols /= 2;
  auto kern = cols == 128 ? recurrence_step_kernel<DELTA, CHANNEL, 128>
                          : (cols == 64 ? recurrence_step_kernel<DELTA, CHANNEL, 64> : recurrence_step_kernel<DELTA, CHANNEL, 32>);
  NVLLM_CUDA(launch_pdl(kern, dim3(a.heads, n_seqs, a.dv / cols), dim3(kThreads), 0, st, a));
  NVLLM_LAUNCH_CHECK("recurrence_step_kernel");
  return 0;
}

bool applies(const float* state, int dk, int dv, int n_seqs, int n_tokens) {
  return n_tokens == n_seqs && n_seqs <= 65535 && dk == kDk && dv % 32 == 0 && dv / 32 <= 65535 && aligned16(state);
}

}  // namespace

bool linear_recurrence_single_applies(const RecArgs& a, int n_seqs, int n_tokens) { return applies(a.state, a.dk, a.dv, n_seqs, n_tokens); }
int linear_recurrence_single(const RecArgs& a, int n_seqs, cudaStream_t st) {
  const StepArgs b{a.y, a.ldy, a.q, a.k, a.v, a.ldq, a.ldk, a.ldv, a.group_div, a.decay, a.decay_ld, a.step, a.step_ld, a.skip, a.state, a.seq_slot,
                   a.cu_tokens, a.positions, a.heads, a.dv, a.q_scale};
  return launch<false, false>(b, n_seqs, st);
}

bool delta_single_applies(const DeltaArgs& a, int n_seqs, int n_tokens) { return applies(a.state, a.dk, a.dv, n_seqs, n_tokens); }
int delta_single(const DeltaArgs& a, bool head_decay, int n_seqs, cudaStream_t st) {
  const StepArgs b{a.y, a.ldy, a.q, a.k, a.v, a.ldq, a.ldk, a.ldv, a.group_div, a.decay, a.ldd, a.beta, a.ldb, nullptr, a.state, a.seq_slot,
                   a.cu_tokens, a.positions, a.heads, a.dv, 1.0f};
  return head_decay ? launch<true, false>(b, n_seqs, st) : launch<true, true>(b, n_seqs, st);
}

}  // namespace nvllm
