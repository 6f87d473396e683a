// sampler.cu — K12: Sampler::forward / sample_single (reference src/layers/sampler.rs:26-219) on the device.
//
// The reference samples one row at a time on the host: a blocking scalar read per parameter, two full sorts of the
// vocabulary (top-k, top-p), a softmax and an unseeded Tensor::rand.  Here one CTA owns one row of the f32 logits and
// never sorts: both filters are *selections*, done MSB-first over the order-preserving integer image of the scaled
// logits with shared-memory histograms (3 passes each over 8 + 12 + 12 key bits, 16-byte loads, warp-aggregated updates):
//   top-k  (sampler.rs:115-149)  k-th largest key by COUNT; ties at the threshold keep the lowest indices (the
//                                reference's stable sort), resolved by an ordered ballot scan only when they straddle k
//   top-p  (sampler.rs:152-191)  smallest prefix of the descending order whose probability mass reaches p, found by
//                                MASS: exp(s - max) in 0.32 fixed point, so every sum is an integer sum (order-free,
//                                deterministic); target = ceil(p * total)
//   Gumbel-max (sampler.rs:194-219) argmax(s + g), g = -log(-log(u)), first maximum wins
// Rows with temperature == 0 take the same final pass without filters or noise (greedy, sampler.rs:79-81,109-112).
// Seeded contract for u (the reference's draws are unseeded and cannot be reproduced): see oracle/layers.py.
// HBM/L2-bound integer + compare work; no tensor cores.
//
// Two short cuts carry the ordinary cases; both select exactly what the radix selection selects, and leave anything unusual
// (NaN or huge values, more candidates than fit, k beyond kShortK) to it:
//   top-k (and top-p behind it)  the k-th largest of the threads' maxima over a sample of the row is a lower bound of the k-th
//                largest value, so ONE pass collects the few hundred values that reach it; ranking, mass and noise then touch
//                those alone.
//   top-p alone  the masses are binned by distance from the maximum (4096 linear bins: neighbouring values spread over bins
//                instead of meeting in one exponent), and only the bin in which the mass reaches p is ranked.
// The radix selection reads the row 3 times per filter and is bound by warp-wide matches in front of its histogram, not by
// memory.  Measured, 256 rows x 151936 f32 (156 MB, 23 us at the copy rate) with top-k 50 and top-p 0.9: 870 us with the radix
// selection, 49 us with the candidates (the row is read once, an eighth of it twice).
#include <math.h>

#include "common.cuh"

namespace nvllm {
namespace {

// A row per CTA: 1024 threads while every row has an SM to itself (148 rows x 151936 without filters: 82 us, with 512 threads 91;
// 32768 values 24 against 41), two CTAs of 512 on an SM beyond that (256 rows x 151936: 140 us).
constexpr int kMaxThreads = 1024;
constexpr int kBins = 4096;  // three selection passes over 8 + 12 + 12 key bits (see radix_select)
constexpr uint64_t kGolden = 0x9E3779B97F4A7C15ull;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27; x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return x;
}
// order-preserving float -> uint32 (larger float <=> larger key); -0 is folded onto +0 first
__device__ __forceinline__ uint32_t okey(float f) {
  const uint32_t u = __float_as_uint(f + 0.0f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float okey_inv(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
__device__ __forceinline__ float scaled(float x, float T) { return T == 1.0f ? x : __fdiv_rn(x, T); }  // sampler.rs:84-88
// exp(s - m) in 0.32 fixed point (s <= m): [0, 2^32 - 1] — the maximum itself is capped one unit below 2^32 so that a
// weight fits 32 bits (two 16-bit warp reductions per histogram update)
__device__ __forceinline__ uint32_t fx_exp(float s, float m) {
  const unsigned long long w = __float2ull_rz(expf(s - m) * 4294967296.0f);
  return w > 0xffffffffull ? 0xffffffffu : static_cast<uint32_t>(w);
}

// keep(key, i) <=> key > sel.key || (key == sel.key && i <= sel.cut)
struct Sel {
  uint32_t key, cut;
};
__device__ __forceinline__ bool keeps(const Sel& s, uint32_t key, uint32_t i) {
  return key > s.key || (key == s.key && i <= s.cut);
}

constexpr int kCand = 4096;    // candidates the short cuts rank (they share the histogram's memory)
constexpr int kShortK = 256;   // largest k of the candidate short cut: expected candidates are ~10 k

struct Shared {
  unsigned long long hist[kBins];   // or the candidates, (~key, index) packed so that ascending order is the descending order of the row
  unsigned long long need, eq;
  float redf[32];
  int redi[32];
  uint32_t cnt[kMaxThreads / 32];
  int sel_bin;
  uint32_t cut;
  int ncand, odd;
  uint32_t kmin, kmax;
};
static_assert(kCand <= kBins, "the candidates share the histogram's memory");

// Visits the row with 16-byte loads (two in flight per thread).  f(v, i0, n): v[0..n) are elements i0 .. i0+n-1; f is
// called the SAME number of times by every thread of the CTA (n == 0 for idle slots), so it may use full-warp intrinsics.
template <int NTH, typename F>
__device__ __forceinline__ void for_each4(const float* __restrict__ row, int V, F f) {
  const int tid = threadIdx.x;
  if ((reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
    const int nvec = V >> 2;
    const float4* r4 = reinterpret_cast<const float4*>(row);
    for (int base = 0; base < nvec; base += 2 * NTH) {
      const int j0 = base + tid, j1 = j0 + NTH;
      float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
      if (j0 < nvec) q0 = __ldg(r4 + j0);
      if (j1 < nvec) q1 = __ldg(r4 + j1);
      const float v0[4] = {q0.x, q0.y, q0.z, q0.w}, v1[4] = {q1.x, q1.y, q1.z, q1.w};
      f(v0, 4 * j0, j0 < nvec ? 4 : 0);
      if (base + NTH < nvec) f(v1, 4 * j1, j1 < nvec ? 4 : 0);  // block-uniform condition
    }
    const int t0 = nvec << 2;
    if (t0 < V) {  // V % 4 trailing elements: thread 0 takes them, everybody makes the call
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      int n = 0;
      if (tid == 0) { n = V - t0; for (int e = 0; e < n; ++e) v[e] = row[t0 + e]; }
      f(v, t0, n);
    }
  } else {
    for (int base = 0; base < V; base += NTH) {
      const int i = base + tid;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (i < V) v[0] = row[i];
      f(v, i, i < V ? 1 : 0);
    }
  }
}

// MSB-first radix selection over the keys of one row, largest first, 8 + 12 + 12 bits.  weight(key, i) is the element's
// contribution (0 = not a candidate).  Finds the key K with  sum{w : key > K} < target <= sum{w : key >= K}  and returns
// how much of the target the group key == K has to supply (`need`, >= 1) and that group's total weight (`eq`).
// MASS == true: weights are 32-bit masses and the target is ceil(p * total), fixed after the first pass; MASS == false:
// weights are 0/1.  Histogram updates are aggregated per warp (match_any on the bin: logits cluster in a handful of
// exponent bins, un-aggregated shared-memory atomics serialise on them).  row_max (optional) receives max(scaled row).
template <int NTH, bool MASS, typename WF>
__device__ void radix_select(Shared& sh, const float* __restrict__ row, int V, float T, WF weight, unsigned long long target,
                             double p, uint32_t& out_key, unsigned long long& out_need, unsigned long long& out_eq,
                             float* row_max) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t prefix = 0, mask = 0;
  unsigned long long rem = target;
  float mx = -INFINITY;
#pragma unroll 1
  for (int pass = 0; pass < 3; ++pass) {
    // First digit = sign + 7 exponent bits only: every element takes part in the first pass, and the warp-aggregated
    // update costs ~ the number of DISTINCT bins in a warp (a handful at this width); later passes see few candidates.
    const int shift = pass == 0 ? 24 : (pass == 1 ? 12 : 0);
    const int nbins = pass == 0 ? 256 : 4096;
    for (int b = tid; b < nbins; b += NTH) sh.hist[b] = 0ull;
    __syncthreads();
    for_each4<NTH>(row, V, [&](const float (&v)[4], int i0, int n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        bool part = e < n;
        const float s = scaled(v[e], T);
        const uint32_t key = okey(s);
        if (pass == 0 && row_max != nullptr && part) mx = fmaxf(mx, s);
        part = part && (key & mask) == prefix;
        const uint32_t w = part ? static_cast<uint32_t>(weight(key, static_cast<uint32_t>(i0 + e))) : 0u;
        part = part && w != 0u;
        if (__any_sync(kFull, part)) {
          const uint32_t bin = part ? ((key >> shift) & static_cast<uint32_t>(nbins - 1)) : 0xffffffffu;
          const unsigned peers = __match_any_sync(kFull, bin);
          unsigned long long sum;
          if (MASS) {
            const uint32_t lo = __reduce_add_sync(peers, w & 0xffffu), hi = __reduce_add_sync(peers, w >> 16);
            sum = (static_cast<unsigned long long>(hi) << 16) + lo;
          } else {
            sum = static_cast<unsigned long long>(__popc(peers));
          }
          if (part && lane == __ffs(peers) - 1) atomicAdd(&sh.hist[bin], sum);
        }
      }
    });
    __syncthreads();
    if (warp == 0) {  // lane l owns bins nbins-1-per*l .. nbins-per*(l+1), scanned from the top
      const int per = nbins / 32, top = nbins - 1 - per * lane;
      unsigned long long s = 0ull;
      for (int j = 0; j < per; ++j) s += sh.hist[top - j];
      unsigned long long incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
      }
      const unsigned long long total = __shfl_sync(kFull, incl, 31);
      if (MASS && pass == 0) {
        const double t = ceil(p * static_cast<double>(total));
        rem = t < 1.0 ? 1ull : static_cast<unsigned long long>(t);
      }
      if (rem > total) rem = total;  // cannot happen for valid inputs; keeps the search well defined
      if (rem < 1ull) rem = 1ull;
      if (total == 0ull && lane == 0) { sh.sel_bin = 0; sh.need = 1ull; sh.eq = 0ull; }  // no candidate at all
      const unsigned long long excl = incl - s;
      if (excl < rem && rem <= incl) {  // exactly one lane
        unsigned long long c = excl;
        for (int j = 0; j < per; ++j) {
          const unsigned long long h = sh.hist[top - j];
          if (c + h >= rem) { sh.sel_bin = top - j; sh.need = rem - c; sh.eq = h; break; }
          c += h;
        }
      }
    }
    __syncthreads();
    prefix |= static_cast<uint32_t>(sh.sel_bin) << shift;
    mask |= static_cast<uint32_t>(nbins - 1) << shift;
    rem = sh.need;
    out_eq = sh.eq;
    __syncthreads();
  }
  out_key = prefix;
  out_need = rem;
  if (row_max != nullptr) *row_max = mx;  // per-thread partial; the caller reduces it
}

// Smallest index I with #{i <= I : pred(i)} == need (pred true for at least `need` elements).  Each warp counts a
// contiguous chunk with ballots, the warp holding the need-th match walks its chunk again.
template <int NTH, typename PF>
__device__ uint32_t ordered_cut(Shared& sh, int V, PF pred, uint32_t need) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = ((V + (NTH / 32) - 1) / (NTH / 32) + 31) & ~31;
  const int start = warp * chunk, end = min(V, start + chunk);
  uint32_t cnt = 0;
  for (int base = start; base < end; base += 32) {
    const int i = base + lane;
    cnt += __popc(__ballot_sync(kFull, i < end && pred(static_cast<uint32_t>(i))));
  }
  if (lane == 0) sh.cnt[warp] = cnt;
  if (tid == 0) sh.cut = 0xffffffffu;
  __syncthreads();
  uint32_t run = 0;
  int wsel = -1;
  for (int w = 0; w < (NTH / 32); ++w) {
    if (wsel < 0) {
      if (run + sh.cnt[w] >= need) wsel = w; else run += sh.cnt[w];
    }
  }
  if (warp == wsel) {
    uint32_t c = run;
    for (int base = start; base < end; base += 32) {
      const int i = base + lane;
      const bool p = i < end && pred(static_cast<uint32_t>(i));
      const unsigned bal = __ballot_sync(kFull, p);
      const uint32_t n = __popc(bal);
      if (c + n >= need) {
        const uint32_t r = need - c;  // 1-based rank inside this ballot
        if (p && static_cast<uint32_t>(__popc(bal & (kFull >> (31 - lane)))) == r) sh.cut = static_cast<uint32_t>(i);
        break;
      }
      c += n;
    }
  }
  __syncthreads();
  const uint32_t cut = sh.cut;
  __syncthreads();
  return cut;
}

// Sorts sh.hist[0 .. n) ascending (n <= kCand), bitonic over the next power of two.
template <int NTH>
__device__ void sort_candidates(Shared& sh, int n) {
  const int tid = threadIdx.x;
  int n2 = 2;
  while (n2 < n) n2 <<= 1;
  for (int i = n + tid; i < n2; i += NTH) sh.hist[i] = ~0ull;
  __syncthreads();
  for (int size = 2; size <= n2; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = tid; i < n2 / 2; i += NTH) {
        const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
        const bool up = (lo & size) == 0;
        const unsigned long long x = sh.hist[lo], y = sh.hist[hi];
        if ((x > y) == up) { sh.hist[lo] = y; sh.hist[hi] = x; }
      }
      __syncthreads();
    }
}
__device__ __forceinline__ unsigned long long pack_candidate(uint32_t key, uint32_t i) {
  return (static_cast<unsigned long long>(~key) << 32) | i;
}
__device__ __forceinline__ uint32_t candidate_key(unsigned long long c) { return ~static_cast<uint32_t>(c >> 32); }

// Position (in the sorted candidates 0 .. n - 1) of the first one at which the summed mass reaches `need`; the mass of candidate
// j is fx_exp(value - m).  Every thread returns it.
__device__ int mass_position(Shared& sh, int n, float m, unsigned long long need, bool from_share, double p) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (warp == 0) {
    unsigned long long total = 0ull;
    if (from_share) {   // need = ceil(p * total)
      for (int j = lane; j < n; j += 32) total += fx_exp(okey_inv(candidate_key(sh.hist[j])), m);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(kFull, total, o);
      const double t = ceil(p * static_cast<double>(total));
      need = t < 1.0 ? 1ull : static_cast<unsigned long long>(t);
      if (need > total) need = total;
      if (need < 1ull) need = 1ull;
    }
    unsigned long long run = 0ull;
    int pos = n - 1;
    for (int base = 0; base < n; base += 32) {
      const int j = base + lane;
      unsigned long long w = j < n ? fx_exp(okey_inv(candidate_key(sh.hist[j])), m) : 0ull;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, w, o);
        if (lane >= o) w += t;
      }
      const unsigned hit = __ballot_sync(kFull, j < n && run + w >= need);
      if (hit) { pos = base + __ffs(hit) - 1; break; }
      run += __shfl_sync(kFull, w, 31);
    }
    if (lane == 0) sh.sel_bin = pos;
  }
  __syncthreads();
  const int pos = sh.sel_bin;
  __syncthreads();
  return pos;
}

// Visits the row like for_each4 with four loads in flight per thread; f(v, i0, n) may be called different numbers of times by
// different threads.  Blocks of 4 NTH values; every `step`-th block is visited (1: all of them).
template <int NTH, typename F>
__device__ __forceinline__ void for_each4_free(const float* __restrict__ row, int V, int step, F f) {
  const int tid = threadIdx.x;
  if ((reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
    const int nvec = V >> 2;
    const float4* r4 = reinterpret_cast<const float4*>(row);
    int j = tid;
    const int hop = step * NTH;
    for (; j + 3 * hop < nvec; j += 4 * hop) {
      float4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = __ldg(r4 + j + u * hop);
#pragma unroll
      for (int u = 0; u < 4; ++u) { const float v[4] = {q[u].x, q[u].y, q[u].z, q[u].w}; f(v, 4 * (j + u * hop), 4); }
    }
    for (; j < nvec; j += hop) { const float4 q = __ldg(r4 + j); const float v[4] = {q.x, q.y, q.z, q.w}; f(v, 4 * j, 4); }
    const int t0 = nvec << 2;
    if (step == 1 && t0 + tid < V) { const float v[4] = {row[t0 + tid], 0.f, 0.f, 0.f}; f(v, t0 + tid, 1); }
  } else {
    for (int i = tid; i < V; i += step * NTH) { const float v[4] = {row[i], 0.f, 0.f, 0.f}; f(v, i, 1); }
  }
}

// (apart: beside the rest it costs every launch 0.2 us, taken or not)
__device__ __noinline__ uint32_t bound_low_bits(uint32_t mine, uint32_t t, int k) {
#pragma unroll 1
  for (int b = 12; b >= 0; --b) {
    const uint32_t mid = t | (1u << b);
    if (__syncthreads_count(mine >= mid) >= k) t = mid;
  }
  return t;
}

// The candidates of top-k: every value that can be among the k largest SCALED ones, ranked in sh.hist.  Returns their number,
// or 0 when the row is one for the radix selection.  T > 0.
template <int NTH>
__device__ int rank_top_k(Shared& sh, const float* __restrict__ row, int V, float T, int k) {
  const int tid = threadIdx.x;
  if (!(T >= 9.5e-7f && T <= 1.05e6f)) return 0;   // values stay normal numbers under the division (with the bound on t below)
  // the k-th largest of the threads' maxima over every 8th block (short rows: all of it): k values of the row reach it
  const int step = V >= 65536 ? 8 : (V >= 16384 ? 2 : 1);
  float mx = -INFINITY;
  for_each4_free<NTH>(row, V, step, [&](const float (&v)[4], int, int n) {
    mx = fmaxf(mx, v[0]);
    if (n == 4) mx = fmaxf(mx, fmaxf(v[1], fmaxf(v[2], v[3])));
  });
  const uint32_t mine = okey(mx);
  uint32_t t = 0;
#pragma unroll 1
  for (int b = 31; b >= 13; --b) {
    const uint32_t mid = t | (1u << b);
    if (__syncthreads_count(mine >= mid) >= k) t = mid;
  }
  if (tid == 0) { sh.ncand = 0; sh.odd = 0; }
  // The low 13 bits, 2^-10 of the value, cost a barrier each and mostly spare a few candidates.  Where many more maxima than k reach t the values lie so
  // close that they do count (10 +- 0.01, 256 x 151936, top-k of 50: 64 us without them, 44 with them).
  if (__syncthreads_count(mine >= t) > k + k / 8 + 4) t = bound_low_bits(mine, t, k);
  // Two values 5 or more units in the last place apart cannot meet in one quotient: values that much below t are out whatever
  // the ties of the scaled row (t and the quotients are normal numbers).
  const float tf = okey_inv(t - 4u);
  if (!(fabsf(tf) >= 1e-30f && fabsf(tf) <= 1e30f)) return 0;
  for_each4_free<NTH>(row, V, 1, [&](const float (&v)[4], int i0, int n) {
    if (n == 4 && v[0] < tf && v[1] < tf && v[2] < tf && v[3] < tf) return;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < n && !(v[e] < tf)) {   // NaN compares false: it is collected, seen and left to the radix selection
        if (!(fabsf(v[e]) <= 1e30f)) sh.odd = 1;
        const int at = atomicAdd(&sh.ncand, 1);
        if (at < kCand) sh.hist[at] = pack_candidate(okey(scaled(v[e], T)), static_cast<uint32_t>(i0 + e));
      }
  });
  __syncthreads();
  const int n = sh.ncand;
  const bool bad = sh.odd != 0 || n > kCand || n < k;
  __syncthreads();
  if (bad) return 0;
  sort_candidates<NTH>(sh, n);
  return n;
}

// Top-p alone (no top-k): the threshold that the radix selection finds, from masses in linear bins; false: a row for the radix
// selection.  T > 0.
template <int NTH>
__device__ bool select_mass_linear(Shared& sh, const float* __restrict__ row, int V, float T, double p, float m, Sel& sp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!(T >= 9.5e-7f && T <= 1.05e6f) || !(fabsf(m) <= 1e30f)) return false;
  for (int b = tid; b < kBins; b += NTH) sh.hist[b] = 0ull;
  if (tid == 0) { sh.ncand = 0; sh.odd = 0; }
  __syncthreads();
  // a mass is zero once the value lies 32 ln 2 = 22.18 below the maximum; equal values share a bin, larger ones are in lower bins
  constexpr float kPerUnit = kBins / 22.2f;
  auto bin_of = [&](float s) { return min(kBins - 1, static_cast<int>((m - s) * kPerUnit)); };
  for_each4_free<NTH>(row, V, 1, [&](const float (&v)[4], int, int n) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < n) {
        const float s = scaled(v[e], T);
        if (m - s < 22.5f) {   // (the difference is exact where it matters; m - 22.5 is not, for large m)
          const uint32_t w = fx_exp(s, m);
          if (w != 0u) {   // two 32-bit adds, the second on a carry: a 64-bit one is a loop that tied values fight over
            uint32_t* at = reinterpret_cast<uint32_t*>(&sh.hist[bin_of(s)]);
            if (atomicAdd(at, w) > ~w) atomicAdd(at + 1, 1u);
          }
        } else if (!(s <= m)) {
          sh.odd = 1;   // NaN
        }
      }
  });
  __syncthreads();
  if (warp == 0) {   // lane l owns the bins [l * per, (l + 1) * per): the first bin at which the sum reaches ceil(p * total)
    constexpr int per = kBins / 32;
    unsigned long long s = 0ull;
    for (int j = 0; j < per; ++j) s += sh.hist[lane * per + j];
    unsigned long long incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    const unsigned long long total = __shfl_sync(kFull, incl, 31), excl = incl - s;
    const double t = ceil(p * static_cast<double>(total));
    unsigned long long rem = t < 1.0 ? 1ull : static_cast<unsigned long long>(t);
    if (rem > total) rem = total;
    if (rem < 1ull) rem = 1ull;
    if (total == 0ull && lane == 0) sh.odd = 1;
    if (excl < rem && rem <= incl) {
      unsigned long long c = excl;
      for (int j = 0; j < per; ++j) {
        const unsigned long long h = sh.hist[lane * per + j];
        if (c + h >= rem) { sh.sel_bin = lane * per + j; sh.need = rem - c; break; }
        c += h;
      }
    }
  }
  __syncthreads();
  const int bin = sh.sel_bin;
  const unsigned long long need = sh.need;
  const bool odd = sh.odd != 0;
  __syncthreads();
  if (odd) return false;
  uint32_t kmin = ~0u, kmax = 0u;   // keys of the bin
  for_each4_free<NTH>(row, V, 1, [&](const float (&v)[4], int i0, int n) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < n) {
        const float s = scaled(v[e], T);
        if (m - s < 22.5f && bin_of(s) == bin && fx_exp(s, m) != 0u) {
          const uint32_t key = okey(s);
          kmin = min(kmin, key);
          kmax = max(kmax, key);
          if (*static_cast<volatile int*>(&sh.ncand) > kCand) continue;
          const int at = atomicAdd(&sh.ncand, 1);
          if (at < kCand) sh.hist[at] = pack_candidate(key, static_cast<uint32_t>(i0 + e));
        }
      }
  });
  __syncthreads();
  const int n = sh.ncand;
  if (n > kCand) {   // more values than the rank holds: a group of ties (logits of a coarse type) is cut by index, the rest is unusual
    if (tid == 0) { sh.kmin = ~0u; sh.kmax = 0u; }
    __syncthreads();
    kmin = __reduce_min_sync(kFull, kmin);
    kmax = __reduce_max_sync(kFull, kmax);
    if (lane == 0) { atomicMin(&sh.kmin, kmin); atomicMax(&sh.kmax, kmax); }
    __syncthreads();
    const uint32_t key = sh.kmin;
    if (key != sh.kmax) return false;
    const unsigned long long w = fx_exp(okey_inv(key), m);
    sp.key = key;
    sp.cut = ordered_cut<NTH>(sh, V, [&](uint32_t i) { return okey(scaled(row[i], T)) == key; }, static_cast<uint32_t>((need + w - 1ull) / w));
    return true;
  }
  __syncthreads();
  if (n < 1) return false;
  sort_candidates<NTH>(sh, n);
  const unsigned long long last = sh.hist[mass_position(sh, n, m, need, false, 0.0)];
  sp.key = candidate_key(last);
  sp.cut = static_cast<uint32_t>(last);
  return true;
}

// u of the seeded contract, and the Gumbel noise it stands for
__device__ __forceinline__ float uniform(uint64_t seed, uint32_t i) {
  const uint64_t h = mix64(seed + static_cast<uint64_t>(i + 1) * kGolden);
  const float u = (static_cast<float>(h >> 41) + 0.5f) * 1.1920928955078125e-07f;  // 2^-23; in (0, 1)
  return fminf(fmaxf(u, 1e-8f), 1.0f - 1e-8f);                                     // sampler.rs:211-212
}
__device__ __forceinline__ float gumbel_of(float u) { return -logf(-logf(u)); }

template <int NTH>
__device__ float block_max(Shared& sh, float v) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_max(v);
  if (lane == 0) sh.redf[warp] = v;
  __syncthreads();
  float r = sh.redf[0];
  for (int w = 1; w < (NTH / 32); ++w) r = fmaxf(r, sh.redf[w]);
  __syncthreads();
  return r;
}

// The row's winner over the CTA (first maximum) and the number of survivors.
template <int NTH>
__device__ void finish_row(Shared& sh, float best, int bidx, int kept, int64_t* out_id, int32_t* kept_count) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(kFull, best, o);
    const int oi = __shfl_xor_sync(kFull, bidx, o);
    kept += __shfl_xor_sync(kFull, kept, o);
    if (ov > best || (ov == best && oi < bidx)) { best = ov; bidx = oi; }
  }
  if (lane == 0) { sh.redf[warp] = best; sh.redi[warp] = bidx; sh.cnt[warp] = static_cast<uint32_t>(kept); }
  __syncthreads();
  if (tid == 0) {
    int total = 0;
    for (int w = 0; w < (NTH / 32); ++w) {
      total += static_cast<int>(sh.cnt[w]);
      if (sh.redf[w] > best || (sh.redf[w] == best && sh.redi[w] < bidx)) { best = sh.redf[w]; bidx = sh.redi[w]; }
    }
    *out_id = bidx == 0x7fffffff ? 0 : bidx;
    if (kept_count != nullptr) *kept_count = total;
  }
}

template <int NTH>
__global__ void __launch_bounds__(NTH, kMaxThreads / NTH)
sample_kernel(int64_t* __restrict__ out_ids, const float* __restrict__ logits, int V, int64_t ld,
              const float* __restrict__ temperatures, const int32_t* __restrict__ top_k, const float* __restrict__ top_p,
              const uint64_t* __restrict__ row_seeds, int32_t* __restrict__ kept_count, uint8_t* __restrict__ kept_mask) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ Shared sh;
  const int tid = threadIdx.x;
  const int b = blockIdx.x;
  const float* __restrict__ row = logits + b * ld;
  const float T = temperatures[b];
  const bool greedy = T == 0.0f;
  bool filtered = false;
  Sel sk{0u, 0xffffffffu}, sp{0u, 0xffffffffu};  // key >= 0 always holds: no filtering

  if (!greedy) {
    const int k = top_k != nullptr ? top_k[b] : 0;
    const float p = top_p != nullptr ? top_p[b] : 0.0f;
    const bool do_k = k > 0 && k < V, do_p = p > 0.0f && p < 1.0f;
    filtered = do_k || do_p;
    float m = -INFINITY;  // max of the scaled row (it always survives top-k), needed by top-p only
    bool have_m = false;
    const int cand = do_k && k <= kShortK ? rank_top_k<NTH>(sh, row, V, T, k) : 0;
    if (cand > 0) {   // the k first of the ranked candidates, cut where their mass reaches p, are the survivors
      int r = k;
      if (do_p) r = mass_position(sh, k, okey_inv(candidate_key(sh.hist[0])), 0ull, true, static_cast<double>(p)) + 1;
      if (kept_mask != nullptr) {
        for (int i = tid; i < V; i += NTH) kept_mask[static_cast<int64_t>(b) * V + i] = 0;
        __syncthreads();
      }
      float best = -INFINITY;
      int bidx = 0x7fffffff;
      for (int j = tid; j < r; j += NTH) {
        const uint32_t i = static_cast<uint32_t>(sh.hist[j]);
        const float score = okey_inv(candidate_key(sh.hist[j])) + gumbel_of(uniform(row_seeds[b], i));
        if (kept_mask != nullptr) kept_mask[static_cast<int64_t>(b) * V + i] = 1;
        if (score > best || (score == best && static_cast<int>(i) < bidx)) { best = score; bidx = static_cast<int>(i); }
      }
      finish_row<NTH>(sh, best, bidx, tid == 0 ? r : 0, out_ids + b, kept_count != nullptr ? kept_count + b : nullptr);
      return;
    }
    // ---- top-k: the k-th largest key by count (sampler.rs:115-149) ----
    if (do_k) {
      uint32_t key;
      unsigned long long need, eq;
      radix_select<NTH, false>(sh, row, V, T, [](uint32_t, uint32_t) { return 1u; }, static_cast<unsigned long long>(k), 0.0, key,
                          need, eq, do_p ? &m : nullptr);
      have_m = do_p;
      sk.key = key;
      if (need < eq)  // ties straddle k: the stable sort keeps the lowest indices
        sk.cut = ordered_cut<NTH>(sh, V, [&](uint32_t i) { return okey(scaled(row[i], T)) == key; }, static_cast<uint32_t>(need));
    }
    // ---- top-p: smallest descending prefix whose softmax mass reaches p (sampler.rs:152-191) ----
    if (do_p) {
      if (!have_m) {
        if (T > 0.0f) {   // the division keeps the order
          for_each4_free<NTH>(row, V, 1, [&](const float (&v)[4], int, int n) {
            m = fmaxf(m, v[0]);
            if (n == 4) m = fmaxf(m, fmaxf(v[1], fmaxf(v[2], v[3])));
          });
          m = scaled(m, T);
        } else {
          for_each4<NTH>(row, V, [&](const float (&v)[4], int, int n) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (e < n) m = fmaxf(m, scaled(v[e], T));
          });
        }
      }
      m = block_max<NTH>(sh, m);
      if (do_k || !(T > 0.0f) || !select_mass_linear<NTH>(sh, row, V, T, static_cast<double>(p), m, sp)) {
        const Sel skc = sk;
        auto w_of = [&](uint32_t key, uint32_t i) { return keeps(skc, key, i) ? fx_exp(okey_inv(key), m) : 0u; };
        uint32_t key;
        unsigned long long need, eq;
        radix_select<NTH, true>(sh, row, V, T, w_of, 0ull, static_cast<double>(p), key, need, eq, nullptr);
        sp.key = key;
        const unsigned long long w1 = fx_exp(okey_inv(key), m);  // every element of the tie group weighs the same
        if (w1 > 0ull) {
          const unsigned long long need_cnt = (need + w1 - 1ull) / w1, eq_cnt = eq / w1;
          if (need_cnt < eq_cnt)
            sp.cut = ordered_cut<NTH>(sh, V, [&](uint32_t i) { const uint32_t kk = okey(scaled(row[i], T)); return kk == key && keeps(skc, kk, i); },
                                 static_cast<uint32_t>(need_cnt));
        }
      }
    }
  }

  // ---- final pass: Gumbel-max over the survivors (sampler.rs:194-219), or plain argmax for greedy rows ----
  const uint64_t seed = greedy ? 0ull : row_seeds[b];
  float best = -INFINITY;
  int bidx = 0x7fffffff, kept = 0;
  if (!filtered && !greedy && kept_mask == nullptr && kept_count == nullptr && V >= 64 * NTH) {
    // Nothing filtered: a value that cannot win is skipped before its noise.  g = -log(w), w = -log(u) >= 1 - u, so it cannot win where
    // 1 - u > exp(s - best), which costs one fast exponential of an approximate quotient instead of a division and two logarithms (1 %
    // is far beyond the approximations' error; 1e4 bounds the rounding of s + g against it).  Short rows end before a thread's own
    // best prunes much: 32768 values on 1024 threads 22 us without the test, 24 with it.
    const float inv_t = 1.0f / T;
    for_each4_free<NTH>(row, V, 1, [&](const float (&v)[4], int i0, int n) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < n) {
          const int i = i0 + e;
          const float near = v[e] * inv_t, u = uniform(seed, static_cast<uint32_t>(i));
          if (fabsf(near) < 1e4f && 1.0f - u > 1.01f * __expf(near - best)) continue;
          const float score = scaled(v[e], T) + gumbel_of(u);
          if (score > best || (score == best && i < bidx)) { best = score; bidx = i; }
        }
    });
  } else {
    for_each4_free<NTH>(row, V, 1, [&](const float (&v)[4], int i0, int n) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < n) {
          const int i = i0 + e;
          float score = v[e];
          bool keep = true;
          if (!greedy) {
            const float s = scaled(v[e], T);
            const uint32_t key = okey(s);
            keep = keeps(sk, key, static_cast<uint32_t>(i)) && keeps(sp, key, static_cast<uint32_t>(i));
            score = keep ? s + gumbel_of(uniform(seed, static_cast<uint32_t>(i))) : -INFINITY;
          }
          if (kept_mask != nullptr) kept_mask[static_cast<int64_t>(b) * V + i] = keep ? 1 : 0;
          kept += keep ? 1 : 0;
          if (score > best || (score == best && i < bidx)) { best = score; bidx = i; }
        }
    });
  }
  finish_row<NTH>(sh, best, bidx, kept, out_ids + b, kept_count != nullptr ? kept_count + b : nullptr);
}

}  // namespace
}  // namespace nvllm

// Sampler::forward (sampler.rs:26-67) for a whole batch in one launch; all pointers are device pointers.
extern "C" int nvllm_sample(int64_t* out_ids, const float* logits, int32_t batch, int32_t vocab, int64_t ld,
                            const float* temperatures, const int32_t* top_k, const float* top_p, const uint64_t* row_seeds,
                            int32_t* kept_count, uint8_t* kept_mask, void* stream) {
  using namespace nvllm;
  NVLLM_CHECK_ARG(batch >= 0 && vocab > 0 && ld >= vocab, NVLLM_ERR_ARG, "sample: batch=%d vocab=%d ld=%lld", batch, vocab,
                  (long long)ld);
  if (batch == 0) return 0;
  NVLLM_CHECK_ARG(out_ids && logits && temperatures && row_seeds, NVLLM_ERR_ARG, "sample: NULL pointer");
  const int threads = batch <= sm_count() ? kMaxThreads : kMaxThreads / 2;
  NVLLM_CUDA(launch_pdl(threads == kMaxThreads ? sample_kernel<kMaxThreads> : sample_kernel<kMaxThreads / 2>, dim3(batch), dim3(threads), 0,
                        static_cast<cudaStream_t>(stream), out_ids, logits, static_cast<int>(vocab), ld, temperatures, top_k, top_p, row_seeds,
                        kept_count, kept_mask));
  return 0;
}
