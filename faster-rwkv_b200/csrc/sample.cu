// Sampling on the device: Sampler::Sample (sampler.cpp:38-101) without copying the [V] logits to the host and
// without the host's std::sort over V entries per token.
//   probs = softmax(logits)   (kernels/cpu/softmax.cpp:6-21, temperature 1)
//   sort descending; keep the shortest prefix whose cumulative probability reaches top_p; cut to top_k if top_k > 0;
//   weights = probs ^ (1 / clamp(temperature, 0.1, 5)); draw the first index whose running sum reaches u * total.
// The uniform draw u in [0, 1] comes from the caller (the reference takes (g() - min) / (max - min) of a
// std::minstd_rand0, sampler.cpp:20-22), so a host that seeds the same generator reproduces the reference's picks.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "internal.h"

namespace frb {

namespace {

// Nothing is sorted.  Both decisions -- where the top-p / top-k prefix ends, and which entry the draw lands on -- are
// "the first entry, in descending order of probability, at which a running sum reaches a target", and such an entry is
// found by narrowing an interval: histogram the weights over 1024 bins of d = max - logit (monotone in probability),
// find the bin in which the sum crosses, repeat inside it until at most 1024 entries are left, and rank those against
// each other.  The sums are fixed-point integers (2^-40 of the largest weight), so the result does not depend on the
// order in which threads add.
// One CTA per row.  A row is read from L2 five times (maximum; histogram and members, twice); sorting it with a
// segmented radix sort took 16 rows of 65536 logits 0.84 ms (one CTA per segment and digit pass), this takes 0.06 ms.
constexpr int SM_T = 1024;                    // threads = histogram bins = most members ranked directly
constexpr int SM_LEVELS = 6;                  // narrowings, 1024 times finer each; a bin of equal values ends it
constexpr float SM_SPAN = 32.f;               // first histogram: the row's spread, at most this far in the exponent (e^-32 has no weight)
constexpr float SM_ONE = 1099511627776.f;     // 2^40
constexpr unsigned long long SM_NEVER = 1ull << 62;   // more than any sum of weights

constexpr int SM_RD = 4;

struct SampleSmem {
  unsigned long long mass[SM_T];   // the members' weights
  unsigned lo32[SM_T], hi32[SM_T]; // histogram: low and high words of the sums
  unsigned count[SM_T];            // histogram of entries, then the members' indices
  float d[SM_T];                   // members
  unsigned long long wsum[32];
  unsigned csum[32];
  unsigned n;                      // members found (may exceed SM_T)
  float dmin, dmax;
  int found;                       // bin, or member
  unsigned long long before;       // sum ahead of it
  unsigned cbefore;
  float fmax[32], fmin[32];
  float lo[SM_LEVELS], scale[SM_LEVELS];   // the narrowings so far: an entry is inside if it falls into bin[q] of each
  int bin[SM_LEVELS];
};

// fixed-point weight of an entry d below the maximum
__device__ __forceinline__ unsigned long long fx_weight(float d, float inv_t) {
  return __float2ull_rn(expf(-d * inv_t) * SM_ONE);
}

// 64-bit sum in two words with native 32-bit atomics (a 64-bit atomicAdd on shared memory is a compare-and-swap loop,
// and the bulk of the vocabulary shares a few bins): the thread whose addition wraps the low word carries
__device__ __forceinline__ void add64(unsigned &lo, unsigned &hi, unsigned long long v) {
  const unsigned l = (unsigned)v, h = (unsigned)(v >> 32);
  const unsigned old = atomicAdd(&lo, l), carry = old + l < old ? 1u : 0u;
  if (h + carry) atomicAdd(&hi, h + carry);
}
// order-preserving maximum / minimum of non-negative floats in shared memory
__device__ __forceinline__ void atomic_max_pos(float *p, float v) { atomicMax(reinterpret_cast<int *>(p), __float_as_int(v)); }
__device__ __forceinline__ void atomic_min_pos(float *p, float v) { atomicMin(reinterpret_cast<int *>(p), __float_as_int(v)); }

// f(value, index) for every entry of the row; four 16-byte loads in flight per thread
template <typename F>
__device__ __forceinline__ void for_row(const float *row, int V, F f) {
  const int V4 = V >> 2;
  for (int base = threadIdx.x; base < V4; base += SM_RD * SM_T) {
    float4 v[SM_RD];
#pragma unroll
    for (int i = 0; i < SM_RD; ++i)
      if (base + i * SM_T < V4) v[i] = reinterpret_cast<const float4 *>(row)[base + i * SM_T];
#pragma unroll
    for (int i = 0; i < SM_RD; ++i) {
      const int j = (base + i * SM_T) * 4;
      if (base + i * SM_T < V4) { f(v[i].x, j); f(v[i].y, j + 1); f(v[i].z, j + 2); f(v[i].w, j + 3); }
    }
  }
  for (int j = V4 * 4 + threadIdx.x; j < V; j += SM_T) f(row[j], j);
}

// inclusive block scan of (a, c), one pair per thread
__device__ __forceinline__ void block_scan(SampleSmem &s, unsigned long long &a, unsigned &c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long ta = __shfl_up_sync(0xffffffffu, a, o);
    const unsigned tc = __shfl_up_sync(0xffffffffu, c, o);
    if (lane >= o) { a += ta; c += tc; }
  }
  __syncthreads();
  if (lane == 31) { s.wsum[warp] = a; s.csum[warp] = c; }
  __syncthreads();
  if (warp == 0) {
    unsigned long long wa = s.wsum[lane];
    unsigned wc = s.csum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long ta = __shfl_up_sync(0xffffffffu, wa, o);
      const unsigned tc = __shfl_up_sync(0xffffffffu, wc, o);
      if (lane >= o) { wa += ta; wc += tc; }
    }
    s.wsum[lane] = wa; s.csum[lane] = wc;
  }
  __syncthreads();
  if (warp > 0) { a += s.wsum[warp - 1]; c += s.csum[warp - 1]; }
}

// Distance of a logit below the row's maximum.  What a caller masks (-inf) lies infinitely far below: no weight, and not
// among the candidates.  +inf is at distance 0 of itself, a row of -inf alone is a row of equals; NaN is no candidate either.
__device__ __forceinline__ float below(float mx, float v) { return v == mx ? 0.f : mx - v; }

struct Entry { float d; int id; };
__device__ __forceinline__ bool precedes(float d, int id, const Entry &e) { return d < e.d || (d == e.d && id <= e.id); }

// First entry, in order of (d, index), at which the running weight reaches frac * (total weight) or the running count
// reaches k (k > 0), among the entries that do not come after `last`; the last of them if there are fewer than k.
// frac > 1 is a target that no sum reaches (the count alone decides).
__device__ __noinline__ Entry select_entry(SampleSmem &s, const float *row, int V, float mx, float span, float inv_t, double frac,
                                              unsigned k, const Entry &last) {
  unsigned long long target = 0, before = 0;   // weight and entries ahead of the interval
  unsigned cbefore = 0;
  float wlo = 0.f, wscale = (float)SM_T / fmaxf(fminf(span, SM_SPAN / inv_t), 1e-30f);
  auto bin_of = [](float d, float l, float sc) {
    const float x = (d - l) * sc;
    return x >= (float)(SM_T - 1) ? SM_T - 1 : x > 0.f ? (int)x : 0;
  };
  for (int level = 0; level < SM_LEVELS; ++level) {
    auto inside = [&](float d, int id) {
      for (int q = 0; q < level; ++q)
        if (bin_of(d, s.lo[q], s.scale[q]) != s.bin[q]) return false;
      return d < INFINITY && precedes(d, id, last);
    };
    s.lo32[threadIdx.x] = 0; s.hi32[threadIdx.x] = 0; s.count[threadIdx.x] = 0;
    __syncthreads();
    for_row(row, V, [&](float v, int id) {
      const float d = below(mx, v);
      if (!inside(d, id)) return;
      const int b = bin_of(d, wlo, wscale);
      const unsigned long long w = fx_weight(d, inv_t);
      if (w) add64(s.lo32[b], s.hi32[b], w);
      if (k > 0) atomicAdd(&s.count[b], 1u);
    });
    __syncthreads();
    const unsigned long long m = (unsigned long long)s.hi32[threadIdx.x] << 32 | s.lo32[threadIdx.x];
    const unsigned c = s.count[threadIdx.x];
    unsigned long long a = m;
    unsigned ca = c;
    block_scan(s, a, ca);
    if (level == 0) {
      const unsigned long long total = s.wsum[31];
      const double t = ceil(frac * (double)total);
      target = !(frac <= 1.0) ? SM_NEVER : t >= (double)total ? total : t > 0.0 ? (unsigned long long)t : 0ull;
      k = min(k, s.csum[31]);            // (candidates in all)
    }
    if (threadIdx.x == 0) s.found = SM_T;
    __syncthreads();
    const bool reached = before + a >= target || (k > 0 && cbefore + ca >= k);
    if (reached && (threadIdx.x == 0 || m > 0 || c > 0)) atomicMin(&s.found, (int)threadIdx.x);
    __syncthreads();
    const int fb = min(s.found, SM_T - 1);
    if (threadIdx.x == fb) { s.before = before + a - m; s.cbefore = cbefore + ca - c; s.n = 0; s.lo[level] = wlo; s.scale[level] = wscale; s.bin[level] = fb; s.dmin = 3.0e38f; s.dmax = 0.f; }
    __syncthreads();
    before = s.before; cbefore = s.cbefore;
    // the members of that bin
    for_row(row, V, [&](float v, int id) {
      const float d = below(mx, v);
      if (!inside(d, id) || bin_of(d, wlo, wscale) != fb) return;
      const unsigned at = atomicAdd(&s.n, 1u);
      if (at < SM_T) { s.d[at] = d; s.count[at] = (unsigned)id; }
      atomic_min_pos(&s.dmin, d); atomic_max_pos(&s.dmax, d);
    });
    __syncthreads();
    const unsigned n = s.n;
    const float dmin = s.dmin, dmax = s.dmax;
    if (n == 0) return Entry{0.f, 0};   // a row without candidates (nothing but NaN)
    if (n <= SM_T) {
      // rank the members: running weight and count up to and including each one
      const bool mine = threadIdx.x < n;
      const float d = mine ? s.d[threadIdx.x] : 0.f;
      const int id = mine ? (int)s.count[threadIdx.x] : 0;
      const unsigned long long w = mine ? fx_weight(d, inv_t) : 0ull;
      s.mass[threadIdx.x] = w;
      if (threadIdx.x == 0) s.found = -1;
      __syncthreads();
      Entry e{d, id};
      unsigned long long run = before;
      unsigned rank = 0;                 // members up to and including this one
      if (mine)
        for (unsigned j = 0; j < n; ++j)
          if (precedes(s.d[j], (int)s.count[j], e)) { run += s.mass[j]; ++rank; }
      const bool hit = run >= target || (k > 0 && cbefore + rank >= k);
      const bool hit_before = rank > 1 && (run - w >= target || (k > 0 && cbefore + rank - 1 >= k));
      if (mine && hit && !hit_before) s.found = (int)threadIdx.x;
      __syncthreads();
      if (s.found < 0 && mine && rank == n) s.found = (int)threadIdx.x;   // not reached: the last one
      __syncthreads();
      const int f = max(s.found, 0);
      Entry r{s.d[f], (int)s.count[f]};
      __syncthreads();
      return r;
    }
    if (dmin == dmax || level == SM_LEVELS - 1) {
      // more equal entries than can be ranked: the m-th of them in index order
      const unsigned long long w = fx_weight(dmin, inv_t);
      unsigned long long need = target > before ? target - before : 1;
      unsigned want = w > 0 ? (unsigned)min((need + w - 1) / w, (unsigned long long)n) : (target > before ? n : 1u);
      if (k > 0) want = min(want, k > cbefore ? k - cbefore : 1u);
      want = max(want, 1u);
      const int S = (V + SM_T - 1) / SM_T, i0 = min(V, (int)threadIdx.x * S), i1 = min(V, i0 + S);
      auto member = [&](int i) { const float d = below(mx, row[i]); return inside(d, i) && bin_of(d, wlo, wscale) == fb; };
      unsigned here = 0;
      for (int i = i0; i < i1; ++i) here += member(i);
      unsigned long long dummy = 0;
      unsigned upto = here;
      block_scan(s, dummy, upto);
      if (upto - here < want && upto >= want) {
        unsigned q = upto - here;
        for (int i = i0; i < i1; ++i)
          if (member(i) && ++q == want) { s.found = i; s.dmax = below(mx, row[i]); }
      }
      __syncthreads();
      Entry r{s.dmax, s.found};
      __syncthreads();
      return r;
    }
    // narrow: the bin's own extent, cut into 1024 again
    wlo = dmin;
    wscale = (float)SM_T / fmaxf(dmax - dmin, 1e-30f);
    __syncthreads();
  }
  return last;   // not reached: the last level returns above
}

struct SampleArgs {
  const float *logits;
  int V, ld, top_k;
  float temperature, top_p;
  const float *u_dev;   // [rows], or null: u holds the draws
  int32_t *out;         // [rows], device or pinned host memory
  float u[SAMPLE_INLINE_U];
};

__global__ void __launch_bounds__(SM_T) sample_rows_kernel(const __grid_constant__ SampleArgs a) {
  __shared__ SampleSmem s;
  const float *row = a.logits + (size_t)blockIdx.x * a.ld;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float mx = -INFINITY, mn = INFINITY;
  for_row(row, a.V, [&](float v, int) { mx = fmaxf(mx, v); mn = fminf(mn, v); });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  if (lane == 0) { s.fmax[warp] = mx; s.fmin[warp] = mn; }
  __syncthreads();
  mx = s.fmax[0]; mn = s.fmin[0];
#pragma unroll
  for (int w = 1; w < 32; ++w) { mx = fmaxf(mx, s.fmax[w]); mn = fminf(mn, s.fmin[w]); }
  const Entry all{INFINITY, a.V};
  Entry cut = all;
  const unsigned k = a.top_k > 0 ? (unsigned)a.top_k : 0u;
  if (a.top_p < 1.f || (k > 0 && k < (unsigned)a.V)) cut = select_entry(s, row, a.V, mx, mx - mn, 1.f, (double)a.top_p, k, all);
  const float inv_t = 1.f / fminf(fmaxf(a.temperature, 0.1f), 5.f);
  float u = a.u_dev ? a.u_dev[blockIdx.x] : a.u[blockIdx.x];
  u = u <= 1.f ? u : 1.f;
  if (inv_t > 1.f) {
    // the reference raises the probabilities themselves: where even the largest one's power underflows, all weights are
    // zero and its walk stops at the first entry
    float e = 0.f;
    for_row(row, a.V, [&](float v, int) { e += expf(v - mx); });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    __syncthreads();
    if (lane == 0) s.fmax[warp] = e;
    __syncthreads();
    e = 0.f;
#pragma unroll
    for (int w = 0; w < 32; ++w) e += s.fmax[w];
    if (powf(1.f / e, inv_t) == 0.f) u = 0.f;
  }
  const Entry pick = select_entry(s, row, a.V, mx, mx - mn, inv_t, (double)u, 0u, cut);
  if (threadIdx.x == 0) a.out[blockIdx.x] = pick.id;
}

// logits[stream[i]][token[i]] += delta[i]: the sparse adjustments a chat loop makes before sampling (frequency /
// presence penalties and the end-of-text / newline biases of chat.cpp:57-75), without the logits leaving the device
__global__ void logits_add_kernel(float *logits, int ld, const int32_t *stream, const int32_t *token, const float *delta, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(logits + (size_t)stream[i] * ld + token[i], delta[i]);
}

}  // namespace

// out: device or pinned host memory [rows]; u: host [rows] if u_on_host (at most SAMPLE_INLINE_U rows), else device
cudaError_t launch_sample_rows(const float *logits, int rows, int V, int ld, float temperature, int top_k, float top_p,
                               const float *u, bool u_on_host, int32_t *out, cudaStream_t st) {
  if (u_on_host && rows > SAMPLE_INLINE_U) return cudaErrorInvalidValue;
  SampleArgs a;
  a.logits = logits; a.V = V; a.ld = ld; a.top_k = top_k; a.temperature = temperature; a.top_p = top_p;
  a.u_dev = u_on_host ? nullptr : u; a.out = out;
  memset(a.u, 0, sizeof(a.u));
  if (u_on_host) memcpy(a.u, u, (size_t)rows * 4);
  sample_rows_kernel<<<rows, SM_T, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_logits_add(float *logits, int ld, const int32_t *stream, const int32_t *token, const float *delta, int n, cudaStream_t st) {
  if (n > 0) logits_add_kernel<<<(n + 255) / 256, 256, 0, st>>>(logits, ld, stream, token, delta, n);
  return cudaGetLastError();
}

}  // namespace frb
