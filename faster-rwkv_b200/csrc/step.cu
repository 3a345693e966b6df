// Persistent whole-token decode kernel for sm_100a: one token of 1 .. 4 independent streams (fp16 weights; quantised RWKV-4:
// 1 and 2) in one cooperative launch, one CTA per SM, all layers and the head.
//
// A token is a chain of 4 L + 1 (RWKV-4) or 5 L + 1 (RWKV-5) matrix-vector phases, each of which needs every output of
// the one before it.  At batch 1 the chain, not the weight stream, decides the time of all but the widest fp16 models:
// an all-to-all hand-over through L2 takes about 2,400 clocks (measured; 2,048 words, 148 CTAs), and the instructions
// around it took several times that.  What they cost is mostly instruction fetch: straight-line code runs at 1 clock per
// instruction and warp from the innermost cache, at 2.5 up to 32 KB and at 5.7 from 64 KB on (measured), and a layer walks
// through all of its code once.  Hence the shape of this kernel:
//   * one copy of every piece of code, whatever phase it serves: gather the input words, make the operand, multiply, finish.
//     Rare parts of the waits are out of line, other model versions are other instances;
//   * 8 consumer warps split K: warp w owns the 64-input chunks w, w + 8, ... of every vector and every matrix.  It
//     polls, converts and multiplies only those, so an operand never crosses warps and plain vectors need no CTA barrier
//     (16 warps issue the fixed part of a phase twice as often: 10 - 30 % slower; 4 leave latency uncovered: 15 - 45 %);
//   * 3 epilogue warps take the row blocks in turn: they fetch the epilogue's inputs (state, residual, bonus) ahead,
//     wait for the partial sums, add them, apply the epilogue and publish, while the consumers are already at the next
//     row block or polling for the next phase;
//   * 1 producer thread keeps a ring of shared-memory slots full of weight tiles (1-D TMA bulk copies, L2 evict-first)
//     and asks L2 for tiles further ahead.  Weights do not depend on activations: it never waits for a phase;
//   * quantised weights are multiplied as integers: 3 instructions per 8 int4 weights, 4 per 8 int8 weights, where
//     their expansion to fp16 took 9 and 8.
//
// Phases are not separated by barriers.  Every value that crosses CTAs is one 32-bit word: the fp32 value rounded to 16
// significant bits, its low 8 mantissa bits replaced by the writing phase's tag; a reader polls the words it needs until
// they carry the expected tag.  Because each phase needs all outputs of the one before it, a CTA can only overwrite a
// vector after every reader of its previous contents has moved on; a CTA that owns no row block in a phase skips the
// phase.  The token-shift states are double-buffered for the same reason.  Every wait is bounded: after WAIT_LIMIT_NS the
// CTA records a status and drains.
#include "common.cuh"
#include "internal.h"

namespace frb {

namespace {

constexpr int SW = 8;                    // consumer warps
constexpr int SCONS = SW * 32;           // consumer threads
constexpr int EW = 3;                    // epilogue warps, one buffer of partial sums each
constexpr int STHREADS = SCONS + 128;    // + producer warp + epilogue warps
constexpr int SBAR = 1;                  // named barrier of the consumer warps
constexpr int STEP_MAX_STAGES = 12;

// One tile of 8 MMA columns.  fp16: stream b is columns 2 b (hi) and 2 b + 1 (lo), so that an accumulator pair is a stream;
// integers: columns 4 b .. 4 b + 2 are the digits of stream b
template <int FMT, int NS> __host__ __device__ constexpr bool fits_tile() { return FMT == FMT_FP16 ? NS <= 4 : NS <= 2; }
// operand bytes of one 64-input chunk
template <int NS> __host__ __device__ constexpr uint32_t chunk_operand_bytes() { return 256u * NS; }

__host__ __device__ inline size_t up_to(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Chunks of a K-input vector that warp w owns, and the chunks of operand its private area holds: the vectors of a
// LayerNorm phase, or the one vector of the widest phase.
__host__ __device__ inline int own_chunks(int K, int w) { const int n = K >> 6; return n > w ? (n - w + SW - 1) / SW : 0; }
__host__ __device__ inline int operand_chunks(int C, int F, int nvec, int w) {
  const int a = nvec * own_chunks(C, w), b = own_chunks(F, w);
  return a > b ? a : b;
}
constexpr uint32_t PARAM_OFF = 512, QUEUE_OFF = 1536, LN_OFF = 2048;   // barriers; kernel parameters; tile queue; LayerNorm sums
struct StepSmem { size_t part, xs, ring, total; };   // byte offsets
template <int NS>
__host__ __device__ inline StepSmem step_layout(int fmt, int C, int F, int nvec, int n_stages) {
  StepSmem o;
  o.part = up_to(LN_OFF + 2 * SW * NS * 8, 128);                       // [EW][SW][3][16 NS] float
  o.xs = o.part + (size_t)EW * SW * 3 * ROWS * NS * 4;
  size_t n = 8;                                                        // (the RWKV-5 state phase uses the first 2 KB as scratch)
  int sum = 0;
  for (int w = 0; w < SW; ++w) sum += operand_chunks(C, F, nvec, w);
  if ((size_t)sum > n) n = sum;
  o.ring = up_to(o.xs + n * chunk_operand_bytes<NS>(), 1024);
  o.total = o.ring + (size_t)n_stages * slot_bytes(fmt);
  return o;
}

// ---- tagged exchange words ----------------------------------------------------------------------
__device__ __forceinline__ unsigned tag_of(const StepParams &p, int pi) { return 1u + (p.seq_base + (unsigned)pi) % 255u; }
__device__ __forceinline__ unsigned tag_before(unsigned t) { return t > 1u ? t - 1u : 255u; }
__device__ __forceinline__ unsigned tag_after(unsigned t) { return t < 255u ? t + 1u : 1u; }
__device__ __forceinline__ void x_store(exch_t *dst, float v, unsigned tag) {
  unsigned u = __float_as_uint(v);
  u = ((u & 0x7f800000u) == 0x7f800000u ? u : u + 0x80u) & 0xffffff00u;   // round to nearest; inf / nan keep their class
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(dst), "r"(u | tag) : "memory");
}
__device__ __forceinline__ exch_t x_load(const exch_t *src) {
  exch_t w;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(w) : "l"(src) : "memory");
  return w;
}
__device__ __forceinline__ uint4 x_load4(const exch_t *src) {
  uint4 w;
  asm volatile("ld.relaxed.gpu.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "l"(src) : "memory");
  return w;
}
__device__ __forceinline__ float x_value(exch_t w) { return __uint_as_float(w & 0xffffff00u); }
__device__ __forceinline__ float4 x_value4(const uint4 &w) { return make_float4(x_value(w.x), x_value(w.y), x_value(w.z), x_value(w.w)); }
// the four tag bytes against tag * 0x01010101
__device__ __forceinline__ bool x_ready4(const uint4 &w, unsigned tag4) {
  return prmt(prmt(w.x, w.y, 0x0040), prmt(w.z, w.w, 0x0040), 0x5410) == tag4;
}

struct Cx {
  const StepParams *p;
  uint8_t *smem;
  uint64_t *full, *empty, *part_full, *part_empty;
  volatile int *abort_flag;
  uint32_t ln, part, xs, ring, queue;   // shared-space addresses
  size_t ring_off;
  uint32_t xw, xo;                 // this warp's operand area; the area of warp (tid / 16) % 8
  int tid, warp, lane, cta, G;
  int n_stages;
  int slot;                        // ring position of the next stage and the parity of its full barrier
  uint32_t parity;
  uint32_t item;                   // row blocks this CTA has started: row block n uses partial-sum buffer n % EW
  uint32_t ln_buf;
};

// Bounded polling: gives up after WAIT_LIMIT_NS, or as soon as another thread of the CTA gave up.
constexpr unsigned long long GIVE_UP = ~0ull;
__device__ __noinline__ unsigned long long patience_check(volatile int *abort_flag, int *status, unsigned long long t0, int code) {
  if (*abort_flag) return GIVE_UP;
  const unsigned long long now = globaltimer_ns();
  if (t0 == 0) t0 = now;
  if (now - t0 > WAIT_LIMIT_NS || __ldcg(status) != 0) {
    *abort_flag = 1;
    atomicCAS(status, 0, code);
    return GIVE_UP;
  }
  return t0;
}
struct Patience {
  unsigned long long t0 = 0;
  int it = 0;
  __device__ __forceinline__ bool more(const Cx &cx, int phase) {
    if ((++it & 63) != 0) return true;
    t0 = patience_check(cx.abort_flag, cx.p->status, t0, ST_TIMEOUT_DATA + 1000 * phase);
    return t0 != GIVE_UP;
  }
};
// a word that may not be there yet
__device__ __noinline__ float x_wait(const exch_t *src, unsigned tag, volatile int *abort_flag, int *status, int code) {
  exch_t w = x_load(src);
  unsigned long long t0 = 0;
  for (int it = 1; (w & 0xffu) != tag; ++it) {
    if ((it & 63) == 0 && (t0 = patience_check(abort_flag, status, t0, code)) == GIVE_UP) break;
    w = x_load(src);
  }
  return x_value(w);
}
__device__ __noinline__ bool bar_wait_slow(uint64_t *b, uint32_t parity, volatile int *abort_flag, int *status, int code) {
  return mbar_wait(b, parity, abort_flag, status, code);
}
__device__ __forceinline__ bool bar_wait(const Cx &cx, uint64_t *b, uint32_t parity, int code) {
  return mbar_try(b, parity) || bar_wait_slow(b, parity, cx.abort_flag, cx.p->status, code);
}

__device__ __forceinline__ int step_token(const StepParams &p, int b) {
  return p.ids_packed ? (int)(0xffffffffu - (unsigned)__ldcg(p.ids_packed + b)) : p.ids_val[b];
}
__device__ __forceinline__ float4 half4_f(const uint2 &u) {
  const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __noinline__ float4 emb4(const StepParams &p, int b, int i4) {
  if (p.emb_f32) return __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p.emb) + (size_t)step_token(p, b) * p.C) + i4);
  return half4_f(__ldg(reinterpret_cast<const uint2 *>(reinterpret_cast<const __half *>(p.emb) + (size_t)step_token(p, b) * p.C) + i4));
}
// Four consecutive activations as they lie in memory, 16 bytes of fp32 or 8 of fp16.  Conversion happens at the use, so
// that loads issued together stay in flight together.
template <bool H>
__device__ __forceinline__ uint4 raw_act(const uint8_t *base, int i4) {
  if (H) { const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(base) + i4); return make_uint4(u.x, u.y, 0u, 0u); }
  return __ldcg(reinterpret_cast<const uint4 *>(base) + i4);
}
template <bool H>
__device__ __forceinline__ float4 raw_f(const uint4 &w) {
  return H ? half4_f(make_uint2(w.x, w.y)) : make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
}
__device__ __forceinline__ void put_act4(uint8_t *base, int i4, bool half, const float4 &v) {
  if (half) {
    const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    reinterpret_cast<uint2 *>(base)[i4] = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
  } else {
    reinterpret_cast<float4 *>(base)[i4] = v;
  }
}

// ---- operands -------------------------------------------------------------------------------------
// Slots: a warp's chunks w, w + 8, ... in order are its local chunks; slot s of lane l is the four inputs
// 4 (l & 15) .. + 3 of local chunk 2 s + (l >> 4), so that one 16-byte load per lane fetches two chunks.
struct Slots {
  int n_own, n_slot;     // chunks and slots of this warp
  int sub;               // float4 inside the chunk
  int hi;                // upper half of the warp
  int c0;                // chunk of slot 0
  __device__ __forceinline__ Slots(const Cx &cx, int K) {
    n_own = own_chunks(K, cx.warp);
    n_slot = (n_own + 1) >> 1;
    hi = cx.lane >> 4;
    sub = cx.lane & 15;
    c0 = cx.warp + hi * SW;
  }
  __device__ __forceinline__ int local(int s) const { return hi + 2 * s; }
  __device__ __forceinline__ bool has(int s) const { return hi + 2 * s < n_own; }
  __device__ __forceinline__ int chunk(int s) const { return c0 + s * (2 * SW); }
  __device__ __forceinline__ int i4(int s) const { return chunk(s) * 16 + sub; }
};

// Operand of one chunk and nvec <= NV vectors: four inputs of stream b per lane, the 16 lanes of a half warp together.
//   fp16 weights: columns hi = fp16(x), lo = fp16(x - hi), ~22 mantissa bits:    [MMA pair][column][q][16 B]
//   int weights:  x as a 23-bit fixed-point number relative to the chunk's largest magnitude, three signed base-256
//                 digits = three s8 columns, and the scale that undoes it:       [column][q][16 B], 4 columns a stream
// (In two steps: the chunk's largest magnitude first.)
template <int FMT, int NV>
__device__ __forceinline__ unsigned chunk_max(int lane, const float4 (&x)[NV]) {
  if constexpr (FMT == FMT_FP16) return 0u;
  unsigned m = 0;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const unsigned m0 = max(__float_as_uint(fabsf(x[v].x)), __float_as_uint(fabsf(x[v].y)));
    const unsigned m1 = max(__float_as_uint(fabsf(x[v].z)), __float_as_uint(fabsf(x[v].w)));
    m = max(m, max(m0, m1));
  }
  return __reduce_max_sync(lane < 16 ? 0x0000ffffu : 0xffff0000u, m);
}
template <int FMT, int NS, int NV>
__device__ __forceinline__ void put_operand(uint32_t at, uint32_t vstride, int sub, int b, int nvec, unsigned m, const float4 (&x)[NV]) {
  const int j = sub >> 2, q = sub & 3;
  if constexpr (FMT == FMT_FP16) {
    uint32_t a = at + (uint32_t)(j >> 1) * (2u * NS * 64u) + (uint32_t)(2 * b) * 64u + (uint32_t)q * 16u + (uint32_t)(j & 1) * 8u;
#pragma unroll
    for (int v = 0; v < NV; ++v, a += vstride) {
      if (v >= nvec) break;
      const __half2 h0 = __floats2half2_rn(x[v].x, x[v].y), h1 = __floats2half2_rn(x[v].z, x[v].w);
      const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
      const __half2 l0 = __floats2half2_rn(x[v].x - f0.x, x[v].y - f0.y), l1 = __floats2half2_rn(x[v].z - f1.x, x[v].w - f1.y);
      sts64(a, make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1)));
      sts64(a + 64u, make_uint2(*reinterpret_cast<const uint32_t *>(&l0), *reinterpret_cast<const uint32_t *>(&l1)));
    }
  } else {
    // |x| < 2^(e - 126): times 2^(148 - e) it is below 2^22; the last bit of the fixed-point number is 2^(e - 148)
    const unsigned e = min(max(m >> 23, 32u), 254u);
    const float up = __uint_as_float((275u - e) << 23), down = m >= 0x7f800000u ? __uint_as_float(0x7fffffffu) : __uint_as_float((e - 21u) << 23);
    uint32_t a = at + (uint32_t)(4 * b) * 64u;
    if (sub < nvec) sts_f32(a + (uint32_t)sub * vstride + 192u, down);
    a += (uint32_t)q * 16u + (uint32_t)j * 4u;
#pragma unroll
    for (int v = 0; v < NV; ++v, a += vstride) {
      if (v >= nvec) break;
      // x * up + 1.5 * 2^23: the integer sits in the low mantissa bits; + 128 in every digit makes the digits signed
      const float M = 12582912.f;
      const unsigned O = 0x00808080u - 0x4b400000u;
      const unsigned y0 = __float_as_uint(fmaf(x[v].x, up, M)) + O, y1 = __float_as_uint(fmaf(x[v].y, up, M)) + O;
      const unsigned y2 = __float_as_uint(fmaf(x[v].z, up, M)) + O, y3 = __float_as_uint(fmaf(x[v].w, up, M)) + O;
      // byte order of the tiles' k positions: int4 0 2 1 3, int8 0 1 2 3
      const unsigned p0 = y0, p1 = FMT == FMT_INT4 ? y2 : y1, p2 = FMT == FMT_INT4 ? y1 : y2, p3 = y3;
      const unsigned t01 = prmt(p0, p1, 0x5140), t23 = prmt(p2, p3, 0x5140), u01 = prmt(p0, p1, 0x0062), u23 = prmt(p2, p3, 0x0062);
      sts_u32(a, prmt(t01, t23, 0x5410) ^ 0x80808080u);
      sts_u32(a + 64u, prmt(t01, t23, 0x7632) ^ 0x80808080u);
      sts_u32(a + 128u, prmt(u01, u23, 0x5410) ^ 0x80808080u);
    }
  }
}

// The words of an exchange vector [B][K] that this warp's operands need, as they are, into the operand areas: 16 bytes a
// lane, 256 a chunk and stream -- the size of the operand that replaces them.  R words a lane are asked for together, and
// again until their tags are there (a word asked for ahead of its time comes back stale and costs another round trip).
template <int NS>
__device__ __forceinline__ void gather(const Cx &cx, const Slots &sl, const exch_t *src, int K, unsigned tag4, int phase) {
  constexpr int R = 4, SR = R / NS;                 // word r of a round: slot s0 + r / NS, stream r % NS
#pragma unroll 1
  for (int s0 = 0; s0 < sl.n_slot; s0 += SR) {
    uint4 w[R];
    unsigned pending = 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (sl.has(s0 + r / NS) && (NS == 1 || r % NS < cx.p->B)) pending |= 1u << r;
    const unsigned all = pending;
    const exch_t *at = src + (size_t)sl.i4(s0) * 4;
    Patience pt;
    while (true) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((pending >> r) & 1u) w[r] = x_load4(at + (size_t)(r % NS) * K + (r / NS) * (2 * SW * 64));
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (((pending >> r) & 1u) && x_ready4(w[r], tag4)) pending &= ~(1u << r);
      if (!pending || !pt.more(cx, phase)) break;
    }
    const uint32_t d = cx.xw + (uint32_t)sl.local(s0) * chunk_operand_bytes<NS>() + (uint32_t)sl.sub * 16u;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((all >> r) & 1u) sts128(d + (uint32_t)(r / NS) * (2u * chunk_operand_bytes<NS>()) + (uint32_t)(r % NS) * 256u, w[r]);
  }
  __syncwarp();
}

// The gathered words -> operand vectors 0 .. nvec - 1 (nvec <= NV).  One copy of this code serves every phase of a layer:
//   LayerNorm + token-shift mix, and, on the CTA that owns the row block of a channel, the new shift state;
//   `plain`: the value itself (the head: the normalised value; ln == false: the vector as it came);
//   `gn`: GroupNorm of the RWKV-5 readout (a head is a chunk: 16 lanes hold its 64 values) times the gate.
struct Operand {
  uint32_t g, b, mix[4];           // element offsets in the vector blob
  const uint8_t *sx_rd;
  uint8_t *sx_wr;
  int own;                         // row blocks own, own + G, ... of the channels belong to this CTA
  int nvec;
  bool ln, layer0, plain, gn;
  unsigned gtag4;
};
template <int FMT, int NS, int NV, bool V5>
__device__ __forceinline__ void make_operand(Cx &cx, const Slots &sl, int K, const Operand &a, int phase) {
  const StepParams &p = *cx.p;
  constexpr bool ACT16 = FMT == FMT_FP16;          // (the strategy decides both: fp16 weights <-> fp16 shift states)
  constexpr uint32_t CB = chunk_operand_bytes<NS>();
  const int B = NS == 1 ? 1 : p.B;
  const bool gn = V5 && a.gn;
  // parameters of a slot, one slot ahead (of slot 0: before the statistics)
  float4 gw, gb, mx[NV];
  uint4 sx;
  auto params = [&](int s) {
    const int i4 = sl.has(s) ? sl.i4(s) : 0;
    const float4 *vb = reinterpret_cast<const float4 *>(p.vecs32) + i4;
    gw = __ldg(vb + (a.g >> 2)); gb = __ldg(vb + (a.b >> 2));
    if (!a.plain) {
#pragma unroll
      for (int v = 0; v < NV; ++v) mx[v] = __ldg(vb + (a.mix[v] >> 2));
      sx = raw_act<ACT16>(a.sx_rd, i4);
    }
  };
  const unsigned keep = a.layer0 ? 0xffffffffu : 0xffffff00u;   // (without the tags)
  auto x_of = [&](uint32_t at) {
    const uint4 w = lds128(at + (uint32_t)sl.sub * 16u);
    return make_float4(__uint_as_float(w.x & keep), __uint_as_float(w.y & keep), __uint_as_float(w.z & keep), __uint_as_float(w.w & keep));
  };
  float mean = 0.f, rstd = 1.f;
  if (a.ln) {
    // Thread t sums the float4 t, t + 256, ... of x, which other warps gathered (they lie in the operand areas until these
    // are written, behind the second barrier), shifted by the first element.  Lane l keeps the result of stream l % NS.
    params(0);
    bar_sync(SBAR, SCONS);
    static_assert(SW == 8, "chunk c belongs to warp c % 8: thread t's float4 are all in the area of warp (t / 16) % 8");
    const uint32_t lnb = cx.ln + cx.ln_buf * (SW * NS * 8u);
    cx.ln_buf ^= 1u;
    const uint32_t x0 = cx.xs + (uint32_t)(cx.lane % NS) * 256u;
    const float piv = lds_f32(x0), pivot = __uint_as_float(__float_as_uint(piv) & keep);
#pragma unroll 1
    for (int b = 0; b < B; ++b) {
      const float pv = NS == 1 ? pivot : __shfl_sync(0xffffffffu, pivot, b);
      float s1 = 0.f, s2 = 0.f;
      uint32_t at = cx.xo + (uint32_t)(cx.tid >> 7) * CB;
#pragma unroll 1
      for (int i = cx.tid; i < (p.C >> 2); i += SCONS, at += 2u * CB) {
        const float4 v = x_of(at + (uint32_t)b * 256u);
        const float d0 = v.x - pv, d1 = v.y - pv, d2 = v.z - pv, d3 = v.w - pv;
        s1 += (d0 + d1) + (d2 + d3);
        s2 += (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
      }
      __syncwarp();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      }
      if (cx.lane == 0) sts64(lnb + (uint32_t)(b * SW + cx.warp) * 8u, make_uint2(__float_as_uint(s1), __float_as_uint(s2)));
    }
    bar_sync(SBAR, SCONS);
    float t1 = 0.f, t2 = 0.f;
#pragma unroll
    for (int w = 0; w < SW; w += 2) {              // two warps' sums per load
      const float4 f = lds_f32x4(lnb + (uint32_t)((NS == 1 ? 0 : cx.lane % NS) * SW + w) * 8u);
      t1 += f.x; t2 += f.y;
      t1 += f.z; t2 += f.w;
    }
    const float inv = 1.f / (float)p.C, m = t1 * inv;
    float var = t2 * inv - m * m;
    var = var > 0.f ? var : 0.f;
    mean = pivot + m;
    rstd = rsqrtf(var + 1e-5f);
  } else if (gn) {
    params(0);
  }
  const uint32_t vb = (uint32_t)sl.n_own * CB;     // bytes of this warp's part of an operand vector
#pragma unroll 1
  for (int s = 0; s < sl.n_slot; ++s) {
    const bool has = sl.has(s);
    const uint32_t at = cx.xw + (uint32_t)sl.local(s) * CB;
    bool own = false;
    if (!a.plain && has)
      for (int t = a.own; t < (p.C >> 4); t += cx.G) own = own || sl.chunk(s) * 4 + (sl.sub >> 2) == t;
    // the chunk's words leave its operand area before the first operand is written
    float4 xs[NS];
#pragma unroll
    for (int b = 0; b < NS; ++b)
      if (has) xs[b] = x_of(at + (uint32_t)b * 256u);
    __syncwarp();
#pragma unroll 1
    for (int b = 0; b < B; ++b) {
      float4 xx = xs[0];
      if (NS > 1) {
#pragma unroll
        for (int q = 1; q < NS; ++q)
          if (b == q) xx = xs[q];
      }
      if (a.ln || gn) {
        float mu = NS == 1 ? mean : __shfl_sync(0xffffffffu, mean, b), rs = NS == 1 ? rstd : __shfl_sync(0xffffffffu, rstd, b);
        if (gn) {
          float t = (xx.x + xx.y) + (xx.z + xx.w);
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          mu = t * (1.f / 64.f);
          const float d0 = xx.x - mu, d1 = xx.y - mu, d2 = xx.z - mu, d3 = xx.w - mu;
          float e = (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
          rs = rsqrtf(e * (1.f / 64.f) + 1e-5f);
        }
        xx = make_float4((xx.x - mu) * rs * gw.x + gb.x, (xx.y - mu) * rs * gw.y + gb.y, (xx.z - mu) * rs * gw.z + gb.z, (xx.w - mu) * rs * gw.w + gb.w);
        if (gn && p.version >= 51) {
          const exch_t *gp = p.g5 + (size_t)b * K + (size_t)(has ? sl.i4(s) : 0) * 4;
          uint4 gv = x_load4(gp);
          Patience pt;
          while (has && !x_ready4(gv, a.gtag4) && pt.more(cx, phase)) gv = x_load4(gp);
          __syncwarp();
          const float4 g = x_value4(gv);
          xx.x *= g.x; xx.y *= g.y; xx.z *= g.z; xx.w *= g.w;
        }
      }
      float4 y[NV];
      y[0] = xx;
      if (!a.plain) {
        const float4 z = raw_f<ACT16>(sx);
        if (NS > 1 && b + 1 < B) sx = raw_act<ACT16>(a.sx_rd + (size_t)(b + 1) * p.state_stride, has ? sl.i4(s) : 0);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const float4 m = mx[v];
          y[v] = make_float4(xx.x * m.x + z.x * (1.f - m.x), xx.y * m.y + z.y * (1.f - m.y), xx.z * m.z + z.z * (1.f - m.z), xx.w * m.w + z.w * (1.f - m.w));
        }
      } else {
#pragma unroll
        for (int v = 1; v < NV; ++v) y[v] = xx;      // (not stored)
      }
      if ((a.ln || gn) && b == B - 1 && s + 1 < sl.n_slot) params(s + 1);
      const unsigned m = chunk_max<FMT, NV>(cx.lane, y);
      if (has) put_operand<FMT, NS, NV>(at, vb, sl.sub, b, a.nvec, m, y);
      if (own) put_act4(a.sx_wr + (size_t)b * p.state_stride, sl.i4(s), ACT16, xx);
    }
  }
  __syncwarp();
}

// ---- multiply ---------------------------------------------------------------------------------------
// One chunk: 16 output rows x 64 inputs of the streamed tile, and the operand.  acc: this lane's share of rows g and
// g + 8, which sum_lanes() turns into the sums of a stream:
//   fp16:  four m16n8k16 MMAs into two accumulator sets (no MMA waits for the one before it); lane q holds stream q (hi +
//          lo columns).  Sums are taken in the order of the batched-prologue kernel, the results are the same bit by bit
//   int:   [0][0], [1][0]; two m16n8k32 int8 MMAs, exact; lane q holds digits 0, 1 (q even: low) or 2 (q odd: high) of stream q / 2.
//          int4 keeps the codes times 16 (the nibble stays in the upper half of its byte); one MMA is one scale group.

// what a chunk's MMAs read from shared memory
template <int FMT, int NS>
struct Frag {
  uint4 a[FMT == FMT_FP16 ? 4 : FMT == FMT_INT8 ? 2 : 1];
  uint4 b[FMT == FMT_FP16 ? 2 : 1];
  uint2 sc;                                 // int4: group scales of rows g, g + 8
  float down;
};
template <int FMT, int NS>
__device__ __forceinline__ void fetch_chunk(Frag<FMT, NS> &f, uint32_t A, uint32_t scales, uint32_t B, int lane) {
  // lanes of the columns in use: the others feed zeros and read nothing
  const bool b_lane = FMT == FMT_FP16 ? NS >= 4 || lane < 8 * NS : NS > 1 || lane < 12;
#pragma unroll
  for (int i = 0; i < (FMT == FMT_FP16 ? 4 : FMT == FMT_INT8 ? 2 : 1); ++i) f.a[i] = lds128(A + 512u * i);
  f.b[0] = make_uint4(0, 0, 0, 0);
  if constexpr (FMT == FMT_FP16) f.b[1] = f.b[0];
  if (b_lane) {
    f.b[0] = lds128(B + (uint32_t)lane * 16u);
    if constexpr (FMT == FMT_FP16) f.b[1] = lds128(B + 2u * NS * 64u + (uint32_t)lane * 16u);
  }
  if constexpr (FMT != FMT_FP16) f.down = lds_f32(B + (NS > 1 ? (uint32_t)(lane & 2) * 128u : 0u) + 192u);
  if constexpr (FMT == FMT_INT4) f.sc = lds64(scales);
}
template <int FMT, int NS>
__device__ __forceinline__ void mul_chunk(const Frag<FMT, NS> &f, int lane, float (&acc)[2][4]) {
  if constexpr (FMT == FMT_FP16) {
    mma16816(acc[0], f.a[0].x, f.a[0].y, f.a[0].z, f.a[0].w, f.b[0].x, f.b[0].y);
    mma16816(acc[1], f.a[1].x, f.a[1].y, f.a[1].z, f.a[1].w, f.b[0].z, f.b[0].w);
    mma16816(acc[0], f.a[2].x, f.a[2].y, f.a[2].z, f.a[2].w, f.b[1].x, f.b[1].y);
    mma16816(acc[1], f.a[3].x, f.a[3].y, f.a[3].z, f.a[3].w, f.b[1].z, f.b[1].w);
  } else {
    const float m256 = lane & 1 ? 0.f : 256.f;       // column 3 of a stream is not a digit
    uint32_t a[8];                                   // A fragments of the two MMAs
    float2 s0, s1;
    if constexpr (FMT == FMT_INT8) {
      const uint32_t S = 0x80808080u;                // byte + 128 -> signed byte
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[4 * i] = prmt(f.a[i].x, f.a[i].y, 0x5410) ^ S; a[4 * i + 1] = prmt(f.a[i].x, f.a[i].y, 0x7632) ^ S;
        a[4 * i + 2] = prmt(f.a[i].z, f.a[i].w, 0x5410) ^ S; a[4 * i + 3] = prmt(f.a[i].z, f.a[i].w, 0x7632) ^ S;
      }
    } else {
      s0 = __half22float2(*reinterpret_cast<const __half2 *>(&f.sc.x));   // group 0: rows g, g + 8
      s1 = __half22float2(*reinterpret_cast<const __half2 *>(&f.sc.y));   // group 1
      const uint32_t H = 0xf0f0f0f0u, S = 0x80808080u;                    // nibble + 8 -> signed upper nibble
      const uint32_t w[4] = {f.a[0].x, f.a[0].y, f.a[0].z, f.a[0].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[2 * i] = lop3_and_xor(w[i] << 4, H, S); a[2 * i + 1] = lop3_and_xor(w[i], H, S); }
    }
    int u[4] = {0, 0, 0, 0}, v[4] = {0, 0, 0, 0};
    mma16832_s8(u, a[0], a[1], a[2], a[3], f.b[0].x, f.b[0].y);
    if constexpr (FMT == FMT_INT8) {
      mma16832_s8(u, a[4], a[5], a[6], a[7], f.b[0].z, f.b[0].w);
      acc[0][0] += f.down * fmaf(m256, (float)u[1], (float)u[0]);
      acc[1][0] += f.down * fmaf(m256, (float)u[3], (float)u[2]);
    } else {
      mma16832_s8(v, a[4], a[5], a[6], a[7], f.b[0].z, f.b[0].w);
      const float r0 = fmaf(s1.x, fmaf(m256, (float)v[1], (float)v[0]), s0.x * fmaf(m256, (float)u[1], (float)u[0]));
      const float r1 = fmaf(s1.y, fmaf(m256, (float)v[3], (float)v[2]), s0.y * fmaf(m256, (float)u[3], (float)u[2]));
      acc[0][0] += f.down * r0;
      acc[1][0] += f.down * r1;
    }
  }
}

// sum of row g + 8 r of a stream over this warp's K share
template <int FMT>
__device__ __forceinline__ float sum_lanes(int lane, const float (&a)[2][4], int r) {
  if constexpr (FMT == FMT_FP16) return (a[0][2 * r] + a[1][2 * r]) + (a[0][2 * r + 1] + a[1][2 * r + 1]);
  // low digits + 2^16 x high digit; int4 codes are 16 times too large
  const float v = a[r][0] * (lane & 1 ? 65536.f : 1.f) * (FMT == FMT_INT4 ? 0.0625f : 1.f);
  return v + __shfl_xor_sync(0xffffffffu, v, 1);
}

// All row blocks of a phase that belong to this CTA: this warp's share of K, partial sums to the epilogue warps.  Matrix u
// of a fused row block reads operand vector u; else the vector is the row block's class: its index / split, at most last_vec.
template <int FMT, int NS>
__device__ __forceinline__ void multiply_items(Cx &cx, int K, int n_items, int n_sub, int split, uint32_t last_vec, int first) {
  static_assert(fits_tile<FMT, NS>(), "the streams' columns fit one MMA tile");
  constexpr int CH = FMT == FMT_FP16 ? 16 : 32;      // chunks of a full stage
  constexpr uint32_t CB = chunk_operand_bytes<NS>(), WB = FMT == FMT_FP16 ? 2048u : FMT == FMT_INT8 ? 1024u : 512u;
  const int n_ch = K >> 6, nst = num_stages(FMT, K);
  const uint32_t vb = (uint32_t)own_chunks(K, cx.warp) * CB;
  const int g = cx.lane >> 2, q = cx.lane & 3;
  const uint32_t lane_a = (uint32_t)cx.warp * WB + (uint32_t)cx.lane * 16u;
  bool ready = false;                                // the next stage was seen complete by an earlier look
#pragma unroll 1
  for (int it = first; it < n_items; it += cx.G) {
    const uint32_t buf = cx.item % EW;
    const uint32_t dst = cx.part + ((buf * SW + (uint32_t)cx.warp) * 3u) * (ROWS * NS * 4u);
#pragma unroll 1
    for (int u = 0; u < n_sub; ++u) {
      const uint32_t vec = n_sub > 1 ? (uint32_t)u : split == 0 || it < split ? 0u : min(it < 2 * split ? 1u : it < 3 * split ? 2u : 3u, last_vec);
      uint32_t bop = cx.xw + vec * vb;
      float acc[2][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { acc[0][i] = 0.f; acc[1][i] = 0.f; }
      int left = n_ch;                               // chunks from this stage on
#pragma unroll 1
      for (int s = 0; s < nst; ++s, left -= CH) {
        if (!ready) bar_wait(cx, &cx.full[cx.slot], cx.parity, ST_TIMEOUT_FULL);
        const int cur = cx.slot;
        if (++cx.slot == cx.n_stages) { cx.slot = 0; cx.parity ^= 1u; }
        ready = mbar_test(&cx.full[cx.slot], cx.parity);
        const uint32_t st = cx.ring + (uint32_t)cur * slot_bytes(FMT);
        const int nch = left < CH ? left : CH;
        // two chunks at a time: both are fetched before the first is multiplied
#pragma unroll
        for (int h0 = 0; h0 < CH / SW; h0 += 2) {
          const int c0 = cx.warp + h0 * SW;
          if (c0 >= nch) break;
          Frag<FMT, NS> f[2];
          const uint32_t A = st + lane_a + (uint32_t)h0 * (SW * WB), S = st + (uint32_t)nch * 512u + (uint32_t)c0 * 64u + (uint32_t)g * 8u;
          const bool two = c0 + SW < nch;
          fetch_chunk<FMT, NS>(f[0], A, S, bop + (uint32_t)h0 * CB, cx.lane);
          if (two) fetch_chunk<FMT, NS>(f[1], A + SW * WB, S + SW * 64u, bop + (uint32_t)(h0 + 1) * CB, cx.lane);
          mul_chunk<FMT, NS>(f[0], cx.lane, acc);
          if (two) mul_chunk<FMT, NS>(f[1], cx.lane, acc);
        }
        bop += (uint32_t)(CH / SW) * CB;
        __syncwarp();
        if (cx.lane == 0) mbar_arrive(&cx.empty[cur]);
      }
      if (u == 0) bar_wait(cx, &cx.part_empty[buf], (cx.item / EW & 1u) ^ 1u, ST_TIMEOUT_EMPTY);
      // fp16: lane q of a row holds stream q; int: lanes 2 s and 2 s + 1 hold stream s
      const int sq = FMT == FMT_FP16 ? q : q >> 1;
      const float r0 = sum_lanes<FMT>(cx.lane, acc, 0), r1 = sum_lanes<FMT>(cx.lane, acc, 1);
      if (FMT == FMT_FP16 ? q < NS : (q & 1) == 0 && sq < NS) {
        const uint32_t d = dst + (uint32_t)u * (ROWS * NS * 4u) + (uint32_t)(g * NS + sq) * 4u;
        sts_f32(d, r0);
        sts_f32(d + (uint32_t)(8 * NS) * 4u, r1);
      }
    }
    __syncwarp();
    if (cx.lane == 0) mbar_arrive(&cx.part_full[buf]);
    ++cx.item;
  }
}

// ---- RWKV-5 state update + readout: units of (stream, head, 32 value columns), all consumer warps of a CTA ----------
// A thread owns one key row and NC of the columns.  (16-column units would be more than there are SMs: a second round for
// a few CTAs costs more than the longer rows.)
__device__ __forceinline__ int wkv5_units(const StepParams &p) { return p.B * p.H * 2; }
__device__ __forceinline__ void state_v5(Cx &cx, int layer, int pi, unsigned tag, int first) {
  const StepParams &p = *cx.p;
  constexpr int TR = SCONS / 64, NC = 32 / TR, NF = NC / 4;   // threads per key row, columns and float4 per thread
  static_assert(NF >= 1 && NF * 4 * TR == 32, "64 key rows x 32 columns over the consumer threads");
  const int C = p.C, H = p.H;
  const unsigned in_tag = tag_before(tag), in_tag4 = in_tag * 0x01010101u;
  const int i = cx.tid / TR, jq = (cx.tid % TR) * NC;
#pragma unroll 1
  for (int un = first; un < wkv5_units(p); un += cx.G) {
    const int b = un / (H * 2), h = (un >> 1) % H, j0 = (un & 1) * 32;
    uint8_t *stb = p.state + (size_t)b * p.state_stride + (size_t)layer * p.layer_stride;
    float4 *sp = reinterpret_cast<float4 *>(reinterpret_cast<float *>(stb + off_mid(C, p.act_fp16)) + (size_t)h * 4096 + i * 64 + j0 + jq);
    float4 s[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) s[f] = sp[f];
    const size_t vo = (size_t)layer * p.vec_stride + (p.version == 50 ? h : h * 64 + i);
    const float u = __ldg(p.vecs32 + p.v_first + vo), w = __ldg(p.vecs32 + p.v_decay + vo);
    const exch_t *kp = p.k5 + (size_t)b * C + h * 64 + i, *rp = p.r5 + (size_t)b * C + h * 64 + i, *vp = p.v5 + (size_t)b * C + h * 64 + j0 + jq;
    exch_t kw, rw;
    uint4 v[NF];
    bool there;
    Patience pt;
    do {
      kw = x_load(kp); rw = x_load(rp);
#pragma unroll
      for (int f = 0; f < NF; ++f) v[f] = x_load4(vp + 4 * f);
      there = (kw & 0xffu) == in_tag && (rw & 0xffu) == in_tag;
#pragma unroll
      for (int f = 0; f < NF; ++f) there = there && x_ready4(v[f], in_tag4);
    } while (!there && pt.more(cx, pi));
    __syncwarp();
    const float ki = x_value(kw), ri = x_value(rw);
    float o[NC];
    auto one = [&](float &st, float vj, float &y) {
      const float a = ki * vj;
      y = ri * (u * a + st);
      st = a + w * st;
    };
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const float4 vj = x_value4(v[f]);
      one(s[f].x, vj.x, o[4 * f]); one(s[f].y, vj.y, o[4 * f + 1]); one(s[f].z, vj.z, o[4 * f + 2]); one(s[f].w, vj.w, o[4 * f + 3]);
      sp[f] = s[f];
    }
    // over the key rows of this warp, then over the warps
#pragma unroll
    for (int d = TR; d < 32; d <<= 1)
#pragma unroll
      for (int e = 0; e < NC; ++e) o[e] += __shfl_xor_sync(0xffffffffu, o[e], d);
    bar_sync(SBAR, SCONS);       // the operand area is free: every warp is past the phase before, or past the last unit
    if (cx.lane < TR) {
#pragma unroll
      for (int f = 0; f < NF; ++f)
        sts128(cx.xs + (uint32_t)(cx.warp * 32 + cx.lane * NC + 4 * f) * 4u,
               make_uint4(__float_as_uint(o[4 * f]), __float_as_uint(o[4 * f + 1]), __float_as_uint(o[4 * f + 2]), __float_as_uint(o[4 * f + 3])));
    }
    bar_sync(SBAR, SCONS);
    if (cx.tid < 32) {
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < SW; ++k) t += lds_f32(cx.xs + (uint32_t)(k * 32 + cx.tid) * 4u);
      x_store(p.o5 + (size_t)b * C + h * 64 + j0 + cx.tid, t, tag);
    }
  }
  if (first < wkv5_units(p)) bar_sync(SBAR, SCONS);   // the sums are read before the next operand overwrites them
}

// ---- epilogue warps ---------------------------------------------------------------------------------
// exp(a - m), exp(b - m) with m = max(a, b)
__device__ __noinline__ float2 exp_pair(float a, float b, float &m) {
  m = fmaxf(a, b);
  return make_float2(expf(a - m), expf(b - m));
}

template <int FMT, int NS>
__device__ __forceinline__ void epilogue_items(Cx &cx, const StepPhase &ph, int layer, int pi, unsigned tag, int first, int e, unsigned long long &best) {
  const StepParams &p = *cx.p;
  constexpr int VPL = NS >= 2 ? NS / 2 : 1;      // outputs per lane and matrix
  constexpr uint32_t MB = ROWS * NS * 4u;        // bytes of one matrix's partial sums of one warp
  const int C = p.C, kind = ph.kind, n_sub = ph.n_sub, split = ph.split;
  const bool halve = p.rescale_every > 0 && (layer + 1) % p.rescale_every == 0;
#pragma unroll 1
  for (int it = first; it < ph.n_items; it += cx.G) {
    const uint32_t n = cx.item++;
    if ((int)(n % EW) != e) continue;
    // what the epilogue reads from global memory is requested before the partial sums are waited for
    int cls = 0, o0 = it * ROWS;                 // class of the row block (ffn receptance; k, v, r, g), channel within it
    for (int t = it; split > 0 && t >= split && cls < (kind == PH_FFN_KR ? 1 : 3); t -= split) { ++cls; o0 -= split * ROWS; }
    float f0[VPL], f1[VPL], f2[VPL], f3[VPL], f4[VPL], r0[VPL], r1[VPL], r2[VPL];
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int idx = NS == 1 ? cx.lane & 15 : cx.lane + 32 * k;
      const int row = idx / NS, b = idx % NS, o = o0 + row;
      const size_t bo = (size_t)b * C + o;
      f0[k] = f1[k] = f2[k] = f3[k] = f4[k] = 0.f;
      r0[k] = r1[k] = r2[k] = 1.f;
      if (NS > 1 && b >= p.B) continue;
      if (FMT == FMT_INT8) {
        const __half *rs = p.rscale + (kind == PH_HEAD ? 0 : (size_t)layer * p.rs_stride) + ph.rs_off + (size_t)it * n_sub * ROWS + row;
        r0[k] = __half2float(__ldg(rs));
        if (n_sub > 1) { r1[k] = __half2float(__ldg(rs + ROWS)); r2[k] = __half2float(__ldg(rs + 2 * ROWS)); }
      }
      if (kind == PH_ATT_KVR) {
        const float *aa = reinterpret_cast<const float *>(p.state + (size_t)b * p.state_stride + (size_t)layer * p.layer_stride + off_mid(C, FMT == FMT_FP16)) + o;
        const float *vp = p.vecs32 + (size_t)layer * p.vec_stride + o;
        f0[k] = aa[0]; f1[k] = aa[C]; f2[k] = aa[2 * C];
        f3[k] = __ldg(vp + p.v_first); f4[k] = __ldg(vp + p.v_decay);
      } else if (kind == PH_FFN_V || kind == PH_ATT_O) {
        // residual and gate words: published before what the consumers wait for
        const bool v = kind == PH_FFN_V;
        if (!v && layer == 0) {
          const size_t eo = (size_t)step_token(p, b) * C + o;
          f0[k] = p.emb_f32 ? __ldg(reinterpret_cast<const float *>(p.emb) + eo) : __half2float(reinterpret_cast<const __half *>(p.emb)[eo]);
        } else {
          const unsigned t1 = tag_before(tag), t2 = tag_before(t1), tx = v || p.version == 4 ? t2 : tag_before(t2);
#pragma unroll 1
          for (int w = 0; w < 1 + (int)v; ++w) {
            const float f = x_wait(w ? p.rr + bo : v ? p.xa + bo : p.x + bo, w ? t1 : tx, cx.abort_flag, p.status, ST_TIMEOUT_DATA + 1000 * pi);
            if (w) f1[k] = f; else f0[k] = f;
          }
        }
      }
    }
    __syncwarp();
    bar_wait(cx, &cx.part_full[e], (n / EW) & 1u, ST_TIMEOUT_FULL);
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int idx = NS == 1 ? cx.lane & 15 : cx.lane + 32 * k;
      const int b = idx % NS, o = o0 + idx / NS;
      const size_t bo = (size_t)b * C + o;
      auto sum = [&](uint32_t u) {
        const uint32_t a = cx.part + (uint32_t)e * SW * 3u * MB + u * MB + (uint32_t)idx * 4u;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < SW; ++w) s += lds_f32(a + (uint32_t)w * 3u * MB);
        return s;
      };
      float v0 = sum(0) * r0[k], v1 = 0.f, v2 = v0;
      if (n_sub > 1) { v1 = sum(1) * r1[k]; v2 = sum(2) * r2[k]; }
      if (k == VPL - 1) {
        __syncwarp();
        if (cx.lane == 0) mbar_arrive(&cx.part_empty[e]);
      }
      if (NS == 1 ? cx.lane >= 16 : b >= p.B) continue;
      if (kind == PH_HEAD) {
        p.logits[(size_t)b * p.Vpad + o] = v0;
        if (p.amax && o < p.V) {
          unsigned u = __float_as_uint(v0);
          u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
          const unsigned long long w = ((unsigned long long)u << 32) | (0xffffffffu - (unsigned)o);
          best = w > best ? w : best;
        }
        continue;
      }
      const float sg = 1.f / (1.f + expf(-v2));  // of r, the receptance row or the gate row, whichever this is
      float pm = 0.f, quo = sg;
      if (kind == PH_ATT_KVR) {
        const float2 e1 = exp_pair(f2[k], f3[k] + v0, pm);
        quo = sg * ((e1.x * f0[k] + e1.y * v1) / (e1.x * f1[k] + e1.y));
      } else if (kind == PH5_KVRG) {
        quo = v0 * sg;
      }
      exch_t *dst = p.x + bo;
      float out = f0[k] + f1[k] * v0;
      if (kind == PH_ATT_KVR) {
        dst = p.rwkv + bo;
        out = quo;
      } else if (kind == PH_FFN_KR) {
        const float t = fmaxf(v0, 0.f);
        dst = cls ? p.rr + bo : p.kk + (size_t)b * p.F + o;
        out = cls ? quo : t * t;
      } else if (kind == PH5_KVRG) {
        dst = (cls == 0 ? p.k5 : cls == 1 ? p.v5 : cls == 2 ? p.r5 : p.g5) + bo;
        out = cls == 3 ? quo : v0;
      } else if (kind == PH_ATT_O) {
        dst = p.xa + bo;
        out = f0[k] + v0;
      } else if (halve) {
        out *= 0.5f;
      }
      x_store(dst, out, tag);
      if (kind == PH_ATT_KVR) {                  // published before the state is updated
        float *aa = reinterpret_cast<float *>(p.state + (size_t)b * p.state_stride + (size_t)layer * p.layer_stride + off_mid(C, FMT == FMT_FP16)) + o;
        const float2 e2 = exp_pair(f4[k] + f2[k], v0, pm);
        aa[0] = e2.x * f0[k] + e2.y * v1;
        aa[C] = e2.x * f1[k] + e2.y;
        aa[2 * C] = pm;
      }
    }
    __syncwarp();
  }
}

// ---- producer: this CTA's weight tiles in the order the consumers use them ---------------------------
template <int FMT>
struct Tiles {
  int layer = 0, k = 0, rot = 0;          // the phase entered next: layer and index within the layer (layer == L: the head)
  int it = 0, n_items = 0, K = 0, u = 0, n_sub = 0, s = 0, nst = 0, G, cta;
  uint32_t at = 0;                        // of the next tile, 16-byte units from the start of the weights
  uint32_t base = 0;
  bool done = false;
  __device__ __forceinline__ uint32_t bytes() const { return stage_bytes(FMT, min(kt_max(FMT), K - s * kt_max(FMT))); }
  // the tile after a tile of b bytes (b == 0: the first one)
  __device__ __forceinline__ void next(const StepParams &p, uint32_t b) {
    at += b >> 4;
    if (b && ++s < nst) return;
    s = 0;
    if (b && ++u < n_sub) return;
    u = 0;
    it += G;
    while (it >= n_items) {               // the next phase in which this CTA owns a row block
      if (layer > p.L) { done = true; return; }
      const bool head = layer == p.L;
      const StepPhase &ph = head ? p.head : p.ph[k];
      it = cta - rot;
      if (it < 0) it += G;
      K = ph.K; n_items = ph.n_items; n_sub = ph.n_sub; nst = num_stages(FMT, K);
      base = (uint32_t)((ph.w_off + (head ? 0 : (size_t)layer * p.w_stride)) >> 4);
      rot += p.rot_step;
      if (rot >= G) rot -= G;
      if (++k == p.n_ph || head) { k = 0; ++layer; }
    }
    at = base + (uint32_t)(((size_t)it * rowblock_bytes(FMT, K) * n_sub) >> 4);
  }
};

// One cursor walks the tiles; it runs up to `window` bytes ahead of the ring, asks L2 for what it passes and leaves the
// addresses in a queue (shared memory) from which the ring is filled.
constexpr int TILE_QUEUE = 64;
template <int FMT>
__device__ __forceinline__ void produce(Cx &cx) {
  const StepParams &p = *cx.p;
  Tiles<FMT> it;
  it.G = cx.G; it.cta = cx.cta;
  it.next(p, 0);
  int ahead = 0;                         // bytes in the queue
  unsigned head = 0, tail = 0;
  const int window = max(p.l2_prefetch_bytes, 1), ring = cx.n_stages * (int)slot_bytes(FMT);
  int slot = 0;
  uint32_t parity = 1;                   // a fresh barrier reads as "previous phase complete"
  const uint64_t pol = l2_evict_first_policy();
#pragma unroll 1
  while (!it.done || head != tail) {
    if (!it.done && ahead < window && tail - head < TILE_QUEUE) {
      const uint32_t b = it.bytes();
      if (ahead >= ring) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.w + ((size_t)it.at << 4)), "r"(b) : "memory");
      sts64(cx.queue + (tail++ % TILE_QUEUE) * 8u, make_uint2(it.at, b));
      ahead += (int)b;
      it.next(p, b);
      continue;
    }
    const uint2 t = lds64(cx.queue + (head++ % TILE_QUEUE) * 8u);
    if (!bar_wait(cx, &cx.empty[slot], parity, ST_TIMEOUT_EMPTY)) {
      // give copies that are still in flight time to land before the CTA's shared memory goes away
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) { }
      break;
    }
    mbar_expect_tx(&cx.full[slot], t.y);
    bulk_g2s_hint(cx.smem + cx.ring_off + (size_t)slot * slot_bytes(FMT), p.w + ((size_t)t.x << 4), t.y, &cx.full[slot], pol);
    ahead -= (int)t.y;
    if (++slot == cx.n_stages) { slot = 0; parity ^= 1u; }
  }
}

// ------------------------------------------------------------------------------------------------------
// Trace (p.prof): warp 0's time stamps of a phase -- start, operand staged, row blocks done (ns), then the clocks from the
// start to the inputs' arrival and from there to the staged operand.
__device__ __forceinline__ void stamp(const Cx &cx, int pi, int i, unsigned long long v) {
  cx.p->prof[((size_t)cx.cta * (cx.p->L * cx.p->n_ph + 1) + pi) * 8 + i] = v;
}
template <int FMT, int NS, int NV, bool V5>
__device__ __forceinline__ void consume(Cx &cx) {
  const StepParams &p = *cx.p;
  int rot = 0, layer = 0, k = 0;
  unsigned tag = tag_before(tag_of(p, 0));           // of the phase before
  const bool trace = p.prof && cx.tid == 0;
#pragma unroll 1
  for (int pi = 0; layer <= p.L; ++pi, tag = tag_after(tag)) {
    const bool head = layer == p.L;
    const StepPhase &ph = head ? p.head : p.ph[k];
    const int kind = ph.kind, lay = layer, K = ph.K, n_items = ph.n_items;
    int first = cx.cta - rot;                        // this CTA's first row block
    if (first < 0) first += cx.G;
    rot += p.rot_step;
    if (rot >= cx.G) rot -= cx.G;
    if (++k == p.n_ph || head) { k = 0; ++layer; }
    if (V5 && kind == PH5_WKV) { state_v5(cx, lay, pi, tag_after(tag), first); continue; }
    if (first >= n_items) continue;                  // no row block here: nothing to read, nothing to write
    const long long t0 = trace ? clock64() : 0;
    if (trace) stamp(cx, pi, 0, globaltimer_ns());
    const uint32_t vo = (uint32_t)lay * p.vec_stride;
    const bool ffn = kind == PH_FFN_KR, ln = kind != PH_FFN_V && kind != PH_ATT_O;
    const Slots sl(cx, K);
    Operand a;
    a.ln = ln; a.layer0 = lay == 0 && ln && !ffn; a.plain = head || !ln; a.gn = kind == PH_ATT_O;
    a.nvec = a.plain ? 1 : ffn ? 2 : NV;
    a.gtag4 = tag_before(tag) * 0x01010101u;
    a.g = head ? p.v_lnout_w : vo + (ffn ? p.v_ln2_w : ln ? p.v_ln1_w : p.v_lnx_w);
    a.b = head ? p.v_lnout_b : vo + (ffn ? p.v_ln2_b : ln ? p.v_ln1_b : p.v_lnx_b);
#pragma unroll
    for (int v = 0; v < NV; ++v) a.mix[v] = vo + (ffn ? p.v_ffn_mix[v > 0] : p.v_att_mix[v]);
    {
      uint8_t *st0 = p.state + (size_t)lay * p.layer_stride + (ffn ? off_ffn_sx(p.C, p.H, V5, FMT == FMT_FP16, 0) : off_sx(p.C, FMT == FMT_FP16, 0));
      const size_t one = (size_t)p.C * act_bytes(FMT == FMT_FP16);
      a.sx_rd = st0 + p.par * one;
      a.sx_wr = st0 + (p.par ^ 1) * one;
    }
    // shift states are written by the CTAs of the key rows (time mix) or the receptance rows (channel mix)
    a.own = ffn ? first - ph.split % cx.G : first;
    if (a.own < 0) a.own += cx.G;
    if (a.layer0) {
      // embedding rows: plain memory, always there
#pragma unroll 1
      for (int s = 0; s < sl.n_slot; ++s)
#pragma unroll 1
        for (int b = 0; b < (NS == 1 ? 1 : p.B); ++b) {
          if (!sl.has(s)) continue;
          const float4 f = emb4(p, b, sl.i4(s));
          sts128(cx.xw + (uint32_t)sl.local(s) * chunk_operand_bytes<NS>() + (uint32_t)b * 256u + (uint32_t)sl.sub * 16u,
                 make_uint4(__float_as_uint(f.x), __float_as_uint(f.y), __float_as_uint(f.z), __float_as_uint(f.w)));
        }
      __syncwarp();
    } else {
      gather<NS>(cx, sl, kind == PH_FFN_V ? p.kk : kind == PH_ATT_O ? (V5 ? p.o5 : p.rwkv) : ffn ? p.xa : p.x, K, tag * 0x01010101u, pi);
    }
    const long long t1 = trace ? clock64() : 0;
    make_operand<FMT, NS, NV, V5>(cx, sl, K, a, pi);
    if (trace) { stamp(cx, pi, 1, globaltimer_ns()); stamp(cx, pi, 5, t1 - t0); stamp(cx, pi, 7, clock64() - t1); }
    multiply_items<FMT, NS>(cx, K, n_items, ph.n_sub, ph.split, ffn ? 1u : 3u, first);
    if (trace) stamp(cx, pi, 2, globaltimer_ns());
  }
}

template <int FMT, int NS>
__device__ __forceinline__ void finish(Cx &cx, int e) {
  const StepParams &p = *cx.p;
  int rot = 0, layer = 0, k = 0;
  unsigned tag = tag_of(p, 0);
  unsigned long long best = 0;                       // head: packed arg-max over this lane's logits
#pragma unroll 1
  for (int pi = 0; layer <= p.L; ++pi, tag = tag_after(tag)) {
    const bool head = layer == p.L;
    const StepPhase &ph = head ? p.head : p.ph[k];
    const int lay = layer;
    int first = cx.cta - rot;
    if (first < 0) first += cx.G;
    rot += p.rot_step;
    if (rot >= cx.G) rot -= cx.G;
    if (++k == p.n_ph || head) { k = 0; ++layer; }
    if (first < ph.n_items) epilogue_items<FMT, NS>(cx, ph, lay, pi, tag, first, e, best);
  }
  if (p.amax) {
    // one candidate per stream and warp: lanes with equal lane % NS hold the same stream
#pragma unroll
    for (int o = 16; o >= NS; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
      best = other > best ? other : best;
    }
    if (cx.lane < NS && cx.lane < p.B && best) atomicMax(p.amax + cx.lane, best);
  }
}

template <int FMT, int NS, int NV, bool V5>
__global__ void __launch_bounds__(STHREADS, 1) step_kernel(const __grid_constant__ StepParams arg) {
  extern __shared__ __align__(1024) uint8_t step_smem[];
  // The parameters are read from shared memory: from the parameter bank the compiler hoists every one of them out of the
  // layer loop and then spills them.
  StepParams &p = *reinterpret_cast<StepParams *>(step_smem + PARAM_OFF);
  static_assert(sizeof(StepParams) <= QUEUE_OFF - PARAM_OFF, "parameter area");
  for (int i = threadIdx.x; i < (int)(sizeof(StepParams) / 4); i += STHREADS)
    reinterpret_cast<uint32_t *>(&p)[i] = reinterpret_cast<const uint32_t *>(&arg)[i];
  __syncthreads();
  const StepSmem o = step_layout<NS>(FMT, p.C, p.F, p.n_att_vec, p.n_stages);
  Cx cx;
  cx.p = &p;
  cx.smem = step_smem;
  cx.full = reinterpret_cast<uint64_t *>(step_smem);
  cx.empty = cx.full + STEP_MAX_STAGES;
  cx.part_full = cx.empty + STEP_MAX_STAGES;
  cx.part_empty = cx.part_full + EW;
  cx.abort_flag = reinterpret_cast<volatile int *>(cx.part_empty + EW);
  cx.tid = threadIdx.x; cx.warp = threadIdx.x >> 5; cx.lane = threadIdx.x & 31;
  cx.cta = blockIdx.x; cx.G = gridDim.x;
  cx.n_stages = p.n_stages;
  cx.slot = 0; cx.parity = 0; cx.item = 0; cx.ln_buf = 0;
  const uint32_t base = smem_u32(step_smem);
  cx.ln = base + LN_OFF; cx.queue = base + QUEUE_OFF;
  cx.part = base + (uint32_t)o.part; cx.xs = base + (uint32_t)o.xs; cx.ring = base + (uint32_t)o.ring;
  cx.ring_off = o.ring;
  cx.xw = cx.xo = cx.xs;
  for (int w = 0; w < SW; ++w) {
    const uint32_t n = (uint32_t)operand_chunks(p.C, p.F, p.n_att_vec, w) * chunk_operand_bytes<NS>();
    if (w < cx.warp) cx.xw += n;
    if (w < ((cx.tid >> 4) & 7)) cx.xo += n;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.n_stages; ++s) { mbar_init(&cx.full[s], 1); mbar_init(&cx.empty[s], SW); }
    for (int e = 0; e < EW; ++e) { mbar_init(&cx.part_full[e], SW); mbar_init(&cx.part_empty[e], 1); }
    *cx.abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  if (cx.warp < SW) consume<FMT, NS, NV, V5>(cx);
  else if (cx.warp > SW) finish<FMT, NS>(cx, cx.warp - SW - 1);
  else if (cx.lane == 0) produce<FMT>(cx);
}

template <int FMT, int NS>
const void *step_instance(int version, int nvec) {
  if constexpr (FMT != FMT_FP16) return version == 4 ? (const void *)step_kernel<FMT, NS, 3, false> : nullptr;
  else return version == 4 ? (const void *)step_kernel<FMT, NS, 3, false>
         : nvec == 3  ? (const void *)step_kernel<FMT, NS, 3, true> : (const void *)step_kernel<FMT, NS, 4, true>;
}
template <int FMT, int NS>
cudaError_t step_launch_t(const StepParams &p, int grid, size_t smem, cudaStream_t st) {
  void *args[] = {const_cast<StepParams *>(&p)};
  const void *kernel = step_instance<FMT, NS>(p.version, p.n_att_vec);
  if (!kernel) return cudaErrorInvalidValue;
  return cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(STHREADS), args, smem, st);
}
template <int FMT, int NS>
cudaError_t step_prepare_t(int version, int nvec, size_t smem, int device, int *grid) {
  const void *kernel = step_instance<FMT, NS>(version, nvec);
  if (!kernel) return cudaErrorInvalidValue;
  cudaError_t e;
  int optin = 0;
  // the limit is the kernel's, not the model's: models of different widths share the instance
  if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin)) != cudaSuccess) return e;
  int per_sm = 0, sms = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, STHREADS, smem);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  *grid = per_sm > 0 ? sms : 0;
  return cudaSuccess;
}

}  // namespace

size_t step_smem_bytes(int fmt, int mode, int C, int F, int nvec, int n_stages) {
  switch (mode) {
    case 0: return step_layout<1>(fmt, C, F, nvec, n_stages).total;
    case 1: return step_layout<2>(fmt, C, F, nvec, n_stages).total;
    default: return step_layout<4>(fmt, C, F, nvec, n_stages).total;
  }
}

#define FRB_STEP_DISPATCH(fn, ...)                              \
  switch (fmt * STEP_MODES + mode) {                            \
    case 0: return fn<FMT_FP16, 1>(__VA_ARGS__);                \
    case 1: return fn<FMT_FP16, 2>(__VA_ARGS__);                \
    case 2: return fn<FMT_FP16, 4>(__VA_ARGS__);                \
    case 3: return fn<FMT_INT8, 1>(__VA_ARGS__);                \
    case 4: return fn<FMT_INT8, 2>(__VA_ARGS__);                \
    case 6: return fn<FMT_INT4, 1>(__VA_ARGS__);                \
    case 7: return fn<FMT_INT4, 2>(__VA_ARGS__);                \
    default: return cudaErrorInvalidValue;                      \
  }

cudaError_t launch_step(const StepParams &p, int fmt, int mode, int grid, size_t smem, cudaStream_t st) {
  FRB_STEP_DISPATCH(step_launch_t, p, grid, smem, st)
}
cudaError_t step_prepare(int fmt, int mode, int version, int nvec, size_t smem, int device, int *grid) {
  FRB_STEP_DISPATCH(step_prepare_t, version, nvec, smem, device, grid)
}
int step_threads() { return STHREADS; }

}  // namespace frb
