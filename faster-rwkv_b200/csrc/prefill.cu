// Seq mode (prompt processing): T tokens of one stream at once.
//
// Replaces the reference's seq path for RWKV-5.x: def::ModelForwardSeq (kernels/default/model_forward_seq.cpp:48-184),
// _ATT_SEQ_V5_2 + rwkv5_2_kernel_forward (kernels/cuda/att_seq.cu:258-322, 368-423) and _FFN_SEQ
// (kernels/cuda/ffn_seq.cu:65-87).  The projections are [T, K] x [K, N] GEMMs on the tcgen05 tensor cores
// (operands staged by TMA, accumulator in TMEM, epilogue fused); LayerNorm + token shift, the per-head state scan
// and GroupNorm + gate are bandwidth-bound row kernels around them.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <utility>

#include "common.cuh"
#include "internal.h"

namespace frb {

// SMs of the current device (asked once per device): grids and split-K factors are sized from it
int device_sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

thread_local long long row_launches = 0;

namespace {

// Every kernel of the seq / batch chain goes through here.  With FR_B200_PDL != 0 (the default) the launch carries
// the programmatic stream-serialisation attribute: the kernel's CTAs may be scheduled, and run their set-up, while the
// kernel before it in the stream drains; each kernel calls pdl_wait() before it touches global memory, so the data
// dependences are those of plain stream order.
bool pdl_enabled() {
  static const int on = [] { const char *v = getenv("FR_B200_PDL"); return !(v && v[0] == '0'); }();
  return on != 0;
}
template <typename... KArgs, typename... Args>
cudaError_t launch_cluster_k(void (*kern)(KArgs...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = (unsigned)cluster; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl_enabled()) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
  if (e == cudaSuccess) ++row_launches;
  return e;
}
template <typename... KArgs, typename... Args>
cudaError_t launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
  return launch_cluster_k(kern, 1, grid, block, smem, st, std::forward<Args>(args)...);
}

// ------------------------------------------------------------------------------------------------
// tcgen05 GEMMs: out[M, N] = epilogue((A + A2)[M, K] . (Bt)[N, K]^T), fp16 operands (both K-major), fp32
// accumulate.  A2 (optional) holds what rounding the activations to fp16 lost.
// All of them put the weights along the MMA rows, so that an accumulator holds out^T (TMEM lane = output channel, column = row
// of X) and the epilogue's lanes run along the channels; K is walked in 64-wide slices through a TMA ring.
//   warp 0: TMA producer          warp 1: MMA issue; it owns the TMEM allocation
//   warps 2..5: epilogue, one TMEM lane quadrant (32 channels) each
// Warps 0 and 1 run their loops whole and elect a lane for each copy or MMA: in a branch of one lane an MMA took 100 clocks to issue.
constexpr int GBM = 128, GBK = 64;
constexpr int G_THREADS = 192;
constexpr uint32_t G_A_BYTES = GBM * GBK * 2;
constexpr int ST_GEMM_TIMEOUT = 201;

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}
// shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes (64 halfs), 128-byte swizzle, eight-row
// groups 1024 bytes apart: start address / 16 in bits 0-13, leading offset (unused for swizzled K-major) = 1 in
// bits 16-29, stride offset 1024 / 16 in bits 32-45, descriptor version 1 in bits 46-47, layout 2 (128B) in bits 61-63
__device__ __forceinline__ uint64_t umma_desc_k128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor, kind::f16: D = f32 (bits 4-5 = 1), A = B = f16 (0), both K-major (0), N / 8 in bits 17-22,
// M / 16 in bits 24-28
// (built per tile width inside the kernel)

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// the tensor maps are launch parameters: their first use would be a cold fetch in front of the first tile
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap *m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// One lane of a converged warp, the same one every time.  The warps that issue MMAs and copies run their loops whole and elect a lane for the
// instruction: inside a branch that one lane took alone, descriptors and addresses move to uniform registers one by one and an MMA took
// about 100 clocks to issue (a slice of int8 over 160 columns 0.34 us, now 0.24; of int4 0.56, now 0.38).
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(one));
  return one != 0;
}

// Place in a ring of barriers.  Its slot and phase are counted: a division by a depth that only the launch knows costs 100
// to 200 clocks of a chain that takes 300 to 1,000 per slice, and every role had two to four of them.
struct Ring {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next(int depth) {
    if (++slot == depth) { slot = 0; phase ^= 1u; }
  }
};

// By the fast exponential (2 + 1.17 |v| ulp by CUDA's bounds) and division (2 ulp): a relative error of up to 5e-7 for v > 0 and 1.7e-6 at
// v = -8, where the value is 3e-4.  The fp16 rounding of a single result (4.9e-4) hides it; where the low half is stored as well (streams, short
// fp16 prompts: 2.4e-7) it is the larger part of the error.
__device__ __forceinline__ float sigmoid_g(float v) { return __fdividef(1.f, 1.f + __expf(-v)); }

template <int EPI>
__device__ __forceinline__ float epi_half_op(float a) {
  if (EPI == GEMM_EPI_SILU_F16) return a * sigmoid_g(a);
  if (EPI == GEMM_EPI_SIGMOID_F16) return sigmoid_g(a);
  if (EPI == GEMM_EPI_RELU2_F16) { a = fmaxf(a, 0.f); return a * a; }
  return a;
}
__device__ __forceinline__ float epi_half_op(int epi, float a) {
  if (epi == GEMM_EPI_SILU_F16) return a * sigmoid_g(a);
  if (epi == GEMM_EPI_SIGMOID_F16) return sigmoid_g(a);
  if (epi == GEMM_EPI_RELU2_F16) { a = fmaxf(a, 0.f); return a * a; }
  return a;
}
// Up to four GEMMs with the same M in one launch (grid.x walks their N tiles back to back, heaviest first): the
// attention projections of a layer, or the two channel-mix projections that read the LayerNorm output.
// Low halves of X in the pair GEMM: in MMA columns of their own beside the high ones (up to 128 rows; the even CTA holds the high
// half, the odd one the low half), after the high half of the same slice, or after all of K.
enum { LO_BESIDE, LO_EACH, LO_AFTER };
struct GemmGroup {
  int n;
  int stages;                           // ring depth; packed-weight GEMM: weight slots
  int estages, xstages;                 // packed-weight GEMM: expanded slices in TMEM, slots of X (stage_bytes each)
  uint32_t acc_cols, tmem_cols;         // packed-weight GEMM: TMEM columns of the accumulator, and in all
  uint32_t stage_bytes;                 // bytes per ring slot
  int split;                            // split-K factor (grid.z); > 1: CTAs write raw partial sums to GemmArgs::raw
  int dual;                             // few-row GEMM: some problem has A2 (the slot holds an X lo tile)
  int bn, m_tiles;                      // pair GEMM: rows of X per tile, row tiles
  bool lock;                            // pair GEMM: two pairs fit the same SMs
  int lo_mode;                          // pair GEMM: where the low halves of X come in
  int tile_start[GEMM_GROUP_MAX + 1];   // first channel tile of each problem
  GemmArgs p[GEMM_GROUP_MAX];
};
struct alignas(64) GemmMaps {
  CUtensorMap a[GEMM_GROUP_MAX], a2[GEMM_GROUP_MAX], b[GEMM_GROUP_MAX];
  CUtensorMap o[GEMM_GROUP_MAX], o_lo[GEMM_GROUP_MAX];   // results (or slabs) in boxes of 32 channels x 32 rows
};

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- epilogue of all of them ----
// A warp turns 32 rows of X at one channel per lane into 32 x 32 results in shared memory, which a tensor store writes to their
// rows (4 to 10 KB apart) on its own.  Stored by the lanes themselves, 128 bytes a row, a 128 x 128 accumulator took 4 us
// behind the last MMA, 2 of them for the address arithmetic alone; staged it takes 1.5.  Outputs whose rows are not multiples of 16 bytes
// are stored by the lanes.
constexpr uint32_t EPI_BUF = 4096;      // a warp has two: one is filled while the other is read
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void sts_u16(uint32_t a, uint16_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(v) : "memory"); }

// residual stream: acc <- x + acc, or x + r * acc.  8 rows' inputs are asked for before the first is used.
template <bool MUL>
__device__ __forceinline__ void tile_add(const GemmArgs &g, int ch, bool ok, int row0, uint32_t (&acc)[32]) {
  const int nr = ok ? g.M - row0 : 0;
  const size_t o = (size_t)row0 * g.ldo + ch, ld = (size_t)g.ldo;
  const float *x = reinterpret_cast<const float *>(g.aux0) + o;
  const __half *r = reinterpret_cast<const __half *>(g.aux1) + o, *rl = g.aux1_lo ? reinterpret_cast<const __half *>(g.aux1_lo) + o : nullptr;
  const float scale = g.scale;
#pragma unroll
  for (int h = 0; h < 32; h += 8) {
    float xv[8], rv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      xv[i] = h + i < nr ? x[(h + i) * ld] : 0.f;
      rv[i] = !MUL ? 1.f : h + i < nr ? __half2float(r[(h + i) * ld]) : 0.f;
    }
    if (MUL && rl) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (h + i < nr) rv[i] += __half2float(rl[(h + i) * ld]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[h + i] = __float_as_uint((xv[i] + rv[i] * __uint_as_float(acc[h + i])) * scale);
  }
}
template <int EPI>
__device__ __forceinline__ void tile_half(uint32_t buf, bool lo, const uint32_t (&acc)[32]) {
  const uint32_t at = buf + (threadIdx.x & 31) * 2;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float e = epi_half_op<EPI>(__uint_as_float(acc[i]));
    const __half h = __float2half_rn(e);
    sts_u16(at + i * 64, __half_as_ushort(h));
    if (lo) sts_u16(at + 2048 + i * 64, __half_as_ushort(__float2half_rn(e - __half2float(h))));
  }
}
// rows row0 .. row0 + 31, channels ch_w .. ch_w + 31 (lane l: ch_w + l) of one problem; RAW: its slab of K range z.  (A kernel is
// compiled for slabs and for finished results apart: with both in one, the slabs of few rows, a dozen microseconds a product, came
// out half a microsecond later -- 10 fp16 tokens of the RWKV-5 3B shape 2.26 ms against 2.14, 16 streams of the 0.1B shape 381 us against 372.)
template <bool RAW>
__device__ __forceinline__ void tile_out(const GemmArgs &g, const CUtensorMap *om, const CUtensorMap *om_lo, int z, int ch_w,
                                         int row0, uint32_t (&acc)[32], uint32_t buf) {
  const int lane = threadIdx.x & 31, ch = ch_w + lane;
  const bool ok = ch < g.N;
  const int epi = RAW ? GEMM_EPI_F32 : g.epi;
  if (epi == GEMM_EPI_ADD_F32) tile_add<false>(g, ch, ok, row0, acc);
  else if (epi == GEMM_EPI_MULADD_F32) tile_add<true>(g, ch, ok, row0, acc);
  const bool f32 = epi == GEMM_EPI_F32 || epi == GEMM_EPI_ADD_F32 || epi == GEMM_EPI_MULADD_F32;
  if (RAW || g.tma_out) {
    if (f32) {
#pragma unroll
      for (int i = 0; i < 32; ++i) sts_u32(buf + i * 128 + lane * 4, acc[i]);
    } else {
      const bool lo = g.out_lo != nullptr;
      if (epi == GEMM_EPI_SILU_F16) tile_half<GEMM_EPI_SILU_F16>(buf, lo, acc);
      else if (epi == GEMM_EPI_SIGMOID_F16) tile_half<GEMM_EPI_SIGMOID_F16>(buf, lo, acc);
      else if (epi == GEMM_EPI_RELU2_F16) tile_half<GEMM_EPI_RELU2_F16>(buf, lo, acc);
      else tile_half<GEMM_EPI_PLAIN_F16>(buf, lo, acc);
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      if (ch_w < g.N) {
        tma_store_3d(om, buf, ch_w, row0, RAW ? z : 0);
        if (!f32 && g.out_lo) tma_store_3d(om_lo, buf + 2048, ch_w, row0, 0);
      }
      asm volatile("cp.async.bulk.commit_group;\ncp.async.bulk.wait_group.read 1;" ::: "memory");   // the other buffer is free again
    }
    __syncwarp();
    return;
  }
  if (!ok) return;
  const size_t o = (size_t)row0 * g.ldo + ch, ld = (size_t)g.ldo;
  const int nr = g.M - row0;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (i >= nr) continue;
    if (f32) {
      reinterpret_cast<float *>(g.out)[o + i * ld] = __uint_as_float(acc[i]);
    } else {
      float e = __uint_as_float(acc[i]);
      e = epi == GEMM_EPI_SILU_F16 ? epi_half_op<GEMM_EPI_SILU_F16>(e) : epi == GEMM_EPI_SIGMOID_F16 ? epi_half_op<GEMM_EPI_SIGMOID_F16>(e)
          : epi == GEMM_EPI_RELU2_F16 ? epi_half_op<GEMM_EPI_RELU2_F16>(e) : e;
      const __half h = __float2half_rn(e);
      reinterpret_cast<__half *>(g.out)[o + i * ld] = h;
      if (g.out_lo) reinterpret_cast<__half *>(g.out_lo)[o + i * ld] = __float2half_rn(e - __half2float(h));
    }
  }
}

// Slabs of up to 32 rows are stored by the lanes: the way through shared memory and a tensor store takes longer than it saves
// (29 int4 tokens of the 1.5B shape 1.50 against 1.53 ms, 16 int8 streams 1.33 against 1.35).
__device__ __forceinline__ void slab_rows(const GemmArgs &g, int z, int ch, int row0, const uint32_t (&acc)[32]) {
  if (ch >= g.N) return;
  float *dst = g.raw + ((size_t)z * g.M + row0) * g.N + ch;
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (row0 + i < g.M) dst[(size_t)i * g.N] = __uint_as_float(acc[i]);
}
// before the CTA may end: its stores have read shared memory
__device__ __forceinline__ void tile_out_end() {
  if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
// the address, in the cluster's shared window, of this CTA's shared address `a` in CTA `rank`
__device__ __forceinline__ uint32_t mapa_u32(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// tile into this CTA's shared memory, bytes counted on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on a barrier of either CTA of the cluster (address from mapa_u32).  Relaxed: it hands over no memory, but columns of TMEM, whose
// writes are complete (tcgen05.wait::st) and ordered by the tcgen05 fences on both sides.  With .release it took 500 to 900 clocks, a slice of
// int8 0.70 us instead of 0.50.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ---- TMEM of a pair of CTAs ----
// tcgen05.alloc / dealloc with cta_group::2 are one operation of a warp of each CTA, and ask that the other CTA has been launched and has not
// left: they stand between cluster barriers.  An SM lets one CTA at a time allocate, from its allocation until it gives the permit back, so two
// pairs that start on the same two SMs at once could each hold the permit of one SM and wait for that of the other for good (a chain of
// products of 300 and 500 rows with a busy row kernel between them stood still, once in some million launches).  Where two pairs fit the same
// SMs (`lock`) they take turns: the even CTA takes the lock of its SM pair, asked for while the CTA sets up, tells the odd one, and gives
// it back when both have their columns.  The first weights are under way meanwhile.
// Every wait is bounded: the lock's for half of what the odd CTA waits, so that one never allocates without the other.  The kernels
// behind may start (pdl_trigger, by every thread) only then: one that took the columns first would wait for this kernel with them.
struct PairTmem {
  uint64_t go, there;        // the odd CTA may allocate; it has
  uint32_t sm, slot;         // this CTA's SM; address of its columns
  int held, ready;           // they are allocated; in both CTAs
};
constexpr int PAIR_LOCKS = 1024;
constexpr uint32_t PAIR_ALONE_SMEM = 150u << 10;   // of 227 KB: a pair kernel without the lock asks for this much at least, one with it for 80 KB
__device__ int pair_lock[PAIR_LOCKS];

__device__ __forceinline__ uint32_t sm_id() {
  uint32_t sm;
  asm volatile("mov.u32 %0, %smid;" : "=r"(sm));
  return sm;
}
__device__ __forceinline__ void pair_tmem_init(PairTmem *t) {   // one thread, ahead of the fence and the cluster barrier
  mbar_init(&t->go, 1);
  mbar_init(&t->there, 1);
  t->sm = sm_id();
}
// Warp 1, ahead of the cluster barrier.  The lock is that of half the smaller SM id, which is half of this one's where a pair has SMs 2 i and 2 i + 1.
__device__ __forceinline__ int pair_tmem_ask(uint32_t rank, bool lock) {
  return lock && rank == 0 && (threadIdx.x & 31) == 0 ? atomicCAS(&pair_lock[sm_id() / 2 % PAIR_LOCKS], 0, 1) : 0;
}
__device__ __forceinline__ void pair_tmem_get(PairTmem *t, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&t->slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
// one warp of each CTA, after the cluster barrier
__device__ __forceinline__ void pair_tmem_alloc(PairTmem *t, uint32_t rank, bool locked, int asked, uint32_t cols, volatile int *abort_flag, int *status) {
  const int lane = threadIdx.x & 31;
  bool ok = true, ready = true;
  if (rank == 0) {
    int *lock = nullptr;
    if (locked && lane == 0) {
      uint32_t other;
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(other) : "r"(mapa_u32(smem_u32(&t->sm), 1)) : "memory");
      int *guess = &pair_lock[sm_id() / 2 % PAIR_LOCKS];
      lock = &pair_lock[min(t->sm, other) / 2 % PAIR_LOCKS];
      if (lock != guess) {
        if (asked == 0) atomicExch(guess, 0);
        asked = atomicCAS(lock, 0, 1);
      }
      const unsigned long long t0 = globaltimer_ns();
      for (; asked != 0; asked = atomicCAS(lock, 0, 1)) {
        if (globaltimer_ns() - t0 > WAIT_LIMIT_NS / 2) {
          *abort_flag = 1;
          atomicCAS(status, 0, ST_GEMM_TIMEOUT);
          ok = false;
          break;
        }
      }
      if (ok) mbar_arrive_cluster(mapa_u32(smem_u32(&t->go), 1));
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok) {
      pair_tmem_get(t, cols);
      ready = __all_sync(0xffffffffu, mbar_wait(&t->there, 0, abort_flag, status, ST_GEMM_TIMEOUT));
      if (locked && lane == 0) atomicExch(lock, 0);
    }
  } else {
    ok = !locked || __all_sync(0xffffffffu, mbar_wait(&t->go, 0, abort_flag, status, ST_GEMM_TIMEOUT));
    if (ok) {
      pair_tmem_get(t, cols);
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&t->there), 0));
    }
  }
  if (lane == 0) { t->held = ok; t->ready = ok && ready; }
  tc_fence_before();
  __syncwarp();
}
// all threads of the CTA, each role's warps at a place of their own
__device__ __forceinline__ bool pair_tmem_ready(const PairTmem *t) {
  asm volatile("bar.sync 1, %0;" ::"r"(blockDim.x) : "memory");
  tc_fence_after();
  pdl_trigger();
  return t->ready != 0;
}
// all threads of both CTAs; neither leaves while the other's MMAs, commits or deallocation may still reach into it
__device__ __forceinline__ void pair_tmem_end(const PairTmem *t, int warp, uint32_t cols) {
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  if (warp == 1 && t->held) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(t->slot), "r"(cols) : "memory");
  }
  __syncwarp();
  cluster_sync();
}
// arrives on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}

// ------------------------------------------------------------------------------------------------
// fp16 weights, more than 128 rows (64, with low halves): out^T[256 channels, BN rows] per pair of CTAs (BN a multiple of 32 up to 256,
// chosen at launch).  The pair is one tcgen05.mma.cta_group::2: each CTA holds the weights of its own 128 channels and
// half of the X tile, so a slice of 64 inputs costs an SM 16 KB of weights and 16 KB of X for 512 clocks of MMA, where a CTA
// of its own with the same 128 x 256 accumulator would fetch, and read from shared memory at every MMA, all 32 KB of X.
// Two CTAs per SM (3 slots of 32 KB and 256 TMEM columns each): the start and the end of one hide in part behind the main loop
// of the other, and tiles are handed out by the hardware, also across the two row pieces of a long prompt.
// [2048 x 2560] x [2560 x 11520] with the relu^2 epilogue: 104 us back to back (1,160 TFLOP/s; a single launch 94 to 95) at 256 rows a tile; 256 x 256 tiles of single CTAs,
// whose epilogue nothing hid, 182.  Without its epilogue 82, without its loads 100 (of 107 then): the epilogue is what is left.  One
// CTA per SM over all tiles with two accumulators: 92, but products of one wave 10 to 40 % slower, a prompt of 4,096 36.4 ms against 35.0.
//   warp 0: TMA into the own shared memory; the bytes of both CTAs are counted on the even CTA's barrier
//   warp 1: TMEM, and in the even CTA the MMAs of the pair        warps 2..5: epilogue, a TMEM lane quadrant each
// Low halves of X (A2) meet the same weights beside the high ones, after them in the same slot, or in slots of their own after
// all of K (LO_BESIDE, LO_EACH, LO_AFTER): sums in the order they always had, which RWKV-5 asks for.
constexpr int PAIR_MAX_STAGES = 8;
constexpr uint32_t PAIR_TMEM_COLS = 256;

template <bool SLABS>
__global__ void __launch_bounds__(G_THREADS, 2)
gemm_pair_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmGroup grp) {
  const int STAGES = grp.stages, BN = grp.bn;
  const uint32_t STAGE_BYTES = grp.stage_bytes;
  extern __shared__ uint8_t gsm_raw[];
  // the same offsets in both CTAs: barriers in the first KB, tiles from the next 1024-byte boundary
  uint8_t *gsm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gsm_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(gsm);
  uint64_t *empty = full + PAIR_MAX_STAGES;
  uint64_t *acc_full = empty + PAIR_MAX_STAGES;
  PairTmem *tmem = reinterpret_cast<PairTmem *>(acc_full + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem + 1);
  const uint32_t tiles = smem_u32(gsm + 1024);
  const int warp = threadIdx.x >> 5;
  const uint32_t rank = cluster_rank();
  // pairs walk the row tiles of one channel tile before the next channel tile
  const int pair = blockIdx.x >> 1, ct = pair / grp.m_tiles, m0 = (pair - ct * grp.m_tiles) * BN;
  int pi = 0;
  while (pi + 1 < grp.n && ct >= grp.tile_start[pi + 1]) ++pi;
  const GemmArgs &g = grp.p[pi];
  const int ch0 = (ct - grp.tile_start[pi]) * (2 * GBM) + (int)rank * GBM;
  const int num_k1 = g.K / GBK;
  const int kz0 = (int)((long long)blockIdx.z * num_k1 / grp.split), nkz = (int)((long long)(blockIdx.z + 1) * num_k1 / grp.split) - kz0;
  const bool has_lo = g.A2 != nullptr;
  const bool wide = has_lo && grp.lo_mode == LO_BESIDE, lo_now = has_lo && grp.lo_mode == LO_EACH, lo_pass = has_lo && grp.lo_mode == LO_AFTER;
  const int cols = wide ? 2 * BN : BN;                            // MMA columns; this CTA holds half of them
  const uint32_t X_BYTES = (uint32_t)cols * (GBK * 2 / 2);
  const uint32_t IDESC = (1u << 4) | ((uint32_t)(cols >> 3) << 17) | ((uint32_t)(2 * GBM >> 4) << 24);
  const int num_e = lo_pass ? 2 * nkz : nkz;

  if (threadIdx.x == 64) { prefetch_tmap(&maps.b[pi]); prefetch_tmap(&maps.a[pi]); if (has_lo) prefetch_tmap(&maps.a2[pi]); }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    pair_tmem_init(tmem);
    *abort_flag = 0;
    mbar_fence_init();
  }
  const int asked = warp == 1 ? pair_tmem_ask(rank, grp.lock) : 0;
  __syncthreads();
  cluster_sync();      // both CTAs are there, and their barriers exist before either one's copies arrive on them

  if (warp == 0) {
    // the weights do not depend on the kernels before this one: the first round of them is asked for ahead of the wait
    const int pre = num_e < STAGES ? num_e : STAGES;
    for (int e = 0; e < pre; ++e)
      if (elect_one()) tma_load_2d_pair(tiles + (uint32_t)e * STAGE_BYTES, &maps.b[pi], (kz0 + (e < nkz ? e : e - nkz)) * GBK, ch0, mapa_u32(smem_u32(&full[e]), 0));
    pair_tmem_ready(tmem);
    pdl_wait();
    Ring at;
    for (int e = 0; e < num_e; ++e, at.next(STAGES)) {
      const int s = at.slot;
      const uint32_t dst = tiles + (uint32_t)s * STAGE_BYTES, bar = mapa_u32(smem_u32(&full[s]), 0);
      const int kx = (kz0 + (e < nkz ? e : e - nkz)) * GBK, row = wide ? m0 : m0 + (int)rank * (BN / 2);
      if (e >= pre) {
        if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], at.phase ^ 1u, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
        if (elect_one()) tma_load_2d_pair(dst, &maps.b[pi], kx, ch0, bar);
      }
      if (elect_one()) {
        if (rank == 0) mbar_expect_tx(&full[s], 2 * (G_A_BYTES + (lo_now ? 2u : 1u) * X_BYTES));   // (bytes that arrived before are counted, too)
        tma_load_2d_pair(dst + G_A_BYTES, (wide ? rank == 0 : e < nkz) ? &maps.a[pi] : &maps.a2[pi], kx, row, bar);
        if (lo_now) tma_load_2d_pair(dst + G_A_BYTES + X_BYTES, &maps.a2[pi], kx, row, bar);
      }
    }
  } else if (warp == 1) {
    pair_tmem_alloc(tmem, rank, grp.lock, asked, PAIR_TMEM_COLS, abort_flag, g.status);
    const bool there = pair_tmem_ready(tmem);
    const uint32_t tmem_base = tmem->slot;
    if (rank == 0 && there) {
      Ring at;
      for (int e = 0; e < num_e; ++e, at.next(STAGES)) {
        const int s = at.slot;
        if (!__all_sync(0xffffffffu, mbar_wait(&full[s], at.phase, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
        tc_fence_after();
        const uint32_t base = tiles + (uint32_t)s * STAGE_BYTES;
        const uint64_t wd = umma_desc_k128(base), xd = umma_desc_k128(base + G_A_BYTES);
        if (elect_one()) {
#pragma unroll
          for (int k4 = 0; k4 < GBK / 16; ++k4)
            umma_f16_pair(tmem_base, wd + (uint64_t)(k4 * 2), xd + (uint64_t)(k4 * 2), IDESC, (e | k4) != 0);
          if (lo_now) {
            const uint64_t xl = umma_desc_k128(base + G_A_BYTES + X_BYTES);
#pragma unroll
            for (int k4 = 0; k4 < GBK / 16; ++k4) umma_f16_pair(tmem_base, wd + (uint64_t)(k4 * 2), xl + (uint64_t)(k4 * 2), IDESC, 1u);
          }
          umma_commit_pair(&empty[s]);
        }
        __syncwarp();
      }
      if (elect_one()) umma_commit_pair(acc_full);
    }
  } else {
    const int quad = warp & 3;
    const bool there = pair_tmem_ready(tmem);
    const uint32_t tmem_base = tmem->slot;
    pdl_wait();
    const bool ok = there && __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, g.status, ST_GEMM_TIMEOUT));
    tc_fence_after();
    if (ok) {
      const uint32_t buf = tiles + (uint32_t)quad * 2 * EPI_BUF;   // the ring has been read
      uint32_t flip = 0;
      for (int c0 = 0; c0 < BN; c0 += 32, flip ^= EPI_BUF) {
        if (m0 + c0 >= g.M) break;   // warp-uniform
        uint32_t acc[32];
        const uint32_t at_acc = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
        tmem_ld32(at_acc, acc);
        if (wide) {
          uint32_t part[32];
          tmem_ld32(at_acc + (uint32_t)BN, part);
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = __float_as_uint(__uint_as_float(acc[i]) + __uint_as_float(part[i]));
        }
        tile_out<SLABS>(g, &maps.o[pi], &maps.o_lo[pi], blockIdx.z, ch0 + quad * 32, m0 + c0, acc, buf + flip);
      }
      tile_out_end();
    }
  }
  pair_tmem_end(tmem, warp, PAIR_TMEM_COLS);
}

// ------------------------------------------------------------------------------------------------
// Few rows (batched decode: one row per stream, or a short prompt): the same product with the operands' roles
// swapped, out^T[N, M] = W^T[N, K] . X[M, K]^T.  The 128 MMA rows are 128 output channels of the weight matrix, the
// MMA columns are the up to BN = 32, 64 or 128 rows of X, so a ring slot is 16 KB of weights plus a small X tile instead of a
// 128-row X tile that is mostly zero fill plus 8 KB of weights: several times the weight bytes in flight per SM,
// which is what a step that streams every weight once is bound by.  The low halves of X (A2) sit in the same slot.
// The accumulator holds out^T: TMEM lane = output channel, column = row of X; the epilogue warps write with the
// lanes along the channels (coalesced), either the finished values or the split-K slabs gemm_finish_kernel sums.
constexpr int WT_MAX_STAGES = 8;

// grp.dual here: some problem has A2 (the slot holds an X lo tile)
template <int BN, bool SLABS>
__global__ void __launch_bounds__(G_THREADS, 2)
gemm_wt_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmGroup grp) {
  constexpr uint32_t X_BYTES = BN * GBK * 2;
  constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(GBM >> 4) << 24);
  // the hi and lo tiles of X, back to back in the slot, are one B operand of 2 BN rows (accumulator columns [0, BN) and
  // [BN, 2 BN), added up by the epilogue): an MMA with few columns costs about as much as a wide one
  constexpr uint32_t IDESC2 = (1u << 4) | ((uint32_t)((2 * BN) >> 3) << 17) | ((uint32_t)(GBM >> 4) << 24);
  constexpr uint32_t TMEM_COLS = 2 * BN;
  const int STAGES = grp.stages;
  const uint32_t STAGE_BYTES = grp.stage_bytes;
  constexpr uint32_t X_OFF = G_A_BYTES, XLO_OFF = X_OFF + X_BYTES;
  extern __shared__ uint8_t gsm_raw[];
  uint8_t *gsm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gsm_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(gsm);
  uint64_t *empty = full + WT_MAX_STAGES;
  uint64_t *acc_full = empty + WT_MAX_STAGES;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t tiles = smem_u32(gsm + 1024);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int pi = 0;
  while (pi + 1 < grp.n && (int)blockIdx.x >= grp.tile_start[pi + 1]) ++pi;
  const GemmArgs &g = grp.p[pi];
  const int tile_n = blockIdx.x - grp.tile_start[pi];
  const int num_k1 = g.K / GBK;
  const int kz0 = (int)((long long)blockIdx.z * num_k1 / grp.split), nkz = (int)((long long)(blockIdx.z + 1) * num_k1 / grp.split) - kz0;
  const bool x_lo = g.A2 != nullptr;

  if (threadIdx.x == 64) {
    prefetch_tmap(&maps.b[pi]); prefetch_tmap(&maps.a[pi]);
    if (x_lo) prefetch_tmap(&maps.a2[pi]);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  // The weights are constants: the ring's first round of weight tiles is on its way before the kernels ahead of this
  // one have finished.  What they wrote (X, the epilogue's inputs and outputs) is touched only after pdl_wait(): by
  // the X loads and by the epilogue warps.

  if (warp == 0) {
    const uint32_t w_bytes = G_A_BYTES, x_bytes = (x_lo ? 2u : 1u) * X_BYTES;
    const int pre = nkz < STAGES ? nkz : STAGES;
    for (int kb = 0; kb < pre; ++kb) {
      if (!elect_one()) continue;
      mbar_expect_tx_only(&full[kb], w_bytes);
      const uint32_t dst = tiles + (uint32_t)kb * STAGE_BYTES;
      tma_load_2d(dst, &maps.b[pi], (kz0 + kb) * GBK, tile_n * GBM, &full[kb]);
    }
    pdl_wait();
    Ring at;
    for (int kb = 0; kb < nkz; ++kb, at.next(STAGES)) {
      const int s = at.slot;
      const uint32_t dst = tiles + (uint32_t)s * STAGE_BYTES;
      const int kx = (kz0 + kb) * GBK;
      if (kb >= pre) {
        if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], at.phase ^ 1u, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
      }
      if (elect_one()) {
        if (kb >= pre) {
          mbar_expect_tx(&full[s], w_bytes + x_bytes);
          tma_load_2d(dst, &maps.b[pi], kx, tile_n * GBM, &full[s]);
        } else {
          mbar_expect_tx(&full[s], x_bytes);
        }
        tma_load_2d(dst + X_OFF, &maps.a[pi], kx, 0, &full[s]);
        if (x_lo) tma_load_2d(dst + XLO_OFF, &maps.a2[pi], kx, 0, &full[s]);
      }
    }
  } else if (warp == 1) {
    Ring at;
    for (int kb = 0; kb < nkz; ++kb, at.next(STAGES)) {
      const int s = at.slot;
      if (!__all_sync(0xffffffffu, mbar_wait(&full[s], at.phase, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
      tc_fence_after();
      const uint32_t base = tiles + (uint32_t)s * STAGE_BYTES;
      const uint64_t wd = umma_desc_k128(base), xd = umma_desc_k128(base + X_OFF);
      if (elect_one()) {
#pragma unroll
        for (int k4 = 0; k4 < GBK / 16; ++k4)
          umma_f16(tmem_base, wd + (uint64_t)(k4 * 2), xd + (uint64_t)(k4 * 2), x_lo ? IDESC2 : IDESC, (kb | k4) != 0);
        umma_commit(&empty[s]);
      }
      __syncwarp();
    }
    if (elect_one()) umma_commit(acc_full);
  } else {
    const int quad = warp & 3;
    const int ch_w = tile_n * GBM + quad * 32;
    pdl_wait();
    const bool ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, g.status, ST_GEMM_TIMEOUT));
    tc_fence_after();
    if (ok) {
      const uint32_t buf = tiles + (uint32_t)quad * 2 * EPI_BUF;   // the ring has been read
      uint32_t flip = 0;
      for (int c0 = 0; c0 < BN; c0 += 32, flip ^= EPI_BUF) {
        if (c0 >= g.M) break;   // warp-uniform
        uint32_t acc[32];
        tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, acc);
        if (x_lo) {
          uint32_t part[32];
          tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(BN + c0), part);
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = __float_as_uint(__uint_as_float(acc[i]) + __uint_as_float(part[i]));
        }
        if (SLABS && BN == 32) slab_rows(g, blockIdx.z, ch_w + lane, c0, acc);
        else tile_out<SLABS>(g, &maps.o[pi], &maps.o_lo[pi], blockIdx.z, ch_w, c0, acc, buf + flip);
      }
      tile_out_end();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// Expansion of packed weights to fp16 pairs.
// int4: four bytes (8 consecutive inputs) -> hi = fp16(q s), lo = q s - hi (exact); s2 = {s, s}
__device__ __forceinline__ void expand_int4(uint32_t word, uint32_t s2, uint32_t *hi, uint32_t *lo) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    // byte j -> {1024 + low nibble, 64 + high nibble} - {1032, 72} = {q_even, q_odd}
    const uint32_t x = prmt(word, 0u, 0x4040u + (uint32_t)j * 0x0101u);   // bytes [b_j, 0, b_j, 0]
    const uint32_t qv = hsub2_u32(lop3_and_or(x, 0x00f0000fu, 0x54006400u), 0x54806408u);
    hi[j] = hmul2_u32(qv, s2);
    lo[j] = hfma2_u32(qv, s2, hi[j] ^ 0x80008000u);
  }
}
// int8: four codes -> their values, exact
__device__ __forceinline__ void expand_int8(uint32_t word, uint32_t *out) {
  const uint32_t M = 0x64646464u, OFF = 0x64806480u, w = word ^ 0x80808080u;    // 1024 + (code + 128) - 1152 = code
  out[0] = hsub2_u32(prmt(w, M, 0x4140), OFF);
  out[1] = hsub2_u32(prmt(w, M, 0x4342), OFF);
}
// The group scales of one row of int4 weights, slice by slice: straight from global memory, 16 bytes (four slices) at a
// time and four slices ahead of their use, so that the expansion never waits for them; rows whose scales are not 16-byte
// aligned (K not a multiple of 256) take them slice by slice, one ahead.
struct GroupScales {
  const __half *gs;      // null: a row that does not exist
  bool quads;
  int nquads, kz0, kend;
  uint4 scq, scq_next;
  uint32_t sc_next;
  __device__ __forceinline__ void start(const GemmArgs &g, int ch, int k0, int nk) {
    gs = ch < g.N ? g.wq_scale + (size_t)ch * (g.K / 32) : nullptr;
    quads = ((g.K / 32) & 7) == 0;
    nquads = g.K / 256;
    kz0 = k0; kend = k0 + nk;
    scq = scq_next = make_uint4(0x3c003c00u, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u);
    sc_next = 0x3c003c00u;
    if (!gs || nk <= 0) return;
    if (quads) {
      scq = *reinterpret_cast<const uint4 *>(gs + (size_t)(kz0 >> 2) * 8);
      if ((kz0 >> 2) + 1 < nquads) scq_next = *reinterpret_cast<const uint4 *>(gs + (size_t)((kz0 >> 2) + 1) * 8);
    } else {
      sc_next = *reinterpret_cast<const uint32_t *>(gs + (size_t)kz0 * 2);
    }
  }
  __device__ __forceinline__ uint32_t at(int ks) {   // called with ks = kz0, kz0 + 1, ...: scales of the slice's two groups
    uint32_t sc = sc_next;
    if (quads) {
      if (ks > kz0 && (ks & 3) == 0) {
        scq = scq_next;
        if (gs && (ks >> 2) + 1 < nquads) scq_next = *reinterpret_cast<const uint4 *>(gs + (size_t)((ks >> 2) + 1) * 8);
      }
      const int qi = ks & 3;
      sc = qi == 0 ? scq.x : qi == 1 ? scq.y : qi == 2 ? scq.z : scq.w;
    } else if (gs && ks + 1 < kend) {
      sc_next = *reinterpret_cast<const uint32_t *>(gs + (size_t)(ks + 1) * 2);
    }
    return sc;
  }
};

// ------------------------------------------------------------------------------------------------
// Quantised weights, read in their packed form (int8 codes [N, K], or int4 nibbles [N, K/2] with fp16 group scales [N, K/32]: the
// bytes a step has to stream).  Eight warps expand a slice of 64 inputs straight into the MMA's A operand in TMEM (lane =
// channel, a column = two inputs), so shared memory carries X alone.
//   PAIR:  more than 128 rows; out^T[256 channels, BN rows] per pair of SMs as in gemm_pair_kernel, one CTA per SM.  Expanded into
//          shared memory instead (one CTA, 128 x 256), a slice of int4 asked it for 163 bytes a clock where it gives 128.
//   !PAIR: up to 128 rows; out^T[128 channels, BN rows] per CTA, two CTAs per SM where 256 columns of TMEM hold the accumulator
//          and some slices.  A step of few streams is a chain of such products of 3 to 11 slices each: every slice that has a
//          slot is loaded and expanded before the kernels ahead have finished, and what is left behind them is X, its MMAs and the epilogue.
//   warp 0      TMA: X into slot x, counted on the even CTA's barrier (PAIR: X and expanded slices share their slots, and that barrier
//               also counts the expanders of both CTAs: the thread that issues the MMAs has one wait and one commit per slice)
//   warp 1      TMEM; (in the even CTA) the MMAs: acc += W_hi X_hi, W_hi X_lo, and for int4 W_lo X_hi (int8 codes are exact in
//               fp16, the row scale is applied to the accumulator; int4: hi = fp16(q s), lo = q s - hi, an exact pair)
//   EW warps    expanders: warp quadrant = TMEM lane quadrant, two warps share a row's 64 inputs (one scale group each); then epilogue
//   last warp   TMA: packed weights, 128 rows x 128 bytes = 4 (int4) or 2 (int8) slices per slot
// !PAIR: the hi and lo halves of X sit back to back in a slot and are one B operand of 2 BN rows: one MMA gives W X_hi in
// accumulator columns [0, BN) and W X_lo in [BN, 2 BN), which the epilogue adds up (an MMA with few columns costs as much as a
// wide one).  PAIR: the halves multiply into the same accumulator, slice by slice.
__device__ __forceinline__ void umma_f16_ta(bool pair, uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if (pair)
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}

// EW expander warps: 8 where two CTAs share an SM, else 16 in two groups of eight that take the slices in turn: a warp's way through a slice
// (wait, load, expand, wait, store, hand over) is longer than the MMAs of most (512 clocks at 256 columns and one pass).
constexpr int gq_threads(int ew) { return 32 * (3 + ew); }
constexpr int GQ_MAX = 8;                // most slots of any ring

template <int FMT, bool PAIR, int EW, bool SLABS>
__global__ void __launch_bounds__(gq_threads(EW), EW == 8 ? 2 : 1)
gemm_q_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmGroup grp) {
  constexpr uint32_t ROW_B = FMT == FMT_INT8 ? GBK : GBK / 2;          // packed bytes per row and slice
  constexpr int KSH = FMT == FMT_INT8 ? 1 : 2, KSUB = 1 << KSH;        // slices per weight slot
  constexpr uint32_t WS_BYTES = GBM * 128;
  constexpr uint32_t A_COLS = FMT == FMT_INT4 ? 64 : 32;               // expanded slice: hi (+ lo)
  constexpr int CH = PAIR ? 2 * GBM : GBM;
  const int NW = grp.stages, NE = grp.estages, NX = grp.xstages, BN = grp.bn;
  const uint32_t X_BYTES = (uint32_t)(PAIR ? BN / 2 : BN) * (GBK * 2), XS_BYTES = grp.stage_bytes;
  const uint32_t IDESC = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(CH >> 4) << 24);
  const uint32_t IDESC2 = (1u << 4) | ((uint32_t)((2 * BN) >> 3) << 17) | ((uint32_t)(CH >> 4) << 24);
  extern __shared__ uint8_t gsm_raw[];
  uint8_t *gsm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gsm_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t *wfull = reinterpret_cast<uint64_t *>(gsm);
  uint64_t *wempty = wfull + GQ_MAX;
  uint64_t *xfull = wempty + GQ_MAX;
  uint64_t *xempty = xfull + GQ_MAX;
  uint64_t *a_full = xempty + GQ_MAX;
  uint64_t *a_empty = a_full + GQ_MAX;
  uint64_t *acc_full = a_empty + GQ_MAX;
  PairTmem *tmem = reinterpret_cast<PairTmem *>(acc_full + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem + 1);
  const uint32_t xtiles = smem_u32(gsm + 1024), wtiles = xtiles + (uint32_t)NX * XS_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  const int id = PAIR ? blockIdx.x >> 1 : blockIdx.x, ct = id / grp.m_tiles, m0 = (id - ct * grp.m_tiles) * BN;
  int pi = 0;
  while (pi + 1 < grp.n && ct >= grp.tile_start[pi + 1]) ++pi;
  const GemmArgs &g = grp.p[pi];
  const int ch0 = (ct - grp.tile_start[pi]) * CH + (int)rank * GBM;
  const int num_k1 = g.K / GBK;
  const int kz0 = (int)((long long)blockIdx.z * num_k1 / grp.split), nkz = (int)((long long)(blockIdx.z + 1) * num_k1 / grp.split) - kz0;
  const bool x_lo = g.A2 != nullptr;
  const int g0 = kz0 >> KSH, ng = nkz > 0 ? ((kz0 + nkz - 1) >> KSH) - g0 + 1 : 0;   // weight slots of this K range

  if (threadIdx.x == 64) { prefetch_tmap(&maps.b[pi]); prefetch_tmap(&maps.a[pi]); if (x_lo) prefetch_tmap(&maps.a2[pi]); }
  if (threadIdx.x == 0) {
    for (int s = 0; s < NW; ++s) { mbar_init(&wfull[s], 1); mbar_init(&wempty[s], EW); }
    for (int x = 0; x < NX; ++x) { mbar_init(&xfull[x], PAIR ? 1 + 8 + 1 : 1); mbar_init(&xempty[x], 1); }
    for (int e = 0; e < NE; ++e) { mbar_init(&a_full[e], 8); mbar_init(&a_empty[e], 1); }
    mbar_init(acc_full, 1);
    if (PAIR) pair_tmem_init(tmem);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (!PAIR && warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem->slot)), "r"(grp.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();      // both CTAs are there, and their barriers exist before anything arrives on them from the other one
  tc_fence_after();
  uint32_t tmem_base = 0;
  if (!PAIR) {
    tmem_base = tmem->slot;
    pdl_trigger();
  }

  if (warp == 0) {
    if (PAIR) pair_tmem_ready(tmem);
    pdl_wait();
    Ring at;
    for (int kb = 0; kb < nkz; ++kb, at.next(NX)) {
      if (!__all_sync(0xffffffffu, mbar_wait(PAIR ? &a_empty[at.slot] : &xempty[at.slot], at.phase ^ 1u, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
      if (!elect_one()) continue;
      const uint32_t dst = xtiles + (uint32_t)at.slot * XS_BYTES;
      const int kx = (kz0 + kb) * GBK;
      if (PAIR) {
        const uint32_t bar = mapa_u32(smem_u32(&xfull[at.slot]), 0);
        const int row = m0 + (int)rank * (BN / 2);
        if (rank == 0) mbar_expect_tx(&xfull[at.slot], (x_lo ? 4u : 2u) * X_BYTES);   // of both CTAs
        tma_load_2d_pair(dst, &maps.a[pi], kx, row, bar);
        if (x_lo) tma_load_2d_pair(dst + X_BYTES, &maps.a2[pi], kx, row, bar);
      } else {
        mbar_expect_tx(&xfull[at.slot], (x_lo ? 2u : 1u) * X_BYTES);
        tma_load_2d(dst, &maps.a[pi], kx, m0, &xfull[at.slot]);
        if (x_lo) tma_load_2d(dst + X_BYTES, &maps.a2[pi], kx, m0, &xfull[at.slot]);
      }
    }
  } else if (warp == 2 + EW) {
    // PAIR: the slots are filled once before the CTA's warps meet for their columns
    const int pre = PAIR ? min(ng, NW) : 0;
    if (PAIR) {
      for (int kw = 0; kw < pre && lane == 0; ++kw) {
        mbar_expect_tx(&wfull[kw], WS_BYTES);
        tma_load_2d(wtiles + (uint32_t)kw * WS_BYTES, &maps.b[pi], (g0 + kw) * 128, ch0, &wfull[kw]);
      }
      __syncwarp();
      pair_tmem_ready(tmem);
    }
    if (lane == 0) {
      Ring at;
      for (int kw = 0; kw < ng; ++kw, at.next(NW)) {
        if (kw < pre) continue;
        if (!mbar_wait(&wempty[at.slot], at.phase ^ 1u, abort_flag, g.status, ST_GEMM_TIMEOUT)) break;
        mbar_expect_tx(&wfull[at.slot], WS_BYTES);
        tma_load_2d(wtiles + (uint32_t)at.slot * WS_BYTES, &maps.b[pi], (g0 + kw) * 128, ch0, &wfull[at.slot]);
      }
    }
  } else if (warp == 1) {
    if (PAIR) pair_tmem_alloc(tmem, rank, false, 0, grp.tmem_cols, abort_flag, g.status);   // (no other pair fits the SMs: launch_gemm_q)
    const bool there = !PAIR || pair_tmem_ready(tmem);
    if (PAIR) tmem_base = tmem->slot;
    if (rank == 0 && there) {
      Ring ea, xa;
      for (int kb = 0; kb < nkz; ++kb, ea.next(NE), xa.next(NX)) {
        if (!PAIR && !__all_sync(0xffffffffu, mbar_wait(&a_full[ea.slot], ea.phase, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
        if (!__all_sync(0xffffffffu, mbar_wait(&xfull[xa.slot], xa.phase, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
        tc_fence_after();
        const uint32_t xb = xtiles + (uint32_t)xa.slot * XS_BYTES, ta = tmem_base + grp.acc_cols + (uint32_t)ea.slot * A_COLS;
        const uint64_t xd = umma_desc_k128(xb), xl = umma_desc_k128(xb + X_BYTES);
        const bool wide = !PAIR && x_lo;
        if (elect_one()) {
#pragma unroll
          for (int k4 = 0; k4 < GBK / 16; ++k4)       // 16 inputs = 8 columns of A
            umma_f16_ta(PAIR, tmem_base, ta + (uint32_t)k4 * 8, xd + (uint64_t)(k4 * 2), wide ? IDESC2 : IDESC, (kb | k4) != 0);
          if (PAIR && x_lo) {
#pragma unroll
            for (int k4 = 0; k4 < GBK / 16; ++k4) umma_f16_ta(PAIR, tmem_base, ta + (uint32_t)k4 * 8, xl + (uint64_t)(k4 * 2), IDESC, 1u);
          }
          if (FMT == FMT_INT4) {
#pragma unroll
            for (int k4 = 0; k4 < GBK / 16; ++k4) umma_f16_ta(PAIR, tmem_base, ta + 32u + (uint32_t)k4 * 8, xd + (uint64_t)(k4 * 2), IDESC, 1u);
          }
          if (PAIR) { umma_commit_pair(&a_empty[ea.slot]); }
          else { umma_commit(&a_empty[ea.slot]); umma_commit(&xempty[xa.slot]); }
        }
        __syncwarp();
      }
      if (elect_one()) { if (PAIR) umma_commit_pair(acc_full); else umma_commit(acc_full); }
    } else if (PAIR && rank == 1 && there && lane == 0) {
      // An arrive in the other CTA takes some hundred clocks: this thread, which has no MMAs to issue, passes the slices of its
      // CTA's expanders on.
      Ring at;
      for (int kb = 0; kb < nkz; ++kb, at.next(NE)) {
        if (!mbar_wait(&a_full[at.slot], at.phase, abort_flag, g.status, ST_GEMM_TIMEOUT)) break;
        tc_fence_after();
        tc_fence_before();
        mbar_arrive_cluster(mapa_u32(smem_u32(&xfull[at.slot]), 0));
      }
    }
  } else {
    const int quad = warp & 3, nth = (warp - 2) >> 2, part = nth & 1, group = nth >> 1;
    const int row = quad * 32 + lane;
    const uint32_t swz = (uint32_t)(row & 7);
    GroupScales scales;
    if (FMT == FMT_INT4) scales.start(g, ch0 + row, kz0, nkz);
    const bool there = !PAIR || pair_tmem_ready(tmem);
    if (PAIR) tmem_base = tmem->slot;
    const uint32_t ta = tmem_base + ((uint32_t)(quad * 32) << 16) + grp.acc_cols + (uint32_t)part * 16;
    Ring wat, at;
    for (int kb = 0; there && kb < nkz; ++kb, at.next(NE)) {
      const int ks = kz0 + kb, sub = ks & (KSUB - 1);
      uint32_t s2 = 0;
      if (FMT == FMT_INT4) {
        const uint32_t sc = scales.at(ks), s16 = part ? (sc >> 16) : (sc & 0xffffu);
        s2 = s16 | (s16 << 16);
      }
      if (EW == 8 || (kb & 1) == group) {
        if (!__all_sync(0xffffffffu, mbar_wait(&wfull[wat.slot], wat.phase, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
        // 16-byte chunk c of the row's 128 bytes is at (c ^ swz) << 4
        const uint32_t src = wtiles + (uint32_t)wat.slot * WS_BYTES + (uint32_t)row * 128u, c0 = (uint32_t)sub * (ROW_B / 16u);
        uint32_t hi[16], lo[16];
        if (FMT == FMT_INT4) {
          const uint4 w = lds128(src + (((c0 + (uint32_t)part) ^ swz) << 4));
          expand_int4(w.x, s2, hi, lo); expand_int4(w.y, s2, hi + 4, lo + 4);
          expand_int4(w.z, s2, hi + 8, lo + 8); expand_int4(w.w, s2, hi + 12, lo + 12);
        } else {
#pragma unroll
          for (int pp = 0; pp < 2; ++pp) {
            const uint4 w = lds128(src + (((c0 + (uint32_t)(part * 2 + pp)) ^ swz) << 4));
            expand_int8(w.x, hi + pp * 8); expand_int8(w.y, hi + pp * 8 + 2);
            expand_int8(w.z, hi + pp * 8 + 4); expand_int8(w.w, hi + pp * 8 + 6);
          }
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&a_empty[at.slot], at.phase ^ 1u, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
        tc_fence_after();
        tmem_st16(ta + (uint32_t)at.slot * A_COLS, hi);
        if (FMT == FMT_INT4) tmem_st16(ta + (uint32_t)at.slot * A_COLS + 32u, lo);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(PAIR && rank == 0 ? &xfull[at.slot] : &a_full[at.slot]);
      } else if (kb == 0 && sub == KSUB - 1) {
        // The first weight slot of a K range may hold one slice, the other group's.  This group waits for it all the same: where it is
        // back at this slot before the slot's first load is there, its wait for the second one would pass on the phase before both.
        if (!__all_sync(0xffffffffu, mbar_wait(&wfull[0], 0, abort_flag, g.status, ST_GEMM_TIMEOUT))) break;
      }
      if (sub == KSUB - 1) {
        if (lane == 0) mbar_arrive(&wempty[wat.slot]);   // (the last slot of this K range is not asked for again)
        wat.next(NW);
      }
    }
    // epilogue
    const int ch = ch0 + row;
    pdl_wait();
    const bool ok = there && __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, g.status, ST_GEMM_TIMEOUT));
    tc_fence_after();
    if (ok) {
      const float sc = (!SLABS && g.col_scale && ch < g.N) ? __half2float(g.col_scale[ch]) : 1.f;
      const uint32_t buf = xtiles + (uint32_t)(warp - 2) * 2 * EPI_BUF;   // the rings have been read
      uint32_t flip = 0;
      for (int c0 = nth * 32; c0 < BN; c0 += 8 * EW, flip ^= EPI_BUF) {
        if (m0 + c0 >= g.M) break;   // warp-uniform
        const uint32_t at_acc = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
        uint32_t acc[32];
        tmem_ld32(at_acc, acc);
        if (!PAIR && x_lo) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t more[16];
            tmem_ld16(at_acc + (uint32_t)(BN + h * 16), more);
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[h * 16 + i] = __float_as_uint(__uint_as_float(acc[h * 16 + i]) + __uint_as_float(more[i]));
          }
        }
        if (!SLABS && g.col_scale) {
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = __float_as_uint(__uint_as_float(acc[i]) * sc);
        }
        if (SLABS && !PAIR && BN == 32) slab_rows(g, blockIdx.z, ch, m0 + c0, acc);
        else tile_out<SLABS>(g, &maps.o[pi], &maps.o_lo[pi], blockIdx.z, ch0 + quad * 32, m0 + c0, acc, buf + flip);
      }
      tile_out_end();
    }
  }
  if (PAIR) {
    pair_tmem_end(tmem, warp, grp.tmem_cols);
    return;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(grp.tmem_cols) : "memory");
  }
}

// split-K: sum the slabs in a fixed order, then the same epilogue.  One thread per 4 consecutive columns of a row
// (coalesced 16-byte reads of every slab); N is a multiple of 4 for every projection (the head never splits).
// blockIdx.y picks the problem of the group (grid.x covers the largest one).
__global__ void __launch_bounds__(256) gemm_finish_kernel(const __grid_constant__ GemmGroup grp) {
  pdl_trigger();
  const GemmArgs &g = grp.p[blockIdx.y];
  const int split = grp.split;
  const int n4 = g.N >> 2;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.M * n4) return;
  const int row = idx / n4, col = (idx - row * n4) * 4;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f), cs = make_float4(1.f, 1.f, 1.f, 1.f);
  if (g.col_scale)
    cs = make_float4(__half2float(g.col_scale[col]), __half2float(g.col_scale[col + 1]), __half2float(g.col_scale[col + 2]),
                     __half2float(g.col_scale[col + 3]));
  pdl_wait();
  for (int z = 0; z < split; ++z) {
    const float4 p = *reinterpret_cast<const float4 *>(g.raw + ((size_t)z * g.M + row) * g.N + col);
    v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
  }
  if (g.col_scale) { v.x *= cs.x; v.y *= cs.y; v.z *= cs.z; v.w *= cs.w; }
  const size_t o = (size_t)row * g.ldo + col;
  float a[4] = {v.x, v.y, v.z, v.w};
  if (g.epi == GEMM_EPI_F32) {
    *reinterpret_cast<float4 *>(reinterpret_cast<float *>(g.out) + o) = v;
  } else if (g.epi == GEMM_EPI_ADD_F32 || g.epi == GEMM_EPI_MULADD_F32) {
    const float4 x = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(g.aux0) + o);
    float r[4] = {1.f, 1.f, 1.f, 1.f};
    if (g.epi == GEMM_EPI_MULADD_F32) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        r[i] = __half2float(reinterpret_cast<const __half *>(g.aux1)[o + i]);
        if (g.aux1_lo) r[i] += __half2float(reinterpret_cast<const __half *>(g.aux1_lo)[o + i]);
      }
    }
    *reinterpret_cast<float4 *>(reinterpret_cast<float *>(g.out) + o) =
        make_float4((x.x + r[0] * a[0]) * g.scale, (x.y + r[1] * a[1]) * g.scale, (x.z + r[2] * a[2]) * g.scale,
                    (x.w + r[3] * a[3]) * g.scale);
  } else {
    __half *out = reinterpret_cast<__half *>(g.out) + o;
    __half *lo = g.out_lo ? reinterpret_cast<__half *>(g.out_lo) + o : nullptr;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float e = epi_half_op(g.epi, a[i]);
      const __half h = __float2half_rn(e);
      out[i] = h;
      if (lo) lo[i] = __float2half_rn(e - __half2float(h));
    }
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

bool encode_map(CUtensorMap *map, CUtensorMapDataType type, int rank, void *base, const cuuint64_t *dims, const cuuint64_t *strides,
                const cuuint32_t *box, bool swizzle, bool promote) {
  EncodeTiledFn fn = encode_fn();
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn && fn(map, type, (cuuint32_t)rank, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                  promote ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static_assert(sizeof(CUtensorMap) == sizeof(TensorMapBytes), "tensor maps are kept as bytes");
// An activation's map out of the forward pass's cache, or encoded.  (A map takes about 0.2 us, a launch of few rows needs up to 15.)
template <typename Encode>
bool cached_map(GemmMapCache *c, CUtensorMap *map, const GemmMapCache::Key &k, Encode encode) {
  if (c)
    for (int i = 0; i < c->n; ++i)
      if (c->key[i].base == k.base && c->key[i].rows == k.rows && c->key[i].cols == k.cols && c->key[i].box == k.box && c->key[i].kind == k.kind) {
        memcpy(map, &c->map[i], sizeof(*map));
        return true;
      }
  if (!encode()) return false;
  if (c && c->n < GemmMapCache::MAX) {
    c->key[c->n] = k;
    memcpy(&c->map[c->n++], map, sizeof(*map));
  }
  return true;
}
bool encode_rows_f16(CUtensorMap *map, const void *base, int rows, int K, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)GBK, (cuuint32_t)box_rows};
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, true, true);
}
// X [rows, K] fp16 row-major -> tensor map with a (64 x box_rows) box, 128-byte swizzle, zero fill outside
bool make_map_x(CUtensorMap *map, const GemmArgs &g, const __half *X, int box_rows) {
  return cached_map(g.maps, map, {X, g.M, g.K, box_rows, 0}, [&] { return encode_rows_f16(map, X, g.M, g.K, box_rows); });
}
// the weights: [N, K] fp16 row-major in (64 x 128 rows) boxes, or [N, packed row] bytes in (128 bytes x 128 rows) boxes, 128-byte swizzle
bool make_map_w(CUtensorMap *map, const GemmArgs &g) {
  if (g.wmap && g.wmap->set) { memcpy(map, &g.wmap->map, sizeof(*map)); return true; }
  bool ok;
  if (g.Wq) {
    const int row_bytes = g.wfmt == FMT_INT8 ? g.K : g.K / 2;
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)g.N}, strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {128, (cuuint32_t)GBM};
    ok = encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t *>(g.Wq), dims, strides, box, true, true);
  } else {
    ok = encode_rows_f16(map, g.Bt, g.N, g.K, GBM);
  }
  if (ok && g.wmap) { memcpy(&g.wmap->map, map, sizeof(*map)); g.wmap->set = true; }
  return ok;
}
// [planes, rows, cols] of fp16 or fp32 with rows `ld` elements and planes rows x ld elements apart -> tensor map with a
// (32 cols x 32 rows) box
bool make_map_out(CUtensorMap *map, const GemmArgs &g, void *base, bool f32, int planes, int ld) {
  return cached_map(g.maps, map, {base, g.M, g.N, ld, (f32 ? 2 : 1) + 4 * planes}, [&] {
    const size_t elt = f32 ? 4 : 2;
    const cuuint64_t dims[3] = {(cuuint64_t)g.N, (cuuint64_t)g.M, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)ld * elt, (cuuint64_t)ld * elt * g.M};
    const cuuint32_t box[3] = {32, 32, 1};
    return encode_map(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, base, dims, strides, box, false, false);
  });
}
// where a group's results go: slabs when K is split, else the outputs, as tensors when their rows allow it
bool make_out_maps(GemmMaps &maps, GemmGroup &grp) {
  for (int i = 0; i < grp.n; ++i) {
    GemmArgs &g = grp.p[i];
    g.tma_out = 0;
    if (grp.split > 1) {
      if (!make_map_out(&maps.o[i], g, g.raw, true, grp.split, g.N)) return false;
      continue;
    }
    const bool f32 = g.epi == GEMM_EPI_F32 || g.epi == GEMM_EPI_ADD_F32 || g.epi == GEMM_EPI_MULADD_F32;
    if (((size_t)g.ldo * (f32 ? 4 : 2)) % 16 || (reinterpret_cast<uintptr_t>(g.out) | reinterpret_cast<uintptr_t>(g.out_lo)) % 16) continue;
    g.tma_out = 1;
    if (!make_map_out(&maps.o[i], g, g.out, f32, 1, g.ldo)) return false;
    if (!f32 && g.out_lo && !make_map_out(&maps.o_lo[i], g, g.out_lo, false, 1, g.ldo)) return false;
  }
  return true;
}
// X and weights of a group (the maps of problems that do not exist are not read)
bool make_in_maps(GemmMaps &maps, const GemmGroup &grp, int box_rows, int box_rows_lo) {   // boxes of problems without and with A2
  for (int i = 0; i < grp.n; ++i) {
    const GemmArgs &g = grp.p[i];
    const int box = g.A2 ? box_rows_lo : box_rows;
    if (!make_map_x(&maps.a[i], g, g.A, box) || !make_map_w(&maps.b[i], g)) return false;
    if (g.A2 && !make_map_x(&maps.a2[i], g, g.A2, box)) return false;
  }
  return true;
}

}  // namespace

namespace {
// [K, N] -> [N, K], 32 x 32 tiles through shared memory
__global__ void transpose_f16_kernel(const __half *src, int K, int N, __half *dst) {
  __shared__ __half tile[32][33];
  const int k0 = blockIdx.y * 32, n0 = blockIdx.x * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int k = k0 + r, n = n0 + threadIdx.x;
    if (k < K && n < N) tile[r][threadIdx.x] = src[(size_t)k * N + n];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int n = n0 + r, k = k0 + threadIdx.x;
    if (k < K && n < N) dst[(size_t)n * K + k] = tile[threadIdx.x][r];
  }
}
}  // namespace

cudaError_t launch_transpose_f16(const __half *src, int K, int N, __half *dst, cudaStream_t st) {
  dim3 grid((N + 31) / 32, (K + 31) / 32), block(32, 8);
  transpose_f16_kernel<<<grid, block, 0, st>>>(src, K, N, dst);
  return cudaGetLastError();
}

namespace {

// ---- block reductions (blockDim.x = 256) -------------------------------------------------------------
__device__ __forceinline__ float2 block_sum2(float a, float b, float *red /* [16] */) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();   // red may still be read from the previous call
  if (lane == 0) { red[warp * 2] = a; red[warp * 2 + 1] = b; }
  __syncthreads();
  float sa = 0.f, sb = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) { sa += red[w * 2]; sb += red[w * 2 + 1]; }
  return make_float2(sa, sb);
}

// mean and 1/std of one fp32 row (shifted single pass, like the decode prologue)
__device__ __forceinline__ float2 row_stats(const float *x, int C, float *red) {
  const float piv = x[0];
  float s1 = 0.f, s2 = 0.f;
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    const float d = x[i] - piv;
    s1 += d; s2 += d * d;
  }
  const float2 s = block_sum2(s1, s2, red);
  const float m = s.x / (float)C;
  float var = s.y / (float)C - m * m;
  var = var > 0.f ? var : 0.f;
  return make_float2(piv + m, rsqrtf(var + 1e-5f));
}

// x[t, :] = embedding row of ids[t]
__device__ __forceinline__ void gather_row(const void *emb, int emb_f32, int id, int C, float *x) {
  const size_t row = (size_t)id * C;
  for (int i = threadIdx.x; i < C; i += blockDim.x)
    x[i] = emb_f32 ? reinterpret_cast<const float *>(emb)[row + i] : __half2float(reinterpret_cast<const __half *>(emb)[row + i]);
}
__global__ void gather_emb_kernel(const void *emb, int emb_f32, const int32_t *ids, int C, float *x) {
  pdl_trigger();
  pdl_wait();
  gather_row(emb, emb_f32, ids[blockIdx.x], C, x + (size_t)blockIdx.x * C);
}
// the same for ids that travel with the launch (captured steps: a graph holds them by value)
constexpr int INLINE_IDS = 512;
struct InlineIds { int32_t id[INLINE_IDS]; };
__global__ void gather_emb_inline_kernel(const void *emb, int emb_f32, const __grid_constant__ InlineIds ids, int C, float *x) {
  pdl_trigger();
  pdl_wait();
  gather_row(emb, emb_f32, ids.id[blockIdx.x], C, x + (size_t)blockIdx.x * C);
}

// LayerNorm + token shift + mix for every token row (LN of att_seq.cu:375, the shifted cat of :377-381 and the
// MixWithG of :384; ffn_seq.cu:70-76): op_v[t] = xx[t] * mu_v + prev[t] * (1 - mu_v), prev[0] = the stored shift
// state, prev[t] = xx[t-1]; the new shift state is xx[T-1].  One CTA per token; it normalises its own row and the
// row before it, so no CTA waits for another.
// Batch mode (rows = independent streams, one token each): prev of row b is stream b's stored shift state and every
// row writes its new one.  nvec == 0: plain LayerNorm into op[0] (ln_out before the head).
// Each thread keeps its float4 pieces of the row (and of the row before) in registers: x is read once.
// Sums and products are written as the operations they round to: left to the compiler, which product of a sum becomes a
// fused multiply-add depends on what else an instance contains, and RWKV-5 amplifies the last bit of a row over 32 layers to
// 1.2 - 2 % of quantised logits.  So every instance gives the same bits.
__device__ __forceinline__ float ln_squares(float d0, float d1, float d2, float d3) {
  return __fadd_rn(__fmaf_rn(d0, d0, __fmul_rn(d1, d1)), __fmaf_rn(d2, d2, __fmul_rn(d3, d3)));
}
__device__ __forceinline__ float ln_value(float x, const float2 &stats, float w, float b) {
  return __fmaf_rn(__fmul_rn(__fsub_rn(x, stats.x), stats.y), w, b);
}
__device__ __forceinline__ float4 ln_value4(const float4 &x, const float2 &s, const float4 &w, const float4 &b) {
  return make_float4(ln_value(x.x, s, w.x, b.x), ln_value(x.y, s, w.y, b.y), ln_value(x.z, s, w.z, b.z), ln_value(x.w, s, w.w, b.w));
}
__device__ __forceinline__ float mix_value(float x, float prev, float m) { return __fmaf_rn(x, m, __fmul_rn(prev, __fsub_rn(1.f, m))); }
__device__ __forceinline__ float2 ln_stats(const float2 &sums, float piv, int C) {
  const float m = sums.x / (float)C;
  const float var = __fmaf_rn(-m, m, sums.y / (float)C);
  return make_float2(piv + m, rsqrtf((var > 0.f ? var : 0.f) + 1e-5f));
}
constexpr int LN_MAX4 = 8;   // float4 per thread: n_embd <= 8192
constexpr int LN_FEW_ROWS = 256;   // about two CTAs of 512 threads per SM
template <int NT, int NJ>
__device__ __forceinline__ float2 stats_from_regs(const float4 *v, int n4, float piv, int C, float *red) {
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    if ((int)threadIdx.x + j * NT < n4) {
      const float d0 = v[j].x - piv, d1 = v[j].y - piv, d2 = v[j].z - piv, d3 = v[j].w - piv;
      s1 += (d0 + d1) + (d2 + d3);
      s2 += ln_squares(d0, d1, d2, d3);
    }
  }
  float2 s;
  if (NT == 256) {
    s = block_sum2(s1, s2, red);
  } else {
    // the order of 256 threads with NT / 256 pieces each: the same bits for every launch shape
    float2 *fold = reinterpret_cast<float2 *>(red + 16);
    const int tid = threadIdx.x;
    if (tid >= 256) fold[tid - 256] = make_float2(s1, s2);
    __syncthreads();
    if (tid < 256) {
#pragma unroll
      for (int i = 0; i < NT / 256 - 1; ++i) { const float2 f = fold[tid + i * 256]; s1 += f.x; s2 += f.y; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      }
      if ((tid & 31) == 0) { red[(tid >> 5) * 2] = s1; red[(tid >> 5) * 2 + 1] = s2; }
    }
    __syncthreads();
    s = make_float2(0.f, 0.f);
#pragma unroll
    for (int w = 0; w < 8; ++w) { s.x += red[w * 2]; s.y += red[w * 2 + 1]; }
  }
  return ln_stats(s, piv, C);
}
__device__ __forceinline__ void store_hl4(__half *hi, __half *lo, size_t o, const float4 &v) {
  const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<const uint32_t *>(&h0); u.y = *reinterpret_cast<const uint32_t *>(&h1);
  *reinterpret_cast<uint2 *>(hi + o) = u;
  if (lo) {
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    const __half2 l0 = __floats2half2_rn(v.x - f0.x, v.y - f0.y), l1 = __floats2half2_rn(v.z - f1.x, v.w - f1.y);
    u.x = *reinterpret_cast<const uint32_t *>(&l0); u.y = *reinterpret_cast<const uint32_t *>(&l1);
    *reinterpret_cast<uint2 *>(lo + o) = u;
  }
}
__device__ __forceinline__ float4 load_act_f4(const void *p, int i4, int act_fp16) {
  if (act_fp16) {
    const uint2 u = reinterpret_cast<const uint2 *>(p)[i4];
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
  return reinterpret_cast<const float4 *>(p)[i4];
}
__device__ __forceinline__ float round_h(float v) { return __half2float(__float2half_rn(v)); }

__device__ __forceinline__ float4 half4_value(const uint2 &u) {
  const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// NT threads, NJ float4 pieces of a row per thread.  What a launch does not need costs it registers, and those cost CTAs, so
// there are three kinds: LN_ROWS (streams: one row, its slabs pending or not), LN_PROMPT (the tokens of a prompt, two rows,
// nothing pending: 60 registers instead of 120 at 2,560 channels), LN_PROMPT_PENDING (behind a projection that left its slabs:
// two rows of a CTA to add up).
enum LnKind { LN_ROWS, LN_PROMPT, LN_PROMPT_PENDING };
template <int NT, int NJ, LnKind KIND>
__global__ void __launch_bounds__(NT) ln_mix_seq_kernel(SeqLnArgs a) {
  constexpr bool EARLY = NJ == 1;
  pdl_trigger();
  __shared__ __align__(8) float red[16 + 2 * (NT - 256)];
  const int t = blockIdx.x, C = a.C, n4 = C >> 2;
  // the parameters are constants: one round trip of them is over before the kernel ahead of this one has finished
  float4 ew = make_float4(0.f, 0.f, 0.f, 0.f), eb = ew, em[4], esx = ew;
  uint2 ecs = make_uint2(0u, 0u);
  if (EARLY && (int)threadIdx.x < n4) {
    ew = reinterpret_cast<const float4 *>(a.ln_w)[threadIdx.x];
    eb = reinterpret_cast<const float4 *>(a.ln_b)[threadIdx.x];
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (v < a.nvec) em[v] = reinterpret_cast<const float4 *>(a.mix[v])[threadIdx.x];
    if (a.pend_split > 1 && a.pend_cscale) ecs = reinterpret_cast<const uint2 *>(a.pend_cscale)[threadIdx.x];
  }
  pdl_wait();
  const uint8_t *srd = reinterpret_cast<const uint8_t *>(a.sx_rd) + (a.batch_mode ? (size_t)t * a.state_stride : 0);
  uint8_t *swr = reinterpret_cast<uint8_t *>(a.sx_wr) + (a.batch_mode ? (size_t)t * a.state_stride : 0);
  const float4 *xr = reinterpret_cast<const float4 *>(a.x + (size_t)t * C);
  const bool from_row = KIND != LN_ROWS && t > 0;
  float4 xv[NJ], pv[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int i4 = threadIdx.x + j * NT;
    if (i4 < n4) {
      xv[j] = xr[i4];
      if (from_row) pv[j] = xr[i4 - n4];
      else if (EARLY && a.nvec > 0) esx = load_act_f4(srd, i4, a.act_fp16);
    }
  }
  float piv = a.x[(size_t)t * C], ppiv = from_row ? a.x[(size_t)(t - 1) * C] : 0.f;
  if (KIND != LN_PROMPT && a.pend_split > 1) {
    // the projection before this LayerNorm left its split-K slabs: sum them (in slab order, like gemm_finish_kernel),
    // apply its epilogue x = (x + [r *] sum) * scale, store the finished row and normalise it from the registers; a
    // prompt's CTA does the same for the row before (which its own CTA stores: to another buffer than it is read from)
    __shared__ float piv_s[2];
    const size_t zs = (size_t)a.T * C;
    constexpr int ZB = NJ == 1 && NT <= 512 ? 16 : 4;   // slabs per batch: NJ x ZB 16-byte loads in flight per thread
    auto finish = [&](float4 *rowv, int row, const uint2 &erh, const uint2 &erl) {
      float4 acc[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int z0 = 0; z0 < a.pend_split; z0 += ZB) {
        float4 p[NJ][ZB];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int i4 = threadIdx.x + j * NT;
          const float *slab = a.pend_raw + (size_t)row * C + (size_t)i4 * 4;
#pragma unroll
          for (int i = 0; i < ZB; ++i)
            if (i4 < n4 && z0 + i < a.pend_split) p[j][i] = *reinterpret_cast<const float4 *>(slab + (size_t)(z0 + i) * zs);
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int i = 0; i < ZB; ++i)   // in slab order
            if (z0 + i < a.pend_split) { acc[j].x += p[j][i].x; acc[j].y += p[j][i].y; acc[j].z += p[j][i].z; acc[j].w += p[j][i].w; }
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int i4 = threadIdx.x + j * NT;
        if (i4 >= n4) continue;
        float4 v = acc[j];
        if (a.pend_cscale) {
          const float4 cs = half4_value(EARLY ? ecs : reinterpret_cast<const uint2 *>(a.pend_cscale)[i4]);
          v.x *= cs.x; v.y *= cs.y; v.z *= cs.z; v.w *= cs.w;
        }
        float r[4] = {1.f, 1.f, 1.f, 1.f};
        if (a.pend_r) {
          const float4 rh = half4_value(EARLY ? erh : reinterpret_cast<const uint2 *>(a.pend_r + (size_t)row * C)[i4]);
          r[0] = rh.x; r[1] = rh.y; r[2] = rh.z; r[3] = rh.w;
          if (a.pend_r_lo) {
            const float4 rl = half4_value(EARLY ? erl : reinterpret_cast<const uint2 *>(a.pend_r_lo + (size_t)row * C)[i4]);
            r[0] += rl.x; r[1] += rl.y; r[2] += rl.z; r[3] += rl.w;
          }
        }
        rowv[j] = make_float4(__fmaf_rn(r[0], v.x, rowv[j].x) * a.pend_scale, __fmaf_rn(r[1], v.y, rowv[j].y) * a.pend_scale,
                              __fmaf_rn(r[2], v.z, rowv[j].z) * a.pend_scale, __fmaf_rn(r[3], v.w, rowv[j].w) * a.pend_scale);
        if (row == t) reinterpret_cast<float4 *>(a.x_wr + (size_t)t * C)[i4] = rowv[j];
        if (i4 == 0) piv_s[t - row] = rowv[j].x;
      }
    };
    // the factor is asked for together with the slabs
    uint2 eh[2], el[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (EARLY && a.pend_r && (i == 0 || (KIND == LN_PROMPT_PENDING && from_row)) && (int)threadIdx.x < n4) {
        eh[i] = reinterpret_cast<const uint2 *>(a.pend_r + (size_t)(t - i) * C)[threadIdx.x];
        if (a.pend_r_lo) el[i] = reinterpret_cast<const uint2 *>(a.pend_r_lo + (size_t)(t - i) * C)[threadIdx.x];
      }
    finish(xv, t, eh[0], el[0]);
    if (KIND == LN_PROMPT_PENDING && from_row) finish(pv, t - 1, eh[1], el[1]);
    __syncthreads();
    piv = piv_s[0];
    if (KIND == LN_PROMPT_PENDING) ppiv = piv_s[1];
  }
  const float2 st = stats_from_regs<NT, NJ>(xv, n4, piv, C, red);
  float2 sp = make_float2(0.f, 0.f);
  if (from_row) sp = stats_from_regs<NT, NJ>(pv, n4, ppiv, C, red);
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int i4 = threadIdx.x + j * NT;
    if (i4 >= n4) continue;
    const float4 w = EARLY ? ew : reinterpret_cast<const float4 *>(a.ln_w)[i4], b = EARLY ? eb : reinterpret_cast<const float4 *>(a.ln_b)[i4];
    const float4 xx = ln_value4(xv[j], st, w, b);
    const size_t o = (size_t)t * C + (size_t)i4 * 4;
    if (a.nvec == 0) {
      store_hl4(a.op[0], a.op_lo[0], o, xx);
      continue;
    }
    float4 prev;
    if (from_row) {
      prev = ln_value4(pv[j], sp, w, b);
      // what the token loop would have stored as shift state
      if (a.act_fp16) prev = make_float4(round_h(prev.x), round_h(prev.y), round_h(prev.z), round_h(prev.w));
    } else {
      prev = EARLY ? esx : load_act_f4(srd, i4, a.act_fp16);
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (v < a.nvec) {
        const float4 m = EARLY ? em[v] : reinterpret_cast<const float4 *>(a.mix[v])[i4];
        store_hl4(a.op[v], a.op_lo[v], o,
                  make_float4(mix_value(xx.x, prev.x, m.x), mix_value(xx.y, prev.y, m.y), mix_value(xx.z, prev.z, m.z),
                              mix_value(xx.w, prev.w, m.w)));
      }
    if (a.batch_mode || t == a.T - 1) {
      if (a.act_fp16) {
        const __half2 h0 = __floats2half2_rn(xx.x, xx.y), h1 = __floats2half2_rn(xx.z, xx.w);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t *>(&h0); u.y = *reinterpret_cast<const uint32_t *>(&h1);
        reinterpret_cast<uint2 *>(swr)[i4] = u;
      } else {
        reinterpret_cast<float4 *>(swr)[i4] = xx;
      }
    }
  }
}

// RWKV-4 WKV over rows (WkvForwardOne, att.cu:30-62, with the sigmoid of att.cu:154-159 fused): one thread per
// (stream, channel), row b is the one token of stream b (prompts of one stream: wkv4_seq_kernel).
//   out[row, c] = sigmoid(r) * wkv (fp16, the operand of the output projection); aa, bb, pp updated in place.
// The loads are all asked for at once: the constants before the kernel ahead has finished, then the state and the slabs.
// ZB: slabs per batch of loads.
template <int ZB>
__global__ void __launch_bounds__(256) wkv4_rows_kernel(Wkv4Args a) {
  pdl_trigger();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (c >= a.C) return;
  const float u = a.first[c], w = a.decay[c];
  float ck = 1.f, cv = 1.f, cr = 1.f;
  if (a.split > 1 && a.cs_k) { ck = __half2float(a.cs_k[c]); cv = __half2float(a.cs_v[c]); cr = __half2float(a.cs_r[c]); }
  pdl_wait();
  float *st = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(a.state) + (size_t)b * a.state_stride);
  float aa = st[c], bb = st[a.C + c], pp = st[2 * a.C + c];
  {
    const int t = b;
    const size_t o = (size_t)t * a.C + c;
    float k, v, rp;
    if (a.split > 1) {
      // the projections left their split-K slabs: sum them here, in slab order like gemm_finish_kernel
      k = 0.f; v = 0.f; rp = 0.f;
      for (int z0 = 0; z0 < a.split; z0 += ZB) {
        float pk[ZB], pv[ZB], pr[ZB];
#pragma unroll
        for (int i = 0; i < ZB; ++i)
          if (z0 + i < a.split) {
            const size_t zo = ((size_t)(z0 + i) * a.T + t) * a.C + c;
            pk[i] = a.raw_k[zo]; pv[i] = a.raw_v[zo]; pr[i] = a.raw_r[zo];
          }
#pragma unroll
        for (int i = 0; i < ZB; ++i)
          if (z0 + i < a.split) { k += pk[i]; v += pv[i]; rp += pr[i]; }
      }
      k *= ck; v *= cv; rp *= cr;
    } else {
      k = a.k[o]; v = a.v[o]; rp = a.r[o];
    }
    const float r = 1.f / (1.f + expf(-rp));
    float ww = u + k;
    float pm = fmaxf(pp, ww);
    float e1 = expf(pp - pm), e2 = expf(ww - pm);
    const float wkv = (e1 * aa + e2 * v) / (e1 * bb + e2);
    const __half oh = __float2half_rn(r * wkv);
    a.out[o] = oh;
    if (a.out_lo) a.out_lo[o] = __float2half_rn(r * wkv - __half2float(oh));
    ww = w + pp;
    pm = fmaxf(ww, k);
    e1 = expf(ww - pm);
    e2 = expf(k - pm);
    aa = e1 * aa + e2 * v;
    bb = e1 * bb + e2;
    pp = pm;
  }
  st[c] = aa; st[a.C + c] = bb; st[2 * a.C + c] = pp;
}

// RWKV-4 WKV over the tokens of ONE stream (prompts).  The recurrence is associative -- a run of tokens acts on the
// state as (aa, bb, pp) -> decay by exp(len * w), plus the run's own sums -- so the prompt is cut into 64 chunks that
// are reduced side by side, combined by a prefix scan, and walked again from their start states.  One CTA holds 16
// channels x 64 chunks (a 64-byte piece of each row per half warp) and does all three steps: no scratch in global
// memory, one launch.  Up to 1024 tokens a thread keeps its chunk's k and v between the two walks (LEN tokens, in
// registers; of LEN = 16 eight words do not fit the 64 a thread has.  0: read again).  What bounds it: the serial walk
// it replaces was one dependent expf chain of T steps on C threads, 700 us a layer at T = 1000, C = 2048; this form is
// 2 x ceil(T / 64) steps on 64 C threads.
constexpr int W4_CH = 16, W4_CHUNKS = 64, W4_THREADS = W4_CH * W4_CHUNKS;
// state (a1, b1, p1) followed by a run of decay d = len * w with sums (a2, b2, p2)
__device__ __forceinline__ void wkv4_join(float &a, float &b, float &p, float d, float a2, float b2, float p2) {
  const float pd = p + d, pm = fmaxf(pd, p2);
  const float e1 = expf(pd - pm), e2 = expf(p2 - pm);
  a = e1 * a + e2 * a2;
  b = e1 * b + e2 * b2;
  p = pm;
}
template <int LEN>
__global__ void __launch_bounds__(W4_THREADS) wkv4_seq_kernel(Wkv4Args a) {
  pdl_trigger();
  pdl_wait();
  // [value][channel][chunk], rows padded by one word
  __shared__ float sh[3][W4_CH][W4_CHUNKS + 1];
  __shared__ float half_tot[3][W4_CH];
  const int cl = threadIdx.x & (W4_CH - 1), ck = threadIdx.x >> 4;
  const int c = blockIdx.x * W4_CH + cl;
  const int len = (a.T + W4_CHUNKS - 1) / W4_CHUNKS;           // LEN == 0 or len <= LEN
  const int t0 = min(a.T, ck * len), t1 = min(a.T, t0 + len);
  float *st = reinterpret_cast<float *>(a.state);
  const float u = a.first[c], w = a.decay[c];
  const float *kp = a.k + c, *vp = a.v + c, *rp = a.r + c;
  constexpr int NR = LEN > 0 ? LEN : 1;
  float kr[NR], vr[NR], rsum = 0.f;
  float aa = 0.f, bb = 0.f, pp = -1e30f;
  auto absorb = [&](float k, float v) {
    const float ww = w + pp, pm = fmaxf(ww, k);
    const float e1 = expf(ww - pm), e2 = expf(k - pm);
    aa = e1 * aa + e2 * v;
    bb = e1 * bb + e2;
    pp = pm;
  };
  if (LEN > 0) {
#pragma unroll
    for (int i = 0; i < NR; ++i)
      if (t0 + i < t1) {
        if (LEN == 1 && a.split > 1) {
          // the projections left their split-K slabs: one token per thread sums its own, in slab order
          float k = 0.f, v = 0.f, r = 0.f;
#pragma unroll 4
          for (int z = 0; z < a.split; ++z) {
            const size_t zo = ((size_t)z * a.T + t0) * a.C + c;
            k += a.raw_k[zo]; v += a.raw_v[zo]; r += a.raw_r[zo];
          }
          if (a.cs_k) { k *= __half2float(a.cs_k[c]); v *= __half2float(a.cs_v[c]); r *= __half2float(a.cs_r[c]); }
          kr[0] = k; vr[0] = v; rsum = r;
        } else {
          kr[i] = kp[(size_t)(t0 + i) * a.C]; vr[i] = vp[(size_t)(t0 + i) * a.C];
          if (LEN == 1) rsum = rp[(size_t)t0 * a.C];
        }
      }
#pragma unroll
    for (int i = 0; i < NR; ++i)
      if (t0 + i < t1) absorb(kr[i], vr[i]);
  } else {
#pragma unroll 4
    for (int t = t0; t < t1; ++t) absorb(kp[(size_t)t * a.C], vp[(size_t)t * a.C]);
  }
  sh[0][cl][ck] = aa; sh[1][cl][ck] = bb; sh[2][cl][ck] = pp;
  __syncthreads();
  {
    // inclusive scan over the chunks: warp pair (2 ch, 2 ch + 1) takes channel ch, lanes along the chunks.  The decay
    // of a joined run is the distance between the runs' ends (the last chunks of a ragged prompt are short or empty).
    const int ch = threadIdx.x >> 6, j = threadIdx.x & 63, lane = threadIdx.x & 31;
    const float wc = a.decay[blockIdx.x * W4_CH + ch];
    float xa = sh[0][ch][j], xb = sh[1][ch][j], xp = sh[2][ch][j];
    const int end_j = min(a.T, (j + 1) * len);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      float ya = __shfl_up_sync(0xffffffffu, xa, o), yb = __shfl_up_sync(0xffffffffu, xb, o), yp = __shfl_up_sync(0xffffffffu, xp, o);
      if (lane >= o) {
        wkv4_join(ya, yb, yp, wc * (float)(end_j - min(a.T, (j - o + 1) * len)), xa, xb, xp);
        xa = ya; xb = yb; xp = yp;
      }
    }
    if (j == 31) { half_tot[0][ch] = xa; half_tot[1][ch] = xb; half_tot[2][ch] = xp; }
    __syncthreads();
    if (j >= 32) {
      float ya = half_tot[0][ch], yb = half_tot[1][ch], yp = half_tot[2][ch];
      wkv4_join(ya, yb, yp, wc * (float)(end_j - min(a.T, 32 * len)), xa, xb, xp);
      xa = ya; xb = yb; xp = yp;
    }
    sh[0][ch][j] = xa; sh[1][ch][j] = xb; sh[2][ch][j] = xp;
  }
  __syncthreads();
  constexpr int RG = LEN > 4 ? 4 : 2;
  float rn[RG];
  if (LEN > 1) {
#pragma unroll
    for (int i = 0; i < RG; ++i) rn[i] = i < NR && t0 + i < t1 ? rp[(size_t)(t0 + i) * a.C] : 0.f;
  }
  // this chunk's start state: the stream's state followed by all chunks before
  aa = st[c]; bb = st[a.C + c]; pp = st[2 * a.C + c];
  __syncthreads();                       // every thread has read the state the last chunk overwrites
  if (ck > 0) wkv4_join(aa, bb, pp, w * (float)t0, sh[0][cl][ck - 1], sh[1][cl][ck - 1], sh[2][cl][ck - 1]);
  auto step = [&](int t, float k, float v, float r_pre) {
    const float r = 1.f / (1.f + expf(-r_pre));
    const float ww = u + k, pm = fmaxf(pp, ww);
    const float e1 = expf(pp - pm), e2 = expf(ww - pm);
    const float y = r * ((e1 * aa + e2 * v) / (e1 * bb + e2));
    const __half oh = __float2half_rn(y);
    a.out[(size_t)t * a.C + c] = oh;
    if (a.out_lo) a.out_lo[(size_t)t * a.C + c] = __float2half_rn(y - __half2float(oh));
    absorb(k, v);
  };
  if (LEN == 1) {
    if (t0 < t1) step(t0, kr[0], vr[0], rsum);
  } else if (LEN > 0) {
    // r comes a group of tokens ahead of its use: asked for token by token it waits behind the stores of the one before
#pragma unroll
    for (int i0 = 0; i0 < NR; i0 += RG) {
      float r[RG];
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        r[i] = rn[i];
        if (i0 + RG + i < NR && t0 + i0 + RG + i < t1) rn[i] = rp[(size_t)(t0 + i0 + RG + i) * a.C];
      }
#pragma unroll
      for (int i = 0; i < RG; ++i)
        if (i0 + i < NR && t0 + i0 + i < t1) step(t0 + i0 + i, kr[i0 + i], vr[i0 + i], r[i]);
    }
  } else {
#pragma unroll 4
    for (int t = t0; t < t1; ++t) step(t, kp[(size_t)t * a.C], vp[(size_t)t * a.C], rp[(size_t)t * a.C]);
  }
  if (ck == W4_CHUNKS - 1) { st[c] = aa; st[a.C + c] = bb; st[2 * a.C + c] = pp; }
}

// greedy sample of every row: index of the largest logit (lowest index on ties).  ctl (optional): the id also goes
// to row ctl->step of the history ctl->hist -- fixed kernel arguments, so that a captured graph can be replayed.
// A cluster of CTAs per row (gridDim.x of them), each over its part of the vocabulary: one CTA has 64 KB in flight at most, and a row of
// 65536 logits took it 29 us.  A step of 16 streams: 410 -> 396 us (0.1B shape), 1185 -> 1154 (1.5B).
__global__ void __launch_bounds__(256) argmax_rows_kernel(const float *logits, int V, int ld, int32_t *out, const GreedyCtl *ctl) {
  pdl_trigger();
  cluster_sync();      // the first CTA is there to be written to
  pdl_wait();
  __shared__ unsigned long long best[8], parts[8];
  const int b = blockIdx.y;
  const float *row = logits + (size_t)b * ld;
  unsigned long long m = 0;
  auto take = [&](float f, int i) {
    unsigned u = __float_as_uint(f);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    const unsigned long long w = ((unsigned long long)u << 32) | (0xffffffffu - (unsigned)i);
    m = w > m ? w : m;
  };
  const int V4 = ((ld & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) ? (V & ~3) : 0;
  // 16-byte loads, eight in flight per thread
#pragma unroll 8
  for (int i = (blockIdx.x * 256 + threadIdx.x) * 4; i < V4; i += gridDim.x * 1024) {
    const float4 f = *reinterpret_cast<const float4 *>(row + i);
    take(f.x, i); take(f.y, i + 1); take(f.z, i + 2); take(f.w, i + 3);
  }
  for (int i = V4 + blockIdx.x * 256 + threadIdx.x; i < V; i += gridDim.x * 256) take(row[i], i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, m, o);
    m = other > m ? other : m;
  }
  if ((threadIdx.x & 31) == 0) best[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w8 = 1; w8 < 8; ++w8) m = best[w8] > m ? best[w8] : m;
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(mapa_u32(smem_u32(&parts[blockIdx.x]), 0)), "l"(m) : "memory");
  }
  __syncwarp();
  cluster_sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    m = parts[0];
    for (int r = 1; r < (int)gridDim.x; ++r) m = parts[r] > m ? parts[r] : m;
    const int32_t id = (int32_t)(0xffffffffu - (unsigned)m);
    out[b] = id;
    if (ctl) ctl->hist[(size_t)ctl->step * gridDim.y + b] = id;
  }
}
__global__ void greedy_bump_kernel(GreedyCtl *ctl) { pdl_trigger(); pdl_wait(); ctl->step += 1; }
__global__ void greedy_start_kernel(GreedyCtl *ctl, int32_t *hist) { pdl_trigger(); pdl_wait(); ctl->hist = hist; ctl->step = 0; }


// RWKV-5 state scan over the tokens of one head (rwkv5_2_kernel_forward, att_seq.cu:258-322; per-head decay for 5.0):
//   y[t, j] = sum_i r[t,i] * (u_i * k[t,i] * v[t,j] + s[i,j]);   s[i,j] = w_i * s[i,j] + k[t,i] * v[t,j]
// r, k, v of 16 tokens at a time arrive in shared memory by cp.async, the next 16 while the current ones are used.
// The sequence is cut into n_chunks pieces that run in parallel (the reference walks it serially):
//   mode 0  state only, from zero, over chunk c               -> E[h][c]        (grid H x n_chunks)
//   mode 1  S_in[h][0] = state; S_in[h][c+1] = w^len(c) * S_in[h][c] + E[h][c]; state = the last one   (grid H)
//   mode 2  full recurrence over chunk c from S_in[h][c]       -> y              (grid H x n_chunks)
// With n_chunks == 1 mode 2 alone reads and writes the model state directly.
constexpr int WKV_TT = 16;

__device__ __forceinline__ void wkv_stage(float (*sr)[64], float (*sk)[64], float (*sv)[64], const SeqWkvArgs &a, int h, int t0,
                                          int nt, bool with_r) {
  // 16 floats = 4 x 16 bytes per (token, vector) quarter row: 3 vectors x nt tokens x 16 pieces
  for (int e = threadIdx.x; e < nt * 16; e += blockDim.x) {
    const int tt = e >> 4, c = (e & 15) * 4;
    const size_t g = (size_t)(t0 + tt) * a.C + h * 64 + c;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&sk[tt][c])), "l"(a.k + g) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&sv[tt][c])), "l"(a.v + g) : "memory");
    if (with_r) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&sr[tt][c])), "l"(a.r + g) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// 64 threads per CTA: thread (jg, iq) owns value columns jg, jg + 16, jg + 32, jg + 48 and key rows 16 iq .. 16 iq + 15,
// i.e. 64 state entries in registers; the r / k values it reads from shared memory serve four columns each.
constexpr int WKV_THREADS = 64;
// Packed fp32 pairs (fma.rn.f32x2 / mul.rn.f32x2: two fp32 operations per instruction on sm_100).  The scan is bound
// by the issue rate of its multiply-adds, so the state is kept as pairs over neighbouring key rows: k, r and the decay
// then come out of shared memory already paired, and only v needs a broadcast pair per token.
__device__ __forceinline__ unsigned long long pack_f2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f2(unsigned long long v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long mul_f2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// y_t[j] = sum_i r_i (u_i k_i v_j + s_ij) = v_j (sum_i r_i u_i k_i) + sum_i r_i s_ij;  s_ij <- w_i s_ij + k_i v_j.
// Thread (jg, iq) owns key rows iq*16 .. +15 of value columns jg + 16 q (q = 0..3): 32 pairs.
template <int MODE>
__global__ void __launch_bounds__(WKV_THREADS) wkv5_seq_kernel(SeqWkvArgs a) {
  pdl_trigger();
  pdl_wait();
  __shared__ __align__(16) float sr[2][WKV_TT][64], sk[2][WKV_TT][64], sv[2][WKV_TT][64];
  const int h = blockIdx.x, c = blockIdx.y, C = a.C;
  const int jg = threadIdx.x >> 2, iq = threadIdx.x & 3;
  const int t_begin = c * a.chunk_len, t_end = min(a.T, t_begin + a.chunk_len);
  unsigned long long s2[4][8], w2[8], u2[8];   // pairs over key rows (iq*16 + 2 p, + 2 p + 1)
  float *Sown = a.state + (size_t)h * 4096;
  const float *Sin = a.n_chunks == 1 ? Sown : a.s_in + ((size_t)h * a.n_chunks + c) * 4096;
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const int ii = iq * 16 + 2 * p;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      s2[q][p] = MODE == 0 ? 0ull : pack_f2(Sin[ii * 64 + jg + 16 * q], Sin[(ii + 1) * 64 + jg + 16 * q]);
    w2[p] = a.per_head ? pack_f2(a.decay[h], a.decay[h]) : pack_f2(a.decay[h * 64 + ii], a.decay[h * 64 + ii + 1]);
    u2[p] = a.per_head ? pack_f2(a.first[h], a.first[h]) : pack_f2(a.first[h * 64 + ii], a.first[h * 64 + ii + 1]);
  }
  int buf = 0;
  if (t_begin < t_end) wkv_stage(sr[0], sk[0], sv[0], a, h, t_begin, min(WKV_TT, t_end - t_begin), MODE == 2);
  for (int t0 = t_begin; t0 < t_end; t0 += WKV_TT) {
    const int nt = min(WKV_TT, t_end - t0);
    const int tn = t0 + WKV_TT;
    if (tn < t_end) {
      wkv_stage(sr[buf ^ 1], sk[buf ^ 1], sv[buf ^ 1], a, h, tn, min(WKV_TT, t_end - tn), MODE == 2);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    for (int tt = 0; tt < nt; ++tt) {
      float vj[4];
      unsigned long long v2[4], y2[4] = {0ull, 0ull, 0ull, 0ull}, ruk2 = 0ull;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        vj[q] = sv[buf][tt][jg + 16 * q];
        v2[q] = pack_f2(vj[q], vj[q]);
      }
#pragma unroll
      for (int p = 0; p < 8; p += 2) {
        // four key rows = two pairs per 16-byte load
        const ulonglong2 k4 = *reinterpret_cast<const ulonglong2 *>(&sk[buf][tt][iq * 16 + 2 * p]);
        ulonglong2 r4 = make_ulonglong2(0ull, 0ull);
        if (MODE == 2) r4 = *reinterpret_cast<const ulonglong2 *>(&sr[buf][tt][iq * 16 + 2 * p]);
        const unsigned long long kk[2] = {k4.x, k4.y}, rr[2] = {r4.x, r4.y};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (MODE == 2) ruk2 = fma_f2(mul_f2(rr[e], u2[p + e]), kk[e], ruk2);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (MODE == 2) y2[q] = fma_f2(rr[e], s2[q][p + e], y2[q]);
            s2[q][p + e] = fma_f2(s2[q][p + e], w2[p + e], mul_f2(kk[e], v2[q]));
          }
        }
      }
      if (MODE == 2) {
        float ra, rb;
        unpack_f2(ruk2, ra, rb);
        const float ruk = ra + rb;
        float y[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float ya, yb;
          unpack_f2(y2[q], ya, yb);
          y[q] = fmaf(vj[q], ruk, ya + yb);
          y[q] += __shfl_xor_sync(0xffffffffu, y[q], 1);
          y[q] += __shfl_xor_sync(0xffffffffu, y[q], 2);
        }
        if (iq == 0) {
#pragma unroll
          for (int q = 0; q < 4; ++q) a.y[(size_t)(t0 + tt) * C + h * 64 + jg + 16 * q] = y[q];
        }
      }
    }
    __syncthreads();   // the buffer just read is the one the next staging overwrites
    buf ^= 1;
  }
  if (MODE == 0 || a.n_chunks == 1) {
    float *S = MODE == 0 ? a.e_out + ((size_t)h * a.n_chunks + c) * 4096 : Sown;
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float lo, hi;
        unpack_f2(s2[q][p], lo, hi);
        const int ii = iq * 16 + 2 * p;
        S[ii * 64 + jg + 16 * q] = lo;
        S[(ii + 1) * 64 + jg + 16 * q] = hi;
      }
  }
}

// mode 1: chain the chunk states; one thread per state entry (grid = H * 16 CTAs of 256 threads), the chunk end
// states are fetched eight at a time ahead of the dependent multiply-adds
__global__ void __launch_bounds__(256) wkv5_combine_kernel(SeqWkvArgs a) {
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x >> 4, e = (blockIdx.x & 15) * 256 + threadIdx.x;
  const int i = e >> 6;
  const float w = a.per_head ? a.decay[h] : a.decay[h * 64 + i];
  const float lw = log2f(w);
  const float wl = exp2f(lw * (float)a.chunk_len);
  float *S = a.state + (size_t)h * 4096;
  float s = S[e];
  const size_t base = (size_t)h * a.n_chunks * 4096 + e;
  for (int c0 = 0; c0 < a.n_chunks; c0 += 8) {
    float ev[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) ev[q] = c0 + q < a.n_chunks ? a.e_out[base + (size_t)(c0 + q) * 4096] : 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int c = c0 + q;
      if (c < a.n_chunks) {
        a.s_in[base + (size_t)c * 4096] = s;
        const int len = min(a.T, (c + 1) * a.chunk_len) - c * a.chunk_len;
        s = (len == a.chunk_len ? wl : exp2f(lw * (float)len)) * s + ev[q];
      }
    }
  }
  S[e] = s;
}

// GroupNorm over a head's 64 values and the gate: lane l of a warp has values 2 l, 2 l + 1 (group_norm.cu:322-357, att.cu:145-152).  Written as
// what it rounds to, so that the two kernels that do it give the same bits.
__device__ __forceinline__ float2 gn_gate_pair(const float2 &v, const float2 &w, const float2 &b, bool gated, const float2 &gg) {
  float s = v.x + v.y;
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
  const float mean = s * (1.f / 64.f);
  const float d0 = v.x - mean, d1 = v.y - mean;
  float q = __fmaf_rn(d0, d0, __fmul_rn(d1, d1));
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) q += __shfl_xor_sync(0xffffffffu, q, k);
  const float rstd = rsqrtf(__fmaf_rn(q, 1.f / 64.f, 1e-5f));
  float2 o = make_float2(__fmaf_rn(__fmul_rn(d0, rstd), w.x, b.x), __fmaf_rn(__fmul_rn(d1, rstd), w.y, b.y));
  if (gated) { o.x *= gg.x; o.y *= gg.y; }
  return o;
}
__device__ __forceinline__ void store_pair(__half *out, __half *out_lo, size_t o, const float2 &v) {
  const __half2 h = __floats2half2_rn(v.x, v.y);
  *reinterpret_cast<__half2 *>(out + o) = h;
  if (out_lo) {
    const float2 f = __half22float2(h);
    *reinterpret_cast<__half2 *>(out_lo + o) = __floats2half2_rn(v.x - f.x, v.y - f.y);
  }
}

// RWKV-5 over rows (streams, one token each): the step of wkv5_seq_kernel<2>, with the projections' split-K slabs summed ahead of it (in slab
// order, as gemm_finish_kernel does) and GroupNorm and gate behind it.  One CTA per (head, stream); a chain of few streams has two
// launches fewer per layer (16 fp16 streams of the 3B shape: finishing pass 4.1 us, state 9.4, GroupNorm 2.7).
__global__ void __launch_bounds__(WKV_THREADS) wkv5_rows_kernel(Wkv5RowsArgs a) {
  pdl_trigger();
  __shared__ __align__(16) float sr[64], sk[64], sv[64], sg[64], sy[64];
  const int h = blockIdx.x, row = blockIdx.y, C = a.C, tid = threadIdx.x, jg = tid >> 2, iq = tid & 3, c = h * 64 + tid;
  unsigned long long s2[4][8], w2[8], u2[8];   // pairs over key rows (iq*16 + 2 p, + 2 p + 1)
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const int ii = iq * 16 + 2 * p;
    w2[p] = a.per_head ? pack_f2(a.decay[h], a.decay[h]) : pack_f2(a.decay[h * 64 + ii], a.decay[h * 64 + ii + 1]);
    u2[p] = a.per_head ? pack_f2(a.first[h], a.first[h]) : pack_f2(a.first[h * 64 + ii], a.first[h * 64 + ii + 1]);
  }
  float cs[4] = {1.f, 1.f, 1.f, 1.f};
  if (a.split > 1)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (a.cs[i]) cs[i] = __half2float(a.cs[i][c]);
  pdl_wait();
  float *S = a.state + (size_t)row * a.state_stride + (size_t)h * 4096;
#pragma unroll
  for (int p = 0; p < 8; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int ii = iq * 16 + 2 * p;
      s2[q][p] = pack_f2(S[ii * 64 + jg + 16 * q], S[(ii + 1) * 64 + jg + 16 * q]);
    }
  const size_t o = (size_t)row * C + c;
  if (a.split > 1) {
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    const size_t zs = (size_t)a.rows * C;
    for (int z = 0; z < a.split; ++z)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < 3 || a.gated) x[i] += a.raw[i][z * zs + o];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (a.cs[i]) x[i] *= cs[i];
    sk[tid] = x[0]; sv[tid] = x[1]; sr[tid] = x[2];
    const float e = epi_half_op<GEMM_EPI_SILU_F16>(x[3]);
    const __half gh = __float2half_rn(e);
    sg[tid] = __half2float(gh) + __half2float(__float2half_rn(e - __half2float(gh)));
  } else {
    sk[tid] = a.k[o]; sv[tid] = a.v[o]; sr[tid] = a.r[o];
    sg[tid] = a.gated ? __half2float(a.g[o]) + __half2float(a.g_lo[o]) : 0.f;
  }
  __syncthreads();
  float vj[4];
  unsigned long long v2[4], y2[4] = {0ull, 0ull, 0ull, 0ull}, ruk2 = 0ull;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    vj[q] = sv[jg + 16 * q];
    v2[q] = pack_f2(vj[q], vj[q]);
  }
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const unsigned long long kk = *reinterpret_cast<const unsigned long long *>(&sk[iq * 16 + 2 * p]);
    const unsigned long long rr = *reinterpret_cast<const unsigned long long *>(&sr[iq * 16 + 2 * p]);
    ruk2 = fma_f2(mul_f2(rr, u2[p]), kk, ruk2);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      y2[q] = fma_f2(rr, s2[q][p], y2[q]);
      s2[q][p] = fma_f2(s2[q][p], w2[p], mul_f2(kk, v2[q]));
    }
  }
  float ra, rb;
  unpack_f2(ruk2, ra, rb);
  const float ruk = ra + rb;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float ya, yb;
    unpack_f2(y2[q], ya, yb);
    float y = fmaf(vj[q], ruk, ya + yb);
    y += __shfl_xor_sync(0xffffffffu, y, 1);
    y += __shfl_xor_sync(0xffffffffu, y, 2);
    if (iq == 0) sy[jg + 16 * q] = y;
  }
#pragma unroll
  for (int p = 0; p < 8; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float lo, hi;
      unpack_f2(s2[q][p], lo, hi);
      const int ii = iq * 16 + 2 * p;
      S[ii * 64 + jg + 16 * q] = lo;
      S[(ii + 1) * 64 + jg + 16 * q] = hi;
    }
  __syncthreads();
  if (tid < 32) {
    const int cc = h * 64 + 2 * tid;
    const float2 w = make_float2(a.lnx_w[cc], a.lnx_w[cc + 1]), b = make_float2(a.lnx_b[cc], a.lnx_b[cc + 1]);
    store_pair(a.out, a.out_lo, (size_t)row * C + cc,
               gn_gate_pair(make_float2(sy[2 * tid], sy[2 * tid + 1]), w, b, a.gated, make_float2(sg[2 * tid], sg[2 * tid + 1])));
  }
}

// GroupNorm over each head's 64 readout values (eps 1e-5, fp32 affine), times the gate where the version has one
// (att_seq.cu:406-415): one warp per (token, head)
__global__ void __launch_bounds__(256) gn_gate_seq_kernel(const float *y, const float *lnx_w, const float *lnx_b, const __half *g,
                                                          const __half *g_lo, int T, int H, __half *out, __half *out_lo) {
  pdl_trigger();
  pdl_wait();
  const int unit = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (unit >= T * H) return;
  const int t = unit / H, h = unit - t * H;
  const size_t o = (size_t)t * H * 64 + h * 64 + lane * 2;
  const int c = h * 64 + lane * 2;
  float2 gg = make_float2(0.f, 0.f);
  if (g) {
    gg = __half22float2(*reinterpret_cast<const __half2 *>(g + o));
    if (g_lo) {
      const float2 gl = __half22float2(*reinterpret_cast<const __half2 *>(g_lo + o));
      gg.x += gl.x; gg.y += gl.y;
    }
  }
  store_pair(out, out_lo, o, gn_gate_pair(*reinterpret_cast<const float2 *>(y + o), make_float2(lnx_w[c], lnx_w[c + 1]),
                                          make_float2(lnx_b[c], lnx_b[c + 1]), g != nullptr, gg));
}

// plain LayerNorm of one row -> fp32 vector (ln_out before the head, model_forward_seq.cpp:171-175)
__global__ void __launch_bounds__(256) ln_row_kernel(const float *x, const float *w, const float *b, int C, float *out) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[16];
  const float2 st = row_stats(x, C, red);
  for (int i = threadIdx.x; i < C; i += blockDim.x) out[i] = (x[i] - st.x) * st.y * w[i] + b[i];
}

}  // namespace

cudaError_t launch_gather_emb(const void *emb, int emb_f32, const int32_t *ids, int T, int C, float *x, cudaStream_t st) {
  launch_k(gather_emb_kernel, dim3(T), dim3(256), 0, st, emb, emb_f32, ids, C, x);
  return cudaGetLastError();
}
cudaError_t launch_gather_emb_host(const void *emb, int emb_f32, const int32_t *ids, int T, int C, float *x, cudaStream_t st) {
  for (int t0 = 0; t0 < T; t0 += INLINE_IDS) {
    const int n = std::min(T - t0, INLINE_IDS);
    InlineIds in = {};
    memcpy(in.id, ids + t0, (size_t)n * 4);
    const cudaError_t e = launch_k(gather_emb_inline_kernel, dim3(n), dim3(256), 0, st, emb, emb_f32, in, C, x + (size_t)t0 * C);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
namespace {
template <LnKind KIND>
void launch_ln_mix_t(const SeqLnArgs &a, bool few, cudaStream_t st) {
  const int n4 = a.C >> 2;
  const dim3 grid(a.T);
  if (few && n4 <= 256) launch_k(ln_mix_seq_kernel<256, 1, KIND>, grid, dim3(256), 0, st, a);
  else if (few && n4 <= 512) launch_k(ln_mix_seq_kernel<512, 1, KIND>, grid, dim3(512), 0, st, a);
  else if (few && n4 <= 768) launch_k(ln_mix_seq_kernel<768, 1, KIND>, grid, dim3(768), 0, st, a);
  else if (n4 <= 2 * 256) launch_k(ln_mix_seq_kernel<256, 2, KIND>, grid, dim3(256), 0, st, a);
  else if (n4 <= 4 * 256) launch_k(ln_mix_seq_kernel<256, 4, KIND>, grid, dim3(256), 0, st, a);
  else launch_k(ln_mix_seq_kernel<256, LN_MAX4, KIND>, grid, dim3(256), 0, st, a);
}
}  // namespace
cudaError_t launch_ln_mix_seq(const SeqLnArgs &a, cudaStream_t st) {
  const int n4 = a.C >> 2;
  const dim3 grid(a.T);
  // Few rows: one piece of the row per thread, everything the row needs asked for at once (16 streams of the 1.5B shape:
  // 1.46 ms a step against 1.63; 100: 1.69 against 1.85; a 29 token prompt: 1.68 against 1.80).  Many rows hide the round trips
  // behind one another, and small CTAs with several pieces per thread pack better (a prompt of 1,000: 6.56 ms against 6.67).
  const bool few = a.T <= LN_FEW_ROWS;
  if (!a.batch_mode && a.pend_split > 1) {   // (short prompts of models up to 2,048 channels: PROMPT_DEFER_ROWS, _C)
    if (!few || n4 > 512) return cudaErrorInvalidValue;
    if (n4 <= 256) launch_k(ln_mix_seq_kernel<256, 1, LN_PROMPT_PENDING>, grid, dim3(256), 0, st, a);
    else launch_k(ln_mix_seq_kernel<512, 1, LN_PROMPT_PENDING>, grid, dim3(512), 0, st, a);
  } else if (!a.batch_mode) {
    launch_ln_mix_t<LN_PROMPT>(a, few, st);
  } else {
    launch_ln_mix_t<LN_ROWS>(a, few, st);
  }
  return cudaGetLastError();
}
// CTAs of the readout pass of the scan that are resident at once on the device: one wave of (head, chunk) pairs is what
// a prompt should be cut into (a second, partly filled wave costs as much as a full one)
int wkv5_scan_slots() {
  static int slots = 0;
  if (!slots) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wkv5_seq_kernel<2>, WKV_THREADS, 0) != cudaSuccess || per_sm < 1) per_sm = 4;
    slots = per_sm * device_sm_count();
  }
  return slots;
}

cudaError_t launch_wkv5_seq(const SeqWkvArgs &a, int H, cudaStream_t st) {
  if (a.n_chunks <= 1) {
    launch_k(wkv5_seq_kernel<2>, dim3(dim3(H, 1)), dim3(WKV_THREADS), 0, st, a);
    return cudaGetLastError();
  }
  launch_k(wkv5_seq_kernel<0>, dim3(dim3(H, a.n_chunks)), dim3(WKV_THREADS), 0, st, a);
  launch_k(wkv5_combine_kernel, dim3(H * 16), dim3(256), 0, st, a);
  launch_k(wkv5_seq_kernel<2>, dim3(dim3(H, a.n_chunks)), dim3(WKV_THREADS), 0, st, a);
  return cudaGetLastError();
}
cudaError_t launch_wkv5_rows(const Wkv5RowsArgs &a, int H, cudaStream_t st) {
  return launch_k(wkv5_rows_kernel, dim3(H, a.rows), dim3(WKV_THREADS), 0, st, a);
}
cudaError_t launch_wkv4_rows(const Wkv4Args &a, cudaStream_t st) {
  if (!a.batch_mode) {
    const dim3 grid(a.C / W4_CH), block(W4_THREADS);
    const int len = (a.T + W4_CHUNKS - 1) / W4_CHUNKS;
    // The fewest tokens kept per thread that cover a chunk: every slot is a pass through the code, taken or not.  This kernel
    // alone at 2,048 channels, us: 256 tokens <4> 7.1, <0> 11.7; 300 tokens <12> 8.9, <16> 10.2, <0> 13.3; 640 tokens 12.9, 14.1,
    // 21.4; 1,000 tokens <16> 19.1, <0> 30.6.  (With more CTAs than SMs <0>, of which two fit an SM, is the faster one: 5,120
    // channels, 640 tokens 31 against 36, 1,000 tokens 49 against 61.)
    if (len <= 1) launch_k(wkv4_seq_kernel<1>, grid, block, 0, st, a);
    else if (len <= 4) launch_k(wkv4_seq_kernel<4>, grid, block, 0, st, a);
    else if (len <= 12) launch_k(wkv4_seq_kernel<12>, grid, block, 0, st, a);
    else if (len <= 16) launch_k(wkv4_seq_kernel<16>, grid, block, 0, st, a);
    else launch_k(wkv4_seq_kernel<0>, grid, block, 0, st, a);
    return cudaGetLastError();
  }
  dim3 grid((a.C + 255) / 256, a.T);
  // Up to 64 rows of a 2,048 channel model a CTA per SM or two has to cover the whole round trip by itself; beyond, fewer
  // registers and more CTAs are better.  This kernel alone, <8> against <4>, us: 6 slabs, 32 rows 3.0 / 4.0, 64 rows 3.55 /
  // 4.24, 80 rows 4.12 / 4.24, 100 rows 4.61 / 4.22, 256 rows 9.1 / 8.3; 3 slabs, 32 rows 2.8 / 3.1, 64 rows 3.27 / 3.32, 80 rows
  // 3.75 / 3.42, 256 rows 8.4 / 6.6.  (768 channels cross at the same T C; up to 16 rows of 2,048 channels the two are within 0.8 us
  // of one another either way.)
  if ((long long)a.T * a.C <= 64 * 2048) launch_k(wkv4_rows_kernel<8>, dim3(grid), dim3(256), 0, st, a);
  else launch_k(wkv4_rows_kernel<4>, dim3(grid), dim3(256), 0, st, a);
  return cudaGetLastError();
}
cudaError_t launch_greedy_start(GreedyCtl *ctl, int32_t *hist, cudaStream_t st) {
  return launch_k(greedy_start_kernel, dim3(1), dim3(1), 0, st, ctl, hist);
}
cudaError_t launch_argmax_rows(const float *logits, int rows, int V, int ld, int32_t *out, GreedyCtl *ctl, cudaStream_t st) {
  // as many CTAs per row as about four per SM allow
  const int slots = 4 * device_sm_count() / std::max(rows, 1), cluster = slots >= 8 ? 8 : slots >= 4 ? 4 : slots >= 2 ? 2 : 1;
  const cudaError_t e = launch_cluster_k(argmax_rows_kernel, cluster, dim3(cluster, rows), dim3(256), 0, st, logits, V, ld, out, (const GreedyCtl *)ctl);
  if (e != cudaSuccess) return e;
  if (ctl) launch_k(greedy_bump_kernel, dim3(1), dim3(1), 0, st, ctl);
  return cudaGetLastError();
}
cudaError_t launch_gn_gate_seq(const float *y, const float *lnx_w, const float *lnx_b, const __half *g, const __half *g_lo, int T,
                               int H, __half *out, __half *out_lo, cudaStream_t st) {
  launch_k(gn_gate_seq_kernel, dim3((T * H + 7) / 8), dim3(256), 0, st, y, lnx_w, lnx_b, g, g_lo, T, H, out, out_lo);
  return cudaGetLastError();
}
cudaError_t launch_ln_row(const float *x, const float *w, const float *b, int C, float *out, cudaStream_t st) {
  launch_k(ln_row_kernel, dim3(1), dim3(256), 0, st, x, w, b, C, out);
  return cudaGetLastError();
}

namespace {

// In how many pieces K is cut for `ctas` tiles of which a device holds `slots`: the cost of a split, in K slices of one CTA, is
// waves x (slices per CTA + fill and drain) + the slabs it adds.
int split_of(int ctas, int slots, int min_k1) {
  const int max_split = std::max(1, std::min(GEMM_SPLIT_MAX, min_k1 / 2));
  int split = 1;
  float best = 0.f;
  for (int sp = 1; sp <= max_split; ++sp) {
    const int waves = (ctas * sp + slots - 1) / slots;
    const float cost = (float)waves * (float)((min_k1 + sp - 1) / sp + 2) + 0.25f * (float)sp;
    if (sp == 1 || cost < best) { best = cost; split = sp; }
  }
  return split;
}
// the cut of a product of RWKV-5 over more than 64 (quantised: 128) rows: that of one 128 x 256 tile per SM
int keep_split(int ctas, int min_k1) { return split_of(ctas, device_sm_count(), min_k1); }

// up to 128 rows: gemm_wt_kernel, split-K into slabs when scratch was given
cudaError_t launch_gemm_wt(const GemmArgs *probs, int n, cudaStream_t st, int *defer_split) {
  const int M = probs[0].M;
  const int bn = M <= 32 ? 32 : M <= 64 ? 64 : 128;
  GemmMaps maps;
  GemmGroup grp;
  memset(&grp, 0, sizeof(grp));
  grp.n = n;
  int tiles = 0, min_k1 = 1 << 30;
  bool raw_ok = true;
  for (int i = 0; i < n; ++i) {
    const GemmArgs &g = probs[i];
    if (g.K % GBK != 0 || g.M < 1 || g.N < 1 || g.M != M || M > 128 || g.col_scale) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(g.A) & 15) || (reinterpret_cast<uintptr_t>(g.Bt) & 15) || (reinterpret_cast<uintptr_t>(g.A2) & 15))
      return cudaErrorInvalidValue;
    grp.p[i] = g;
    grp.tile_start[i] = tiles;
    tiles += (g.N + GBM - 1) / GBM;
    min_k1 = std::min(min_k1, g.K / GBK);
    raw_ok = raw_ok && g.raw != nullptr && (g.N & 3) == 0 && (g.ldo & 3) == 0;
    if (g.A2) grp.dual = 1;
  }
  if (!make_in_maps(maps, grp, bn, bn)) return cudaErrorNotSupported;
  grp.tile_start[n] = tiles;
  // one CTA per SM, none waiting for a second wave: split K until the tiles about cover the SMs
  // (up to 64 rows the slabs are small next to the weights and two CTAs fit an SM: twice the slots, so that every SM
  // streams even when the group has few tiles)
  grp.split = 1;
  const int sms = device_sm_count();
  const int slots = bn <= 64 ? 2 * sms : sms;
  if (raw_ok) grp.split = split_of(tiles, slots, min_k1);
  grp.stage_bytes = G_A_BYTES + (grp.dual ? 2u : 1u) * (uint32_t)bn * GBK * 2;
  // two CTAs per SM with rings of >= 3 slots where they fit (shorter tail when there are more tiles than SMs),
  // else one CTA with as deep a ring as fits
  int stages = (int)((100u << 10) / grp.stage_bytes);
  if (stages < 3) stages = (int)((200u << 10) / grp.stage_bytes);
  grp.stages = std::max(2, std::min(stages, WT_MAX_STAGES));
  if (!make_out_maps(maps, grp)) return cudaErrorNotSupported;
  const size_t smem = 1024 + (size_t)grp.stages * grp.stage_bytes + 1024;
  dim3 grid(tiles, 1, grp.split);
  auto kern = grp.split > 1 ? (bn == 32 ? gemm_wt_kernel<32, true> : bn == 64 ? gemm_wt_kernel<64, true> : gemm_wt_kernel<128, true>)
                            : (bn == 32 ? gemm_wt_kernel<32, false> : bn == 64 ? gemm_wt_kernel<64, false> : gemm_wt_kernel<128, false>);
  cudaError_t e = launch_k(kern, grid, dim3(G_THREADS), smem, st, maps, grp);
  if (e != cudaSuccess) return e;
  if (defer_split) *defer_split = grp.split;
  if (grp.split > 1 && !defer_split) {
    int max_n = 0;
    for (int i = 0; i < n; ++i) max_n = std::max(max_n, probs[i].N);
    launch_k(gemm_finish_kernel, dim3(dim3((M * (max_n / 4) + 255) / 256, n)), dim3(256), 0, st, grp);
  }
  return cudaGetLastError();
}
// Costs in clocks, fitted to products of 256 and 1000 rows (2048 x 2048 up to 65536 x 2048 and 2048 x 8192) with 64 to 256 columns
// and 1 to 9 cuts, within 10 % of the times of these.  Products of other widths are cut by the same constants; whether another cut would
// be faster there has not been looked at.
// Slabs: the next kernel reads them at about 2,500 bytes a clock; without one that does, a finishing pass is launched.
float slab_cost(int split, int M, int sum_n, bool deferred) {
  return split > 1 ? (deferred ? 0.f : 8000.f) + (float)split * (float)M * (float)sum_n * 4.f / 2500.f : 0.f;
}
// `tiles` pair tiles of nk slices: rounds of two CTAs per SM, the last one alone on its SMs where it is at most half full
float pair_cost(int tiles, int nk, int bn, float passes, int num_pairs) {
  const float start_end = 11000.f + 16.f * (float)bn;
  const float shared = 2.f * (float)nk * std::max(2.3f * passes * (float)bn, 256.f + passes * (float)bn) + start_end;
  const float alone = (float)nk * std::max(2.05f * passes * (float)bn, 420.f + 150.f * passes) + start_end;
  const int rounds = tiles / (2 * num_pairs), rest = tiles - rounds * 2 * num_pairs;
  return (float)rounds * shared + (rest > num_pairs ? shared : rest > 0 ? alone : 0.f);
}

// fp16 weights, more than 128 rows of X, or more than 64 with low halves: gemm_pair_kernel
cudaError_t launch_gemm_pair(const GemmArgs *probs, int n, cudaStream_t st, int *defer_split) {
  const int M = probs[0].M, num_pairs = device_sm_count() / 2;
  GemmMaps maps;
  GemmGroup grp;
  memset(&grp, 0, sizeof(grp));
  grp.n = n;
  int tiles = 0, tiles128 = 0, units = 0, min_k1 = 1 << 30, sum_n = 0;
  bool raw_ok = M <= GEMM_SMALL_M, any_lo = false;
  for (int i = 0; i < n; ++i) {
    const GemmArgs &g = probs[i];
    any_lo = any_lo || g.A2;
    if (g.K % GBK != 0 || g.M < 1 || g.N < 1 || g.M != M || g.col_scale) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(g.A) & 15) || (reinterpret_cast<uintptr_t>(g.Bt) & 15) || (reinterpret_cast<uintptr_t>(g.A2) & 15))
      return cudaErrorInvalidValue;
    grp.p[i] = g;
    grp.tile_start[i] = tiles;
    const int t = (g.N + 2 * GBM - 1) / (2 * GBM);
    tiles += t;
    tiles128 += (g.N + GBM - 1) / GBM;
    units += t * (g.A2 ? 2 : 1);
    sum_n += g.N;
    min_k1 = std::min(min_k1, g.K / GBK);
    raw_ok = raw_ok && g.raw != nullptr && (g.N & 3) == 0 && (g.ldo & 3) == 0;
  }
  grp.tile_start[n] = tiles;
  // The sums of a result follow from how K is cut.  RWKV-5 amplifies a changed last bit to percents of its logits, so its
  // products keep the cut of keep_split(); else a cut and a row tile are chosen together.
  const int fixed = raw_ok && probs[0].fixed_split ? keep_split(tiles128 * ((M + 255) / 256), min_k1) : 0;
  const int max_split = raw_ok ? std::max(1, std::min(GEMM_SPLIT_MAX, min_k1 / 4)) : 1;
  grp.split = 1;
  grp.bn = 256;
  float best = 0.f;
  const float passes = (float)units / (float)tiles;
  const bool beside = M <= 128;
  for (int rt = (M + 255) / 256; rt <= (M + 127) / 128; ++rt) {
    const int bn = ((M + rt - 1) / rt + 31) / 32 * 32;
    for (int sp = fixed ? fixed : 1; sp <= (fixed ? fixed : max_split); ++sp) {
      const float cost = (beside ? pair_cost(tiles * sp, (min_k1 + sp - 1) / sp, any_lo ? 2 * bn : bn, 1.f, num_pairs)
                                 : pair_cost(tiles * rt * sp, (min_k1 + sp - 1) / sp, bn, passes, num_pairs)) + slab_cost(sp, M, sum_n, defer_split != nullptr);
      if (best == 0.f || cost < best) { best = cost; grp.split = sp; grp.bn = bn; }
    }
  }
  grp.m_tiles = (M + grp.bn - 1) / grp.bn;
  grp.lo_mode = beside ? LO_BESIDE : M <= GEMM_SMALL_M ? LO_EACH : LO_AFTER;
  if (!make_in_maps(maps, grp, grp.bn / 2, beside ? grp.bn : grp.bn / 2)) return cudaErrorNotSupported;
  grp.stage_bytes = G_A_BYTES + (grp.lo_mode != LO_AFTER && any_lo ? 2u : 1u) * (uint32_t)grp.bn * GBK;
  // tiles that have an SM each to themselves take a ring of twice the depth
  const bool alone = tiles * grp.m_tiles * grp.split <= num_pairs;
  grp.stages = std::min<int>(PAIR_MAX_STAGES, (int)((alone ? 200u << 10 : 110u << 10) / grp.stage_bytes));
  if (!make_out_maps(maps, grp)) return cudaErrorNotSupported;
  const size_t smem = std::max<size_t>(1024 + (size_t)grp.stages * grp.stage_bytes + 1024, alone ? PAIR_ALONE_SMEM : 0);
  grp.lock = smem < PAIR_ALONE_SMEM;
  cudaError_t e = launch_cluster_k(grp.split > 1 ? gemm_pair_kernel<true> : gemm_pair_kernel<false>, 2, dim3(2 * tiles * grp.m_tiles, 1, grp.split), dim3(G_THREADS), smem, st, maps, grp);
  if (e != cudaSuccess) return e;
  if (defer_split) *defer_split = grp.split;
  if (grp.split > 1 && !defer_split) {
    int max_n = 0;
    for (int i = 0; i < n; ++i) max_n = std::max(max_n, probs[i].N);
    launch_k(gemm_finish_kernel, dim3((M * (max_n / 4) + 255) / 256, n), dim3(256), 0, st, grp);
  }
  return cudaGetLastError();
}

using GemmKernel = void (*)(GemmMaps, GemmGroup);
template <bool SLABS>
GemmKernel gemm_q_kern(int fmt, bool pair, bool two_per_sm) {
  if (pair) return fmt == FMT_INT4 ? gemm_q_kernel<FMT_INT4, true, 16, SLABS> : gemm_q_kernel<FMT_INT8, true, 16, SLABS>;
  if (two_per_sm) return fmt == FMT_INT4 ? gemm_q_kernel<FMT_INT4, false, 8, SLABS> : gemm_q_kernel<FMT_INT8, false, 8, SLABS>;
  return fmt == FMT_INT4 ? gemm_q_kernel<FMT_INT4, false, 16, SLABS> : gemm_q_kernel<FMT_INT8, false, 16, SLABS>;
}

// quantised weights in packed form (GemmArgs::Wq): gemm_q_kernel, on pairs of SMs above 128 rows
cudaError_t launch_gemm_q(const GemmArgs *probs, int n, cudaStream_t st, int *defer_split) {
  const int M = probs[0].M, fmt = probs[0].wfmt, sms = device_sm_count(), num_pairs = sms / 2;
  const bool pair = M > 128;
  if (fmt != FMT_INT8 && fmt != FMT_INT4) return cudaErrorInvalidValue;
  GemmMaps maps;
  GemmGroup grp;
  memset(&grp, 0, sizeof(grp));
  grp.n = n;
  int tiles = 0, tiles128 = 0, units = 0, min_k1 = 1 << 30, sum_n = 0;
  bool raw_ok = M <= GEMM_SMALL_M, any_lo = false;
  for (int i = 0; i < n; ++i) {
    const GemmArgs &g = probs[i];
    if (g.K % GBK != 0 || g.M < 1 || g.N < 1 || g.M != M || !g.Wq || g.wfmt != fmt) return cudaErrorInvalidValue;
    if (fmt == FMT_INT4 && !g.wq_scale) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(g.A) & 15) || (reinterpret_cast<uintptr_t>(g.Wq) & 15) || (reinterpret_cast<uintptr_t>(g.A2) & 15))
      return cudaErrorInvalidValue;
    grp.p[i] = g;
    grp.tile_start[i] = tiles;
    const int t128 = (g.N + GBM - 1) / GBM, t = pair ? (t128 + 1) / 2 : t128;
    tiles += t;
    tiles128 += t128;
    units += t * ((fmt == FMT_INT4 ? 2 : 1) + (g.A2 ? 1 : 0));
    sum_n += g.N;
    min_k1 = std::min(min_k1, g.K / GBK);
    raw_ok = raw_ok && g.raw != nullptr && (g.N & 3) == 0 && (g.ldo & 3) == 0;
    any_lo = any_lo || g.A2;
  }
  grp.tile_start[n] = tiles;
  grp.split = 1;
  const uint32_t a_cols = fmt == FMT_INT4 ? 64u : 32u;
  bool two_per_sm = false;
  if (pair) {
    const int fixed = raw_ok && probs[0].fixed_split ? keep_split(tiles128 * ((M + 255) / 256), min_k1) : 0;   // (as in launch_gemm_pair)
    const int max_split = raw_ok ? std::max(1, std::min(GEMM_SPLIT_MAX, min_k1 / 2)) : 1;
    const float passes = (float)units / (float)tiles;
    float best = 0.f;
    for (int rt = (M + 255) / 256; rt <= (M + 127) / 128; ++rt) {
      const int bn = ((M + rt - 1) / rt + 31) / 32 * 32;
      for (int sp = fixed ? fixed : 1; sp <= (fixed ? fixed : max_split); ++sp) {
        // in clocks: a slice is bound by its MMAs or by its expansion, a wave starts and ends
        const int waves = (tiles * rt * sp + num_pairs - 1) / num_pairs;
        const float cost = (float)waves * ((float)((min_k1 + sp - 1) / sp) * std::max(2.05f * (float)bn * passes, 460.f) + 11000.f + 14.f * (float)bn) +
                           slab_cost(sp, M, sum_n, defer_split != nullptr);
        if (best == 0.f || cost < best) { best = cost; grp.split = sp; grp.bn = bn; }
      }
    }
    grp.acc_cols = 256;
    grp.tmem_cols = 512;
  } else {
    grp.bn = M <= 32 ? 32 : M <= 64 ? 64 : 128;
    // K is cut for two CTAs per SM where their accumulators are narrow
    if (raw_ok) grp.split = split_of(tiles, (grp.bn <= 64 || !any_lo) ? 2 * sms : sms, min_k1);
    grp.acc_cols = (any_lo ? 2u : 1u) * (uint32_t)grp.bn;
    two_per_sm = grp.acc_cols <= 128;
    grp.tmem_cols = two_per_sm ? 256 : 512;
  }
  grp.m_tiles = (M + grp.bn - 1) / grp.bn;
  const int xrows = pair ? grp.bn / 2 : grp.bn;
  if (!make_in_maps(maps, grp, xrows, xrows)) return cudaErrorNotSupported;
  grp.stage_bytes = (any_lo ? 2u : 1u) * (uint32_t)xrows * GBK * 2;
  grp.estages = std::min<int>(GQ_MAX, (int)((grp.tmem_cols - grp.acc_cols) / a_cols));
  const uint32_t avail = (two_per_sm ? 110u : 220u) << 10, ws = GBM * 128;
  grp.stages = two_per_sm ? ((avail - 3 * ws) / grp.stage_bytes >= 4 ? 3 : 2) : 4;
  grp.xstages = std::min<int>(GQ_MAX, (int)((avail - grp.stages * ws) / grp.stage_bytes));
  if (pair) grp.xstages = grp.estages = std::min(grp.xstages, grp.estages);
  if (!make_out_maps(maps, grp)) return cudaErrorNotSupported;
  const size_t rings = (size_t)grp.xstages * grp.stage_bytes + (size_t)grp.stages * ws;
  const int ew = two_per_sm ? 8 : 16;
  size_t smem = 1024 + std::max<size_t>(rings, ew * 2 * EPI_BUF) + 1024;
  // No CTA of another pair kernel shares an SM with one of these (gemm_pair_kernel's take 82 KB at least), which therefore need no lock for
  // their allocation.
  if (pair) smem = std::max(smem, (size_t)PAIR_ALONE_SMEM);
  auto kern = grp.split > 1 ? gemm_q_kern<true>(fmt, pair, two_per_sm) : gemm_q_kern<false>(fmt, pair, two_per_sm);
  const dim3 grid((pair ? 2 : 1) * tiles * grp.m_tiles, 1, grp.split);
  cudaError_t e = launch_cluster_k(kern, pair ? 2 : 1, grid, dim3(gq_threads(ew)), smem, st, maps, grp);
  if (e != cudaSuccess) return e;
  if (defer_split) *defer_split = grp.split;
  if (grp.split > 1 && !defer_split) {
    int max_n = 0;
    for (int i = 0; i < n; ++i) max_n = std::max(max_n, probs[i].N);
    launch_k(gemm_finish_kernel, dim3((M * (max_n / 4) + 255) / 256, n), dim3(256), 0, st, grp);
  }
  return cudaGetLastError();
}
}  // namespace

// defer_split (optional): the caller's next kernel sums the split-K slabs itself (ln_mix_seq_kernel, wkv4_rows_kernel, wkv4_seq_kernel, wkv5_rows_kernel);
// it receives the split that was chosen, 1 meaning that the outputs are already complete.
cudaError_t launch_gemm_group(const GemmArgs *probs, int n, cudaStream_t st, int *defer_split) {
  if (n < 1 || n > GEMM_GROUP_MAX) return cudaErrorInvalidValue;
  const int M = probs[0].M;
  if (defer_split) *defer_split = 1;
  if (probs[0].Wq) return launch_gemm_q(probs, n, st, defer_split);
  // 65 to 128 rows: X as hi + lo pairs is worth a pair of SMs (every CTA reads half of it), X of single halves is not.  1.5B shape, ms:
  // 100 streams 1.53 on pairs, 1.61 without; a prompt of 100 tokens 1.70 and 1.61, 1.65 with its key / value
  // / receptance alone on pairs (of which two have low halves).
  bool pairs = M > 64;
  for (int i = 0; i < n && M <= 128; ++i) pairs = pairs && probs[i].A2;
  return pairs ? launch_gemm_pair(probs, n, st, defer_split) : launch_gemm_wt(probs, n, st, defer_split);
}

cudaError_t gemm_prepare(int device) {
  int optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  const GemmKernel f16[] = {gemm_wt_kernel<32, false>, gemm_wt_kernel<64, false>, gemm_wt_kernel<128, false>, gemm_pair_kernel<false>,
                            gemm_wt_kernel<32, true>, gemm_wt_kernel<64, true>, gemm_wt_kernel<128, true>, gemm_pair_kernel<true>};
  for (GemmKernel k : f16)
    if (e == cudaSuccess) e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  for (int fmt : {(int)FMT_INT8, (int)FMT_INT4})
    for (int way = 0; way < 3; ++way) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute((const void *)gemm_q_kern<false>(fmt, way == 0, way == 1), cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
      if (e == cudaSuccess) e = cudaFuncSetAttribute((const void *)gemm_q_kern<true>(fmt, way == 0, way == 1), cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    }
  return e;
}

cudaError_t launch_gemm_f16(const GemmArgs &g, cudaStream_t st) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = gemm_prepare(device);
  return e != cudaSuccess ? e : launch_gemm_group(&g, 1, st, nullptr);   // no raw scratch: no split-K
}

}  // namespace frb
