// Fused denoiser inference on the 5th-generation tensor cores (tcgen05).
//
// Same function as inferKernel in mlp.cu (feature rows from the feature-render
// statistics, 112 -> 128 -> 128 -> 128 -> 8 network with bf16 operands and
// fp32 accumulation, bias + ReLU between layers, residual add), laid out for
// sm_103a's MMA unit as a two-role pipeline in one persistent block of 1024
// threads per SM:
//   * all weights are staged once in shared memory as K-major UMMA operands
//     (transposed to [out][in]) in the canonical no-swizzle layout: 8-row x
//     16-byte core matrices, core matrices along K 128 bytes apart (leading
//     byte offset) and 8-row groups K*16 bytes apart (stride byte offset);
//   * feature warps 0-15 build the 112 features of each row of a 128-row
//     tile from statistics derived once per row (deriveKernel: three float4)
//     and unit axes (axesKernel), into one of three tile buffers, and signal
//     it full on an mbarrier.  A warp holds one quarter of the features of 32
//     rows, in whole 16-byte pieces (features 0-31, 32-63, 64-87, 88-111), so
//     every store is a 16-byte row of a core matrix, without bank conflicts;
//   * two groups of eight network warps (16-23 and 24-31) take the tiles in
//     turn, each with a 128-column TMEM accumulator of its own: one elected
//     thread of the group issues each layer's tcgen05.mma instructions (M =
//     128, N = 128, K = 16 each) and commits them to the group's mbarrier.
//     Warps q and 4 + q of a group read accumulator lanes 32 q .. +31,
//     columns 0-63 and 64-127, with tcgen05.ld, add the bias, apply ReLU,
//     round to bf16 and write the next layer's operand into the same tile
//     buffer (the MMAs that read it are done);
//     the last layer (N padded to 16) adds the residual base and writes the
//     output, and its commit hands the buffer back to the feature warps.
// A layer is a chain of waits (MMA, accumulator read, barrier) that leaves the
// SM idle; with two tiles in flight one group's waits are the other's work,
// and the third buffer lets the feature warps run ahead of both.  1.5 M rows
// take 451 us with one group, two buffers, two-byte feature stores and a
// 64-bit division a row, 358 us in this form, and 326 us with the statistics by
// slot (deriveKernel); without any feature work 285 us: what is left is the
// network side, whose operand reads, bias loads and activation stores share the
// shared-memory pipe.
// Every mbarrier wait is bounded: on timeout the waiting side records an error
// bit and stops; the other side then times out too, the network warps wait
// (bounded) for their last commit, and the TMEM is freed.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_api.hpp"
#include "features.cuh"

namespace cr {
namespace {

constexpr int kTcRows = 128;
constexpr int kFeatThreads = 512;  // feature warps 0-15: four threads per row
constexpr int kNetThreads = 256;   // a network group's warps: two per accumulator lane quarter
constexpr int kNetGroups = 2;
constexpr int kTcThreads = kFeatThreads + kNetGroups * kNetThreads;
constexpr int kTcBuffers = 3;
constexpr int kTmemCols = 128 * kNetGroups;
constexpr uint32_t kSpinLimit = 1u << 26;  // bounded waits (far longer than one layer's MMAs)

// Byte offset of element (r, k) in a K-major no-swizzle operand with K
// elements per row: 8x8 core matrices of bf16.
__host__ __device__ constexpr uint32_t coreOffset(uint32_t r, uint32_t k, uint32_t K) {
  return (r >> 3) * (K * 16u) + (k >> 3) * 128u + (r & 7u) * 16u + (k & 7u) * 2u;
}

// Shared-memory matrix descriptor: start address, leading byte offset
// (between core matrices along K), stride byte offset (between 8-row
// groups), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smemDesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;  // version
  return d;
}

// Instruction descriptor of kind::f16: fp32 accumulator, bf16 A and B, both
// K-major, N and M.
__host__ __device__ constexpr uint32_t instrDesc(uint32_t M, uint32_t N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ uint32_t smemAddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mmaBf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void commitTo(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ bool tryWait(uint32_t mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool waitParity(uint32_t mbar, uint32_t parity) {
  for (uint32_t i = 0; i < kSpinLimit; ++i)
    if (tryWait(mbar, parity)) return true;
  return false;
}

__device__ __forceinline__ void fenceAsyncShared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tcFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive fp32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmemLoad32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmemLoad4(uint32_t taddr, float* v) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}

// Two floats to a bf16 pair, round to nearest even: one paired conversion
// (the conversion pipe's throughput limited the epilogue with two single
// ones).
__device__ __forceinline__ uint32_t packBf16(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}

// Shared memory plan (bytes).
constexpr uint32_t kW1Bytes = kMlpHidden * kFeatureWidth * 2;  // 128 x 112
constexpr uint32_t kWBytes = kMlpHidden * kMlpHidden * 2;      // 128 x 128
constexpr uint32_t kW4Rows = 16;                               // N of the last layer, padded
constexpr uint32_t kW4Bytes = kW4Rows * kMlpHidden * 2;
constexpr uint32_t kActBytes = kTcRows * kMlpHidden * 2;
constexpr uint32_t kOffW1 = 0;
constexpr uint32_t kOffW2 = kOffW1 + kW1Bytes;
constexpr uint32_t kOffW3 = kOffW2 + kWBytes;
constexpr uint32_t kOffW4 = kOffW3 + kWBytes;
// Tile buffers: features (K = 112 layout), then in place the hidden
// activations of layers 1-3 (K = 128 layout).
constexpr uint32_t kOffB0 = kOffW4 + kW4Bytes;
constexpr uint32_t kOffBias = kOffB0 + kTcBuffers * kActBytes;      // 3 x 128 + 16 floats
constexpr uint32_t kBars = 2 * kTcBuffers + kNetGroups;             // full, empty, one per group's MMAs
constexpr uint32_t kOffBar = kOffBias + (3 * kMlpHidden + 16) * 4;  // mbarriers (8 B each) + TMEM address
constexpr uint32_t kTcSmem = kOffBar + 8 * kBars + 8 + 128;         // + alignment slack
static_assert(kTcSmem <= 227 * 1024, "shared memory plan exceeds a block's limit");

// Position of a thread's row: poses in order, the ommatidia of a pose in the
// eye's direction order, so that a tile's rows are neighbouring ommatidia whose
// neighbour statistics overlap in L1.  Steps from tile to tile without a
// division.
struct RowWalk {
  uint64_t pos, stride;
  uint32_t p, j, dp, dj, N;
  __device__ __forceinline__ RowWalk(uint64_t first, uint64_t step, uint32_t n) : pos(first), stride(step), N(n) {
    p = static_cast<uint32_t>(first / n);
    j = static_cast<uint32_t>(first - static_cast<uint64_t>(p) * n);
    dp = static_cast<uint32_t>(step / n);
    dj = static_cast<uint32_t>(step - static_cast<uint64_t>(dp) * n);
  }
  __device__ __forceinline__ void next() {
    pos += stride;
    p += dp;
    j += dj;
    if (j >= N) {
      j -= N;
      ++p;
    }
  }
  __device__ __forceinline__ uint32_t omm(const uint32_t* __restrict__ order) const {
    return order ? __ldg(order + j) : j;
  }
};

// Stages W[in x out] (global, bf16, row-major) as a K-major operand of
// `rows` output rows (zero beyond `out`) and `in` columns.
__device__ void stageWeights(unsigned char* dst, const __nv_bfloat16* __restrict__ w, int in, int out, int rows) {
  for (int e = threadIdx.x; e < rows * in; e += blockDim.x) {
    const int n = e / in, k = e % in;
    const __nv_bfloat16 v = n < out ? w[static_cast<size_t>(k) * out + n] : __float2bfloat16(0.f);
    *reinterpret_cast<__nv_bfloat16*>(dst + coreOffset(n, k, in)) = v;
  }
}

// Inputs of the inference in the eye's direction order (slots; order null:
// index order), so that the rows of a tile lie next to each other: derived
// statistics as three float4 planes of P x N, unit axes, and the neighbour
// table as kNeighbours planes of slots.  With the statistics by ommatidium
// index a gather of 32 rows touched 32 cache lines, and the L1's lookups
// bounded the feature warps (358 us for 1.5 M rows, 326 us by slot).
__global__ void deriveKernel(const float* __restrict__ stats, uint64_t rows, uint32_t N,
                             const uint32_t* __restrict__ order, float4* __restrict__ derived) {
  const uint64_t r = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const uint32_t p = static_cast<uint32_t>(r / N), j = static_cast<uint32_t>(r - static_cast<uint64_t>(p) * N);
  const uint32_t o = order ? __ldg(order + j) : j;
  const float4* s = reinterpret_cast<const float4*>(stats + (static_cast<size_t>(p) * N + o) * kFeatureStats);
  const float4 s0 = __ldg(s), s1 = __ldg(s + 1), s2 = __ldg(s + 2);
  const float row[kFeatureStats] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w, s2.x, s2.y, s2.z, s2.w};
  float4 d[3];
  feat::deriveStats(row, d);
#pragma unroll
  for (int k = 0; k < 3; ++k) derived[static_cast<size_t>(k) * rows + r] = d[k];
}

__global__ void axesKernel(const float4* __restrict__ omm, uint32_t N, const uint32_t* __restrict__ order,
                           float4* __restrict__ axes) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  float aa;
  const float3 d = feat::ommAxis(omm, order ? order[j] : j, aa);
  axes[j] = make_float4(d.x, d.y, d.z, aa);
}

__global__ void slotOfKernel(const uint32_t* __restrict__ order, uint32_t N, uint32_t* __restrict__ slotOf) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < N) slotOf[order ? order[j] : j] = j;
}

__global__ void slotNeighboursKernel(const int* __restrict__ nb, const uint32_t* __restrict__ order, uint32_t N,
                                     const uint32_t* __restrict__ slotOf, uint32_t* __restrict__ nbSlots) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  const uint32_t o = order ? order[j] : j;
  for (int k = 0; k < kNeighbours; ++k)
    nbSlots[static_cast<size_t>(k) * N + j] = slotOf[static_cast<uint32_t>(nb[kNeighbours * o + k])];
}

__device__ __forceinline__ void mbarInit(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbarArrive(uint32_t mbar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}\n" ::"r"(mbar) : "memory");
}

// AND of `v` over the threads of network group g (named barrier 1 + g).
__device__ __forceinline__ bool netAll(int g, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %3, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "n"(kNetThreads), "r"(1 + g)
      : "memory");
  return r != 0;
}

// Two bf16 of max(a + b, 0) of two float pairs: one packed addition, one
// paired conversion, one packed maximum (a NaN becomes 0, as with fmaxf; the
// maximum commutes with the rounding).
__device__ __forceinline__ uint32_t biasReluPack(float a0, float a1, float b0, float b1) {
  float s0, s1;
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %3};\n\t"
      "mov.b64 y, {%4, %5};\n\t"
      "add.rn.ftz.f32x2 z, x, y;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}\n"
      : "=f"(s0), "=f"(s1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(packBf16(s0, s1)), "r"(0u));
  return r;
}

// Features 8 c .. 8 c + 7 of tile row r as one 16-byte store.
__device__ __forceinline__ void putChunk(uint32_t buf, uint32_t r, uint32_t c, const float* f) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + coreOffset(r, 8 * c, kFeatureWidth)),
               "r"(packBf16(f[0], f[1])), "r"(packBf16(f[2], f[3])), "r"(packBf16(f[4], f[5])),
               "r"(packBf16(f[6], f[7]))
               : "memory");
}

// One quarter q of the features of slot o of a pose (dp: its first plane of
// derived statistics, the planes `plane` apart): the values of featureRowTo.
// The neighbours whose blocks reach into quarter q: [quarterBegin, quarterEnd).
__host__ __device__ constexpr int quarterBegin(int q) { return q == 0 ? 0 : (q == 1 ? 1 : (q == 2 ? 3 : 4)); }
__host__ __device__ constexpr int quarterEnd(int q) { return q == 0 ? 2 : (q == 1 ? 4 : (q == 2 ? 5 : 6)); }

template <int q>
__device__ __forceinline__ void featureQuarter(const float4* __restrict__ dp, uint64_t plane,
                                               const float4* __restrict__ axes, const uint32_t* near, uint32_t o,
                                               uint32_t buf, uint32_t r) {
  constexpr int kFirst = q == 0 ? 0 : (q == 1 ? 32 : (q == 2 ? 64 : 88)), kCount = q < 2 ? 32 : 24;
  const float4 a0 = __ldg(dp + o), a1 = __ldg(dp + plane + o);
  const float4 ax = __ldg(axes + o);
  const float aa = ax.w;
  const float3 d = make_float3(ax.x, ax.y, ax.z);
  float f[kCount];
#pragma unroll
  for (int k = 0; k < kCount; ++k) f[k] = 0.f;
  auto put = [&](int k, float v) {  // k is a constant wherever this is called
    if (k >= kFirst && k < kFirst + kCount) f[k - kFirst] = v;
  };
  if (q == 0) {
    const float4 a2 = __ldg(dp + 2 * plane + o);
    const float own[kFeatBlock] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z,
                                   d.x,  d.y,  d.z,  aa * 10.0f};
#pragma unroll
    for (int k = 0; k < kFeatBlock; ++k) put(k, own[k]);
  }
  const float inva = 1.0f / fmaxf(aa, 1e-6f);
  float3 t1 = fabsf(d.y) < 0.9f ? make_float3(d.z, 0.f, -d.x) : make_float3(0.f, -d.z, d.y);
  const float il = rsqrtf(fmaxf(t1.x * t1.x + t1.y * t1.y + t1.z * t1.z, 1e-30f));
  t1 = make_float3(t1.x * il, t1.y * il, t1.z * il);
  const float3 t2 = make_float3(d.y * t1.z - d.z * t1.y, d.z * t1.x - d.x * t1.z, d.x * t1.y - d.y * t1.x);
#pragma unroll
  for (int j = quarterBegin(q); j < quarterEnd(q); ++j) {
    const int k0 = kFeatBlock * (j + 1);
    const uint32_t n = near[j - quarterBegin(q)];
    const float4 b0 = __ldg(dp + n), b1 = __ldg(dp + plane + n), b2 = __ldg(dp + 2 * plane + n);
    const float4 e = __ldg(axes + n);
    const float3 g = make_float3(e.x - d.x, e.y - d.y, e.z - d.z);
    const float u = (g.x * t1.x + g.y * t1.y + g.z * t1.z) * inva, v = (g.x * t2.x + g.y * t2.y + g.z * t2.z) * inva;
    const float w[kFeatBlock] = {(b0.x - a0.x) * 4.0f, (b0.y - a0.y) * 4.0f, (b0.z - a0.z) * 4.0f,
                                 b0.w, b1.x, b1.y, b1.z - a1.z, b1.w - a1.w, b2.x, b2.y, b2.z,
                                 u, v, sqrtf(u * u + v * v), e.w * inva};
#pragma unroll
    for (int k = 0; k < kFeatBlock; ++k) put(k0 + k, w[k]);
  }
#pragma unroll
  for (int c = 0; c < kCount / 8; ++c) putChunk(buf, r, static_cast<uint32_t>(kFirst / 8 + c), f + 8 * c);
}

__global__ void __launch_bounds__(kTcThreads, 1)
    inferTcKernel(const float4* __restrict__ derived, const float4* __restrict__ axes,
                  const uint32_t* __restrict__ nb, uint32_t N, uint64_t rows, MlpWeights w, bool residual, float* __restrict__ out,
                  uint32_t* errFlag, const uint32_t* __restrict__ order) {
  extern __shared__ __align__(128) unsigned char smemRaw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smemRaw) + 127) & ~uintptr_t(127));
  float* bias = reinterpret_cast<float*>(sm + kOffBias);  // b1 | b2 | b3 | b4 (16)
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + kOffBar);
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(sm + kOffBar + 8 * kBars);
  const int tid = threadIdx.x, warp = tid >> 5;

  stageWeights(sm + kOffW1, w.w1, kFeatureWidth, kMlpHidden, kMlpHidden);
  stageWeights(sm + kOffW2, w.w2, kMlpHidden, kMlpHidden, kMlpHidden);
  stageWeights(sm + kOffW3, w.w3, kMlpHidden, kMlpHidden, kMlpHidden);
  stageWeights(sm + kOffW4, w.w4, kMlpHidden, kMlpOut, kW4Rows);
  for (int e = tid; e < kMlpHidden; e += kTcThreads) {
    bias[e] = w.b1[e];
    bias[kMlpHidden + e] = w.b2[e];
    bias[2 * kMlpHidden + e] = w.b3[e];
  }
  if (tid < 16) bias[3 * kMlpHidden + tid] = tid < kMlpOut ? w.b4[tid] : 0.f;
  const uint32_t bar0 = smemAddr(bars);
  auto fullBar = [bar0](uint32_t b) { return bar0 + 8u * b; };
  auto emptyBar = [bar0](uint32_t b) { return bar0 + 8u * (kTcBuffers + b); };
  if (tid == 0) {
    for (uint32_t b = 0; b < kTcBuffers; ++b) {
      mbarInit(fullBar(b), kFeatThreads);
      mbarInit(emptyBar(b), 1);
    }
    for (uint32_t g = 0; g < kNetGroups; ++g) mbarInit(bar0 + 8u * (2 * kTcBuffers + g), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kFeatThreads / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tmemSlot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fenceAsyncShared();
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint64_t tiles = (rows + kTcRows - 1) / kTcRows;

  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kTcRows;

  if (tid < kFeatThreads) {
    // Feature warps: tile i of this block into buffer i mod 3.
    const uint32_t r = static_cast<uint32_t>(tid & (kTcRows - 1)), q = static_cast<uint32_t>(tid / kTcRows);
    RowWalk row(static_cast<uint64_t>(blockIdx.x) * kTcRows + r, stride, N);
    // A row's neighbours and their statistics are dependent loads: the
    // indices of a tile are fetched while the tile before is built.
    const int j0 = quarterBegin(static_cast<int>(q)), j1 = quarterEnd(static_cast<int>(q));
    uint32_t near[3];
    auto neighbours = [&]() {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        near[k] = row.pos < rows && j0 + k < j1 ? __ldg(nb + static_cast<size_t>(j0 + k) * N + row.j) : 0u;
    };
    neighbours();
    uint32_t b = 0, round = 0;
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      if (round > 0 && !waitParity(emptyBar(b), (round - 1u) & 1u)) {
        atomicOr(errFlag, kErrMmaTimeout);
        break;
      }
      const uint32_t buf = smemAddr(sm + kOffB0) + b * kActBytes;
      if (row.pos < rows) {
        const float4* dp = derived + static_cast<size_t>(row.p) * N;
        const uint32_t cur[3] = {near[0], near[1], near[2]}, o = row.j;
        row.next();
        neighbours();
        switch (q) {  // the same for a whole warp
          case 0: featureQuarter<0>(dp, rows, axes, cur, o, buf, r); break;
          case 1: featureQuarter<1>(dp, rows, axes, cur, o, buf, r); break;
          case 2: featureQuarter<2>(dp, rows, axes, cur, o, buf, r); break;
          default: featureQuarter<3>(dp, rows, axes, cur, o, buf, r); break;
        }
      } else {
        const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (uint32_t c = q; c < kFeatureWidth / 8; c += 4) putChunk(buf, r, c, zero);
      }
      fenceAsyncShared();  // the tensor cores read the buffer through the async proxy
      mbarArrive(fullBar(b));
      if (++b == kTcBuffers) {
        b = 0;
        ++round;
      }
    }
  } else {
    // Network group g: the four layers of tiles g, g + 2, ... of this block.
    const int g = (tid - kFeatThreads) / kNetThreads;
    const uint32_t tmem = *tmemSlot + 128u * static_cast<uint32_t>(g);
    const int lq = warp & 3;                                            // TMEM lane quarter this warp may read
    const int half = ((warp - kFeatThreads / 32) >> 2) & 1;             // columns 64 half .. +63
    const int m = lq * 32 + (tid & 31);                                 // accumulator lane = tile row
    const uint32_t laneBase = tmem + (static_cast<uint32_t>(lq * 32) << 16);
    const bool issuer = tid == kFeatThreads + g * kNetThreads;
    const uint32_t mmaBar = bar0 + 8u * static_cast<uint32_t>(2 * kTcBuffers + g);
    const uint32_t biasAddr = smemAddr(bias);
    uint32_t phase = 0;
    bool ok = true, pending = false;  // pending: a commit to mmaBar not yet waited for
    const uint64_t first = blockIdx.x + static_cast<uint64_t>(g) * gridDim.x;
    RowWalk row(first * kTcRows + static_cast<uint64_t>(m), kNetGroups * stride, N);
    uint32_t b = static_cast<uint32_t>(g), round = 0;
    for (uint64_t tile = first; tile < tiles; tile += kNetGroups * static_cast<uint64_t>(gridDim.x)) {
      const uint32_t h = smemAddr(sm + kOffB0) + b * kActBytes;
      for (int layer = 0; layer < 4; ++layer) {
        const uint32_t K = layer == 0 ? kFeatureWidth : kMlpHidden;
        const uint32_t Nn = layer == 3 ? kW4Rows : kMlpHidden;
        if (issuer && (layer > 0 || waitParity(fullBar(b), round & 1u))) {
          tcFenceAfter();
          const uint32_t idesc = instrDesc(kTcRows, Nn);
          const uint32_t wOff = layer == 0 ? kOffW1 : (layer == 1 ? kOffW2 : (layer == 2 ? kOffW3 : kOffW4));
          const uint32_t sW = smemAddr(sm) + wOff;
          for (uint32_t ks = 0; ks < K / 16; ++ks) {
            const uint64_t a = smemDesc(h + ks * 256u, 128u, K * 16u);
            const uint64_t bd = smemDesc(sW + ks * 256u, 128u, K * 16u);
            mmaBf16(tmem, a, bd, idesc, ks > 0 ? 1u : 0u);
          }
          if (layer == 3) commitTo(emptyBar(b));  // the tile buffer is free once these MMAs are done
          commitTo(mmaBar);
          pending = true;
        }
        // A wait that times out (also when the issuer had nothing to issue)
        // ends the group at the barrier below; tcgen05.ld wants whole warps.
        ok = __all_sync(0xffffffffu, waitParity(mmaBar, phase));
        phase ^= 1u;
        tcFenceAfter();
        if (ok) {
          pending = false;
          if (layer < 3) {
#pragma unroll 1
            for (uint32_t c0 = 64u * half; c0 < 64u * half + 64u; c0 += 32u) {
              float v[32];
              tmemLoad32(laneBase + c0, v);
              const uint32_t bs = biasAddr + 4u * (static_cast<uint32_t>(layer) * kMlpHidden + c0);
              const uint32_t hs = h + coreOffset(static_cast<uint32_t>(m), c0, kMlpHidden);
#pragma unroll
              for (uint32_t j = 0; j < 4; ++j) {
                float c[8];
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                             : "r"(bs + 32u * j));
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(c[4]), "=f"(c[5]), "=f"(c[6]), "=f"(c[7])
                             : "r"(bs + 32u * j + 16u));
                uint32_t qs[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  qs[k] = biasReluPack(v[8 * j + 2 * k], v[8 * j + 2 * k + 1], c[2 * k], c[2 * k + 1]);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hs + 128u * j), "r"(qs[0]), "r"(qs[1]),
                             "r"(qs[2]), "r"(qs[3])
                             : "memory");
              }
            }
          } else if (half == 0) {
            float v[4];
            tmemLoad4(laneBase, v);
            if (row.pos < rows) {
              const uint64_t at = static_cast<uint64_t>(row.p) * N + row.omm(order);
              const float* b4 = bias + 3 * kMlpHidden;
              const float4 mc = __ldg(derived + row.pos);  // the mean colour, as the statistics hold it
              const float mean[3] = {mc.x, mc.y, mc.z};
              for (int c = 0; c < 3; ++c) {
                const float y = v[c] + b4[c];
                out[3 * at + c] = residual ? mean[c] + y : y;
              }
            }
          }
        }
        // The next MMA reads h (async proxy) and overwrites the accumulator
        // that every thread of the group has just read.
        fenceAsyncShared();
        tcFenceBefore();
        ok = netAll(g, ok);
        tcFenceAfter();
        if (!ok) break;
      }
      if (!ok) {
        if (issuer) atomicOr(errFlag, kErrMmaTimeout);
        break;
      }
      row.next();
      b += kNetGroups;
      if (b >= kTcBuffers) {
        b -= kTcBuffers;
        ++round;
      }
    }
    if (!ok && pending && issuer) waitParity(mmaBar, phase ^ 1u);  // let a late commit land before the TMEM is freed
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  if (warp == kFeatThreads / 32) {
    const uint32_t tmem = *tmemSlot;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// The bounded wait, on an mbarrier that nothing arrives on.
__global__ void waitProbeKernel(uint32_t polls, uint32_t* errFlag) {
  __shared__ uint64_t bar;
  const uint32_t mbar = smemAddr(&bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  bool landed = false;
  for (uint32_t i = 0; i < polls && !landed; ++i) landed = tryWait(mbar, 0);
  if (!landed && threadIdx.x == 0) atomicOr(errFlag, kErrMmaTimeout);
}

// ---------------------------------------------------------------------------
// Training GEMMs on the tcgen05 tensor cores: C[M x N] = sum_k a(m, k) b(n, k)
// with the operand conventions of gemmBf16 (mlp.cu):
//   a(m, k) = aTrans ? A[k * lda + m] : A[m * lda + k],
//   b(n, k) = bTrans ? B[n * ldb + k] : B[k * ldb + n],
// and its epilogues (0 fp32 store, 1 bias + ReLU to bf16 and the fp32
// pre-activation, 2 ReLU-derivative mask to bf16, 3 bias to fp32).
// One 256-thread block per 128 x 128 output tile (N padded to a multiple of
// 16 for the MMA), K in chunks of 64 staged by the threads into shared
// memory in the canonical K-major no-swizzle layout, 16 bytes per load; one
// thread issues the chunk's four tcgen05.mma (K 16 each) into the TMEM
// accumulator and commits them; warps w and w + 4 read accumulator lanes
// 32 w .. +31, columns 0-63 and 64-127.  grid.z > 1 splits
// K into slices that write partial tiles (ldc = N) for a reduction in slice
// order.  Waits are bounded; a timeout sets g_tcGemmErr.
// ---------------------------------------------------------------------------
constexpr int kGemmTile = 128;
constexpr int kGemmChunk = 64;
constexpr uint32_t kGemmStage = kGemmTile * kGemmChunk * 2;  // bytes per operand stage
// Dynamic shared memory per block, sized so that at most four blocks share
// an SM: their four 128-column accumulators fill its 512 TMEM columns, and
// no block ever waits in tcgen05.alloc.
constexpr uint32_t kGemmSmem = 56 * 1024;
static_assert(2 * kGemmStage + 128 <= kGemmSmem, "staging exceeds the block's shared memory");
constexpr uint32_t kGemmMaskOff = 8 * 32 * 33 * 4;  // after the eight warps' fp32 epilogue tiles
constexpr int kGemmMaskLd = 40;                     // bf16 per mask row: 80 bytes, 16-byte aligned rows
static_assert(kGemmMaskOff % 16 == 0, "mask tiles must start 16-byte aligned");
static_assert(kGemmMaskOff + 8 * 32 * kGemmMaskLd * 2 + 128 <= kGemmSmem,
              "epilogue tiles exceed the block's shared memory");
__device__ uint32_t g_tcGemmErr;

constexpr int kGemmThreads = 256;  // eight warps: two per accumulator lane quarter

// Stages rows [0, rowsValid) x chunk columns of an operand whose element
// (r, c) is at P[(row0 + r) * ld + k0 + c] (K contiguous: 8 elements per
// 16-byte load) or, when `kMajorInMemory` is false, at
// P[(k0 + c) * ld + row0 + r] (rows contiguous: 8 rows per 16-byte load,
// scattered to their core-matrix rows); zero outside rowsValid and kEnd.
__device__ __forceinline__ void stageOperand(unsigned char* dst, const __nv_bfloat16* __restrict__ P, int ld,
                                             bool kMajorInMemory, int row0, int rowsValid, int rowsPadded, int k0,
                                             int kEnd, int tid) {
  const bool vec = (reinterpret_cast<uintptr_t>(P) & 15) == 0 && (ld & 7) == 0;
  if (kMajorInMemory) {
    // groups of 8 consecutive k of one row
    for (int e = tid; e < rowsPadded * (kGemmChunk / 8); e += kGemmThreads) {
      const int r = e / (kGemmChunk / 8), c = (e % (kGemmChunk / 8)) * 8;
      const int k = k0 + c;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < rowsValid) {
        const __nv_bfloat16* src = P + static_cast<size_t>(row0 + r) * ld + k;
        if (vec && k + 8 <= kEnd) {
          v = *reinterpret_cast<const uint4*>(src);
        } else {
          uint16_t t[8];
          for (int j = 0; j < 8; ++j) t[j] = k + j < kEnd ? __bfloat16_as_ushort(src[j]) : 0;
          v = make_uint4(t[0] | (uint32_t(t[1]) << 16), t[2] | (uint32_t(t[3]) << 16), t[4] | (uint32_t(t[5]) << 16),
                         t[6] | (uint32_t(t[7]) << 16));
        }
      }
      *reinterpret_cast<uint4*>(dst + coreOffset(static_cast<uint32_t>(r), static_cast<uint32_t>(c), kGemmChunk)) = v;
    }
  } else {
    // 8 x 8 blocks (8 rows x 8 k), one per group of eight lanes: lane l8
    // loads the block's 8 rows at k = 8 kg + l8 (16 bytes, rows contiguous in
    // memory), the group transposes the block in three exchange rounds, and
    // lane l8 stores row l8's 8 k as one 16-byte row of a core matrix, so the
    // eight lanes of a store phase fill 128 contiguous bytes.
    const int lane = tid & 31, q = lane >> 3, l8 = lane & 7;
    const int groups = rowsPadded / 8, nBlocks = groups * (kGemmChunk / 8);  // nBlocks: a multiple of 4
    for (int base = (tid >> 5) * 4; base < nBlocks; base += kGemmThreads / 8) {
      const int b = base + q;  // < nBlocks for every lane: the warp runs each round whole
      const int g = b % groups, kg = b / groups;
      const int r = g * 8, k = k0 + kg * 8 + l8;
      uint32_t w0 = 0u, w1 = 0u, w2 = 0u, w3 = 0u;
      if (k < kEnd) {
        const __nv_bfloat16* src = P + static_cast<size_t>(k) * ld + row0 + r;
        if (vec && r + 8 <= rowsValid) {
          const uint4 v = *reinterpret_cast<const uint4*>(src);
          w0 = v.x; w1 = v.y; w2 = v.z; w3 = v.w;
        } else {
          uint32_t t[8];
          for (int j = 0; j < 8; ++j) t[j] = r + j < rowsValid ? __bfloat16_as_ushort(src[j]) : 0u;
          w0 = t[0] | (t[1] << 16); w1 = t[2] | (t[3] << 16); w2 = t[4] | (t[5] << 16); w3 = t[6] | (t[7] << 16);
        }
      }
      // Round 1, lanes l8 ^ 4: elements 4-7 of the low lanes for 0-3 of the high ones.
      {
        const bool hi = l8 & 4;
        const uint32_t r0 = __shfl_xor_sync(0xffffffffu, hi ? w0 : w2, 4);
        const uint32_t r1 = __shfl_xor_sync(0xffffffffu, hi ? w1 : w3, 4);
        if (hi) { w0 = r0; w1 = r1; } else { w2 = r0; w3 = r1; }
      }
      // Round 2, lanes l8 ^ 2: element pairs {2,3}, {6,7} against {0,1}, {4,5}.
      {
        const bool hi = l8 & 2;
        const uint32_t r0 = __shfl_xor_sync(0xffffffffu, hi ? w0 : w1, 2);
        const uint32_t r1 = __shfl_xor_sync(0xffffffffu, hi ? w2 : w3, 2);
        if (hi) { w0 = r0; w2 = r1; } else { w1 = r0; w3 = r1; }
      }
      // Round 3, lanes l8 ^ 1: odd elements of the even lane for even
      // elements of the odd lane, two per exchanged word.
      {
        const bool hi = l8 & 1;
        const uint32_t s0 = hi ? __byte_perm(w0, w1, 0x5410) : __byte_perm(w0, w1, 0x7632);
        const uint32_t s1 = hi ? __byte_perm(w2, w3, 0x5410) : __byte_perm(w2, w3, 0x7632);
        const uint32_t r0 = __shfl_xor_sync(0xffffffffu, s0, 1);
        const uint32_t r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
        if (hi) {
          w0 = __byte_perm(r0, w0, 0x7610); w1 = __byte_perm(r0, w1, 0x7632);
          w2 = __byte_perm(r1, w2, 0x7610); w3 = __byte_perm(r1, w3, 0x7632);
        } else {
          w0 = __byte_perm(w0, r0, 0x5410); w1 = __byte_perm(w1, r0, 0x7610);
          w2 = __byte_perm(w2, r1, 0x5410); w3 = __byte_perm(w3, r1, 0x7610);
        }
      }
      *reinterpret_cast<uint4*>(dst + coreOffset(static_cast<uint32_t>(r + l8), static_cast<uint32_t>(kg * 8),
                                                 kGemmChunk)) = make_uint4(w0, w1, w2, w3);
    }
  }
}

template <int kMode>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemmTcKernel(int M, int N, int K, const __nv_bfloat16* __restrict__ A, int lda, bool aTrans,
                 const __nv_bfloat16* __restrict__ B, int ldb, bool bTrans, float* __restrict__ Cf,
                 __nv_bfloat16* __restrict__ Hb, int ldc, const float* __restrict__ bias,
                 const __nv_bfloat16* __restrict__ mask, int kSlice) {
  extern __shared__ __align__(128) unsigned char gemmSmem[];
  unsigned char* stage =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gemmSmem) + 127) & ~uintptr_t(127));
  __shared__ uint64_t bar;
  __shared__ uint32_t tmemSlot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * kGemmTile, n0 = blockIdx.x * kGemmTile;
  const int Mt = min(kGemmTile, M - m0);
  const int Nt = min(kGemmTile, N - n0);
  const uint32_t Nn = static_cast<uint32_t>((Nt + 15) & ~15);  // MMA N: a multiple of 16
  const int kBeg = kSlice ? static_cast<int>(blockIdx.z) * kSlice : 0;
  const int kEnd = kSlice ? min(K, kBeg + kSlice) : K;
  if (kSlice) Cf += static_cast<size_t>(blockIdx.z) * M * N;
  unsigned char* sA = stage;
  unsigned char* sB = stage + kGemmStage;
  const uint32_t mbar = smemAddr(&bar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint32_t tmem = tmemSlot;
  uint32_t phase = 0;
  bool ok = true, pending = false;
  for (int k0 = kBeg; k0 < kEnd && ok; k0 += kGemmChunk) {
    // a(m, k): K contiguous unless aTrans; b(n, k): K contiguous when bTrans.
    stageOperand(sA, A, lda, !aTrans, m0, Mt, kGemmTile, k0, kEnd, tid);
    stageOperand(sB, B, ldb, bTrans, n0, Nt, static_cast<int>(Nn), k0, kEnd, tid);
    fenceAsyncShared();
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    if (tid == 0) {
      const uint32_t idesc = instrDesc(kGemmTile, Nn);
      for (uint32_t ks = 0; ks < kGemmChunk / 16; ++ks) {
        const uint64_t a = smemDesc(smemAddr(sA) + ks * 256u, 128u, kGemmChunk * 16u);
        const uint64_t b = smemDesc(smemAddr(sB) + ks * 256u, 128u, kGemmChunk * 16u);
        mmaBf16(tmem, a, b, idesc, (k0 > kBeg || ks > 0) ? 1u : 0u);
      }
      commitTo(mbar);
    }
    pending = true;
    if (!__syncthreads_and(waitParity(mbar, phase))) {
      ok = false;
      if (tid == 0) atomicOr(&g_tcGemmErr, kErrMmaTimeout);
      break;
    }
    pending = false;
    phase ^= 1u;
    tcFenceAfter();
  }
  if (ok) {
    // Each warp turns its 32 rows x 32 columns through shared memory (the
    // staging area is free once the MMAs are done), so that a store writes
    // 32 consecutive columns of one row.
    const int lq = warp & 3, half = warp >> 2;  // lane quarter, and columns 64 half .. +63
    const uint32_t laneBase = tmem + (static_cast<uint32_t>(lq * 32) << 16);
    const bool empty = kEnd <= kBeg;  // no chunk ran: the accumulator holds nothing
    float* t = reinterpret_cast<float*>(stage) + warp * (32 * 33);
    // kMode 2: the warp's 32 x 32 block of the mask, read in 16-byte pieces
    // while the accumulators load, then turned through shared memory too.
    __nv_bfloat16* mt = reinterpret_cast<__nv_bfloat16*>(stage + kGemmMaskOff) + warp * (32 * kGemmMaskLd);
    const bool maskVec = kMode == 2 && (reinterpret_cast<uintptr_t>(mask) & 15) == 0 && (ldc & 7) == 0;
    for (int c0 = 64 * half; c0 < min(Nt, 64 * half + 64); c0 += 32) {
      uint4 mq[4];
      if (kMode == 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int m = m0 + lq * 32 + (lane >> 2) + 8 * i, cc = c0 + (lane & 3) * 8;
          mq[i] = make_uint4(0u, 0u, 0u, 0u);
          if (m < M) {
            const __nv_bfloat16* src = mask + static_cast<size_t>(m) * ldc + n0 + cc;
            if (maskVec && cc + 8 <= Nt) {
              mq[i] = __ldg(reinterpret_cast<const uint4*>(src));
            } else {
              uint16_t e[8];
              for (int j = 0; j < 8; ++j) e[j] = cc + j < Nt ? __bfloat16_as_ushort(src[j]) : 0;
              mq[i] = make_uint4(e[0] | (uint32_t(e[1]) << 16), e[2] | (uint32_t(e[3]) << 16),
                                 e[4] | (uint32_t(e[5]) << 16), e[6] | (uint32_t(e[7]) << 16));
            }
          }
        }
      }
      float v[32];
      if (!empty) tmemLoad32(laneBase + static_cast<uint32_t>(c0), v);
      else
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) t[lane * 33 + j] = v[j];  // row `lane`, column j
      if (kMode == 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(mt + ((lane >> 2) + 8 * i) * kGemmMaskLd + (lane & 3) * 8) = mq[i];
      }
      __syncwarp();
      const int n = n0 + c0 + lane;
      const bool colOk = c0 + lane < Nt;
      const float bn = (kMode == 1 || kMode == 3) && colOk ? bias[n] : 0.f;
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        const int m = m0 + lq * 32 + r;
        if (m >= M || !colOk) continue;
        const size_t o = static_cast<size_t>(m) * ldc + n;
        const float acc = t[r * 33 + lane];
        if (kMode == 0) {
          Cf[o] = acc;
        } else if (kMode == 1) {
          const float z = acc + bn;
          Cf[o] = z;
          Hb[o] = __float2bfloat16(fmaxf(z, 0.f));
        } else if (kMode == 2) {
          Hb[o] = __float2bfloat16(__bfloat162float(mt[r * kGemmMaskLd + lane]) > 0.f ? acc : 0.f);
        } else {
          Cf[o] = acc + bn;
        }
      }
      __syncwarp();
    }
  }
  if (!ok && pending && tid == 0) waitParity(mbar, phase);  // let a late commit land before the TMEM is freed
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

__global__ void tcSplitReduceKernel(const float* __restrict__ part, int slices, int M, int N, float* __restrict__ C,
                                    int ldc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M * N) return;
  const int m = i / N, n = i % N;
  float s = 0.f;
  for (int k = 0; k < slices; ++k) s += part[static_cast<size_t>(k) * M * N + i];
  C[static_cast<size_t>(m) * ldc + n] = s;
}

float* g_tcSplit = nullptr;
size_t g_tcSplitFloats = 0;

}  // namespace

cudaError_t gemmBf16Tc(int mode, int M, int N, int K, const void* A, int lda, bool aTrans, const void* B, int ldb,
                       bool bTrans, float* Cf, void* Hb, int ldc, const float* bias, const void* mask,
                       cudaStream_t stream) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  if (mode < 0 || mode > 3) return cudaErrorInvalidValue;
  const unsigned gx = static_cast<unsigned>((N + kGemmTile - 1) / kGemmTile);
  const unsigned gy = static_cast<unsigned>((M + kGemmTile - 1) / kGemmTile);
  auto a = static_cast<const __nv_bfloat16*>(A);
  auto b = static_cast<const __nv_bfloat16*>(B);
  auto h = static_cast<__nv_bfloat16*>(Hb);
  auto mk = static_cast<const __nv_bfloat16*>(mask);
  // Weight gradients: a long K over the minibatch and one or two output
  // tiles; K is split into slices of 128 summed afterwards in slice order.
  static bool attrSet = false;
  if (!attrSet) {
    const void* fns[4] = {reinterpret_cast<const void*>(gemmTcKernel<0>), reinterpret_cast<const void*>(gemmTcKernel<1>),
                          reinterpret_cast<const void*>(gemmTcKernel<2>), reinterpret_cast<const void*>(gemmTcKernel<3>)};
    for (const void* f : fns) {
      const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
      if (e != cudaSuccess) return e;
    }
    attrSet = true;
  }
  if (mode == 0 && K >= 1024 && gx * gy < 64) {
    const int slice = 128, slices = (K + slice - 1) / slice;
    const size_t need = static_cast<size_t>(slices) * M * N;
    if (need > g_tcSplitFloats) {
      if (g_tcSplit) cudaFree(g_tcSplit);
      g_tcSplit = nullptr;
      g_tcSplitFloats = 0;
      const cudaError_t e = cudaMalloc(&g_tcSplit, need * sizeof(float));
      if (e != cudaSuccess) return e;
      g_tcSplitFloats = need;
    }
    gemmTcKernel<0><<<dim3(gx, gy, slices), kGemmThreads, kGemmSmem, stream>>>(M, N, K, a, lda, aTrans, b, ldb, bTrans,
                                                                       g_tcSplit, nullptr, N, nullptr, nullptr, slice);
    tcSplitReduceKernel<<<(M * N + 255) / 256, 256, 0, stream>>>(g_tcSplit, slices, M, N, Cf, ldc);
    return cudaGetLastError();
  }
  const dim3 grid(gx, gy);
  switch (mode) {
    case 0: gemmTcKernel<0><<<grid, kGemmThreads, kGemmSmem, stream>>>(M, N, K, a, lda, aTrans, b, ldb, bTrans, Cf, h, ldc, bias, mk, 0); break;
    case 1: gemmTcKernel<1><<<grid, kGemmThreads, kGemmSmem, stream>>>(M, N, K, a, lda, aTrans, b, ldb, bTrans, Cf, h, ldc, bias, mk, 0); break;
    case 2: gemmTcKernel<2><<<grid, kGemmThreads, kGemmSmem, stream>>>(M, N, K, a, lda, aTrans, b, ldb, bTrans, Cf, h, ldc, bias, mk, 0); break;
    default: gemmTcKernel<3><<<grid, kGemmThreads, kGemmSmem, stream>>>(M, N, K, a, lda, aTrans, b, ldb, bTrans, Cf, h, ldc, bias, mk, 0); break;
  }
  return cudaGetLastError();
}

cudaError_t takeTcGemmError(uint32_t* flags) {
  cudaError_t e = cudaMemcpyFromSymbol(flags, g_tcGemmErr, sizeof(uint32_t));
  if (e != cudaSuccess) return e;
  const uint32_t zero = 0;
  return cudaMemcpyToSymbol(g_tcGemmErr, &zero, sizeof(uint32_t));
}

cudaError_t launchWaitProbe(uint32_t polls, uint32_t* errFlag, cudaStream_t stream) {
  waitProbeKernel<<<1, 32, 0, stream>>>(polls, errFlag);
  return cudaGetLastError();
}

cudaError_t slotNeighbours(const int* nb, const uint32_t* order, uint32_t N, uint32_t* slotOf, uint32_t* nbSlots,
                           cudaStream_t stream) {
  if (N == 0) return cudaSuccess;
  slotOfKernel<<<(N + 255) / 256, 256, 0, stream>>>(order, N, slotOf);
  slotNeighboursKernel<<<(N + 255) / 256, 256, 0, stream>>>(nb, order, N, slotOf, nbSlots);
  return cudaGetLastError();
}

cudaError_t deriveFeatureStats(const float* stats, const float4* omm, uint32_t N, uint32_t P, const uint32_t* order,
                               float4* derived, float4* axes, cudaStream_t stream) {
  const uint64_t rows = static_cast<uint64_t>(N) * P;
  if (rows == 0) return cudaSuccess;
  deriveKernel<<<static_cast<unsigned>((rows + 255) / 256), 256, 0, stream>>>(stats, rows, N, order, derived);
  axesKernel<<<(N + 255) / 256, 256, 0, stream>>>(omm, N, order, axes);
  return cudaGetLastError();
}

cudaError_t inferDenoiserTc(const float4* derived, const float4* axes, const uint32_t* nbSlots, uint32_t N, uint32_t P,
                            const MlpWeights& w, float* out, uint32_t* errFlag, cudaStream_t stream, bool residual,
                            const uint32_t* order) {
  const uint64_t rows = static_cast<uint64_t>(N) * P;
  if (rows == 0) return cudaSuccess;
  static int smCount = 0;
  static bool attrSet = false;
  if (!attrSet) {
    cudaError_t e = cudaFuncSetAttribute(inferTcKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kTcSmem));
    if (e != cudaSuccess) return e;
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smCount, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    attrSet = true;
  }
  const uint64_t tiles = (rows + kTcRows - 1) / kTcRows;
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(tiles, static_cast<uint64_t>(smCount)));
  inferTcKernel<<<grid, kTcThreads, kTcSmem, stream>>>(derived, axes, nbSlots, N, rows, w, residual, out, errFlag, order);
  return cudaGetLastError();
}

}  // namespace cr
