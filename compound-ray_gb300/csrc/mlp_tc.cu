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
//     and unit axes (axesKernel), into one of four tile buffers, and signal
//     it full on an mbarrier.  A warp holds one quarter of the features of 32
//     rows, in whole 16-byte pieces (features 0-31, 32-63, 64-87, 88-111), so
//     every store is a 16-byte row of a core matrix, without bank conflicts;
//   * four groups of four network warps (16-19, .. 28-31) take the tiles in
//     turn, each with a 128-column TMEM accumulator of its own: one warp of
//     the group issues each layer's tcgen05.mma instructions (M = 128,
//     N = 128, K = 16 each) and commits them to the group's mbarrier.  The
//     hidden layers compute outputs by rows (A the weights, B the tile), so a
//     thread of warp q reads one output's accumulators for all 128 rows
//     (tcgen05.ld, lane 32 q ..), adds the bias that it holds in a register,
//     applies ReLU, rounds to bf16 and writes 16-byte pieces of eight rows
//     into the same tile buffer (the MMAs that read it are done): the next
//     layer's MN-major operand.  The last layer (N padded to 16) has the rows
//     as M again, adds the residual base and writes the output, and its commit
//     hands the buffer back to the feature warps.
// A layer is a chain of waits (MMA, accumulator read, barrier) that leaves the
// SM idle; with four tiles in flight one group's waits are the others' work.
// 1.5 M rows took 451 us with one group, two buffers, two-byte feature stores
// and a 64-bit division a row; 358 with two groups of eight warps and three
// buffers; 326 with the statistics by slot (deriveKernel); 265 with MMAs
// issued by a converged warp (electLane); 240 with four groups; 218 in this
// form (rows by outputs read the biases from shared memory, whose pipe the
// MMAs' operands fill).  Without feature work it is 58 us less, without the
// hidden layers' epilogue 47, without both 85: the MMAs alone are 80 us at
// their rate.
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
constexpr int kNetThreads = 128;   // a network group's warps: one per accumulator lane quarter
constexpr int kNetGroups = 4;
constexpr int kTcThreads = kFeatThreads + kNetGroups * kNetThreads;
constexpr int kTcBuffers = kNetGroups;  // tile buffers: group g works in buffer g
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

// The same with an MN-major operand.
constexpr uint32_t kAMnMajor = 1u << 15, kBMnMajor = 1u << 16;

__device__ __forceinline__ uint32_t smemAddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One lane of a converged warp.  MMAs are issued by a whole warp with this as
// their predicate: behind a branch on the thread's index the compiler has to
// move every descriptor to a uniform register in a loop over the lanes, and a
// 128 x 128 x 16 MMA took 118 clocks to issue; like this it takes the 64 that
// the MMA itself needs.
__device__ __forceinline__ uint32_t electLane() {
  uint32_t e;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(e));
  return e;
}

__device__ __forceinline__ void mmaBf16(uint32_t elected, uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected));
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

// Two bf16 of max(a + b, 0): one packed addition, one paired conversion, one
// packed maximum (a NaN becomes 0, as with fmaxf; the maximum commutes with
// the rounding).
__device__ __forceinline__ uint32_t biasReluPack(float a0, float a1, float b) {
  float s0, s1;
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %3};\n\t"
      "mov.b64 y, {%4, %4};\n\t"
      "add.rn.ftz.f32x2 z, x, y;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}\n"
      : "=f"(s0), "=f"(s1)
      : "f"(a0), "f"(a1), "f"(b));
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
    // Feature warps: tile i of this block into buffer i mod kTcBuffers.
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
    // Network group g: the four layers of tiles g, g + kNetGroups, ... of this
    // block, in buffer g.
    const int g = (tid - kFeatThreads) / kNetThreads;
    const uint32_t tmem = *tmemSlot + 128u * static_cast<uint32_t>(g);
    const int lq = warp & 3;                                            // TMEM lane quarter this warp may read
    const int m = lq * 32 + (tid & 31);                                 // accumulator lane: an output, last layer a tile row
    const uint32_t laneBase = tmem + (static_cast<uint32_t>(lq * 32) << 16);
    const bool issuer = tid == kFeatThreads + g * kNetThreads;
    const bool issuing = __shfl_sync(0xffffffffu, warp, 0) == (kFeatThreads + g * kNetThreads) / 32;  // the issuer's warp
    const uint32_t mmaBar = bar0 + 8u * static_cast<uint32_t>(2 * kTcBuffers + g);
    uint32_t phase = 0;
    bool ok = true, pending = false;  // pending: a commit to mmaBar not yet waited for
    const uint64_t first = blockIdx.x + static_cast<uint64_t>(g) * gridDim.x;
    RowWalk row(first * kTcRows + static_cast<uint64_t>(m), kNetGroups * stride, N);
    const uint32_t b = static_cast<uint32_t>(g), h = smemAddr(sm + kOffB0) + b * kActBytes;
    uint32_t round = 0;
    for (uint64_t tile = first; tile < tiles; tile += kNetGroups * static_cast<uint64_t>(gridDim.x), ++round) {
      for (int layer = 0; layer < 4; ++layer) {
        const uint32_t K = layer == 0 ? kFeatureWidth : kMlpHidden;
        if (issuing && (layer > 0 || __all_sync(0xffffffffu, waitParity(fullBar(b), round & 1u)))) {
          tcFenceAfter();
          const uint32_t elected = electLane();
          const uint32_t idesc = layer == 3 ? instrDesc(kTcRows, kW4Rows) | kAMnMajor
                                            : instrDesc(kMlpHidden, kTcRows) | (layer > 0 ? kBMnMajor : 0u);
          const uint32_t wOff = layer == 0 ? kOffW1 : (layer == 1 ? kOffW2 : (layer == 2 ? kOffW3 : kOffW4));
          const uint32_t sW = smemAddr(sm) + wOff;
          const uint64_t x = layer == 0 ? smemDesc(h, 128u, K * 16u) : smemDesc(h, kMlpHidden * 16u, 128u);
          const uint64_t w = smemDesc(sW, 128u, K * 16u);
          const uint32_t xStep = layer == 0 ? 16u : 2u * kMlpHidden;  // 16 bytes of address: 16 features on
#pragma unroll
          for (uint32_t ks = 0; ks < kMlpHidden / 16; ++ks)
            if (ks < K / 16)
              mmaBf16(elected, tmem, layer == 3 ? x + ks * xStep : w + 16u * ks, layer == 3 ? w + 16u * ks : x + ks * xStep,
                      idesc, ks > 0 ? 1u : 0u);
          if (elected) {
            if (layer == 3) commitTo(emptyBar(b));  // the tile buffer is free once these MMAs are done
            commitTo(mmaBar);
          }
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
            const float own = bias[layer * kMlpHidden + m];
#pragma unroll
            for (uint32_t c0 = 0; c0 < kTcRows; c0 += 32u) {
              float v[32];
              tmemLoad32(laneBase + c0, v);
              const uint32_t hs = h + coreOffset(static_cast<uint32_t>(m), c0, kMlpHidden);
#pragma unroll
              for (uint32_t j = 0; j < 4; ++j) {
                uint32_t qs[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  qs[k] = biasReluPack(v[8 * j + 2 * k], v[8 * j + 2 * k + 1], own);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hs + 128u * j), "r"(qs[0]), "r"(qs[1]),
                             "r"(qs[2]), "r"(qs[3])
                             : "memory");
              }
            }
          } else {
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
// One training step's forward and backward pass for a tile of 128 rows, in
// one block: the rows are gathered, the four layers, the loss gradient, the
// input gradients and the tile's share of every weight and bias gradient are
// computed without leaving the SM, and only that share is written
// (kParams floats a tile; reduceStep sums the tiles in order).
//
// Every operand stays in shared memory in the canonical no-swizzle layout of
// 8 x 8 core matrices (coreOffset), and each is used twice.  A tile image
// [row][feature] is the K-major A operand of the next layer (K = features)
// and, read with the transpose bit, the MN-major operand of the weight
// gradient (K = rows, so core matrices along MN are 128 bytes apart and those
// along K a row group apart); a weight image [out][in] is the K-major B operand of the
// forward pass and the MN-major one of the input gradient.  So nothing is
// transposed and no second copy of the weights is read.  dz of layer l
// overwrites that layer's activations once the weight gradient that reads
// them is done; the ReLU masks stay in registers (a thread reads the same
// accumulator row and columns in both directions).
//
// 16 warps: warp w reads accumulator lanes 32 (w % 4) .. +31, columns
// 32 (w / 4) .. +31; one thread issues.  TMEM columns: 0-127 the forward and
// input-gradient accumulator, 128-143 dW4 and later 128-255 dW1, 256-383
// dW3, 384-511 dW2.  While the MMAs of a layer run, the warps write out the
// previous weight gradient and sum the bias gradient.
//
// A step is a chain of 8 dependent MMA groups, so its time is their latency
// and not their work: as 23 launches (one GEMM per layer and direction, with
// the activations in memory between them and split-K reductions) 8192 rows
// took 190 us a step; in this form 28 us with the reduction and Adam.
// The rows' sums are formed in the same order as there.  Waits are bounded; a
// timeout sets g_tcGemmErr.
// ---------------------------------------------------------------------------
constexpr int kStepThreads = 512;
constexpr uint32_t kStepXGroup = kFeatureWidth * 16u;  // bytes of 8 feature rows
constexpr uint32_t kStepGroup = kMlpHidden * 16u;      // bytes of 8 rows of a 128-wide image
constexpr uint32_t kOffStepX = 0;
constexpr uint32_t kOffStepH = kOffStepX + kTcRows * kFeatureWidth * 2;  // three layers' activations, then dz
constexpr uint32_t kOffStepW2 = kOffStepH + 3 * kActBytes;
constexpr uint32_t kOffStepW3 = kOffStepW2 + kWBytes;
constexpr uint32_t kOffStepW4 = kOffStepW3 + kWBytes;
constexpr uint32_t kOffStepW1 = kOffStepW4 + kW4Bytes;
constexpr uint32_t kOffStepDy = kOffStepW1 + kW1Bytes;               // 128 x 16 bf16, the upper 8 columns zero
constexpr uint32_t kOffStepBias = kOffStepDy + kTcRows * 16 * 2;     // 3 x 128 + 8 floats; later 3 x 128 of dy in fp32
constexpr uint32_t kStepSmem = kOffStepBias + (3 * kMlpHidden + 8) * 4 + 128;  // + alignment slack
static_assert(kStepSmem + 64 <= 227 * 1024, "shared memory plan exceeds a block's limit");
static_assert(kTcRows == kMlpHidden, "the weight gradients' M is a tile image's width");
constexpr uint32_t kStepTmemCols = 512;
__device__ uint32_t g_tcGemmErr;

// 16 bytes to shared memory, zeros unless `valid`.
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void copyCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void copyWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// The image of `rows` rows (the first `valid` from `src`, row-major with
// `in` columns, the others zero): core matrices in order, so piece e of 16
// bytes lies at 16 e.
__device__ __forceinline__ void copyImage(uint32_t dst, const __nv_bfloat16* __restrict__ src, int in, int rows,
                                          int valid) {
  for (int e = threadIdx.x; e < rows * in / 8; e += kStepThreads) {
    const int g = (e >> 3) / (in / 8), c = (e >> 3) - g * (in / 8), n = g * 8 + (e & 7);
    copy16(dst + 16u * static_cast<uint32_t>(e), src + static_cast<size_t>(n < valid ? n : 0) * in + 8 * c, n < valid);
  }
}

__global__ void __launch_bounds__(kStepThreads, 1) trainTileKernel(TrainTiles a) {
  extern __shared__ __align__(128) unsigned char stepSmem[];
  unsigned char* sm =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(stepSmem) + 127) & ~uintptr_t(127));
  __shared__ uint64_t bar;
  __shared__ uint32_t tmemSlot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lq = warp & 3, cq = warp >> 2;
  const int m = lq * 32 + lane;                           // accumulator lane: tile row, or row of a weight gradient
  const uint32_t c0 = 32u * static_cast<uint32_t>(cq);    // first of this thread's 32 columns
  const int row0 = (a.firstTile + static_cast<int>(blockIdx.x)) * kTcRows;
  const bool valid = row0 + m < a.rows;
  float* part = a.part + static_cast<size_t>(blockIdx.x) * a.stride;
  const uint32_t base = smemAddr(sm);
  const uint32_t mbar = smemAddr(&bar);
  if (tid == 0) {
    mbarInit(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)),
                 "r"(kStepTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // Copies in the order of use: rows and W1, W2, W3 with W4.
  const uint32_t* order = a.order ? a.order + (a.offset ? *a.offset : 0u) : nullptr;
  for (int e = tid; e < kTcRows * kFeatureWidth / 8; e += kStepThreads) {
    const int g = (e >> 3) / (kFeatureWidth / 8), c = (e >> 3) - g * (kFeatureWidth / 8), r = row0 + g * 8 + (e & 7);
    const bool in = r < a.rows;
    const size_t src = in ? (order ? __ldg(order + r) : static_cast<uint32_t>(r)) : 0u;
    copy16(base + kOffStepX + 16u * static_cast<uint32_t>(e), a.X + src * kFeatureWidth + 8 * c, in);
  }
  copyImage(base + kOffStepW1, a.wT + a.w.off[0], kFeatureWidth, kMlpHidden, kMlpHidden);
  copyCommit();
  copyImage(base + kOffStepW2, a.wT + a.w.off[1], kMlpHidden, kMlpHidden, kMlpHidden);
  copyCommit();
  copyImage(base + kOffStepW3, a.wT + a.w.off[2], kMlpHidden, kMlpHidden, kMlpHidden);
  copyImage(base + kOffStepW4, a.wT + a.w.off[3], kMlpHidden, static_cast<int>(kW4Rows), kMlpOut);
  copyCommit();
  float* bias = reinterpret_cast<float*>(sm + kOffStepBias);
  if (tid < 3 * kMlpHidden) bias[tid] = a.params[a.b[tid / kMlpHidden] + tid % kMlpHidden];
  else if (tid < 3 * kMlpHidden + kMlpOut) bias[tid] = a.params[a.b[3] + tid - 3 * kMlpHidden];
  float own[3] = {0.f, 0.f, 0.f}, want[3] = {0.f, 0.f, 0.f};
  if (cq == 0 && valid) {
    const size_t src = order ? __ldg(order + row0 + m) : static_cast<uint32_t>(row0 + m);
    for (int c = 0; c < 3; ++c) {
      own[c] = a.base[3 * src + c];
      want[c] = a.target[3 * src + c];
    }
  }
  bool ok = true;
  uint32_t phase = 0, commits = 0;
  uint32_t tmem = 0;
  // Everything written to shared memory before this is an operand after it,
  // and every accumulator read before it may be overwritten.
  auto meet = [&]() {
    fenceAsyncShared();
    tcFenceBefore();
    ok = __syncthreads_and(ok);
    tcFenceAfter();
  };
  const bool issuing = __shfl_sync(0xffffffffu, warp, 0) == 0;
  auto commit = [&](uint32_t elected) {
    if (elected) commitTo(mbar);
    ++commits;
  };
  auto await = [&]() {
    if (ok) ok = __all_sync(0xffffffffu, waitParity(mbar, phase));
    phase ^= 1u;
    tcFenceAfter();
  };
  const uint32_t laneBits = static_cast<uint32_t>(lq * 32) << 16;
  uint32_t mask[3];
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    if (l == 0) copyWait<2>();
    else if (l == 1) copyWait<1>();
    else copyWait<0>();
    meet();
    if (l == 0) tmem = tmemSlot;
    const uint32_t in = base + (l == 0 ? kOffStepX : kOffStepH + static_cast<uint32_t>(l - 1) * kActBytes);
    const uint32_t out = base + kOffStepH + static_cast<uint32_t>(l) * kActBytes;
    if (ok && issuing) {
      const uint32_t elected = electLane();
      const uint32_t w = base + (l == 0 ? kOffStepW1 : (l == 1 ? kOffStepW2 : kOffStepW3));
      const uint32_t group = l == 0 ? kStepXGroup : kStepGroup;
#pragma unroll
      for (uint32_t ks = 0; ks < (l == 0 ? kFeatureWidth : kMlpHidden) / 16; ++ks)
        mmaBf16(elected, tmem, smemDesc(in + ks * 256u, 128u, group), smemDesc(w + ks * 256u, 128u, group),
                instrDesc(kTcRows, kMlpHidden), ks > 0 ? 1u : 0u);
      commit(elected);
    }
    await();
    mask[l] = 0u;
    if (ok) {
      float v[32];
      tmemLoad32(tmem + laneBits + c0, v);
      const float* bl = bias + l * kMlpHidden + c0;
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        uint32_t q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = 8 * j + 2 * k;
          const uint32_t h = packBf16(fmaxf(v[i] + bl[i], 0.f), fmaxf(v[i + 1] + bl[i + 1], 0.f));
          q[k] = valid ? h : 0u;
          if (q[k] & 0x7fffu) mask[l] |= 1u << i;
          if (q[k] & 0x7fff0000u) mask[l] |= 2u << i;
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                         out + coreOffset(static_cast<uint32_t>(m), c0 + 8 * j, kMlpHidden)),
                     "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3])
                     : "memory");
      }
    }
  }
  // Output layer and the gradient of the mean squared error.
  meet();
  const uint32_t h3 = base + kOffStepH + 2 * kActBytes, dy = base + kOffStepDy;
  if (ok && issuing) {
    const uint32_t elected = electLane();
#pragma unroll
    for (uint32_t ks = 0; ks < kMlpHidden / 16; ++ks)
      mmaBf16(elected, tmem, smemDesc(h3 + ks * 256u, 128u, kStepGroup), smemDesc(base + kOffStepW4 + ks * 256u, 128u, kStepGroup),
              instrDesc(kTcRows, kW4Rows), ks > 0 ? 1u : 0u);
    commit(elected);
  }
  await();
  float* dyf = bias;  // [3][128], over the hidden layers' biases, which nothing reads any more
  if (ok && cq == 0) {
    float v[4];
    tmemLoad4(tmem + laneBits, v);
    const float scale = 2.0f / (3.0f * static_cast<float>(a.rows));
    float e2 = 0.f, g[3];
    for (int c = 0; c < 3; ++c) {
      const float y = v[c] + bias[3 * kMlpHidden + c];
      const float d = own[c] + y - want[c];
      if (valid) e2 += d * d;
      g[c] = valid ? scale * d : 0.f;
      dyf[c * kTcRows + m] = g[c];
    }
    const uint32_t at = dy + coreOffset(static_cast<uint32_t>(m), 0, 16);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %3};" ::"r"(at), "r"(packBf16(g[0], g[1])),
                 "r"(packBf16(g[2], 0.f)), "r"(0u)
                 : "memory");
    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at + 128u), "r"(0u) : "memory");
    if (a.lossSum) {
      for (int s = 16; s >= 1; s >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, s);
      if (lane == 0) atomicAdd(a.lossSum + (a.lossIndex ? *a.lossIndex : 0), e2);
    }
  }
  meet();
  if (ok && issuing) {
    const uint32_t elected = electLane();
#pragma unroll
    for (uint32_t ks = 0; ks < kTcRows / 16; ++ks)  // dW4 = h3^T dy
      mmaBf16(elected, tmem + 128u, smemDesc(h3 + ks * 2 * kStepGroup, kStepGroup, 128u), smemDesc(dy + ks * 512u, 256u, 128u),
              instrDesc(kMlpHidden, kW4Rows) | kAMnMajor | kBMnMajor, ks > 0 ? 1u : 0u);
    // dZ3 = dy W4^T, K = 16
    mmaBf16(elected, tmem, smemDesc(dy, 128u, 256u), smemDesc(base + kOffStepW4, kStepGroup, 128u),
            instrDesc(kTcRows, kMlpHidden) | kBMnMajor, 0u);
    commit(elected);
  }
  if (ok && warp == 0) {
    // db4, in colSum's order: lane 8 c + w sums rows w, w + 16, .. and w + 8,
    // w + 24, .., then the eight sums in order.
    const int c = lane >> 3, w = lane & 7;
    float s0 = 0.f, s1 = 0.f;
    if (c < 3)
      for (int r = w; r < kTcRows; r += 16) {
        s0 += dyf[c * kTcRows + r];
        s1 += dyf[c * kTcRows + r + 8];
      }
    const float s = s0 + s1;
    float t = 0.f;
    for (int k = 0; k < 8; ++k) t += __shfl_sync(0xffffffffu, s, (lane & 24) + k);
    t = __shfl_sync(0xffffffffu, t, (lane & 3) * 8);
    if (lane < kMlpOut) part[a.b[3] + lane] = lane < 3 ? t : 0.f;
  }
  // Columns c0 .. +31 of a weight gradient's row m, from TMEM column `at`:
  // float4 of four columns by row, so that a warp writes 512 bytes in a row.
  auto drain = [&](uint32_t at, int w, int in) {
    float v[32];
    tmemLoad32(tmem + at + laneBits + c0, v);
    if (m < in) {
      float4* dst = reinterpret_cast<float4*>(part + w) + static_cast<size_t>(c0 / 4) * in + m;
#pragma unroll
      for (int j = 0; j < 8; ++j) dst[static_cast<size_t>(j) * in] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  };
#pragma unroll
  for (int l = 2; l >= 0; --l) {
    const uint32_t dz = base + kOffStepH + static_cast<uint32_t>(l) * kActBytes;
    await();
    if (ok) {
      float v[32];
      tmemLoad32(tmem + laneBits + c0, v);
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        uint32_t q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = 8 * j + 2 * k;
          q[k] = packBf16(mask[l] & (1u << i) ? v[i] : 0.f, mask[l] & (2u << i) ? v[i + 1] : 0.f);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                         dz + coreOffset(static_cast<uint32_t>(m), c0 + 8 * j, kMlpHidden)),
                     "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3])
                     : "memory");
      }
    }
    meet();
    if (ok && issuing) {
      const uint32_t elected = electLane();
      const uint32_t in = base + (l == 0 ? kOffStepX : kOffStepH + static_cast<uint32_t>(l - 1) * kActBytes);
      const uint32_t group = l == 0 ? kStepXGroup : kStepGroup;
      const uint32_t acc = tmem + (l == 2 ? 256u : (l == 1 ? 384u : 128u));
      // dW = in^T dz.  For l = 0 accumulator rows 112-127 hold nothing: the
      // 16 columns past a feature row are the next row group's first.
      if (l > 0) {
        const uint32_t w = base + (l == 1 ? kOffStepW2 : kOffStepW3);
#pragma unroll
        for (uint32_t ks = 0; ks < kMlpHidden / 16; ++ks)  // dZ of the layer before: dz W^T
          mmaBf16(elected, tmem, smemDesc(dz + ks * 256u, 128u, kStepGroup), smemDesc(w + ks * 2 * kStepGroup, kStepGroup, 128u),
                  instrDesc(kTcRows, kMlpHidden) | kBMnMajor, ks > 0 ? 1u : 0u);
      }
#pragma unroll
      for (uint32_t ks = 0; ks < kTcRows / 16; ++ks)
        mmaBf16(elected, acc, smemDesc(in + ks * 2 * group, group, 128u), smemDesc(dz + ks * 2 * kStepGroup, kStepGroup, 128u),
                instrDesc(kMlpHidden, kMlpHidden) | kAMnMajor | kBMnMajor, ks > 0 ? 1u : 0u);
      commit(elected);
    }
    if (ok) {
      if (warp < 8) {
        // Bias gradient, in colSum's order: lane = 16 cg + 8 odd + w of warp
        // k sums rows w + 8 i, i odd or even, of the 8 columns of core column
        // 2 k + cg; then s0 + s1, and a column's eight sums in order.
        const int w = lane & 7, odd = (lane >> 3) & 1, cg = 2 * warp + (lane >> 4);
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 q = *reinterpret_cast<const uint4*>(sm + (dz - base) + (2 * i + odd) * kStepGroup + cg * 128 + w * 16);
          const uint32_t x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            s[2 * k] += __uint_as_float(x[k] << 16);
            s[2 * k + 1] += __uint_as_float(x[k] & 0xffff0000u);
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] += __shfl_xor_sync(0xffffffffu, s[k], 8);
        float mine = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float t = 0.f;
#pragma unroll
          for (int r = 0; r < 8; ++r) t += __shfl_sync(0xffffffffu, s[k], (lane & 24) + r);
          if (w == k) mine = t;
        }
        if (!odd) part[a.b[l] + cg * 8 + w] = mine;
      }
      if (l == 2) {
        if (cq == 0) {
          for (uint32_t k = 0; k < kMlpOut / 4; ++k) {
            float v[4];
            tmemLoad4(tmem + 128u + laneBits + 4 * k, v);
            reinterpret_cast<float4*>(part + a.w.off[3])[k * kMlpHidden + m] = make_float4(v[0], v[1], v[2], v[3]);
          }
        }
      } else if (l == 1) {
        drain(256u, a.w.off[2], kMlpHidden);
      } else {
        drain(384u, a.w.off[1], kMlpHidden);
      }
    }
  }
  await();
  if (ok) drain(128u, a.w.off[0], kFeatureWidth);
  if (!ok && lane == 0) atomicOr(&g_tcGemmErr, kErrMmaTimeout);
  if (!ok && tid == 0 && commits > 0) waitParity(mbar, (commits - 1) & 1u);  // let a late commit land before the TMEM is freed
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemSlot), "r"(kStepTmemCols) : "memory");
}

}  // namespace

cudaError_t trainTiles(const TrainTiles& a, int tiles, cudaStream_t stream) {
  if (tiles <= 0) return cudaSuccess;
  static bool attrSet = false;
  if (!attrSet) {
    const cudaError_t e = cudaFuncSetAttribute(trainTileKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kStepSmem));
    if (e != cudaSuccess) return e;
    attrSet = true;
  }
  trainTileKernel<<<static_cast<unsigned>(tiles), kStepThreads, kStepSmem, stream>>>(a);
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
