// Learned DXT1 endpoint proposal: a 48 -> 256 (GELU) -> 256 (GELU) -> 8 MLP trained and run on
// the 5th-generation tensor cores (tcgen05.mma, BF16 operands from shared memory, FP32
// accumulators in tensor memory). This part has no counterpart in the reference; it replaces
// the initial guess and most of the refinement of dxt1_endpoint_optimizer (crnlib/crn_dxt1.cpp)
// for blocks where it is good enough, and the exact optimizer stays the fallback and the arbiter of that error.
//
// Inputs: 16 texels x RGB scaled to [0, 1]. Outputs: y[0..5] = low/high endpoint (r/31, g/63,
// b/31) of the plain optimizer's 4-colour solution, y[6] = log2(1 + block error)/16, the
// network's prediction of the error the plain optimizer reaches (the fallback bound); y[7] unused.
//
// Inference (crngpu_mlp_forward, the learned encode) runs as one fused persistent kernel,
// k_mlp_infer: weights resident in shared memory, activations kept on the SM.
// Training runs in three kernels: k_train_tile (per 128 samples: forward, loss gradient and the
// backward products that stay within the samples), k_train_weight_grads (the products over the
// batch, split over it) and k_train_reduce (the slices' sum and, in a training step, AdamW).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>
#include <vector>

#include "crngpu_internal.h"

namespace crngpu {



namespace mlp {

constexpr int kIn = 48, kHid = 256, kOut = 8, kOutPad = 16;
constexpr int BM = 128;
constexpr uint32_t kWaitLimit = 1u << 24;  // bounded mbarrier polls (~ tens of ms), then error

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// byte offset of element (r, k) of a tile with `kt` K-columns in the no-swizzle K-major layout
__device__ __forceinline__ uint32_t kmaj_off(int r, int k, int kt) {
  return (uint32_t)((r >> 3) * ((kt >> 3) * 128) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// tcgen05 shared-memory matrix descriptor: start, leading (K) and stride (8-row) byte offsets,
// descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}

__device__ __forceinline__ float gelu(float x) {
  const float c = 0.7978845608f;  // sqrt(2/pi), tanh form
  return 0.5f * x * (1.f + tanhf(c * (x + 0.044715f * x * x * x)));
}
// gelu(x) and its derivative from one tanh
__device__ __forceinline__ float gelu_both(float x, float& grad) {
  const float c = 0.7978845608f;
  const float t = tanhf(c * (x + 0.044715f * x * x * x));
  grad = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * c * (1.f + 3.f * 0.044715f * x * x);
  return 0.5f * x * (1.f + t);
}

// Polls of a first wait on a tcgen05.commit (a test hook can lower it to force the timeout path);
// after a timeout the in-flight MMAs are drained with kDrainPolls, which the hook does not change,
// so TMEM and shared memory are never released under a running MMA. Timeouts are counted.
constexpr uint32_t kDrainPolls = 1u << 26;
__device__ uint32_t g_mma_wait_polls = kWaitLimit;
__device__ unsigned int g_mma_wait_timeouts;

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t polls) {
  uint32_t done = 0;
  for (uint32_t it = 0; it < polls && !done; it++) {
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity));
  }
  return done != 0;
}

// ------------------------------------------------------------------------------------------
// Fused inference: the whole 48 -> 256 -> 256 -> 16 forward pass of 128 blocks per tile in one
// persistent CTA per SM. All weights stay in shared memory in the K-major core-matrix layout
// (W2 128 KB, W1 24 KB, W3 8 KB); the activations of a tile never leave the SM: input features
// and hidden layers go through one 64 KB shared-memory tile (features alias its first 12 KB),
// accumulators through 256 TMEM columns reused by all three layers. Same arithmetic as the
// training forward (bf16 operands, fp32 accumulation, bias + tanh-GELU in fp32, bf16 hidden).
// The hidden epilogues (65,536 tanh a tile) are what it spends its time on: a thread per row and
// quarter of the columns, as with half of them the eight warps left the schedulers idle half the time
// (87,000 blocks 68 us, now 63 with the texels loaded ahead).
constexpr int kInferThreads = 512;
constexpr int kInferCols = kHid / (kInferThreads / BM);  // hidden columns of a thread
constexpr uint32_t kSmW2 = 0, kSmW1 = kSmW2 + kHid * kHid * 2, kSmW3 = kSmW1 + kHid * kIn * 2,
                   kSmH = kSmW3 + kOutPad * kHid * 2, kSmB1 = kSmH + BM * kHid * 2, kSmB2 = kSmB1 + kHid * 4,
                   kSmB3 = kSmB2 + kHid * 4, kSmBar = kSmB3 + kOutPad * 4, kSmTmem = kSmBar + 8,
                   kInferSmem = kSmTmem + 8;
static_assert(kInferSmem <= 232448, "fused forward exceeds the 227 KB shared-memory limit");

// byte offset of the 16-byte row segment (row r, K-group kg) in a K-major tile with kt K-columns
__device__ __forceinline__ uint32_t kseg(int r, int kg, int kt) {
  return (uint32_t)((r >> 3) * ((kt >> 3) * 128) + kg * 128 + (r & 7) * 16);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
               "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);  // .x = a (low half), .y = b
  return *reinterpret_cast<const uint32_t*>(&h);
}

// hidden-layer epilogue: TMEM accumulators of this thread's row, columns [c_lo, c_lo + kInferCols),
// + bias, GELU, bf16 into the K-major hidden tile
__device__ __forceinline__ void hidden_epilogue(uint32_t tmem, int quarter, int row, int c_lo, const float* bias,
                                                unsigned char* sH) {
#pragma unroll 1
  for (int c0 = c_lo; c0 < c_lo + kInferCols; c0 += 16) {
    uint32_t r[16];
    tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, r);
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float a = gelu(__uint_as_float(r[2 * j]) + bias[c0 + 2 * j]);
      const float b = gelu(__uint_as_float(r[2 * j + 1]) + bias[c0 + 2 * j + 1]);
      w[j] = pack_bf16(a, b);
    }
    *reinterpret_cast<uint4*>(sH + kseg(row, c0 >> 3, kHid)) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(sH + kseg(row, (c0 >> 3) + 1, kHid)) = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// Waits for the tcgen05.commit of this phase; false (uniform across the CTA) on timeout, after a
// second bounded wait so the tensor core is done with shared memory and TMEM before the caller exits.
__device__ __forceinline__ bool tile_wait(uint32_t bar, uint32_t phase) {
  const bool done = mbar_wait(bar, phase, g_mma_wait_polls);
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (__syncthreads_and(done)) return true;
  if (threadIdx.x == 0) atomicAdd(&g_mma_wait_timeouts, 1u);
  mbar_wait(bar, phase, kDrainPolls);
  asm volatile("tcgen05.fence::after_thread_sync;");
  return false;
}

__global__ void __launch_bounds__(kInferThreads, 1)
    k_mlp_infer(const uint8_t* __restrict__ blocks, int n, const __nv_bfloat16* __restrict__ W1,
                const __nv_bfloat16* __restrict__ W2, const __nv_bfloat16* __restrict__ W3,
                const float* __restrict__ b1, const float* __restrict__ b2, const float* __restrict__ b3,
                float* __restrict__ y, uint32_t* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* sW1 = sm + kSmW1;
  unsigned char* sW2 = sm + kSmW2;
  unsigned char* sW3 = sm + kSmW3;
  unsigned char* sH = sm + kSmH;  // features (first 12 KB) / hidden layer of the current tile
  float* sB1 = reinterpret_cast<float*>(sm + kSmB1);
  float* sB2 = reinterpret_cast<float*>(sm + kSmB2);
  float* sB3 = reinterpret_cast<float*>(sm + kSmB3);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kSmBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kSmTmem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // weights (row-major bf16 [rows x K]) -> K-major core matrices, 16 bytes at a time: the 8 rows of a
  // core matrix to neighbouring lanes, as a row's segments lie 128 bytes apart (32 lanes on the same
  // banks took 6.6 us of a launch)
  auto stage = [&](const __nv_bfloat16* w, unsigned char* dst, int rows, int groups) {
    for (int e = tid; e < rows * groups; e += kInferThreads) {
      const int kg = (e >> 3) % groups, r = (e >> 3) / groups * 8 + (e & 7);
      *reinterpret_cast<uint4*>(dst + kseg(r, kg, groups * 8)) =
          __ldg(reinterpret_cast<const uint4*>(w + (r * groups + kg) * 8));
    }
  };
  stage(W2, sW2, kHid, kHid / 8);
  stage(W1, sW1, kHid, kIn / 8);
  stage(W3, sW3, kOutPad, kHid / 8);
  for (int e = tid; e < kHid; e += kInferThreads) { sB1[e] = b1[e]; sB2[e] = b2[e]; }
  if (tid < kOutPad) sB3[tid] = b3[tid];
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)));
  asm volatile("fence.proxy.async.shared::cta;");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  const uint32_t bar = smem_u32(mbar);
  const uint32_t id256 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kHid >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  const uint32_t id16 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kOutPad >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  const uint32_t aH = smem_u32(sH), aW1 = smem_u32(sW1), aW2 = smem_u32(sW2), aW3 = smem_u32(sW3);
  const int quarter = warp & 3, part = warp >> 2;
  const int erow = quarter * 32 + lane;  // the tile row whose accumulators this thread reads
  uint32_t phase = 0;
  bool ok = true;
  const int ntiles = (n + BM - 1) / BM;
  uint4 v0, v1;  // this thread's texels, loaded a tile ahead
  auto load = [&](int tile) {
    const long long row = (long long)tile * BM + (tid & (BM - 1));
    v0 = v1 = make_uint4(0, 0, 0, 0);
    if (tid < 2 * BM && row < n) {
      const uint4* src = reinterpret_cast<const uint4*>(blocks + row * 64 + (tid >> 7) * 32);
      v0 = __ldg(src);
      v1 = __ldg(src + 1);
    }
  };
  load(blockIdx.x);
#pragma unroll 1
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long row0 = (long long)tile * BM;
    if (tid < 2 * BM) {  // features: thread (row, half) converts texels 8*half .. 8*half+7 (24 features, 3 K-groups)
      const int r = tid & (BM - 1), hf = tid >> 7;
      const uint32_t px[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
      float f[24];
#pragma unroll
      for (int t = 0; t < 8; t++)
#pragma unroll
        for (int c = 0; c < 3; c++) f[t * 3 + c] = (float)((px[t] >> (8 * c)) & 255u) * (1.0f / 255.0f);
#pragma unroll
      for (int g = 0; g < 3; g++)
        *reinterpret_cast<uint4*>(sH + kseg(r, hf * 3 + g, kIn)) =
            make_uint4(pack_bf16(f[g * 8], f[g * 8 + 1]), pack_bf16(f[g * 8 + 2], f[g * 8 + 3]),
                       pack_bf16(f[g * 8 + 4], f[g * 8 + 5]), pack_bf16(f[g * 8 + 6], f[g * 8 + 7]));
    }
    asm volatile("fence.proxy.async.shared::cta;");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0) {  // layer 1: [128 x 48] x [48 x 256]
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int ks = 0; ks < kIn / 16; ks++)
        mma_bf16(tmem, make_desc(aH + ks * 256, 128, (kIn / 8) * 128), make_desc(aW1 + ks * 256, 128, (kIn / 8) * 128),
                 id256, ks > 0);
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar));
    }
    load(min(tile + (int)gridDim.x, ntiles));  // at ntiles every row is past n: nothing is read
    if (!(ok = tile_wait(bar, phase))) break;
    phase ^= 1;
    hidden_epilogue(tmem, quarter, erow, part * kInferCols, sB1, sH);
    asm volatile("fence.proxy.async.shared::cta;");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0) {  // layer 2: [128 x 256] x [256 x 256]
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int ks = 0; ks < kHid / 16; ks++)
        mma_bf16(tmem, make_desc(aH + ks * 256, 128, (kHid / 8) * 128), make_desc(aW2 + ks * 256, 128, (kHid / 8) * 128),
                 id256, ks > 0);
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar));
    }
    if (!(ok = tile_wait(bar, phase))) break;
    phase ^= 1;
    hidden_epilogue(tmem, quarter, erow, part * kInferCols, sB2, sH);
    asm volatile("fence.proxy.async.shared::cta;");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0) {  // layer 3: [128 x 256] x [256 x 16]
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int ks = 0; ks < kHid / 16; ks++)
        mma_bf16(tmem, make_desc(aH + ks * 256, 128, (kHid / 8) * 128), make_desc(aW3 + ks * 256, 128, (kHid / 8) * 128),
                 id16, ks > 0);
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar));
    }
    if (!(ok = tile_wait(bar, phase))) break;
    phase ^= 1;
    if (part == 0) {
      uint32_t r[16];
      tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16), r);
      if (row0 + erow < n) {
        float4* dst = reinterpret_cast<float4*>(y + (row0 + erow) * kOutPad);
#pragma unroll
        for (int q = 0; q < 4; q++)
          dst[q] = make_float4(__uint_as_float(r[4 * q]) + sB3[4 * q], __uint_as_float(r[4 * q + 1]) + sB3[4 * q + 1],
                               __uint_as_float(r[4 * q + 2]) + sB3[4 * q + 2],
                               __uint_as_float(r[4 * q + 3]) + sB3[4 * q + 3]);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();  // TMEM columns and the feature tile are reused by the next tile
  }
  if (!ok && tid == 0) atomicExch(err, 1u);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem));
}

// ------------------------------------------------------------------------------------------
// Training. Everything a sample's forward and backward pass needs of other samples is the weight
// gradients, so a tile of 128 samples runs through all layers, forward and back, in one CTA
// (k_train_tile), its activations in shared and tensor memory; what the weight gradients need of
// it (both hidden layers, their gradients, the features and output gradients, BF16) is written
// transposed, [feature][sample], in the K-major core-matrix layout those products stage as is. The
// weight gradients' K is the batch: k_train_weight_grads gives a run of tiles to each of about 128
// CTAs, k_train_reduce adds the runs' partial sums in a fixed order and applies AdamW. Bias
// gradients and the loss are summed in FP32 per 32 samples with warp shuffles, then in a fixed
// order. A step is bound by the latency of its serial parts (six dependent MMAs and four epilogues
// of 32,768 tanh or products each per tile), not by its 4 GFLOP. A step of batch 8192 with separate
// GEMMs, one thread per column for the bias sums and an AdamW launch per parameter took 1.39 ms.
constexpr int kTrainThreads = 512;
constexpr int kGradCols = kHid + kIn + kOutPad;             // dW2 | dW1 | dW3^T columns of a partial sum
constexpr int kBiasSums = 2 * kHid + kOutPad + 1;           // db1, db2, db3, loss
constexpr uint32_t kTileT = kHid * BM * 2, kTileX = kIn * BM * 2, kTileDy = kOutPad * BM * 2;

// k_train_tile's shared memory. W2's place takes W2^T for the backward product; W1's, once layer 1
// is done, the warps' transposing buffers and W3^T; H is features, h1, h2, dY and dpre2 in turn.
constexpr uint32_t kTrW2 = 0, kTrH = kTrW2 + kHid * kHid * 2, kTrW1 = kTrH + BM * kHid * 2, kTrBuf = kTrW1,
                   kTrW3T = kTrBuf + (kTrainThreads / 32) * 1024, kTrW3 = kTrW1 + kHid * kIn * 2,
                   kTrB1 = kTrW3 + kOutPad * kHid * 2, kTrB2 = kTrB1 + kHid * 4, kTrB3 = kTrB2 + kHid * 4,
                   kTrBar = kTrB3 + kOutPad * 4, kTrTmem = kTrBar + 8, kTrainSmem = kTrTmem + 8;
static_assert(kTrW3T + kHid * kOutPad * 2 <= kTrW3, "transposing buffers and W3^T fit in W1's place");
static_assert(kTrainSmem <= 232448, "k_train_tile exceeds the 227 KB shared-memory limit");

struct TrainArgs {
  const uint8_t* blocks;
  const float* targets;
  int n, tiles;
  float tau, bw;
  const __nv_bfloat16 *W1, *W2, *W2T, *W3, *W3T;
  const float *b1, *b2, *b3;
  unsigned char *h1T, *h2T, *d1T, *d2T, *xT, *dyT;  // per tile: [feature][128 samples] core-matrix tiles
  float *g1, *g2;                                   // per tile: gelu' of both layers, [feature][128 samples]
  float* bias;                                      // [kBiasSums][4 * tiles]: sums of 32 samples
  float* part;                                      // [slices][kGradCols][kHid] partial weight gradients
  int slices, slice_tiles;
  uint32_t* err;
};

__device__ __forceinline__ void async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}

// row-major BF16 [rows x kt] -> K-major core matrices at dst
__device__ __forceinline__ void async_weights(uint32_t dst, const __nv_bfloat16* w, int rows, int kt) {
  const int segs = kt >> 3;
  for (int e = threadIdx.x; e < rows * segs; e += kTrainThreads) {
    const int r = e / segs, kg = e - r * segs;
    async16(dst + kseg(r, kg, kt), w + (size_t)r * kt + kg * 8);
  }
}

// 16 features (first c0) of this warp's 32 samples (`quarter` of the tile), BF16, into the
// [feature][sample] tile: through the warp's 1 KB buffer, then 16 bytes (8 samples) a lane
__device__ __forceinline__ void store_transposed(unsigned char* buf, unsigned char* tile, int quarter, int c0,
                                                 const uint32_t* packed) {
  const int lane = threadIdx.x & 31;
  uint16_t* b16 = reinterpret_cast<uint16_t*>(buf);
#pragma unroll
  for (int j = 0; j < 8; j++) {
    b16[(2 * j) * 32 + lane] = (uint16_t)packed[j];
    b16[(2 * j + 1) * 32 + lane] = (uint16_t)(packed[j] >> 16);
  }
  __syncwarp();
#pragma unroll
  for (int u = lane; u < 64; u += 32) {
    const int c = c0 + (u >> 2), sg = quarter * 4 + (u & 3);
    *reinterpret_cast<uint4*>(tile + (c >> 3) * (BM / 8 * 128) + sg * 128 + (c & 7) * 16) =
        *reinterpret_cast<const uint4*>(buf + u * 16);
  }
  __syncwarp();
}

// sums of v[0..15] over the warp's lanes: lane 2c (and 2c + 1) returns column c's
__device__ __forceinline__ float column_sums(float (&v)[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int half = 8; half > 0; half >>= 1) {
    const bool up = (lane & (2 * half)) != 0;
#pragma unroll
    for (int j = 0; j < half; j++) {
      const float give = up ? v[j] : v[j + half], keep = up ? v[j + half] : v[j];
      v[j] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, 2 * half);
    }
  }
  return v[0] + __shfl_xor_sync(0xFFFFFFFFu, v[0], 1);
}

__global__ void __launch_bounds__(kTrainThreads, 1) k_train_tile(TrainArgs a) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* sH = sm + kTrH;
  float* sB1 = reinterpret_cast<float*>(sm + kTrB1);
  float* sB2 = reinterpret_cast<float*>(sm + kTrB2);
  float* sB3 = reinterpret_cast<float*>(sm + kTrB3);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kTrTmem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, cg = warp >> 2, row = quarter * 32 + lane;  // TMEM lane = tile row; 64 columns
  const int tile = blockIdx.x;
  const long long row0 = (long long)tile * BM;
  unsigned char* buf = sm + kTrBuf + warp * 1024;
  const uint32_t base = smem_u32(sm), bar = base + kTrBar;
  async_weights(base + kTrW1, a.W1, kHid, kIn);
  asm volatile("cp.async.commit_group;");
  async_weights(base + kTrW2, a.W2, kHid, kHid);
  async_weights(base + kTrW3, a.W3, kOutPad, kHid);
  asm volatile("cp.async.commit_group;");
  if (tid < kHid) { sB1[tid] = a.b1[tid]; sB2[tid] = a.b2[tid]; }
  if (tid < kOutPad) sB3[tid] = a.b3[tid];
  if (tid < 2 * BM) {  // features: texels 8 * hf .. + 7 of a sample, and their transposed copy
    const int r = tid & (BM - 1), hf = tid >> 7;
    uint32_t px[8] = {};
    if (row0 + r < a.n) {
      const uint8_t* src = a.blocks + (row0 + r) * 64 + hf * 32;
      if (((uintptr_t)a.blocks & 15) == 0) {
        const uint4 v0 = __ldg(reinterpret_cast<const uint4*>(src)), v1 = __ldg(reinterpret_cast<const uint4*>(src) + 1);
        px[0] = v0.x; px[1] = v0.y; px[2] = v0.z; px[3] = v0.w;
        px[4] = v1.x; px[5] = v1.y; px[6] = v1.z; px[7] = v1.w;
      } else {
#pragma unroll
        for (int t = 0; t < 8; t++) px[t] = (uint32_t)__ldg(src + 4 * t) | (uint32_t)__ldg(src + 4 * t + 1) << 8 | (uint32_t)__ldg(src + 4 * t + 2) << 16;
      }
    }
    uint32_t f[12];
#pragma unroll
    for (int k = 0; k < 12; k++) {
      const int i = 2 * k, j = 2 * k + 1;
      f[k] = pack_bf16((float)((px[i / 3] >> (8 * (i % 3))) & 255u) * (1.0f / 255.0f),
                       (float)((px[j / 3] >> (8 * (j % 3))) & 255u) * (1.0f / 255.0f));
    }
    unsigned char* xt = a.xT + (size_t)tile * kTileX;
#pragma unroll
    for (int k = 0; k < 12; k++) {
      *reinterpret_cast<uint16_t*>(xt + kmaj_off(hf * 24 + 2 * k, r, BM)) = (uint16_t)f[k];
      *reinterpret_cast<uint16_t*>(xt + kmaj_off(hf * 24 + 2 * k + 1, r, BM)) = (uint16_t)(f[k] >> 16);
    }
#pragma unroll
    for (int g = 0; g < 3; g++)
      *reinterpret_cast<uint4*>(sH + kseg(r, hf * 3 + g, kIn)) = make_uint4(f[4 * g], f[4 * g + 1], f[4 * g + 2], f[4 * g + 3]);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
  asm volatile("cp.async.wait_group 1;");
  const uint32_t id256 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kHid >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  const uint32_t id16 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kOutPad >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  auto to_mma = [&]() {  // shared-memory writes and TMEM reads of all threads before the next product
    asm volatile("fence.proxy.async.shared::cta;");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
  };
  to_mma();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  uint32_t phase = 0;
  // TMEM columns 0.. = A [128 x kt] x B [N x kt]^T, both K-major in shared memory; false on a timeout
  auto product = [&](uint32_t at, uint32_t bt, int kt, uint32_t idesc) {
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t sbo = (uint32_t)(kt >> 3) * 128;
      for (int ks = 0; ks < kt / 16; ks++)
        mma_bf16(tmem, make_desc(base + at + ks * 256, 128, sbo), make_desc(base + bt + ks * 256, 128, sbo), idesc, ks > 0);
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar));
    }
    const bool ok = tile_wait(bar, phase);
    phase ^= 1;
    return ok;
  };
  const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
  auto hidden = [&](const float* bias, float* grad, unsigned char* hT) {
#pragma unroll 1
    for (int c0 = cg * 64; c0 < cg * 64 + 64; c0 += 16) {
      uint32_t r[16], w[8];
      tmem_ld16(taddr + (uint32_t)c0, r);
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        float ga, gb;
        const float x = gelu_both(__uint_as_float(r[j]) + bias[c0 + j], ga);
        const float y = gelu_both(__uint_as_float(r[j + 1]) + bias[c0 + j + 1], gb);
        w[j / 2] = pack_bf16(x, y);
        grad[(c0 + j) * BM + row] = ga;  // read back by this thread alone
        grad[(c0 + j + 1) * BM + row] = gb;
      }
      *reinterpret_cast<uint4*>(sH + kseg(row, c0 >> 3, kHid)) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(sH + kseg(row, (c0 >> 3) + 1, kHid)) = make_uint4(w[4], w[5], w[6], w[7]);
      store_transposed(buf, hT, quarter, c0, w);
    }
  };
  auto back = [&](const float* grad, unsigned char* dT, float* bias, bool keep) {
#pragma unroll 1
    for (int c0 = cg * 64; c0 < cg * 64 + 64; c0 += 16) {
      uint32_t r[16], w[8];
      float v[16];
      tmem_ld16(taddr + (uint32_t)c0, r);
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]) * grad[(c0 + j) * BM + row];
#pragma unroll
      for (int j = 0; j < 8; j++) w[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
      if (keep) {
        *reinterpret_cast<uint4*>(sH + kseg(row, c0 >> 3, kHid)) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(sH + kseg(row, (c0 >> 3) + 1, kHid)) = make_uint4(w[4], w[5], w[6], w[7]);
      }
      store_transposed(buf, dT, quarter, c0, w);
      const float s = column_sums(v);
      if (!(lane & 1)) bias[(size_t)(c0 + (lane >> 1)) * 4 * a.tiles] = s;
    }
  };
  float* g1 = a.g1 + (size_t)tile * kHid * BM;
  float* g2 = a.g2 + (size_t)tile * kHid * BM;
  float* bias = a.bias + (size_t)tile * 4 + quarter;
  const size_t bias_row = (size_t)4 * a.tiles;
  bool ok;
  do {
    if (!(ok = product(kTrH, kTrW1, kIn, id256))) break;
    async_weights(base + kTrW3T, a.W3T, kHid, kOutPad);  // into W1's place
    asm volatile("cp.async.commit_group;");
    hidden(sB1, g1, a.h1T + (size_t)tile * kTileT);
    asm volatile("cp.async.wait_group 0;");
    to_mma();
    if (!(ok = product(kTrH, kTrW2, kHid, id256))) break;
    async_weights(base + kTrW2, a.W2T, kHid, kHid);  // into W2's place
    asm volatile("cp.async.commit_group;");
    hidden(sB2, g2, a.h2T + (size_t)tile * kTileT);
    to_mma();
    if (!(ok = product(kTrH, kTrW3, kHid, id16))) break;
    if (cg == 0) {
      // Loss gradient. Outputs 0..5 (endpoints): squared error, dY = 2 (y - t) / B. Output 6 (the
      // error bound): squared error when tau <= 0; otherwise the quantile (pinball) loss
      // bw * max(tau (t - y), (1 - tau) (y - t)), whose minimiser is the tau-quantile of the plain
      // optimizer's error given the block, i.e. an upper bound that holds for a fraction tau of blocks.
      uint32_t r[16], w[8];
      float v[16], loss = 0.f;
      tmem_ld16(taddr, r);
#pragma unroll
      for (int c = 0; c < 16; c++) v[c] = 0.f;
      if (row0 + row < a.n) {
        const float* t = a.targets + (row0 + row) * kOut;
#pragma unroll
        for (int c = 0; c < 7; c++) {
          const float d = __uint_as_float(r[c]) + sB3[c] - __ldg(t + c);
          if (c == 6 && a.tau > 0.f) {
            loss += a.bw * (d > 0.f ? (1.f - a.tau) * d : -a.tau * d);
            v[c] = a.bw * (d > 0.f ? (1.f - a.tau) : -a.tau) / (float)a.n;
          } else {
            loss += d * d;
            v[c] = 2.f * d / (float)a.n;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 8; j++) w[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
      *reinterpret_cast<uint4*>(sH + kseg(row, 0, kOutPad)) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(sH + kseg(row, 1, kOutPad)) = make_uint4(w[4], w[5], w[6], w[7]);
      store_transposed(buf, a.dyT + (size_t)tile * kTileDy, quarter, 0, w);
      const float s = column_sums(v);
      if (!(lane & 1)) bias[(2 * kHid + (lane >> 1)) * bias_row] = s;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o);
      if (lane == 0) bias[(2 * kHid + kOutPad) * bias_row] = loss / (float)a.n;
    }
    to_mma();
    if (!(ok = product(kTrH, kTrW3T, kOutPad, id256))) break;  // dY W3
    back(g2, a.d2T + (size_t)tile * kTileT, bias + kHid * bias_row, true);
    asm volatile("cp.async.wait_group 0;");
    to_mma();
    if (!(ok = product(kTrH, kTrW2, kHid, id256))) break;  // dpre2 W2
    back(g1, a.d1T + (size_t)tile * kTileT, bias, false);
  } while (false);
  if (!ok && tid == 0) atomicExch(a.err, 1u);
  asm volatile("cp.async.wait_group 0;");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem));
}

// blockIdx.x: half of the 256 rows, blockIdx.y: slice of the tiles. Rows [128 half, + 128) of
// dW2 = dpre2^T h1, dW1 = dpre1^T X and dW3^T = h2^T dY over the slice, accumulated in TMEM (columns
// 0.., 256.., 304..), written column by column ([kGradCols][kHid]: 32 rows a warp store).
constexpr uint32_t kWgD2 = 0, kWgH1 = kWgD2 + kTileT / 2, kWgD1 = kWgH1 + kTileT, kWgX = kWgD1 + kTileT / 2,
                   kWgH2 = kWgX + kTileX, kWgDy = kWgH2 + kTileT / 2, kWgBar = kWgDy + kTileDy, kWgTmem = kWgBar + 8,
                   kWgSmem = kWgTmem + 8;
static_assert(kWgSmem <= 232448, "k_train_weight_grads exceeds the 227 KB shared-memory limit");

__global__ void __launch_bounds__(kTrainThreads, 1) k_train_weight_grads(TrainArgs a) {
  extern __shared__ __align__(1024) unsigned char sm[];
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kWgTmem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = smem_u32(sm), bar = base + kWgBar, half = blockIdx.x;
  const int t0 = blockIdx.y * a.slice_tiles, t1 = min(a.tiles, t0 + a.slice_tiles);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  uint32_t phase = 0;
  bool ok = true;
  auto copy = [&](uint32_t dst, const unsigned char* src, uint32_t bytes) {
    for (uint32_t e = tid * 16; e < bytes; e += kTrainThreads * 16) async16(base + dst + e, src + e);
  };
  for (int t = t0; t < t1; t++) {
    const size_t at = (size_t)t * kTileT + half * (kTileT / 2);
    copy(kWgD2, a.d2T + at, kTileT / 2);
    copy(kWgH1, a.h1T + (size_t)t * kTileT, kTileT);
    copy(kWgD1, a.d1T + at, kTileT / 2);
    copy(kWgX, a.xT + (size_t)t * kTileX, kTileX);
    copy(kWgH2, a.h2T + at, kTileT / 2);
    copy(kWgDy, a.dyT + (size_t)t * kTileDy, kTileDy);
    asm volatile("cp.async.commit_group;");
    asm volatile("cp.async.wait_group 0;");
    asm volatile("fence.proxy.async.shared::cta;");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      auto idesc = [](int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24); };
      constexpr uint32_t sbo = BM / 8 * 128;
#pragma unroll
      for (int ks = 0; ks < BM / 16; ks++) {
        const uint32_t acc = t > t0 || ks > 0;
        auto desc = [&](uint32_t o) { return make_desc(base + o + ks * 256, 128, sbo); };
        mma_bf16(tmem, desc(kWgD2), desc(kWgH1), idesc(kHid), acc);
        mma_bf16(tmem + kHid, desc(kWgD1), desc(kWgX), idesc(kIn), acc);
        mma_bf16(tmem + kHid + kIn, desc(kWgH2), desc(kWgDy), idesc(kOutPad), acc);
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar));
    }
    if (!(ok = tile_wait(bar, phase))) break;
    phase ^= 1;
  }
  if (!ok) {
    if (tid == 0) atomicExch(a.err, 1u);
  } else {
    const int quarter = warp & 3, cg = warp >> 2;
    float* dst = a.part + (size_t)blockIdx.y * kGradCols * kHid + half * BM + quarter * 32 + lane;
#pragma unroll 1
    for (int c0 = cg * (kGradCols / 4); c0 < (cg + 1) * (kGradCols / 4); c0 += 16) {
      uint32_t r[16];
      tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, r);
#pragma unroll
      for (int j = 0; j < 16; j++) dst[(size_t)(c0 + j) * kHid] = __uint_as_float(r[j]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// A parameter's buffers: FP32 gradient, weights and Adam moments, BF16 copy and transposed copy.
struct ParamPtrs {
  float *g, *w, *m, *v;
  __nv_bfloat16 *wb, *wbT;
};
struct ReduceArgs {
  const float *part, *bias;
  int slices, bias_sums;
  ParamPtrs W1, b1, W2, b2, W3, b3;
  float* loss;
  const uint32_t* err;
  int update;  // AdamW after the gradients
  float lr, beta1, beta2, eps, wd, bc1, bc2;
};

// AdamW on the FP32 master weight; returns it
__device__ __forceinline__ float adamw(const ReduceArgs& a, const ParamPtrs& p, size_t i, float gi, float wd) {
  const float mi = a.beta1 * p.m[i] + (1.f - a.beta1) * gi;
  const float vi = a.beta2 * p.v[i] + (1.f - a.beta2) * gi * gi;
  p.m[i] = mi;
  p.v[i] = vi;
  float wi = p.w[i] * (1.f - a.lr * wd);
  wi -= a.lr * (mi / a.bc1) / (sqrtf(vi / a.bc2) + a.eps);
  p.w[i] = wi;
  return wi;
}

// Blocks 0..79: a 32 x 32 tile of the weight gradients ([kGradCols][kHid] partial sums, added slice
// after slice); the others: one bias gradient (or the loss) per warp. After a timed-out wait (err)
// nothing is written.
constexpr int kReduceTiles = (kHid / 32) * (kGradCols / 32), kReduceBlocks = kReduceTiles + (kBiasSums + 31) / 32;
static_assert(kGradCols % 32 == 0 && (kHid + kIn) % 32 == 16, "the last column tile is half W1, half W3");

__global__ void __launch_bounds__(1024) k_train_reduce(ReduceArgs a) {
  if (*a.err) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (blockIdx.x >= kReduceTiles) {
    const int o = (blockIdx.x - kReduceTiles) * 32 + warp;
    if (o >= kBiasSums) return;
    const float* src = a.bias + (size_t)o * a.bias_sums;
    float s = 0.f;
    for (int k = lane; k < a.bias_sums; k += 32) s += src[k];
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, k);
    if (lane) return;
    if (o == 2 * kHid + kOutPad) { *a.loss = s; return; }
    const ParamPtrs& p = o < kHid ? a.b1 : o < 2 * kHid ? a.b2 : a.b3;
    const int i = o < kHid ? o : o < 2 * kHid ? o - kHid : o - 2 * kHid;
    p.g[i] = s;
    if (a.update) adamw(a, p, i, s, 0.f);
    return;
  }
  __shared__ float t[32][33];
  const int r0 = (blockIdx.x % (kHid / 32)) * 32, c0 = (blockIdx.x / (kHid / 32)) * 32;
  {
    const float* src = a.part + (size_t)(c0 + warp) * kHid + r0 + lane;
    float s = 0.f;
#pragma unroll 8
    for (int z = 0; z < a.slices; z++) s += src[(size_t)z * kGradCols * kHid];
    const int o = c0 + warp - kHid - kIn;
    if (o >= 0) {  // W3 [16 x 256]: rows 7.. stay zero
      const size_t i = (size_t)o * kHid + r0 + lane;
      a.W3.g[i] = s;
      if (a.update) {
        float w = 0.f;
        if (o < 7) w = adamw(a, a.W3, i, s, a.wd); else a.W3.w[i] = 0.f;
        a.W3.wb[i] = __float2bfloat16(w);
        a.W3.wbT[(size_t)(r0 + lane) * kOutPad + o] = __float2bfloat16(w);
      }
    }
    t[warp][lane] = s;
  }
  __syncthreads();
  const int row = r0 + warp, col = c0 + lane;
  if (col >= kHid + kIn) return;
  const ParamPtrs& p = col < kHid ? a.W2 : a.W1;
  const size_t i = col < kHid ? (size_t)row * kHid + col : (size_t)row * kIn + col - kHid;
  const float s = t[lane][warp];
  p.g[i] = s;
  if (!a.update) return;
  const __nv_bfloat16 w = __float2bfloat16(adamw(a, p, i, s, a.wd));
  p.wb[i] = w;
  if (col < kHid) p.wbT[(size_t)col * kHid + row] = w;
}

// Training targets from the plain optimizer's blocks: endpoints of the 4-colour solution in
// [0, 1] units, and log2(1 + error) / 16.
__global__ void k_make_targets(const uint8_t* __restrict__ blocks8, const uint64_t* __restrict__ err, int n,
                               float* __restrict__ t) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint8_t* b = blocks8 + (long long)i * 8;
    uint32_t lo = b[0] | (b[1] << 8), hi = b[2] | (b[3] << 8);
    if (lo <= hi) { const uint32_t x = lo; lo = hi; hi = x; }  // 3-colour blocks: order as 4-colour
    float* o = t + (long long)i * kOut;
    o[0] = (float)(lo >> 11) / 31.f; o[1] = (float)((lo >> 5) & 63) / 63.f; o[2] = (float)(lo & 31) / 31.f;
    o[3] = (float)(hi >> 11) / 31.f; o[4] = (float)((hi >> 5) & 63) / 63.f; o[5] = (float)(hi & 31) / 31.f;
    o[6] = log2f(1.f + (float)err[i]) / 16.f;
    o[7] = 0.f;
  }
}

// Learned encode, per block: quantise the predicted endpoints, choose selectors, refit the
// endpoints by least squares from those selectors (refine_solution level 0,
// crnlib/crn_dxt1.cpp:525-600), polish with a short greedy search of +-1 steps on the six
// endpoint components, check the 3-colour block on the same endpoints, and keep the block unless
// its error is above `threshold` x the network's predicted bound; those blocks are queued for the
// exact optimizer.
__device__ __forceinline__ int q565(float v, int hi) {
  int x = __float2int_rn(v * (float)hi);
  return x < 0 ? 0 : (x > hi ? hi : x);
}
// Packed FP32 (sm_100 and later): two colours of a block at a time.
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpair(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
// A block in registers: the colours in pairs, as floats, and the sum of their weighted squares.
struct RefitBlock {
  uint64_t r[8], g[8], b[8];
  float wr, wg;
  uint32_t squares;
};
// A palette entry p as the distance of a colour x less |x|^2 is evaluated: -2 w p and w p^2 + kOffset,
// which keeps the whole of it between 2^23 and 2^24 (w p^2 - 2 w p x is between -34 * 255^2 and
// 34 * 255^2): an integer in the low mantissa bits, every step exact.
constexpr float kOffset = 13000000.f, kNoEntry = 16000000.f;
struct RefitEntry {
  float r, g, b, c;
  __device__ __forceinline__ void set(const RefitBlock& B, float pr, float pg, float pb) {
    r = -2.f * B.wr * pr; g = -2.f * B.wg * pg; b = -2.f * pb;
    c = fmaf(B.wr * pr, pr, fmaf(B.wg * pg, pg, fmaf(pb, pb, kOffset)));
  }
};
__device__ __forceinline__ void refit_palette(const RefitBlock& B, uint32_t lo, uint32_t hi, bool three, RefitEntry (&q)[4]) {
  auto e5 = [](uint32_t v) { return (int)((v << 3) | (v >> 2)); };
  auto e6 = [](uint32_t v) { return (int)((v << 2) | (v >> 4)); };
  const int a[3] = {e5(lo >> 11), e6((lo >> 5) & 63u), e5(lo & 31u)}, c[3] = {e5(hi >> 11), e6((hi >> 5) & 63u), e5(hi & 31u)};
  q[0].set(B, (float)a[0], (float)a[1], (float)a[2]);
  q[1].set(B, (float)c[0], (float)c[1], (float)c[2]);
  if (three) {
    q[2].set(B, (float)((a[0] + c[0]) >> 1), (float)((a[1] + c[1]) >> 1), (float)((a[2] + c[2]) >> 1));
    q[3].r = q[3].g = q[3].b = 0.f;
    q[3].c = kNoEntry;
  } else {
    q[2].set(B, (float)((a[0] * 2 + c[0]) / 3), (float)((a[1] * 2 + c[1]) / 3), (float)((a[2] * 2 + c[2]) / 3));
    q[3].set(B, (float)((c[0] * 2 + a[0]) / 3), (float)((c[1] * 2 + a[1]) / 3), (float)((c[2] * 2 + a[2]) / 3));
  }
}
// Error of the 4-colour (three = false) or 3-colour palette of (lo, hi), and with `selectors` the
// selectors in 2-bit slots (the first of equally near entries).
template <bool selectors>
__device__ __forceinline__ uint32_t block_error(const RefitBlock& B, uint32_t lo, uint32_t hi, bool three, uint32_t* sel_out) {
  RefitEntry q[4];
  refit_palette(B, lo, hi, three, q);
  uint64_t qr[4], qg[4], qb[4], qc[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    qr[k] = pair(q[k].r, q[k].r); qg[k] = pair(q[k].g, q[k].g);
    qb[k] = pair(q[k].b, q[k].b); qc[k] = pair(q[k].c, q[k].c);
  }
  uint32_t sum = 0, sel = 0;
#pragma unroll
  for (int p = 0; p < 8; p++) {
    float d[2][4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      unpair(fma_pair(B.r[p], qr[k], fma_pair(B.g[p], qg[k], fma_pair(B.b[p], qb[k], qc[k]))), d[0][k], d[1][k]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const float m = fminf(fminf(d[h][0], d[h][1]), fminf(d[h][2], d[h][3]));
      sum += __float_as_uint(m);
      if (selectors) {
        const uint32_t k = m == d[h][0] ? 0u : m == d[h][1] ? 1u : m == d[h][2] ? 2u : 3u;
        sel |= k << (4 * p + 2 * h);
      }
    }
  }
  if (selectors) *sel_out = sel;
  // a distance's bits are those of 2^23 plus (distance + kOffset - 2^23)
  return sum - 16u * (0x4B000000u + (uint32_t)(kOffset - 8388608.f)) + B.squares;
}

// One thread per block: the error of 14 to 38 endpoint pairs over 16 colours and four entries is what
// it does, in exact packed floats (3 multiply-adds for two colours and an entry, a minimum, an integer
// add), with selectors only where they are used. In integer arithmetic with selectors for every pair
// the proposals of 87,000 blocks took 116 us, now 52.
// y holds the proposals of blocks base .. base + n - 1; indices written to `fallback` are batch-wide
__global__ void k_learned_refit(const uint8_t* __restrict__ blocks, const float* __restrict__ y, uint32_t base, int n,
                                int perceptual, uint8_t* __restrict__ out, uint32_t* __restrict__ fallback,
                                uint32_t* __restrict__ nfall, float threshold) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const long long i = (long long)base + j;
    RefitBlock B;
    B.wr = perceptual ? 8.f : 1.f;
    B.wg = perceptual ? 25.f : 1.f;
    B.squares = 0;
    const uint4* p4 = reinterpret_cast<const uint4*>(blocks + i * 64);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint4 v = __ldg(p4 + q);
      const uint32_t px[4] = {v.x, v.y, v.z, v.w};
      float x[4][3];
#pragma unroll
      for (int t = 0; t < 4; t++) {
#pragma unroll
        for (int k = 0; k < 3; k++) x[t][k] = (float)((px[t] >> (8 * k)) & 255u);
        B.squares += (uint32_t)fmaf(B.wr * x[t][0], x[t][0], fmaf(B.wg * x[t][1], x[t][1], x[t][2] * x[t][2]));
      }
#pragma unroll
      for (int t = 0; t < 2; t++) {
        B.r[2 * q + t] = pair(x[2 * t][0], x[2 * t + 1][0]);
        B.g[2 * q + t] = pair(x[2 * t][1], x[2 * t + 1][1]);
        B.b[2 * q + t] = pair(x[2 * t][2], x[2 * t + 1][2]);
      }
    }
    const float* yi = y + (long long)j * kOutPad;
    auto pk = [](int r, int g, int b) { return (uint32_t)((r << 11) | (g << 5) | b); };
    uint32_t lo = pk(q565(yi[0], 31), q565(yi[1], 63), q565(yi[2], 31));
    uint32_t hi = pk(q565(yi[3], 31), q565(yi[4], 63), q565(yi[5], 31));
    uint32_t sel;
    uint32_t err = block_error<true>(B, lo, hi, false, &sel);
    // least-squares refit from the selectors (points at 1, 0, 2/3, 1/3 of the low endpoint)
    {
      float aa = 0.f, ab = 0.f, bb = 0.f, ax[3] = {0, 0, 0}, bx[3] = {0, 0, 0};
#pragma unroll
      for (int p = 0; p < 16; p++) {
        const uint32_t k = (sel >> (2 * p)) & 3u;
        const float a = k == 0 ? 1.f : k == 1 ? 0.f : k == 2 ? 2.f / 3.f : 1.f / 3.f, b = 1.f - a;
        aa += a * a; ab += a * b; bb += b * b;
        float x[3], other;
        if (p & 1) { unpair(B.r[p / 2], other, x[0]); unpair(B.g[p / 2], other, x[1]); unpair(B.b[p / 2], other, x[2]); }
        else { unpair(B.r[p / 2], x[0], other); unpair(B.g[p / 2], x[1], other); unpair(B.b[p / 2], x[2], other); }
#pragma unroll
        for (int k3 = 0; k3 < 3; k3++) { ax[k3] += a * x[k3]; bx[k3] += b * x[k3]; }
      }
      const float det = aa * bb - ab * ab;
      if (fabsf(det) > 1e-6f) {
        const float inv = 1.f / det;
        int f[6];
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const int lim = k == 1 ? 63 : 31;
          f[k] = q565((ax[k] * bb - bx[k] * ab) * inv / 255.f, lim);
          f[3 + k] = q565((bx[k] * aa - ax[k] * ab) * inv / 255.f, lim);
        }
        const uint32_t flo = pk(f[0], f[1], f[2]), fhi = pk(f[3], f[4], f[5]);
        const uint32_t nerr = block_error<false>(B, flo, fhi, false, nullptr);
        if (nerr < err) { err = nerr; lo = flo; hi = fhi; }
      }
    }
    // greedy polish: up to three rounds of the best single +-1 move over the six components
#pragma unroll 1
    for (int round = 0; round < 3; round++) {
      uint32_t best_err = err, best_lo = lo, best_hi = hi;
#pragma unroll 1
      for (int t = 0; t < 12; t++) {
        const int k = t >> 1, c = k % 3, shift = c == 0 ? 11 : c == 1 ? 5 : 0;
        const uint32_t field = (c == 1 ? 63u : 31u) << shift, from = k < 3 ? lo : hi;
        if ((from & field) == (t & 1 ? field : 0u)) continue;  // at the component's end
        const uint32_t to = t & 1 ? from + (1u << shift) : from - (1u << shift);
        const uint32_t nlo = k < 3 ? to : lo, nhi = k < 3 ? hi : to;
        const uint32_t nerr = block_error<false>(B, nlo, nhi, false, nullptr);
        if (nerr < best_err) { best_err = nerr; best_lo = nlo; best_hi = nhi; }
      }
      if (best_err == err) break;
      err = best_err;
      lo = best_lo;
      hi = best_hi;
    }
    // 4-colour blocks need low > high; equal endpoints are nudged apart as the reference does
    // (crnlib/crn_dxt1.cpp:1563-1583). The selectors are those of the order that was searched: with
    // the endpoints swapped, 0 <-> 1 and 2 <-> 3
    err = block_error<true>(B, lo, hi, false, &sel);
    if (lo < hi) {
      const uint32_t t = lo; lo = hi; hi = t;
      sel ^= 0x55555555u;
    } else if (lo == hi) {
      if ((lo & 31) != 31) lo++; else hi--;
      err = block_error<true>(B, lo, hi, false, &sel);
    }
    // the 3-colour block on the same endpoints (low <= high, mid-point palette)
    {
      const uint32_t err3 = block_error<false>(B, hi, lo, true, nullptr);
      if (err3 < err) {
        err = err3;
        block_error<true>(B, hi, lo, true, &sel);
        const uint32_t t = lo; lo = hi; hi = t;
      }
    }
    const float bound = exp2f(yi[6] * 16.f) - 1.f;
    *reinterpret_cast<uint2*>(out + i * 8) = make_uint2(lo | (hi << 16), sel);
    if (!(threshold > 0.f) || (float)err > threshold * fmaxf(bound, 1.f)) {  // threshold <= 0: all exact
      const uint32_t at = atomicAdd(nfall, 1u);
      fallback[at] = (uint32_t)i;
    }
  }
}

__global__ void k_gather_idx(const uint8_t* __restrict__ blocks, const uint32_t* __restrict__ idx,
                             const uint32_t* __restrict__ count, uint8_t* __restrict__ out) {
  const uint32_t n = *count;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n * 4; t += gridDim.x * blockDim.x) {
    const uint32_t i = t >> 2, q = t & 3;
    reinterpret_cast<uint4*>(out)[t] = reinterpret_cast<const uint4*>(blocks + (long long)idx[i] * 64)[q];
  }
}
__global__ void k_scatter_idx(const uint8_t* __restrict__ enc, const uint32_t* __restrict__ idx,
                              const uint32_t* __restrict__ count, uint8_t* __restrict__ out) {
  const uint32_t n = *count;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    *reinterpret_cast<uint2*>(out + (long long)idx[i] * 8) = reinterpret_cast<const uint2*>(enc)[i];
}

// ------------------------------------------------------------------------------------------
// Host side

struct Param {
  int rows, cols;
  DevBuf w, g, m, v, wb;  // fp32 master, grad, Adam moments, bf16 copy (weights only)
  DevBuf wbT;             // bf16 transposed copy (W2, W3: the backward products)
  size_t n() const { return (size_t)rows * cols; }
};

struct Net {
  uint32_t magic = 0x4D4C5030u;
  int device = -1;
  Param W1, b1, W2, b2, W3, b3;
  int step = 0;
  float bound_tau = 0.f, bound_weight = 1.f;  // loss of the error-bound output (see k_train_tile)
  // training scratch sized for the largest batch seen (tiles of 128 samples, see TrainArgs)
  int cap = 0;
  DevBuf h1T, h2T, d1T, d2T, xT, dyT, g1, g2, bias, part;
  DevBuf errflag;  // [0] a wait timed out, [1] the loss
  // learned encode scratch
  DevBuf fb_idx, fb_count, fb_in, fb_out, chunk_y;
  std::vector<Param*> params() { return {&W1, &b1, &W2, &b2, &W3, &b3}; }
};

int alloc_param(Param& p, int rows, int cols, bool bf16, bool transposed) {
  p.rows = rows; p.cols = cols;
  cudaError_t e;
  if ((e = p.w.ensure(p.n() * 4)) != cudaSuccess) return cuda_check(e, "alloc weights");
  if ((e = p.g.ensure(p.n() * 4)) != cudaSuccess) return cuda_check(e, "alloc grads");
  if ((e = p.m.ensure(p.n() * 4)) != cudaSuccess) return cuda_check(e, "alloc adam m");
  if ((e = p.v.ensure(p.n() * 4)) != cudaSuccess) return cuda_check(e, "alloc adam v");
  cudaMemset(p.m.ptr, 0, p.n() * 4);
  cudaMemset(p.v.ptr, 0, p.n() * 4);
  cudaMemset(p.g.ptr, 0, p.n() * 4);
  if (bf16 && (e = p.wb.ensure(p.n() * 2)) != cudaSuccess) return cuda_check(e, "alloc bf16 weights");
  if (transposed && (e = p.wbT.ensure(p.n() * 2)) != cudaSuccess) return cuda_check(e, "alloc bf16 weights");
  return CRNGPU_OK;
}

int upload(Param& p, const std::vector<float>& host) {
  cudaError_t e = cudaMemcpy(p.w.ptr, host.data(), p.n() * 4, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_check(e, "upload weights");
  if (p.wb.ptr) {
    std::vector<__nv_bfloat16> hb(p.n());
    for (size_t i = 0; i < p.n(); i++) hb[i] = __float2bfloat16(host[i]);
    if ((e = cudaMemcpy(p.wb.ptr, hb.data(), p.n() * 2, cudaMemcpyHostToDevice)) != cudaSuccess)
      return cuda_check(e, "upload bf16 weights");
  }
  if (p.wbT.ptr) {
    std::vector<__nv_bfloat16> hb(p.n());
    for (int r = 0; r < p.rows; r++)
      for (int c = 0; c < p.cols; c++) hb[(size_t)c * p.rows + r] = __float2bfloat16(host[(size_t)r * p.cols + c]);
    if ((e = cudaMemcpy(p.wbT.ptr, hb.data(), p.n() * 2, cudaMemcpyHostToDevice)) != cudaSuccess)
      return cuda_check(e, "upload bf16 weights");
  }
  return CRNGPU_OK;
}

// Slices of the weight gradients' sum: with two halves of the rows each, about as many CTAs as SMs.
constexpr int kMaxSlices = 64;

int ensure_batch(Net& net, int tiles) {
  cudaError_t e;
  if ((e = net.errflag.ensure(16)) != cudaSuccess) return cuda_check(e, "alloc flag");
  if (tiles <= net.cap) return CRNGPU_OK;
  net.cap = 0;  // a buffer that does not get its memory has given up what it had
  // the largest first, so that a batch that does not fit fails before it holds much
  struct { DevBuf* b; size_t bytes; } need[] = {
      {&net.g1, kHid * BM * 4}, {&net.g2, kHid * BM * 4}, {&net.h1T, kTileT}, {&net.h2T, kTileT}, {&net.d1T, kTileT},
      {&net.d2T, kTileT}, {&net.xT, kTileX}, {&net.dyT, kTileDy}, {&net.bias, kBiasSums * 4 * 4}};
  for (auto& n : need)
    if ((e = n.b->ensure(n.bytes * (size_t)tiles)) != cudaSuccess) return cuda_check(e, "alloc training scratch");
  if ((e = net.part.ensure((size_t)std::min(tiles, kMaxSlices) * kGradCols * kHid * 4)) != cudaSuccess)
    return cuda_check(e, "alloc partial gradients");
  net.cap = tiles;
  return CRNGPU_OK;
}

// inference over n blocks (device) -> y [n x 16] with the fused kernel, one persistent CTA per SM
int infer(Net& net, const uint8_t* blocks, uint32_t n, float* y, cudaStream_t s) {
  static bool attr_done[64] = {};
  static int sms[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_check(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) { set_error("device index out of range"); return CRNGPU_E_DEVICE; }
  {
    std::lock_guard<std::mutex> lock(device_setup_mutex());
    if (!attr_done[dev]) {
      e = cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInferSmem);
      if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return cuda_check(e, "set up k_mlp_infer");
      attr_done[dev] = true;
    }
  }
  if ((e = net.errflag.ensure(16)) != cudaSuccess) return cuda_check(e, "alloc flag");
  if (!n) return CRNGPU_OK;
  const uint32_t tiles = (n + BM - 1) / BM;
  const uint32_t grid = tiles < (uint32_t)sms[dev] ? tiles : (uint32_t)sms[dev];
  k_mlp_infer<<<grid, kInferThreads, kInferSmem, s>>>(
      blocks, (int)n, static_cast<__nv_bfloat16*>(net.W1.wb.ptr), static_cast<__nv_bfloat16*>(net.W2.wb.ptr),
      static_cast<__nv_bfloat16*>(net.W3.wb.ptr), static_cast<float*>(net.b1.w.ptr), static_cast<float*>(net.b2.w.ptr),
      static_cast<float*>(net.b3.w.ptr), y, static_cast<uint32_t*>(net.errflag.ptr));
  return cuda_check(cudaGetLastError(), "launch k_mlp_infer");
}

struct Adam {
  float lr, wd;
};

// Loss and gradients of B samples, and with `adam` one AdamW step (betas 0.9/0.999, eps 1e-8); the
// loss goes to errflag[1].
int train_pass(Net& net, const uint8_t* blocks, const float* targets, uint32_t n, const Adam* adam, cudaStream_t s) {
  if (n > (1u << 28)) { set_error("training: at most 2^28 blocks per batch"); return CRNGPU_E_PARAM; }
  const int B = (int)n;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_check(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) { set_error("device index out of range"); return CRNGPU_E_DEVICE; }
  {
    std::lock_guard<std::mutex> lock(device_setup_mutex());
    if (!attr_done[dev]) {
      e = cudaFuncSetAttribute(k_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_train_weight_grads, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgSmem);
      if (e != cudaSuccess) return cuda_check(e, "set up the training kernels");
      attr_done[dev] = true;
    }
  }
  const int tiles = (B + BM - 1) / BM;
  int rc = ensure_batch(net, tiles);
  if (rc != CRNGPU_OK) return rc;
  auto f32 = [](DevBuf& b) { return static_cast<float*>(b.ptr); };
  auto bf = [](DevBuf& b) { return static_cast<__nv_bfloat16*>(b.ptr); };
  auto u8 = [](DevBuf& b) { return static_cast<unsigned char*>(b.ptr); };
  uint32_t* err = static_cast<uint32_t*>(net.errflag.ptr);
  TrainArgs t;
  t.blocks = blocks;
  t.targets = targets;
  t.n = B;
  t.tiles = tiles;
  t.tau = net.bound_tau;
  t.bw = net.bound_weight;
  t.W1 = bf(net.W1.wb); t.W2 = bf(net.W2.wb); t.W2T = bf(net.W2.wbT); t.W3 = bf(net.W3.wb); t.W3T = bf(net.W3.wbT);
  t.b1 = f32(net.b1.w); t.b2 = f32(net.b2.w); t.b3 = f32(net.b3.w);
  t.h1T = u8(net.h1T); t.h2T = u8(net.h2T); t.d1T = u8(net.d1T); t.d2T = u8(net.d2T); t.xT = u8(net.xT); t.dyT = u8(net.dyT);
  t.g1 = f32(net.g1); t.g2 = f32(net.g2);
  t.bias = f32(net.bias);
  t.part = f32(net.part);
  t.slice_tiles = (tiles + kMaxSlices - 1) / kMaxSlices;
  t.slices = (tiles + t.slice_tiles - 1) / t.slice_tiles;
  t.err = err;
  ReduceArgs r;
  auto ptrs = [&](Param& p) { return ParamPtrs{f32(p.g), f32(p.w), f32(p.m), f32(p.v), bf(p.wb), bf(p.wbT)}; };
  r.W1 = ptrs(net.W1); r.b1 = ptrs(net.b1); r.W2 = ptrs(net.W2); r.b2 = ptrs(net.b2); r.W3 = ptrs(net.W3); r.b3 = ptrs(net.b3);
  r.part = t.part;
  r.bias = t.bias;
  r.slices = t.slices;
  r.bias_sums = 4 * tiles;
  r.loss = reinterpret_cast<float*>(err + 1);
  r.err = err;
  r.update = adam != nullptr;
  r.beta1 = 0.9f;
  r.beta2 = 0.999f;
  r.eps = 1e-8f;
  r.lr = adam ? adam->lr : 0.f;
  r.wd = adam ? adam->wd : 0.f;
  r.bc1 = 1.f - std::pow(r.beta1, (float)(net.step + 1));
  r.bc2 = 1.f - std::pow(r.beta2, (float)(net.step + 1));
  if ((e = cudaMemsetAsync(err, 0, 8, s)) != cudaSuccess) return cuda_check(e, "clear flag");
  k_train_tile<<<tiles, kTrainThreads, kTrainSmem, s>>>(t);
  k_train_weight_grads<<<dim3(2, t.slices), kTrainThreads, kWgSmem, s>>>(t);
  k_train_reduce<<<kReduceBlocks, 1024, 0, s>>>(r);
  return cuda_check(cudaGetLastError(), "launch the training kernels");
}

// Waits for the stream; the flag (and with `loss` the loss) of what ran on it.
int check_flag(Net& net, cudaStream_t s, float* loss = nullptr) {
  uint32_t f[2] = {};
  cudaError_t e = cudaMemcpyAsync(f, net.errflag.ptr, loss ? 8 : 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_check(e, "read mma status");
  if (f[0]) { set_error("tensor-core wait timed out"); return CRNGPU_E_DEVICE; }
  if (loss) std::memcpy(loss, &f[1], 4);
  return CRNGPU_OK;
}

}  // namespace mlp
// Test hook for the tcgen05 commit waits: polls per first wait (drains are not affected).
int set_mma_wait_polls(uint32_t polls) {
  return cuda_check(cudaMemcpyToSymbol(mlp::g_mma_wait_polls, &polls, sizeof(polls)), "set mma wait polls");
}

// Number of first waits that ran out since the last reset.
int mma_wait_counter(uint32_t* out, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out, mlp::g_mma_wait_timeouts, sizeof(uint32_t));
  if (e == cudaSuccess && reset) {
    const uint32_t z = 0;
    e = cudaMemcpyToSymbol(mlp::g_mma_wait_timeouts, &z, sizeof(z));
  }
  return cuda_check(e, "read mma wait counter");
}

}  // namespace crngpu

using namespace crngpu;
using namespace crngpu::mlp;

extern "C" void* crngpu_mlp_create(uint64_t seed) try {
  clear_error();
  Net* net = new Net();
  cudaGetDevice(&net->device);
  std::mt19937_64 rng(seed);
  auto init = [&](Param& p, int rows, int cols, int rows_live, bool is_bias, int fan_in) {
    if (alloc_param(p, rows, cols, !is_bias, &p == &net->W2 || &p == &net->W3) != CRNGPU_OK) return false;
    std::vector<float> h(p.n(), 0.f);
    if (!is_bias) {
      const float bound = std::sqrt(6.0f / (float)fan_in) * 0.5f;
      std::uniform_real_distribution<float> u(-bound, bound);
      for (int r = 0; r < rows_live; r++)
        for (int c = 0; c < cols; c++) h[(size_t)r * cols + c] = u(rng);
    }
    return upload(p, h) == CRNGPU_OK;
  };
  if (!init(net->W1, kHid, kIn, kHid, false, kIn) || !init(net->b1, 1, kHid, 1, true, 1) ||
      !init(net->W2, kHid, kHid, kHid, false, kHid) || !init(net->b2, 1, kHid, 1, true, 1) ||
      !init(net->W3, kOutPad, kHid, 7, false, kHid) || !init(net->b3, 1, kOutPad, 1, true, 1)) {
    delete net;
    return nullptr;
  }
  cudaDeviceSynchronize();
  return net;
} catch (...) {
  crngpu::exception_status();
  return nullptr;
}

extern "C" int crngpu_mlp_destroy(void* h) try {
  Net* net = static_cast<Net*>(h);
  if (!net || net->magic != 0x4D4C5030u) return CRNGPU_E_PARAM;
  net->magic = 0;
  delete net;
  return CRNGPU_OK;
} catch (...) {
  return crngpu::exception_status();
}

// Parameter access for checkpoints and gradient checks. which: 0 W1, 1 b1, 2 W2, 3 b2, 4 W3, 5 b3;
// what: 0 weights, 1 gradients. count = number of floats in the buffer.
extern "C" int crngpu_mlp_param(void* h, int which, int what, float* host, uint32_t count, int write) try {
  Net* net = static_cast<Net*>(h);
  if (!net || net->magic != 0x4D4C5030u || which < 0 || which > 5 || !host) return CRNGPU_E_PARAM;
  Param* p = net->params()[which];
  if (count != p->n()) { set_error("size mismatch"); return CRNGPU_E_PARAM; }
  void* dev = what ? p->g.ptr : p->w.ptr;
  if (write) {
    std::vector<float> v(host, host + count);
    if (what == 0) return upload(*p, v);
    return cuda_check(cudaMemcpy(dev, host, count * 4, cudaMemcpyHostToDevice), "write param");
  }
  return cuda_check(cudaMemcpy(host, dev, count * 4, cudaMemcpyDeviceToHost), "read param");
} catch (...) {
  return crngpu::exception_status();
}

// Loss of the error-bound output: tau <= 0 squared error (weight ignored); 0 < tau < 1 the
// tau-quantile (pinball) loss scaled by `weight`.
extern "C" int crngpu_mlp_set_bound_loss(void* h, float tau, float weight) try {
  Net* net = static_cast<Net*>(h);
  if (!net || net->magic != 0x4D4C5030u || !(tau < 1.f) || !(weight > 0.f)) return CRNGPU_E_PARAM;
  net->bound_tau = tau > 0.f ? tau : 0.f;
  net->bound_weight = weight;
  return CRNGPU_OK;
} catch (...) {
  return crngpu::exception_status();
}

// Forward pass over n blocks (device RGBA8, n x 64) -> y (device, n x 16 fp32).
extern "C" int crngpu_mlp_forward(void* h, const uint8_t* d_blocks, uint32_t n, float* d_y, void* stream) try {
  clear_error();
  Net* net = static_cast<Net*>(h);
  if (!net || net->magic != 0x4D4C5030u || !d_blocks || !d_y) return CRNGPU_E_PARAM;
  if (n > (1u << 28)) { set_error("crngpu_mlp_forward: at most 2^28 blocks per call"); return CRNGPU_E_PARAM; }
  cudaStream_t s = as_stream(stream);
  cudaError_t e = net->errflag.ensure(16);
  if (e != cudaSuccess) return cuda_check(e, "alloc flag");
  cudaMemsetAsync(net->errflag.ptr, 0, 4, s);
  int rc = infer(*net, d_blocks, n, d_y, s);
  if (rc != CRNGPU_OK) return rc;
  return check_flag(*net, s);
} catch (...) {
  return crngpu::exception_status();
}

// Gradients of the loss for n blocks and targets (device, n x 8 fp32) into the gradient buffers;
// *loss (host) receives the loss. Does not update the weights.
extern "C" int crngpu_mlp_gradients(void* h, const uint8_t* d_blocks, const float* d_targets, uint32_t n, float* loss,
                                    void* stream) try {
  clear_error();
  Net* net = static_cast<Net*>(h);
  if (!net || net->magic != 0x4D4C5030u || !d_blocks || !d_targets || !n) return CRNGPU_E_PARAM;
  cudaStream_t s = as_stream(stream);
  int rc = train_pass(*net, d_blocks, d_targets, n, nullptr, s);
  return rc != CRNGPU_OK ? rc : check_flag(*net, s, loss);
} catch (...) {
  return crngpu::exception_status();
}

// One AdamW step (betas 0.9/0.999, eps 1e-8) on a batch: forward, backward, update.
extern "C" int crngpu_mlp_train_step(void* h, const uint8_t* d_blocks, const float* d_targets, uint32_t n, float lr,
                                     float weight_decay, float* loss, void* stream) try {
  clear_error();
  Net* net = static_cast<Net*>(h);
  if (!net || net->magic != 0x4D4C5030u || !d_blocks || !d_targets || !n) return CRNGPU_E_PARAM;
  cudaStream_t s = as_stream(stream);
  const Adam adam = {lr, weight_decay};
  int rc = train_pass(*net, d_blocks, d_targets, n, &adam, s);
  if (rc != CRNGPU_OK || (rc = check_flag(*net, s, loss)) != CRNGPU_OK) return rc;
  net->step++;
  return CRNGPU_OK;
} catch (...) {
  return crngpu::exception_status();
}

// Training targets from plain-optimizer output (device): blocks8 (n x 8) + errors (n) -> n x 8.
extern "C" int crngpu_mlp_make_targets(const uint8_t* d_blocks8, const uint64_t* d_err, uint32_t n, float* d_targets,
                                       void* stream) try {
  if (!d_blocks8 || !d_err || !d_targets) return CRNGPU_E_PARAM;
  k_make_targets<<<(n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096, 256, 0, as_stream(stream)>>>(d_blocks8, d_err,
                                                                                                  (int)n, d_targets);
  return cuda_check(cudaGetLastError(), "launch k_make_targets");
} catch (...) {
  return crngpu::exception_status();
}

// Learned DXT1 encode of n blocks (device RGBA8 in, device dxt1 out): MLP proposal, one
// selector refit, and the exact optimizer for blocks whose error exceeds threshold x the
// predicted bound. *fallbacks (host, optional) receives how many blocks fell back.
extern "C" int crngpu_dxt1_learned_ex(void* h, const uint8_t* d_blocks, uint32_t n, int perceptual, float threshold,
                                      uint32_t fallback_quality, uint8_t* d_out, uint32_t* fallbacks, void* stream) try {
  clear_error();
  Net* net = static_cast<Net*>(h);
  if (!net || net->magic != 0x4D4C5030u || !d_blocks || !d_out) return CRNGPU_E_PARAM;
  if (fallback_quality > kDxtQualityUber) { set_error("crngpu_dxt1_learned: bad fallback quality"); return CRNGPU_E_PARAM; }
  if (!n) return CRNGPU_OK;
  if (n > (1u << 28)) { set_error("crngpu_dxt1_learned: at most 2^28 blocks per call"); return CRNGPU_E_PARAM; }
  cudaStream_t s = as_stream(stream);
  const uint32_t chunk = 1u << 20;
  int rc;
  cudaError_t e;
  if ((e = net->errflag.ensure(16)) != cudaSuccess) return cuda_check(e, "alloc flag");
  if ((e = net->chunk_y.ensure((size_t)(n < chunk ? n : chunk) * kOutPad * 4)) != cudaSuccess)
    return cuda_check(e, "alloc proposals");
  if ((e = net->fb_idx.ensure((size_t)n * 4)) != cudaSuccess) return cuda_check(e, "alloc fallback list");
  if ((e = net->fb_count.ensure(16)) != cudaSuccess) return cuda_check(e, "alloc fallback count");
  uint32_t* idx = static_cast<uint32_t*>(net->fb_idx.ptr);
  uint32_t* cnt_d = static_cast<uint32_t*>(net->fb_count.ptr);
  cudaMemsetAsync(cnt_d, 0, 4, s);
  cudaMemsetAsync(net->errflag.ptr, 0, 4, s);
  if (fallbacks) *fallbacks = 0;
  // proposals for every block (chunked to bound the activation buffers); blocks above the bound
  // are appended to one list of indices into the whole batch
  for (uint32_t c0 = 0; c0 < n; c0 += chunk) {
    const uint32_t cn = n - c0 < chunk ? n - c0 : chunk;
    if ((rc = infer(*net, d_blocks + (size_t)c0 * 64, cn, static_cast<float*>(net->chunk_y.ptr), s)) != CRNGPU_OK)
      return rc;
    k_learned_refit<<<(cn + 127) / 128, 128, 0, s>>>(d_blocks, static_cast<float*>(net->chunk_y.ptr), c0, (int)cn,
                                                      perceptual, d_out, idx, cnt_d, threshold);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_check(e, "launch k_learned_refit");
  }
  // blocks above the bound: the exact optimizer on a compacted copy, scattered back. The count
  // stays on the device: the gather, both encoder kernels and the scatter read it there, so the
  // call never waits for the host between the proposals and the fallback.
  if ((e = net->fb_in.ensure((size_t)n * 64)) != cudaSuccess) return cuda_check(e, "alloc fallback blocks");
  if ((e = net->fb_out.ensure((size_t)n * 8)) != cudaSuccess) return cuda_check(e, "alloc fallback out");
  const uint32_t sweep = (uint32_t)std::min<uint64_t>(((uint64_t)n * 4 + 255) / 256, 8192);
  k_gather_idx<<<sweep, 256, 0, s>>>(d_blocks, idx, cnt_d, static_cast<uint8_t*>(net->fb_in.ptr));
  if ((rc = launch_dxt1_count(static_cast<uint8_t*>(net->fb_in.ptr), n, cnt_d,
                              dxt1_options(perceptual != 0, true, fallback_quality, false, false, 128),
                              static_cast<uint8_t*>(net->fb_out.ptr), 8, s)) != CRNGPU_OK)
    return rc;
  k_scatter_idx<<<(sweep + 3) / 4, 256, 0, s>>>(static_cast<uint8_t*>(net->fb_out.ptr), idx, cnt_d, d_out);
  uint32_t cnt = 0;
  if (fallbacks && (e = cudaMemcpyAsync(&cnt, cnt_d, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cuda_check(e, "read fallback count");
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_check(e, "learned encode kernels");
  rc = check_flag(*net, s);  // synchronises the stream
  if (rc != CRNGPU_OK) return rc;
  if (fallbacks) {
    if (cnt > n) { set_error("crngpu_dxt1_learned: fallback count out of range"); return CRNGPU_E_DEVICE; }
    *fallbacks = cnt;
  }
  return CRNGPU_OK;
} catch (...) {
  return crngpu::exception_status();
}

extern "C" int crngpu_dxt1_learned(void* h, const uint8_t* d_blocks, uint32_t n, int perceptual, float threshold,
                                   uint8_t* d_out, uint32_t* fallbacks, void* stream) try {
  return crngpu_dxt1_learned_ex(h, d_blocks, n, perceptual, threshold, kDxtQualityUber, d_out, fallbacks, stream);
} catch (...) {
  return crngpu::exception_status();
}
