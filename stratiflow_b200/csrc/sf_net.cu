// The learned predictor of pseudo-arclength continuation: a stack of 1D
// convolutions along z over the spectral coefficients of converged branch
// states (no counterpart in the reference, whose predictor is the secant of
// PseudoArclength.cpp:33-61). Training and inference run on the tensor
// cores with BF16 operands and FP32 accumulation; master weights, gradients
// and the Adam moments stay FP32.
//
// Tensors are channel-last: an activation is [batch][Z][C] (BF16), the
// weights of a layer W[Cout][tap][Cin] (tap < 5, zero padding of 2 levels at
// both ends of z) followed by its bias[Cout]. Every contraction is one
// implicit GEMM, C[m][n] = sum_k A(m,k) B(n,k):
//   forward          m = co, n = (b,z),        k = (tap,ci)
//   backward data    m = ci, n = (b,z),        k = (tap,co)
//   backward weights m = co, n = (tap,ci),     k = (b,z)
// issued as tcgen05.mma on 128 x 64 tiles with the accumulator in tensor
// memory, the operands brought in by tensor-map copies (k_conv_gemm_tc).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <string>
#include <vector>

#include "../../include/stratiflow_b200.h"

extern void sf_set_error_message(const std::string& msg);
extern void* sf_host_dma(const void* p);

namespace {

constexpr int kTaps = 5, kPad = 2;

enum GemmMode { G_FWD = 0, G_BWD_DATA = 1, G_BWD_W = 2 };

struct ConvGemm {
  int B, Z, Cin, Cout;
  int M;                     // rows of C
  const float* bias;         // forward
  float* outF;               // FP32 result (forward output layer, dW)
  __nv_bfloat16* outB;       // BF16 result (activation, dP of the layer below)
  int relu;                  // forward: ReLU on the BF16 result
  const __nv_bfloat16* mask; // backward data: keep where mask > 0 (ReLU')
};

// ---------------------------------------------------------------- tcgen05 --
// The implicit GEMMs on the 5th-generation tensor cores. A CTA of four warps
// computes a 128 x 64 tile of C: a tile's n are 64 levels of one sample
// (forward, backward data) or 64 input channels of one tap (backward weights).
// Every K slice of 64 is one tap's run of 64 channels, or one sample's run of
// 64 levels, so both operands of a slice are boxes of the tensors as they lie
// in memory: X and dP as [B][Z][C], W as [Cout][tap][Cin]. Thread 0 brings
// them in by cp.async.bulk.tensor (levels outside 0..Z-1 and channels past C
// arrive as zeros: the convolution's padding and the tiles' edges need no
// code), thread 32 issues tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, M =
// 128, N = 64, K = 16) with the accumulator in tensor memory, all four warps
// read it back. A slice's operands lie in shared memory in the 128-byte
// swizzle, with K contiguous (forward; backward data's dP) or with M or N
// contiguous (backward data's W, both operands of the weight gradient: the
// instruction's transpose bits), as the tensors have them.
//
// Bound by the operands' way from L2: 24 KB a slice and SM, which takes about
// 840 cycles on 104 SMs at once (6.0 TB/s over the GPU) against the
// instructions' 128; four slices in flight per CTA, two CTAs per SM (eight
// slices measured the same). Measured, 13 samples of 256 levels: 1024 -> 256
// channels forward 34 us under ncu, the 11 GEMMs of one gradient 0.18 ms in 8 launches,
// where the version that gathered operands through registers took 3.29 ms.
//
// The K slices, and the runs of 16 of an instruction within them, go in the
// order of (tap, channel), one accumulator per tile: a result does not depend
// on the tiling. Every wait is bounded; one that runs out sets *err, the other
// waits of the block then give up at once, and the block waits, with the same
// bound, for its copies and instructions in flight and frees its tensor memory.
constexpr int TM = 128, TN = 64, TK = 64, kTcThreads = 128, kTcStages = 4, kMaxLayers = 16;
constexpr int kTcABytes = TM * TK * 2, kTcBBytes = TN * TK * 2, kTcStageBytes = kTcABytes + kTcBBytes;
// the stages, and room to align the first to the swizzle's 1024-byte period
static_assert(TN == TK, "the X and dP maps' boxes serve as N tiles and as K slices");
constexpr size_t kTcSmem = (size_t)kTcStages * kTcStageBytes + 1024;
constexpr int kTcSpin = 1 << 22;                                   // bounded mbarrier waits

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor (sm_100) of the 128-byte swizzle: start
// address and the byte offsets in 16-byte units, descriptor version 1, layout
// type 2 (SWIZZLE_128B). K contiguous: rows of 64 K values, 8-row groups SBO =
// 1024 bytes apart (LBO unused). M or N contiguous: rows of 64 M or N values,
// one per k, 8-k groups SBO = 1024 bytes apart, the next 64 M or N values
// LBO = 8192 bytes on (64 k rows of 128 bytes).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t addr, bool mn) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(mn ? 8192 >> 4 : 1) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

// instruction descriptor of kind::f16: D FP32, A and B BF16, N and M of the
// instruction; a_mn / b_mn: the operand has M / N contiguous
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N, bool a_mn, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(b)) : "memory");
}
// false when the wait ran out, or (give_up) another of the block has
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, volatile int* failed, bool give_up = true) {
  const uint32_t a = smem_u32(bar);
  for (int i = 0; i < kTcSpin; i++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(phase)
        : "memory");
    if (done) return true;
    if (give_up && *failed) return false;
  }
  return false;
}
__device__ __forceinline__ void tma3(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// A block whose wait ran out: the copies in flight, of slices that no
// instruction has waited for, and the instructions in flight, before their
// operands and the accumulator go. Not inlined: out of the way of the loops'
// code, inside which they cost 5 us of a gradient's 418.
__device__ __noinline__ void drain_copies(uint64_t* full, int issued, volatile int* failed) {
  for (int i = issued > kTcStages ? issued - kTcStages : 0; i < issued; i++)
    mbar_wait(&full[i % kTcStages], (i / kTcStages) & 1, failed, false);
}
__device__ __noinline__ void drain_instructions(uint64_t* drain, volatile int* failed, int* err) {
  *failed = 1;
  atomicExch(err, 1);
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(drain))
               : "memory");
  mbar_wait(drain, 0, failed, false);
}

// tile (tn, m0) of one GEMM
template <int MODE>
__device__ __forceinline__ void conv_tile(const CUtensorMap& mapA, const CUtensorMap& mapB, const ConvGemm& p,
                                          const int tn, const int m0, int* err) {
  extern __shared__ __align__(128) unsigned char tsm[];
  unsigned char* stage0 = tsm + ((1024 - (smem_u32(tsm) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t full[kTcStages], empty[kTcStages], done, drain;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int ns = kTcStages;
  constexpr bool a_mn = MODE != G_FWD, b_mn = MODE == G_BWD_W;
  // the tile's n: levels z0 .. of sample nb, or channels c0n .. of a tap
  const int per = MODE == G_BWD_W ? (p.Cin + TN - 1) / TN : (p.Z + TN - 1) / TN;
  const int nb = tn / per, n0 = (tn - nb * per) * TN;
  // the K slices: (tap, 64 channels), or (sample, 64 levels)
  const int ks = MODE == G_BWD_W ? (p.Z + TK - 1) / TK : ((MODE == G_FWD ? p.Cin : p.Cout) + TK - 1) / TK;
  const int nk = (MODE == G_BWD_W ? p.B : kTaps) * ks;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(TN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    failed = 0;
    for (int s = 0; s < ns; s++) {
      mbar_init(&full[s]);
      mbar_init(&empty[s]);
    }
    mbar_init(&done);
    mbar_init(&drain);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  int issued = 0;   // thread 0: the slices whose copies it has issued
  if (warp == 0) {
    if (lane == 0) {
      int kt = 0, s = 0, ph = 1;   // ph: the parity of the slot's last use
      for (; kt < nk; kt++, s = s + 1 == ns ? 0 : s + 1, ph ^= s == 0) {
        const int k1 = kt / ks, k0 = (kt - k1 * ks) * TK;
        if (kt >= ns && !mbar_wait(&empty[s], ph, &failed)) {
          failed = 1;
          atomicExch(err, 1);
          break;
        }
        unsigned char *A = stage0 + (size_t)s * kTcStageBytes, *Bt = A + kTcABytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[s])),
                     "r"(kTcStageBytes)
                     : "memory");
        if (MODE == G_FWD) {
          tma3(A, &mapA, k0, k1, m0, &full[s]);
          tma3(Bt, &mapB, k0, n0 + k1 - kPad, nb, &full[s]);
        } else if (MODE == G_BWD_DATA) {
          tma3(A, &mapA, m0, k1, k0, &full[s]);
          tma3(A + kTcABytes / 2, &mapA, m0 + 64, k1, k0, &full[s]);
          tma3(Bt, &mapB, k0, n0 - k1 + kPad, nb, &full[s]);
        } else {
          tma3(A, &mapA, m0, k0, k1, &full[s]);
          tma3(A + kTcABytes / 2, &mapA, m0 + 64, k0, k1, &full[s]);
          tma3(Bt, &mapB, n0, k0 + nb - kPad, k1, &full[s]);
        }
      }
      issued = kt;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(TM, TN, a_mn, b_mn);
      int kt = 0, s = 0, ph = 0;
      for (; kt < nk; kt++, s = s + 1 == ns ? 0 : s + 1, ph ^= s == 0) {
        if (!mbar_wait(&full[s], ph, &failed)) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t a0 = smem_u32(stage0) + s * kTcStageBytes, b0 = a0 + kTcABytes;
#pragma unroll
        for (int kk = 0; kk < TK / 16; kk++) {
          // K = 16 per instruction: 32 bytes of every row, or 16 rows of 128
          const uint64_t da = umma_desc_sw128(a0 + (a_mn ? 2048 : 32) * kk, a_mn);
          const uint64_t db = umma_desc_sw128(b0 + (b_mn ? 2048 : 32) * kk, b_mn);
          const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
              ::"r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(kt + 1 < nk ? &empty[s] : &done))
                     : "memory");   // the last covers every instruction before it
      }
      if (__builtin_expect(kt < nk, 0)) drain_instructions(&drain, &failed, err);
    }
    __syncwarp();
  }
  const bool ok = mbar_wait(&done, 0, &failed);
  if (!ok && !failed) {
    failed = 1;
    atomicExch(err, 1);
  }
  if (__builtin_expect(!ok && tid == 0, 0)) drain_copies(full, issued, &failed);
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (__all_sync(0xffffffffu, ok)) {
    // warp w reads tensor-memory lanes 32w..32w+31: row m0 + 32w + lane
    const int m = m0 + 32 * warp + lane;
    const int nend = (MODE == G_BWD_W ? p.Cin : p.Z) - n0;   // columns of the tile inside C
    for (int c = 0; c < TN; c += 8) {
      if (c >= nend) break;
      uint32_t v[8];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
          : "r"(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (m >= p.M) continue;
      if (MODE == G_BWD_W) {   // channel counts are multiples of 8: 8 whole columns, 32-byte aligned
        float4* o = reinterpret_cast<float4*>(p.outF + ((size_t)m * kTaps + nb) * p.Cin + n0 + c);
        o[0] = make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3]));
        o[1] = make_float4(__uint_as_float(v[4]), __uint_as_float(v[5]), __uint_as_float(v[6]), __uint_as_float(v[7]));
        continue;
      }
      const size_t o0 = ((size_t)nb * p.Z + n0 + c) * p.M + m;
      if (MODE == G_FWD) {
        const float bias = p.bias[m];
#pragma unroll
        for (int e = 0; e < 8; e++) {
          if (c + e >= nend) break;
          const float x = __uint_as_float(v[e]) + bias;
          const size_t o = o0 + (size_t)e * p.M;
          if (p.outF) p.outF[o] = x;
          if (p.outB) p.outB[o] = __float2bfloat16(p.relu ? fmaxf(x, 0.f) : x);
        }
      } else {
        __nv_bfloat16 k[8];
#pragma unroll
        for (int e = 0; e < 8; e++)
          if (c + e < nend) k[e] = p.mask[o0 + (size_t)e * p.M];
#pragma unroll
        for (int e = 0; e < 8; e++) {
          if (c + e >= nend) break;
          const float x = __bfloat162float(k[e]) > 0.f ? __uint_as_float(v[e]) : 0.f;
          p.outB[o0 + (size_t)e * p.M] = __float2bfloat16(x);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN));
}

template <int MODE>
__global__ void __launch_bounds__(kTcThreads) k_conv_gemm_tc(const __grid_constant__ CUtensorMap mapA,
                                                              const __grid_constant__ CUtensorMap mapB,
                                                              const __grid_constant__ ConvGemm p, int* err) {
  conv_tile<MODE>(mapA, mapB, p, blockIdx.x, blockIdx.y * TM, err);
}

// the weight gradients of every layer in one launch, once the last dP is
// known: a layer alone has 40 to 160 tiles, each a chain of B * Z / 64 slices
// (four launches of 23 to 28 us at 13 samples of 256 levels; together 48 us)
struct DwLayers {
  CUtensorMap dp[kMaxLayers], x[kMaxLayers];
  ConvGemm g[kMaxLayers];
  int first[kMaxLayers + 1];   // first block of each layer
};
__global__ void __launch_bounds__(kTcThreads) k_conv_gemm_tc_dw(const __grid_constant__ DwLayers d, int* err) {
  int l = 0;
  while ((int)blockIdx.x >= d.first[l + 1]) l++;
  const ConvGemm& p = d.g[l];
  const int t = blockIdx.x - d.first[l], nt = kTaps * ((p.Cin + TN - 1) / TN);
  conv_tile<G_BWD_W>(d.dp[l], d.x[l], p, t % nt, (t / nt) * TM, err);
}

__global__ void k_to_bf16(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

// loss = mean (out - target)^2; dP = bf16(2 (out - target) / count)
__global__ void k_mse(const float* __restrict__ out, const float* __restrict__ tgt, __nv_bfloat16* __restrict__ dP,
                      size_t n, double* loss) {
  double s = 0.0;
  const float inv = 2.0f / (float)n;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float d = out[i] - tgt[i];
    s += (double)d * d;
    dP[i] = __float2bfloat16(inv * d);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tsum = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) tsum += red[w];
    atomicAdd(loss, tsum / (double)n);
  }
}

// dbias[co] = sum over (b,z) of dP[b][z][co], every layer in one launch. A
// block takes 16 channels: two threads read a row's 32 bytes, 128 rows at a
// time, and the block's partial sums are added as a tree (one thread per
// channel over all rows was one chain of dependent additions: 765 us for 3328
// rows and four layers; now 19).
constexpr int kBiasThreads = 256;
struct BiasLayers {
  const __nv_bfloat16* dP[kMaxLayers];
  float* db[kMaxLayers];
  int C[kMaxLayers];
};
__global__ void __launch_bounds__(kBiasThreads) k_bias_grad(const __grid_constant__ BiasLayers a, int rows) {
  const int C = a.C[blockIdx.y];
  if (16 * (int)blockIdx.x >= C) return;
  const __nv_bfloat16* __restrict__ dP = a.dP[blockIdx.y];
  float* __restrict__ db = a.db[blockIdx.y];
  __shared__ float red[kBiasThreads / 2][17];
  const int half = threadIdx.x & 1, r0 = threadIdx.x >> 1, c = 16 * blockIdx.x + 8 * half;
  float s[8] = {};
  if (c < C)   // channel counts are multiples of 8
#pragma unroll 4
    for (int r = r0; r < rows; r += kBiasThreads / 2) {
      const uint4 v = *reinterpret_cast<const uint4*>(dP + (size_t)r * C + c);
      const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
      for (int k = 0; k < 8; k++) s[k] += __bfloat162float(e[k]);
    }
#pragma unroll
  for (int k = 0; k < 8; k++) red[r0][8 * half + k] = s[k];
  __syncthreads();
  for (int n = kBiasThreads / 4; n > 0; n >>= 1) {
    for (int i = threadIdx.x; i < n * 16; i += kBiasThreads) red[i >> 4][i & 15] += red[(i >> 4) + n][i & 15];
    __syncthreads();
  }
  if (threadIdx.x < 16 && 16 * (int)blockIdx.x + (int)threadIdx.x < C) db[16 * blockIdx.x + threadIdx.x] = red[0][threadIdx.x];
}

// Adam (Kingma & Ba 2015) on the FP32 master weights; refreshes the BF16
// copy of each weight (biases stay FP32)
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ gr, float* __restrict__ m1,
                       float* __restrict__ m2, size_t n, float lr, float b1, float b2, float c1, float c2,
                       float eps) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gv = gr[i];
    const float a = b1 * m1[i] + (1.f - b1) * gv, b = b2 * m2[i] + (1.f - b2) * gv * gv;
    m1[i] = a;
    m2[i] = b;
    w[i] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
  }
}

unsigned blocks_for(size_t n, int t) {
  size_t b = (n + t - 1) / t;
  return (unsigned)(b > 8192 ? 8192 : (b < 1 ? 1 : b));
}

}  // namespace

struct sf_net {
  int nl = 0, Z = 0, maxb = 0;
  std::vector<int> ch;               // ch[0] inputs .. ch[nl] outputs
  std::vector<size_t> woff, boff;    // offsets of W_l and b_l in the parameter vector
  size_t nparam = 0;
  float *w = nullptr, *gr = nullptr, *m1 = nullptr, *m2 = nullptr;
  __nv_bfloat16* wb = nullptr;       // BF16 copy of the whole parameter vector
  std::vector<__nv_bfloat16*> act;   // act[l]: input of layer l, [maxb][Z][ch[l]]
  std::vector<__nv_bfloat16*> dP;    // dP[l]: gradient of layer l's pre-activation
  float* out = nullptr;              // [maxb][Z][ch[nl]]
  float* xin = nullptr;              // FP32 staging of the input
  float* tgt = nullptr;              // training targets
  int nb_data = 0;                   // samples held in act[0] / tgt
  double* loss = nullptr;
  long long t = 0;                   // Adam steps taken
  cudaStream_t st = nullptr;
  int* err = nullptr;                // set by a GEMM block whose bounded wait ran out
  // tensor maps of each layer: W in boxes of 128 and of 64 output channels,
  // the layer's input and the gradient of its pre-activation
  struct Maps {
    CUtensorMap wf, wb, x, dp;
  };
  std::vector<Maps> maps;
};

namespace {

int nfail(int code, const std::string& m) {
  sf_set_error_message(m);
  return code;
}

#define NCK(x)                                                                       \
  do {                                                                               \
    cudaError_t e_ = (x);                                                            \
    if (e_ != cudaSuccess) return nfail(SF_ECUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// a BF16 tensor [d2][d1][d0] in boxes of 64 x b1 x b2 with the 128-byte swizzle
int conv_map(CUtensorMap* m, const __nv_bfloat16* base, int d0, int d1, int d2, int b1, int b2) {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn)
    return -1;
  const cuuint64_t dims[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
  const cuuint64_t strides[2] = {(cuuint64_t)d0 * 2, (cuuint64_t)d0 * d1 * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)b1, (cuuint32_t)b2}, es[3] = {1, 1, 1};
  const CUresult r = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn)(
      m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(base), dims, strides, box, es,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -1;
}

unsigned tiles(int a, int b) { return (unsigned)((a + b - 1) / b); }

int gemm(sf_net* n, int l, GemmMode mode, ConvGemm p) {
  const sf_net::Maps& t = n->maps[l];
  p.M = mode == G_FWD ? p.Cout : p.Cin;
  const dim3 grid(p.B * tiles(p.Z, TN), tiles(p.M, TM));
  if (mode == G_FWD) k_conv_gemm_tc<G_FWD><<<grid, kTcThreads, kTcSmem, n->st>>>(t.wf, t.x, p, n->err);
  else k_conv_gemm_tc<G_BWD_DATA><<<grid, kTcThreads, kTcSmem, n->st>>>(t.wb, t.dp, p, n->err);
  NCK(cudaGetLastError());
  return SF_OK;
}

int forward(sf_net* n, int B, bool keep_out) {
  for (int l = 0; l < n->nl; l++) {
    ConvGemm p{};
    p.B = B; p.Z = n->Z; p.Cin = n->ch[l]; p.Cout = n->ch[l + 1];
    p.bias = n->w + n->boff[l];
    const bool last = l == n->nl - 1;
    p.outF = last ? n->out : nullptr;
    p.outB = last ? nullptr : n->act[l + 1];
    p.relu = last ? 0 : 1;
    int rc = gemm(n, l, G_FWD, p);
    if (rc) return rc;
  }
  (void)keep_out;
  return SF_OK;
}

// gradients of the mean-square loss against n->tgt into n->gr
int backward(sf_net* n, int B) {
  const size_t nout = (size_t)B * n->Z * n->ch[n->nl];
  NCK(cudaMemsetAsync(n->loss, 0, sizeof(double), n->st));
  k_mse<<<std::min(blocks_for(nout, 256), 592u), 256, 0, n->st>>>(n->out, n->tgt, n->dP[n->nl - 1], nout, n->loss);
  for (int l = n->nl - 1; l > 0; l--) {   // dP of layer l-1 = (W^T * dP_l) where its ReLU was active
    ConvGemm p{};
    p.B = B; p.Z = n->Z; p.Cin = n->ch[l]; p.Cout = n->ch[l + 1];
    p.outB = n->dP[l - 1];
    p.mask = n->act[l];
    int rc = gemm(n, l, G_BWD_DATA, p);
    if (rc) return rc;
  }
  DwLayers d;
  BiasLayers bl;
  int blocks = 0, cmax = 0;
  for (int l = 0; l < n->nl; l++) {
    ConvGemm& p = d.g[l] = ConvGemm{};
    p.B = B; p.Z = n->Z; p.Cin = n->ch[l]; p.M = p.Cout = n->ch[l + 1];
    p.outF = n->gr + n->woff[l];
    d.dp[l] = n->maps[l].dp;
    d.x[l] = n->maps[l].x;
    d.first[l] = blocks;
    blocks += (int)(kTaps * tiles(p.Cin, TN) * tiles(p.M, TM));
    bl.dP[l] = n->dP[l];
    bl.db[l] = n->gr + n->boff[l];
    bl.C[l] = p.Cout;
    cmax = std::max(cmax, p.Cout);
  }
  d.first[n->nl] = blocks;
  k_conv_gemm_tc_dw<<<blocks, kTcThreads, kTcSmem, n->st>>>(d, n->err);
  k_bias_grad<<<dim3(tiles(cmax, 16), n->nl), kBiasThreads, 0, n->st>>>(bl, B * n->Z);
  NCK(cudaGetLastError());
  return SF_OK;
}

int refresh_bf16(sf_net* n) {
  k_to_bf16<<<blocks_for(n->nparam, 256), 256, 0, n->st>>>(n->w, n->wb, n->nparam);
  NCK(cudaGetLastError());
  return SF_OK;
}

int upload_input(sf_net* n, const float* x, int B) {
  const size_t nin = (size_t)B * n->Z * n->ch[0];
  NCK(cudaMemcpyAsync(n->xin, x, sizeof(float) * nin, cudaMemcpyHostToDevice, n->st));
  k_to_bf16<<<blocks_for(nin, 256), 256, 0, n->st>>>(n->xin, n->act[0], nin);
  NCK(cudaGetLastError());
  return SF_OK;
}

}  // namespace

extern "C" {

// waits for the stream; a GEMM whose tensor-core wait ran out is an error
static int net_status(sf_net* n) {
  int h = 0;
  NCK(cudaMemcpyAsync(&h, n->err, sizeof(int), cudaMemcpyDeviceToHost, n->st));
  NCK(cudaStreamSynchronize(n->st));
  if (h) {
    NCK(cudaMemset(n->err, 0, sizeof(int)));
    return nfail(SF_ECUDA, "a tensor-core GEMM block gave up waiting for its MMAs");
  }
  return SF_OK;
}

int sf_net_create(int nlayers, const int* channels, int Z, int max_batch, unsigned long long seed, void* stream,
                  sf_net** out) {
  if (!out || nlayers < 1 || nlayers > kMaxLayers || !channels || Z < 1 || max_batch < 1)
    return nfail(SF_EINVAL, "bad argument");
  for (int l = 0; l <= nlayers; l++)
    if (channels[l] < 1 || channels[l] % 8) return nfail(SF_EINVAL, "channel counts must be positive multiples of 8");
  sf_net* n = new sf_net();
  n->nl = nlayers;
  n->Z = Z;
  n->maxb = max_batch;
  n->ch.assign(channels, channels + nlayers + 1);
  n->st = (cudaStream_t)stream;
  for (int l = 0; l < nlayers; l++) {
    n->woff.push_back(n->nparam);
    n->nparam += (size_t)n->ch[l + 1] * kTaps * n->ch[l];
    n->boff.push_back(n->nparam);
    n->nparam += (size_t)n->ch[l + 1];
  }
  // He-normal weights (std sqrt(2 / fan_in)), zero biases, from the seed;
  // the output layer starts at zero so that an untrained net predicts no
  // correction
  std::vector<float> h(n->nparam, 0.f);
  std::mt19937_64 rng(seed);
  for (int l = 0; l < nlayers - 1; l++) {
    std::normal_distribution<float> nd(0.f, std::sqrt(2.f / (kTaps * n->ch[l])));
    for (size_t i = 0; i < (size_t)n->ch[l + 1] * kTaps * n->ch[l]; i++) h[n->woff[l] + i] = nd(rng);
  }
  auto bail = [&](const char* what) {
    sf_net_destroy(n);
    return nfail(SF_ENOMEM, what);
  };
  if (cudaMalloc(&n->w, sizeof(float) * n->nparam) != cudaSuccess) return bail("cudaMalloc weights");
  if (cudaMalloc(&n->gr, sizeof(float) * n->nparam) != cudaSuccess) return bail("cudaMalloc gradients");
  if (cudaMalloc(&n->m1, sizeof(float) * n->nparam) != cudaSuccess) return bail("cudaMalloc moments");
  if (cudaMalloc(&n->m2, sizeof(float) * n->nparam) != cudaSuccess) return bail("cudaMalloc moments");
  if (cudaMalloc(&n->wb, sizeof(__nv_bfloat16) * n->nparam) != cudaSuccess) return bail("cudaMalloc bf16 weights");
  n->act.assign(nlayers, nullptr);
  n->dP.assign(nlayers, nullptr);
  const size_t rows = (size_t)max_batch * Z;
  for (int l = 0; l < nlayers; l++) {
    if (cudaMalloc(&n->act[l], sizeof(__nv_bfloat16) * rows * n->ch[l]) != cudaSuccess) return bail("cudaMalloc act");
    if (cudaMalloc(&n->dP[l], sizeof(__nv_bfloat16) * rows * n->ch[l + 1]) != cudaSuccess) return bail("cudaMalloc dP");
  }
  if (cudaMalloc(&n->out, sizeof(float) * rows * n->ch[nlayers]) != cudaSuccess) return bail("cudaMalloc out");
  if (cudaMalloc(&n->tgt, sizeof(float) * rows * n->ch[nlayers]) != cudaSuccess) return bail("cudaMalloc targets");
  if (cudaMalloc(&n->xin, sizeof(float) * rows * n->ch[0]) != cudaSuccess) return bail("cudaMalloc input");
  if (cudaMalloc(&n->loss, sizeof(double)) != cudaSuccess) return bail("cudaMalloc loss");
  if (cudaMalloc(&n->err, sizeof(int)) != cudaSuccess) return bail("cudaMalloc status");
  bool set = cudaMemset(n->err, 0, sizeof(int)) == cudaSuccess;
  const int lim = (int)kTcSmem;
  for (auto* k : {k_conv_gemm_tc<G_FWD>, k_conv_gemm_tc<G_BWD_DATA>})
    set = set && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) == cudaSuccess;
  set = set && cudaFuncSetAttribute(k_conv_gemm_tc_dw, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) == cudaSuccess;
  n->maps.resize(nlayers);
  for (int l = 0; l < nlayers && set; l++) {
    const int ci = n->ch[l], co = n->ch[l + 1];
    sf_net::Maps& t = n->maps[l];
    const __nv_bfloat16* W = n->wb + n->woff[l];
    set = conv_map(&t.wf, W, ci, kTaps, co, 1, TM) == 0 && conv_map(&t.wb, W, ci, kTaps, co, 1, TK) == 0 &&
          conv_map(&t.x, n->act[l], ci, Z, max_batch, TN, 1) == 0 && conv_map(&t.dp, n->dP[l], co, Z, max_batch, TN, 1) == 0;
  }
  if (!set) {
    sf_net_destroy(n);
    return nfail(SF_ECUDA, "setting up the tensor-core GEMM");
  }
  if (cudaMemcpy(n->w, h.data(), sizeof(float) * n->nparam, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(n->m1, 0, sizeof(float) * n->nparam) != cudaSuccess ||
      cudaMemset(n->m2, 0, sizeof(float) * n->nparam) != cudaSuccess ||
      cudaMemset(n->gr, 0, sizeof(float) * n->nparam) != cudaSuccess) {
    sf_net_destroy(n);
    return nfail(SF_ECUDA, "initialising the weights");
  }
  int rc = refresh_bf16(n);
  if (rc) {
    sf_net_destroy(n);
    return rc;
  }
  *out = n;
  return SF_OK;
}

int sf_net_destroy(sf_net* n) {
  if (!n) return SF_OK;
  for (auto p : n->act) cudaFree(p);
  for (auto p : n->dP) cudaFree(p);
  for (void* p : {(void*)n->w, (void*)n->gr, (void*)n->m1, (void*)n->m2, (void*)n->wb, (void*)n->out,
                  (void*)n->tgt, (void*)n->xin, (void*)n->loss, (void*)n->err})
    cudaFree(p);
  delete n;
  return SF_OK;
}

int sf_net_num_params(sf_net* n, long long* count) {
  if (!n || !count) return nfail(SF_EINVAL, "bad argument");
  *count = (long long)n->nparam;
  return SF_OK;
}

int sf_net_get_params(sf_net* n, float* host) {
  if (!n || !host) return nfail(SF_EINVAL, "bad argument");
  NCK(cudaMemcpyAsync(host, n->w, sizeof(float) * n->nparam, cudaMemcpyDeviceToHost, n->st));
  NCK(cudaStreamSynchronize(n->st));
  return SF_OK;
}

int sf_net_set_params(sf_net* n, const float* host) {
  if (!n || !host) return nfail(SF_EINVAL, "bad argument");
  NCK(cudaMemcpyAsync(n->w, host, sizeof(float) * n->nparam, cudaMemcpyHostToDevice, n->st));
  NCK(cudaMemsetAsync(n->m1, 0, sizeof(float) * n->nparam, n->st));
  NCK(cudaMemsetAsync(n->m2, 0, sizeof(float) * n->nparam, n->st));
  n->t = 0;
  int rc = refresh_bf16(n);
  if (rc) return rc;
  NCK(cudaStreamSynchronize(n->st));
  return SF_OK;
}

int sf_net_forward(sf_net* n, const float* x, int batch, float* y) {
  if (!n || !x || !y || batch < 1 || batch > n->maxb) return nfail(SF_EINVAL, "bad argument");
  int rc = upload_input(n, x, batch);
  if (!rc) rc = forward(n, batch, true);
  if (rc) return rc;
  n->nb_data = 0;   // act[0] no longer holds the training inputs
  NCK(cudaMemcpyAsync(sf_host_dma(y), n->out, sizeof(float) * batch * n->Z * n->ch[n->nl], cudaMemcpyDeviceToHost, n->st));
  return net_status(n);
}

int sf_net_set_data(sf_net* n, const float* x, const float* target, int batch) {
  if (!n || !x || !target || batch < 1 || batch > n->maxb) return nfail(SF_EINVAL, "bad argument");
  int rc = upload_input(n, x, batch);
  if (rc) return rc;
  NCK(cudaMemcpyAsync(n->tgt, target, sizeof(float) * batch * n->Z * n->ch[n->nl], cudaMemcpyHostToDevice,
                      n->st));
  // the caller may change x and target from here on, page-locked or not
  NCK(cudaStreamSynchronize(n->st));
  n->nb_data = batch;
  return SF_OK;
}

int sf_net_gradient(sf_net* n, float* grad, double* loss) {
  if (!n || n->nb_data < 1) return nfail(SF_ESTATE, "sf_net_set_data first");
  int rc = forward(n, n->nb_data, true);
  if (!rc) rc = backward(n, n->nb_data);
  if (rc) return rc;
  if (grad) NCK(cudaMemcpyAsync(sf_host_dma(grad), n->gr, sizeof(float) * n->nparam, cudaMemcpyDeviceToHost, n->st));
  if (loss) NCK(cudaMemcpyAsync(loss, n->loss, sizeof(double), cudaMemcpyDeviceToHost, n->st));
  return net_status(n);
}

int sf_net_train(sf_net* n, int steps, double lr, double* losses) {
  if (!n || steps < 0) return nfail(SF_EINVAL, "bad argument");
  if (n->nb_data < 1) return nfail(SF_ESTATE, "sf_net_set_data first");
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int s = 0; s < steps; s++) {
    int rc = forward(n, n->nb_data, true);
    if (!rc) rc = backward(n, n->nb_data);
    if (rc) return rc;
    n->t++;
    const float c1 = 1.f - std::pow(b1, (float)n->t), c2 = 1.f - std::pow(b2, (float)n->t);
    k_adam<<<blocks_for(n->nparam, 256), 256, 0, n->st>>>(n->w, n->gr, n->m1, n->m2, n->nparam, (float)lr, b1, b2,
                                                           c1, c2, eps);
    rc = refresh_bf16(n);
    if (rc) return rc;
    if (losses) NCK(cudaMemcpyAsync(losses + s, n->loss, sizeof(double), cudaMemcpyDeviceToHost, n->st));
  }
  return net_status(n);
}

}  // extern "C"
