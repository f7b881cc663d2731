// Ensembles of 2D solvers on different grids (sf_ensemble_*): one RK stage of
// every member in one launch.
//
// Blocks of 12 warps, one per SM, claim work items from counters[0] in order:
// all x-pass items first (largest members first), then all z items. An x item
// is 12 warps' worth of a member's level segments, marched by xmarch_rows
// (sf_xmarch.cuh); a z item is 8 modes of a member, by z_step_f_body
// (sf_zstep_f.cuh) whose 12 warps are 3 fields x 4; a member whose own z kernel
// is k_z_step or k_z_step_tma has z_step_body instead (sf_zstep_k.cuh, 16 modes
// by 12 chunks, at every other item). A z item of member r
// starts once member r's x items have all finished (counters[1 + r] reaches
// xneed[r]). A block claims its next item as it starts the current one, so
// the claim's latency hides behind the work; every wait still ends: an item
// claimed ahead always has a higher index than the claiming block's current
// item, so every x item is being run or is next after an x item being run,
// and x items wait on nothing. The waits are bounded all the same: one that
// runs out sets *err and skips its item. The host clears the counters before
// each step.
//
// 64 runs, N1 in {64, 128, 256}, N3 in {128, 256, 384}, per stage: 153 us (x items
// 70, z items 93, each alone in a launch); with slab x items and one field
// after the other in the z items, two blocks of 8 warps per SM, 243 (135, 108).
#include <algorithm>

#include "sf_xmarch.cuh"
#include "sf_zstep_f.cuh"
#include "sf_zstep_k.cuh"

namespace sf {

constexpr int kEnsWarps = kEnsThreads / 32;
constexpr long long kEnsSpin = 1ll << 24;   // x 64 ns: about a second
static_assert(kEnsThreads == ZfShape<3, 4>::THREADS, "a z item is three fields of four warps");

// warps that march in a block of one grid width (as many as the shared memory takes)
template <int N1>
constexpr int ens_warps() { return std::min(kEnsWarps, XMShape<N1, false, 0, false>::WARPS); }

template <int N1>
__device__ __forceinline__ void ens_x(const StageArgs& a, unsigned char* sm, const EnsItem& it, bool tables) {
  if (tables) {
    xmarch_tables<N1>(sm, a.tw);
    __syncthreads();
  }
  const int w = threadIdx.x >> 5;
  const StageArgs la = a;   // out of shared memory, which the march's stores might alias
  if (w < it.iters) xmarch_rows<N1, false, 0, false>(la, sm, 1, 0, a.g.N3, it.S, it.x + w, it.x + w + 1);
}

__global__ void __launch_bounds__(kEnsThreads, 1) k_ens_stage(const StageArgs* __restrict__ args,
                                                              const EnsItem* __restrict__ xitems, int nx,
                                                              const EnsItem* __restrict__ zitems, int nz,
                                                              int* counters, const int* __restrict__ xneed, int* err) {
  extern __shared__ __align__(16) unsigned char esm[];
  __shared__ __align__(16) StageArgs sa;
  __shared__ int next, have, ok;
  static_assert(sizeof(StageArgs) % sizeof(int) == 0, "StageArgs copied as words");
  if (threadIdx.x == 0) {
    next = atomicAdd(&counters[0], 1);
    have = -1;
  }
  int tables = 0;   // the grid width whose transform tables this block holds
  __syncthreads();
  for (;;) {
    const int i = next;
    if (i >= nx + nz) break;
    const bool xp = i < nx;
    const EnsItem it = xp ? xitems[i] : zitems[i - nx];
    const bool fresh = it.run != have;
    __syncthreads();   // everyone has read next and have
    if (threadIdx.x == 0) {
      next = atomicAdd(&counters[0], 1);
      have = it.run;
      ok = 1;
    }
    if (fresh) {   // this member's stage arguments, copied by the block's threads
      const int* src = reinterpret_cast<const int*>(args + it.run);
      int* dst = reinterpret_cast<int*>(&sa);
      for (int w = threadIdx.x; w < (int)(sizeof(StageArgs) / sizeof(int)); w += blockDim.x) dst[w] = src[w];
    }
    if (!xp && threadIdx.x == 0) {
      const volatile int* done = counters + 1 + it.run;
      long long n = 0;
      while (*done < xneed[it.run] && n < kEnsSpin) {
        __nanosleep(64);
        n++;
      }
      if (*done < xneed[it.run]) {
        ok = 0;
        atomicExch(err, 1);
      }
      __threadfence();   // the member's x-pass results before its z step reads them
    }
    __syncthreads();
    if (xp) {
      const bool fill = sa.g.N1 != tables;
      tables = sa.g.N1;
      switch (sa.g.N1) {
        case 16: ens_x<16>(sa, esm, it, fill); break;
        case 32: ens_x<32>(sa, esm, it, fill); break;
        case 64: ens_x<64>(sa, esm, it, fill); break;
        case 128: ens_x<128>(sa, esm, it, fill); break;
        case 256: ens_x<256>(sa, esm, it, fill); break;
        case 512: ens_x<512>(sa, esm, it, fill); break;
        default: break;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();   // this item's r rows, before it counts as done
        atomicAdd(&counters[1 + it.run], 1);
      }
    } else if (ok && sa.zkernel != 2) {   // the member asks for the other z kernels' solves
      tables = 0;
      const int N3 = sa.g.N3, per = N3 <= kEnsFusedN3 ? 2 : 1;   // items per 16 modes
      if (it.x % per == 0) {
        if ((N3 + kEnsWarps - 1) / kEnsWarps >= 48) z_step_body<kEnsWarps, true>(sa, it.x / per, 0);
        else z_step_body<kEnsWarps, false>(sa, it.x / per, 0);
      }
    } else if (ok) {   // the shapes of k_z_step_f that 12 warps make (sf_zstep3.cu), else k_z_step_c's
      tables = 0;
      const int N3 = sa.g.N3;
      const StageArgs la = sa;   // as in ens_x
      if (N3 <= 64) z_step_f_body<3, 4, 4, 2, 4, false, false, false>(la, it.x, 0);
      else if (N3 <= kEnsFusedN3) z_step_f_body<3, 4, 0, 12, 4, true, true, false>(la, it.x, 0);
      else z_step_c_body<2 * kEnsWarps, true>(sa, it.x, 0);
    }
    __syncthreads();
  }
}

// modes per z item of a member
int ensemble_z_modes(int N3) { return N3 <= kEnsFusedN3 ? kFM : 16; }

// x items of a member: warps of an item, and segments per warp
int ensemble_x_warps(int N1) {
  switch (N1) {
    case 16: return ens_warps<16>();
    case 32: return ens_warps<32>();
    case 64: return ens_warps<64>();
    case 128: return ens_warps<128>();
    case 256: return ens_warps<256>();
    default: return ens_warps<512>();
  }
}
int ensemble_x_rows(int N1) {
  switch (N1) {
    case 16: return XMT<16>::W;
    case 32: return XMT<32>::W;
    case 64: return XMT<64>::W;
    case 128: return XMT<128>::W;
    default: return 1;
  }
}

size_t ensemble_smem(int N1, int N3) {
  size_t x = 0;
  switch (N1) {
    case 16: x = XMShape<16, false, 0, false>::smem(ens_warps<16>()); break;
    case 32: x = XMShape<32, false, 0, false>::smem(ens_warps<32>()); break;
    case 64: x = XMShape<64, false, 0, false>::smem(ens_warps<64>()); break;
    case 128: x = XMShape<128, false, 0, false>::smem(ens_warps<128>()); break;
    case 256: x = XMShape<256, false, 0, false>::smem(ens_warps<256>()); break;
    default: x = XMShape<512, false, 0, false>::smem(ens_warps<512>()); break;
  }
  const size_t z = N3 > kEnsFusedN3 ? zc_smem_bytes<2 * kEnsWarps>(N3)
                                    : ZfShape<3, 4>::smem(N3, N3 > 64, N3 > 64);
  const size_t k = sizeof(float) * ((size_t)N3 * 32 + 3 * kEnsWarps * 32);   // z_step_body
  return std::max(x, std::max(z, k));
}

int launch_ens_stage(const StageArgs* args, const EnsItem* xitems, int nx, const EnsItem* zitems, int nz,
                     int* counters, const int* xneed, int* err, int blocks, size_t smem, cudaStream_t st) {
  k_ens_stage<<<blocks, kEnsThreads, smem, st>>>(args, xitems, nx, zitems, nz, counters, xneed, err);
  return 1;
}
int ensemble_stage_blocks() { return sm_count(); }

int prepare_ensemble_kernels() {
  const int lim = 227 * 1024 - (int)sizeof(StageArgs) - 64;
  return cudaFuncSetAttribute(k_ens_stage, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) == cudaSuccess ? 0 : -1;
}

}  // namespace sf
