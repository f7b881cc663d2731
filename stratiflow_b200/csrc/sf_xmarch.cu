// The x pass as level-marching lane groups (BuildRHS, IMEXRK.cpp:136-193:
// ToNodal's x part, the nodal products, ToModal's x part with 1/(N1 N2) and the
// 2/3 truncation, then the x derivatives and the z stencils that follow each
// product; and the same about a base flow).
//
// One lane group (XMT<N1>::G lanes) owns one row, a y row in 3D, and walks up a
// range of z levels. At level t it inverse-transforms the fields of level t
// (u1 + i u3 and b + i u2, packed as one two-transform pair, sf_xmt.cuh), keeps
// them in registers and the fields of level t-1 in its own shared memory, forms
// the eleven products of level t (with P4 of level t-1, the one product that
// needs u3 of the level above), forward-transforms them as three packed pairs
// and finishes the combinations:
//   level t-1: c1, cB, c2 get their ddz(D->N) term from Q1, QB, Q2 of level t,
//              c3 its ddz(N->D) term from P4 of level t-1; written out;
//   level t:   c1y, c2y, c3y, cBy written out; c1, cB, c2, c3 started and
//              carried to the next level.
// The nodal values a lane forms after the inverse transform are those of the
// x positions it feeds into the forward transforms, so the products need no
// exchange between lanes; the only shared memory traffic is the transforms'
// transposes, the level below and the staged input rows. No block-wide barrier
// after set-up: the groups of a warp march in step, warps are independent.
//
// The shared-memory pipe bounds it (81 % busy at 256x128x384). So the
// nonlinear step carries its combinations in registers where a lane keeps three
// modes or fewer, and forms the first batch of products from the inverse
// transform's own registers: 230 us a stage with both in shared memory, 208
// with the first, 197 with both; 2 x 128x64x180: 66, 61, 58; 32 x 256x256 in 2D:
// 43, 41, 36. The linear and tangent modes need the base flow's registers too:
// carried there as well, they gained 3 % at some sizes and lost 4 % at others.
#include "sf_xmarch.cuh"

namespace sf {

// the units split evenly over the launch's warps
template <int N1, bool D3, int MODE>
__global__ void __launch_bounds__(XMShape<N1, D3, MODE>::WARPS * 32, 1) k_xmarch(const __grid_constant__ StageArgs a, int nruns,
                                                                         int t_lo, int t_hi, int seg) {
  constexpr int W = XMT<N1>::W;
  extern __shared__ __align__(16) unsigned char xsm[];
  xmarch_tables<N1>(xsm, a.tw);
  chain_begin();
  __syncthreads();
  const int L = t_hi - t_lo, nwarps = blockDim.x >> 5;
  const long long NW = (long long)gridDim.x * nwarps, wid = (long long)blockIdx.x * nwarps + (threadIdx.x >> 5);
  const long long U = D3 ? (long long)nruns * (a.g.N2 / W) * L : ((long long)nruns * ((L + seg - 1) / seg) + W - 1) / W;
  xmarch_rows<N1, D3, MODE>(a, xsm, nruns, t_lo, t_hi, seg, U * wid / NW, U * (wid + 1) / NW);
}

template <int N1, bool D3, int MODE>
static void xmarch_launch(const StageArgs& a, int nruns, int t_lo, int t_hi, cudaStream_t st) {
  using X = XMShape<N1, D3, MODE>;
  const int nsm = sm_count();
  if (D3) {
    launch_chained(k_xmarch<N1, D3, MODE>, dim3(nsm), X::WARPS * 32, X::smem(X::WARPS), st, a.chained, a, nruns, t_lo, t_hi, 0);
    return;
  }
  // 2D: the shortest segments that all the launch's groups together hold at
  // once, spread over the SMs
  const long long L = t_hi - t_lo, room = (long long)nsm * X::WARPS * X::W;
  const int seg = (int)((nruns * L + room - 1) / room);
  const long long warps = (nruns * ((L + seg - 1) / seg) + X::W - 1) / X::W;
  const int wb = (int)std::min<long long>(X::WARPS, (warps + nsm - 1) / nsm);
  launch_chained(k_xmarch<N1, D3, MODE>, dim3((unsigned)((warps + wb - 1) / wb)), wb * 32, X::smem(wb), st, a.chained, a, nruns,
                 t_lo, t_hi, seg);
}

// mode 0 nonlinear, 1 frozen base, 2 live base. 3D: every grid whose row has a
// shape here. 2D: where the slab kernel's blocks do not spread a few levels over
// more SMs, from 2^17 points of the launch's runs, 2^13 at N1 = 128, whose rows
// march two to a warp at 8 points a lane; always in mode 1, whose slabs copy the base's
// rows as well. Near 2^17 points the two are even. Measured, a whole step (us), slab and march:
//   N1 = 128      64 levels 37.8 36.9; 128 levels 47.1 45.1; 4 x 256 76.7 72.4; 1 + 2 tangents, 128 levels 83.4 73.8
//   others        64x64 32.8 34.9; 256x64 36.9 38.9; 64x64 x 4 33.8 36.9; 256x128 47.1 49.5; 64x128 x 8 45.1 46.0;
//                 256x256 x 2 75.8 75.8; 256x256 x 3 79.9 80.7; 512x388 110.9 107.6; 32x256 x 16 71.7 69.7
// and per launch:
//   2D nonlinear  4 x 256x256 17.9 15.8; 16 x 64x256 20.9 14.0; 6 x 512x388 57.6 36.5; 32 x 256x256 61.0 37.8
//   2D frozen     1 x 64x64 13.5 13.2; 1 x 128x128 15.9 13.8; 4 x 256x256 29.0 17.8
//   2D live base  1 + 2 x 512x200 55.0 54.8; 1 + 4 x 256x256 40.6 29.9
//   3D            2 x 128x64x180 131 58; frozen 2 x 128x64x192 258 95; frozen 256x64x128 172 68
bool xmarch_supported(const StageArgs& a, int mode, int nruns) {
  const Geo& g = a.g;
  if (a.adjoint) return false;
  const int N1 = g.N1;
  if (g.dim3) return (N1 == 64 || N1 == 128 || N1 == 256) && g.N2 % 4 == 0;
  return N1 <= 512 && (mode == 1 || (long long)N1 * g.N3 * nruns >= (N1 == 128 ? 1 << 13 : 1 << 17));
}

template <int N1, bool D3>
static void xmarch_mode(const StageArgs& a, int mode, int nruns, int t_lo, int t_hi, cudaStream_t st) {
  switch (mode) {
    case 0: xmarch_launch<N1, D3, 0>(a, nruns, t_lo, t_hi, st); break;
    case 1: xmarch_launch<N1, D3, 1>(a, nruns, t_lo, t_hi, st); break;
    default: xmarch_launch<N1, D3, 2>(a, nruns, t_lo, t_hi, st); break;
  }
}

int launch_xmarch(const StageArgs& a, int mode, int nruns, int t_lo, int t_hi, cudaStream_t st) {
  const bool d3 = a.g.dim3 != 0;
  switch (a.g.N1) {
    case 16: xmarch_mode<16, false>(a, mode, nruns, t_lo, t_hi, st); break;
    case 32: xmarch_mode<32, false>(a, mode, nruns, t_lo, t_hi, st); break;
    case 64: d3 ? xmarch_mode<64, true>(a, mode, nruns, t_lo, t_hi, st) : xmarch_mode<64, false>(a, mode, nruns, t_lo, t_hi, st); break;
    case 128: d3 ? xmarch_mode<128, true>(a, mode, nruns, t_lo, t_hi, st) : xmarch_mode<128, false>(a, mode, nruns, t_lo, t_hi, st); break;
    case 256: d3 ? xmarch_mode<256, true>(a, mode, nruns, t_lo, t_hi, st) : xmarch_mode<256, false>(a, mode, nruns, t_lo, t_hi, st); break;
    case 512: xmarch_mode<512, false>(a, mode, nruns, t_lo, t_hi, st); break;
    default: return 0;
  }
  return 1;
}

template <int N1, bool D3>
static cudaError_t xmarch_attr() {
  cudaError_t e = cudaFuncSetAttribute(k_xmarch<N1, D3, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)XMShape<N1, D3, 0>::smem(XMShape<N1, D3, 0>::WARPS));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_xmarch<N1, D3, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)XMShape<N1, D3, 1>::smem(XMShape<N1, D3, 1>::WARPS));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_xmarch<N1, D3, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)XMShape<N1, D3, 2>::smem(XMShape<N1, D3, 2>::WARPS));
  return e;
}
int prepare_xmarch_kernels() {
  for (cudaError_t e : {xmarch_attr<64, true>(), xmarch_attr<128, true>(), xmarch_attr<256, true>(),
                        xmarch_attr<16, false>(), xmarch_attr<32, false>(), xmarch_attr<64, false>(), xmarch_attr<128, false>(),
                        xmarch_attr<256, false>(), xmarch_attr<512, false>()})
    if (e != cudaSuccess) return -1;
  return 0;
}

}  // namespace sf
