// The z pass with one lane per real component, a field after the other: the
// device code of k_z_step and k_z_proj_chunked (sf_kernels.cu), shared with
// the ensembles' stage kernel (sf_ens.cu) for members that ask for it.
#pragma once
#include <climits>

#include "sf_internal.cuh"

namespace sf {

constexpr int kZU = 8;   // levels of every input loaded ahead per thread

// ------------------------------------------------ chunked z solves ----
// The Thomas sweeps are first-order affine recurrences: D_j = al_j D_{j-1} +
// be_j (al_j = -a_j/den_j, be_j = R_j/den_j) upward, x_j = D_j - C_j x_{j+1}
// downward. A block of ZW warps (8, or 16 for grids too small to fill the
// GPU) splits N3 into ZW z-chunks, one per warp,
// and covers 16 modes x {real, imag} per warp: every chunk composes its
// affine map, one warp scans the ZW maps in z order, and every chunk then
// replays its levels from the right incoming value. be_j and D_j stay in
// shared memory ([N3][32] floats per block). The result equals the sequential
// sweep up to rounding.
constexpr int kZU2 = 4;   // levels of every input loaded ahead in the chunked z kernels' first sweep
constexpr int kZI = 16;   // levels of inverse pivots loaded ahead in their later sweeps
constexpr int kZP = 4;    // levels of the fields loaded ahead in the projection's last sweep

template <int ZW>
__device__ __forceinline__ void zscan_up(float* sA, float* sB, float* sIn, int w, int lane, float A, float B) {
  sA[w * 32 + lane] = A;
  sB[w * 32 + lane] = B;
  __syncthreads();
  if (w == 0) {
    float v = 0.f;
    for (int k = 0; k < ZW; k++) {
      sIn[k * 32 + lane] = v;
      v = sA[k * 32 + lane] * v + sB[k * 32 + lane];
    }
  }
  __syncthreads();
}
template <int ZW>
__device__ __forceinline__ void zscan_down(float* sA, float* sB, float* sIn, int w, int lane, float A, float B) {
  sA[w * 32 + lane] = A;
  sB[w * 32 + lane] = B;
  __syncthreads();
  if (w == 0) {
    float v = 0.f;
    for (int k = ZW - 1; k >= 0; k--) {
      sIn[k * 32 + lane] = v;
      v = sA[k * 32 + lane] * v + sB[k * 32 + lane];
    }
  }
  __syncthreads();
}

// the inverse pivots of levels j0, j0 + step, ... (K of them, those in
// [lo, hi)) loaded ahead of their use in the serial sweeps
template <int K>
__device__ __forceinline__ void load_iden(float (&bi)[K], const float* __restrict__ iden, int Pp, int j0, int step,
                                          int lo, int hi) {
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int j = j0 + step * i;
    bi[i] = (j >= lo && j < hi) ? iden[(size_t)j * Pp] : 0.f;
  }
}

// the CN solve of k_z_step for field f of family FAM (0: u1 and u2,
// 1: u3, Dirichlet; 2: b), so that each family's loads and terms are fixed
// at compile time; IC: chunks clear of the ends take sweeps without the
// per-level end tests
template <int ZW, int FAM, bool IC>
__device__ __forceinline__ void z_cn_body(const StageArgs& a, const int f, const int bx, const int bz) {
  const Geo g = a.g;
  extern __shared__ float zsm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int m0 = bx * 16 + (lane >> 1), c = lane & 1;
  const bool act = m0 < g.P;
  const int m = act ? m0 : 0;
  const int run = bz;
  const int N3 = g.N3, Pp = g.Pp;
  const int chunk = (N3 + ZW - 1) / ZW;
  const int js = min(N3, w * chunk), je = min(N3, js + chunk);
  float* sD = zsm;                      // [N3][32]: be_j, then D_j
  float* sA = zsm + (size_t)N3 * 32;    // [ZW][32]
  float* sB = sA + ZW * 32;
  float* sIn = sB + ZW * 32;
  const int q = m / g.K1, j1 = m - q * g.K1;
  const float kxv = a.kx[j1], kyv = a.ky[q];
  const float d1 = -(kxv * kxv), d2 = -(kyv * kyv);
  const float sc = c == 0 ? -1.f : 1.f;   // (i k z)_c = sc * k * z_{1-c}
  constexpr bool dir = (FAM == 1);
  const int fs = (FAM == 2 ? 1 : (dir ? 2 : 0)) * 3 + a.stage;   // factor sets: velocity, buoyancy, u3
  const float* __restrict__ fa = a.fa + (size_t)fs * N3;
  const float* __restrict__ fc = a.fc + (size_t)fs * N3;
  const float* __restrict__ iden = a.inv_den + (size_t)fs * N3 * Pp + m;
  const float* __restrict__ zc = a.zc;
  const float* __restrict__ lo2 = zc + (dir ? ZC_D2D_LO : ZC_D2N_LO) * N3;
  const float* __restrict__ di2 = zc + (dir ? ZC_D2D_DI : ZC_D2N_DI) * N3;
  const float* __restrict__ up2 = zc + (dir ? ZC_D2D_UP : ZC_D2N_UP) * N3;
  const float* __restrict__ dnd_lo = zc + ZC_DND_LO * N3;
  const float* __restrict__ dnd_di = zc + ZC_DND_DI * N3;
  const float* __restrict__ full_lo = zc + ZC_FULL_LO * N3;
  const float* __restrict__ full_di = zc + ZC_FULL_DI * N3;
  const float cco = (FAM == 2) ? a.cb : a.cv;
  const float Ri = a.Ri[run];
  const float* __restrict__ dB = a.dBdz + (size_t)run * N3;
  const bool zmode = (m == 0);   // the (0,0) mode: no buoyancy force (IMEXRK.cpp:141-143)
  const size_t fo = (size_t)(run * 5 + f) * N3 * Pp + m;
  const float* uc = reinterpret_cast<const float*>(a.S + fo) + c;
  const float* pc = reinterpret_cast<const float*>(a.S + (size_t)(run * 5 + 4) * N3 * Pp + m) + c;
  const float* po = reinterpret_cast<const float*>(a.S + (size_t)(run * 5 + 4) * N3 * Pp + m) + (1 - c);
  const float* bc = reinterpret_cast<const float*>(a.S + (size_t)(run * 5 + 3) * N3 * Pp + m) + c;
  const float* wc = reinterpret_cast<const float*>(a.S + (size_t)(run * 5 + 2) * N3 * Pp + m) + c;
  const float* rc = reinterpret_cast<const float*>(a.rnl + (size_t)(run * 4 + f) * N3 * Pp + m) + c;
  float* rold = reinterpret_cast<float*>(a.rold + (size_t)(run * 4 + f) * N3 * Pp + m) + c;
  float* out = reinterpret_cast<float*>(a.Sn + fo) + c;
  const bool use_rold = (a.hz != 0.f);
  const float kgrad = (f == 0) ? kxv : kyv;
  const size_t S2 = 2 * (size_t)Pp;

  // ---- forward, pass 1: right-hand side, be_j, chunk map ----
  float um = js >= 1 && js < N3 ? uc[(js - 1) * S2] : 0.f;
  float u0 = js < N3 ? uc[js * S2] : 0.f;
  float pm1 = (FAM == 1 && js >= 1 && js < N3) ? pc[(js - 1) * S2] : 0.f;
  float bm1 = (FAM == 1 && js >= 1 && js < N3) ? bc[(js - 1) * S2] : 0.f;
  float w0 = (FAM == 2 && js < N3) ? wc[js * S2] : 0.f;
  float A = 1.f, B = 0.f;
  // a chunk clear of both ends (levels 3..N3-4) and a whole number of batches
  // of each sweep takes the sweeps without the per-level end tests
  const bool interior = IC && js >= 3 && je <= N3 - 4 && (je - js) % kZI == 0;
  static_assert(kZI % kZU2 == 0, "the first sweep's batches tile the later sweeps'");
  auto sweep1 = [&](auto tag) {
  constexpr bool IN = decltype(tag)::value;
  for (int j0 = js; j0 < je; j0 += kZU2) {
    float bu[kZU2], br[kZU2], bo[kZU2], bp[kZU2], bx[kZU2], bi[kZU2];
#pragma unroll
    for (int i = 0; i < kZU2; i++) {
      const int j = j0 + i;
      const bool in = IN || j < je, nx = IN || (j + 1 < N3 && in);
      bu[i] = nx ? uc[(j + 1) * S2] : 0.f;
      br[i] = in ? rc[j * S2] : 0.f;
      bo[i] = (in && use_rold) ? rold[j * S2] : 0.f;
      bi[i] = in ? iden[(size_t)j * Pp] : 0.f;
      bp[i] = 0.f;
      bx[i] = 0.f;
      if (FAM == 0) bp[i] = in ? po[j * S2] : 0.f;
      if (FAM == 1) {
        bp[i] = in ? pc[j * S2] : 0.f;
        bx[i] = in ? bc[j * S2] : 0.f;
      }
      if (FAM == 2) bx[i] = nx ? wc[(j + 1) * S2] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kZU2; i++) {
      const int j = j0 + i;
      if (!IN && j >= je) break;
      const float up = bu[i];
      float rt = br[i];
      float gp = 0.f;
      if (FAM == 0) {
        gp = sc * kgrad * bp[i];   // (i k p)_c
      } else if (FAM == 1) {
        if (IN || j >= 2) gp = dnd_lo[j] * pm1 + dnd_di[j] * bp[i];
        pm1 = bp[i];
        if ((IN || j >= 1) && !zmode && !a.adjoint) rt += Ri * (full_lo[j] * bm1 + full_di[j] * bx[i]);   // r3 += Ri Full(b - <b>)
        bm1 = bx[i];
      } else {
        const float w1 = bx[i];
        const float dw = (IN || j + 1 < N3) ? 0.5f * w0 + 0.5f * w1 : 0.5f * w0;
        if (!a.adjoint) rt -= dB[j] * dw;   // rB -= dB/dz ReinterpolateDirichlet(u3)
        w0 = w1;
      }
      float R = u0;
      if (use_rold) R += a.hz * bo[i];
      R += -a.h * gp;
      R += a.hb * rt;
      const bool band = IN || (dir ? (j >= 2 && j <= N3 - 2) : (j >= 1 && j <= N3 - 2));
      const float d2u = band ? lo2[j] * um + di2[j] * u0 + up2[j] * up : 0.f;
      R += cco * ((d1 * u0 + d2 * u0) + d2u);
      const bool zend = !IN && ((j <= 1) || (j >= N3 - 2) || (dir && j == 2));   // ZeroEnds (Field.h:475-486)
      if (zend) R = 0.f;
      const float be = R * bi[i];
      const float al = (!IN && j == 0) ? 0.f : -fa[j] * bi[i];
      sD[j * 32 + lane] = be;
      if (act) rold[j * S2] = rt;
      A = al * A;
      B = al * B + be;
      um = u0;
      u0 = up;
    }
  }
  };
  if (interior) sweep1(std::true_type{});
  else sweep1(std::false_type{});
  zscan_up<ZW>(sA, sB, sIn, w, lane, A, B);
  // ---- forward, pass 2: D_j, and with it the chunk map of the backward
  // sweep x_j = D_j - C_j x_{j+1}, composed upwards: x_js = B + A x_je ----
  float D = sIn[w * 32 + lane];
  A = 1.f;
  B = 0.f;
  auto sweep2 = [&](auto tag) {
    constexpr bool IN = decltype(tag)::value;
    for (int j0 = js; j0 < je; j0 += kZI) {
      float bi[kZI];
      load_iden(bi, iden, Pp, j0, 1, IN ? INT_MIN : js, IN ? INT_MAX : je);
#pragma unroll
      for (int i = 0; i < kZI; i++) {
        const int j = j0 + i;
        if (!IN && j >= je) break;
        const float al = (!IN && j == 0) ? 0.f : -fa[j] * bi[i];
        D = al * D + sD[j * 32 + lane];
        sD[j * 32 + lane] = D;
        B = B + A * D;
        A = -A * (fc[j] * bi[i]);
      }
    }
  };
  if (interior) sweep2(std::true_type{});
  else sweep2(std::false_type{});
  __syncthreads();
  zscan_down<ZW>(sA, sB, sIn, w, lane, A, B);
  // ---- backward, pass 2: the solution ----
  float x = sIn[w * 32 + lane];
  auto sweep3 = [&](auto tag) {
    constexpr bool IN = decltype(tag)::value;
    for (int j0 = je - 1; j0 >= js; j0 -= kZI) {
      float bi[kZI];
      load_iden(bi, iden, Pp, j0, -1, IN ? INT_MIN : js, IN ? INT_MAX : je);
#pragma unroll
      for (int i = 0; i < kZI; i++) {
        const int j = j0 - i;
        if (!IN && j < js) break;
        const float Cj = fc[j] * bi[i];
        x = sD[j * 32 + lane] - Cj * x;
        if (act) out[j * S2] = x;
      }
    }
  };
  if (interior) sweep3(std::true_type{});
  else sweep3(std::false_type{});
}

// RemoveDivergence with the chunked solve, for 16 modes per block: the
// divergence and the Laplacian factors upward, q downward, then u -= grad q
// and p += pm q. The two components of a mode are adjacent lanes and
// exchange q; u3_{j+1} at a chunk's top uses the next chunk's q from the scan.
template <int ZW>
__device__ __forceinline__ void z_proj_body(const Geo& g, float2* U, const float2* Psrc, float2* Pdst,
                                            const float* zc, const float* fa, const float* fc,
                                            const float* inv_den, const float* kx, const float* ky, float pm,
                                            const int bx, const int bz) {
  extern __shared__ float zsm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int m0 = bx * 16 + (lane >> 1), c = lane & 1;
  const bool act = m0 < g.P;
  const int m = act ? m0 : 0;
  const int run = bz;
  const int N3 = g.N3, Pp = g.Pp;
  const int chunk = (N3 + ZW - 1) / ZW;
  const int js = min(N3, w * chunk), je = min(N3, js + chunk);
  float* sD = zsm;
  float* sA = zsm + (size_t)N3 * 32;
  float* sB = sA + ZW * 32;
  float* sIn = sB + ZW * 32;
  const int q = m / g.K1, j1 = m - q * g.K1;
  const float kxv = kx[j1], kyv = g.dim3 ? ky[q] : 0.f;
  const float sc = c == 0 ? -1.f : 1.f;
  const size_t S2 = 2 * (size_t)Pp;
  float* u1 = reinterpret_cast<float*>(U + (size_t)(run * 5 + 0) * N3 * Pp + m);
  float* u2 = reinterpret_cast<float*>(U + (size_t)(run * 5 + 1) * N3 * Pp + m);
  float* u3 = reinterpret_cast<float*>(U + (size_t)(run * 5 + 2) * N3 * Pp + m) + c;
  const float* ps = reinterpret_cast<const float*>(Psrc + (size_t)(run * 5 + 4) * N3 * Pp + m) + c;
  float* pd = reinterpret_cast<float*>(Pdst + (size_t)(run * 5 + 4) * N3 * Pp + m) + c;
  const float* __restrict__ a_ = fa + (size_t)kFS_Lap * N3;
  const float* __restrict__ c_ = fc + (size_t)kFS_Lap * N3;
  const float* __restrict__ iden = inv_den + (size_t)kFS_Lap * N3 * Pp + m;
  const float* __restrict__ ddn_di = zc + ZC_DDN_DI * N3;
  const float* __restrict__ ddn_up = zc + ZC_DDN_UP * N3;
  const float* __restrict__ dnd_lo = zc + ZC_DND_LO * N3;
  const float* __restrict__ dnd_di = zc + ZC_DND_DI * N3;
  const float* u1o = u1 + (1 - c);   // u1_{1-c}
  const float* u2o = u2 + (1 - c);
  float* u1c = u1 + c;
  float* u2c = u2 + c;

  // ---- forward, pass 1: divergence, be_j, chunk map ----
  float w0 = js < N3 ? u3[js * S2] : 0.f;
  float A = 1.f, B = 0.f;
  for (int j0 = js; j0 < je; j0 += kZU) {
    float b1[kZU], b2[kZU], b3[kZU], bi[kZU];
#pragma unroll
    for (int i = 0; i < kZU; i++) {
      const int j = j0 + i;
      const bool in = j < je;
      b1[i] = in ? u1o[j * S2] : 0.f;
      b2[i] = (in && g.dim3) ? u2o[j * S2] : 0.f;
      b3[i] = (in && j + 1 < N3) ? u3[(j + 1) * S2] : 0.f;
      bi[i] = in ? iden[(size_t)j * Pp] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kZU; i++) {
      const int j = j0 + i;
      if (j >= je) break;
      const float w1 = b3[i];
      float dv = 0.f;
      if (j >= 2 && j <= N3 - 3) dv = sc * (kxv * b1[i] + kyv * b2[i]) + (ddn_di[j] * w0 + ddn_up[j] * w1);
      const float be = dv * bi[i];
      const float al = (j == 0) ? 0.f : -a_[j] * bi[i];
      sD[j * 32 + lane] = be;
      A = al * A;
      B = al * B + be;
      w0 = w1;
    }
  }
  zscan_up<ZW>(sA, sB, sIn, w, lane, A, B);
  // D_j, and with it the chunk map of the backward sweep, composed upwards
  auto Cof = [&](int j, float bij) {
    float Cj = c_[j] * bij;
    if (m == 0 && j == 1) Cj = 0.f;   // (0,0) mode: row 1 pinned (IMEXRK.h:68-74)
    return Cj;
  };
  float D = sIn[w * 32 + lane];
  A = 1.f;
  B = 0.f;
  for (int j0 = js; j0 < je; j0 += kZI) {
    float bi[kZI];
    load_iden(bi, iden, Pp, j0, 1, js, je);
#pragma unroll
    for (int i = 0; i < kZI; i++) {
      const int j = j0 + i;
      if (j >= je) break;
      const float al = (j == 0) ? 0.f : -a_[j] * bi[i];
      D = al * D + sD[j * 32 + lane];
      sD[j * 32 + lane] = D;
      B = B + A * D;
      A = -A * Cof(j, bi[i]);
    }
  }
  __syncthreads();
  zscan_down<ZW>(sA, sB, sIn, w, lane, A, B);
  // ---- backward, pass 2: q_j, projection, p ----
  float qn = sIn[w * 32 + lane];   // q at level je (0 above the top)
  // every row of u1, u2, u3, p is written once, by the step of one level,
  // so the loads of a batch may all go ahead of its stores
  for (int j0 = je - 1; j0 >= js; j0 -= kZP) {
    float bi[kZP], pv[kZP], v1[kZP], v2[kZP], v3[kZP];
    load_iden(bi, iden, Pp, j0, -1, js, je);
#pragma unroll
    for (int i = 0; i < kZP; i++) {
      const int j = j0 - i, jj = j + 1;
      const bool in = j >= js && act;
      pv[i] = in ? ps[j * S2] : 0.f;
      v1[i] = in ? u1c[j * S2] : 0.f;
      v2[i] = (in && g.dim3) ? u2c[j * S2] : 0.f;
      v3[i] = (in && jj >= 2 && jj <= N3 - 1) ? u3[jj * S2] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kZP; i++) {
      const int j = j0 - i;
      if (j < js) break;
      const float qj = sD[j * 32 + lane] - Cof(j, bi[i]) * qn;
      const float qo = __shfl_xor_sync(0xffffffffu, qj, 1);
      if (act) {
        u1c[j * S2] = v1[i] - sc * kxv * qo;
        if (g.dim3) u2c[j * S2] = v2[i] - sc * kyv * qo;
        pd[j * S2] = pv[i] + pm * qj;
        const int jj = j + 1;   // u3_{j+1} -= ddz(q)_{j+1}, rows 2..N-1
        if (jj >= 2 && jj <= N3 - 1) u3[jj * S2] = v3[i] - (dnd_lo[jj] * qj + dnd_di[jj] * qn);
      }
      qn = qj;
    }
  }
}

// The whole z pass of a stage for 16 modes per block: the CN solves of every
// field (ExplicitRK, linear buoyancy terms, FinishRHS, CrankNicolson and the
// Thomas solve, IMEXRK.cpp:75-134), then RemoveDivergence on the new
// velocities (IMEXRK.cpp:43-73). The projection reads the velocities this
// block has just written (visible to the block after the barrier, and still
// in L2), so the pass makes one trip through HBM instead of two kernels'.
// Every field's solve uses the same shared-memory rows: a thread reads and
// writes only its own rows of sD, and the chunk scans synchronise the block.
template <int ZW, bool IC>
__device__ __forceinline__ void z_step_body(const StageArgs& a, const int bx, const int bz) {
  if (a.g.dim3) {
    z_cn_body<ZW, 0, IC>(a, 0, bx, bz);
    z_cn_body<ZW, 0, IC>(a, 1, bx, bz);
  } else {
    z_cn_body<ZW, 0, IC>(a, 0, bx, bz);
  }
  z_cn_body<ZW, 1, IC>(a, 2, bx, bz);
  z_cn_body<ZW, 2, IC>(a, 3, bx, bz);
  __syncthreads();
  z_proj_body<ZW>(a.g, a.Sn, a.S, a.Sn, a.zc, a.fa, a.fc, a.inv_den, a.kx, a.ky, a.pm, bx, bz);
}

}  // namespace sf
