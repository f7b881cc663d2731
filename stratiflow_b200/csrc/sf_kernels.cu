// CUDA kernels of one IMEX-RK stage (IMEXRK.cpp:8-24 / 26-41) for sm_100a.
//
// A stage runs as
//   [3D] k_ifft_y   modal u1,u2,u3,b -> (kx, y) rows          (ModalField::ToNodal, y part)
//        k_xmarch   (sf_xmarch.cu; small 2D launches: k_xpass, per y row and
//                   slab of z levels): c2r along x, the nodal products of
//                   BuildRHS / BuildRHSLinear, r2c along x, 1/(N1 N2), 2/3
//                   truncation and the z stencils and x-derivatives that
//                   follow each product
//   [3D] k_fft_y    (kx, y) -> (kx, ky), y-derivatives, sum into r
//        k_z_step_f (sf_zstep3.cu; also k_z_step here and sf_zstep*.cu) per group
//                   of modes: for every field ExplicitRK + linear buoyancy terms
//                   + FinishRHS + CrankNicolson right-hand side + Thomas solve,
//                   then the divergence, Laplacian solve, projection and p
//                   update (k_z_proj_chunked alone serves RemoveDivergence
//                   outside a step)
// Every kernel touches only kept (dealiased) modes, which is all the reference's
// ModalField arithmetic touches (Field.h:1129-1166).

#include <algorithm>
#include <climits>
#include <type_traits>
#include "sf_internal.cuh"
#include "sf_fft.cuh"
#include "sf_fft2.cuh"
#include "sf_zstep_c.cuh"
#include "sf_zstep_k.cuh"

namespace sf {

// ===================================================== y transforms (3D) ====
constexpr int kYThreads = 128;

__device__ __forceinline__ int n2_of_q(int q, int Ky, int K2, int N2) { return q < Ky ? q : q + N2 - K2; }

// kx columns handled by one block of the y transforms: one per lane group
template <int N2>
__host__ __device__ constexpr int ycols() { return (kYThreads / 32) * (32 / FFTShape<N2>::G); }

// the same in the pair kernels
template <int N2>
__host__ __device__ constexpr int ypcols() { return (kYThreads / 32) * (32 / YT<N2>::G); }

// modal [q][j1] of (run, field f, level j) -> plain rows [y][j1] of that field,
// inverse c2c in y (the nodal fields of files, bases and diagnostics). One lane
// group per kx column; consecutive columns in consecutive groups so that a
// warp's loads of one y row cover whole 32-byte sectors.
template <int N2>
__global__ void __launch_bounds__(kYThreads, 8) k_ifft_y(StageArgs a) {
  constexpr int G = FFTShape<N2>::G, E = FFTShape<N2>::E, BUF = fft_buf_stride<N2>();
  const Geo g = a.g;
  __shared__ float2 fbuf[(kYThreads / G) * BUF];
  const int lane = threadIdx.x & 31, grp = threadIdx.x / G, l = threadIdx.x % G;
  const int j1 = blockIdx.x * ycols<N2>() + grp;
  const int j = blockIdx.y + a.lvl0;
  const int run = blockIdx.z >> 2, f = blockIdx.z & 3;
  const bool act = j1 < g.K1;
  const float2* src = a.S + ((size_t)(run * 5 + f) * g.N3 + j) * g.Pp;
  float2 x[E];
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int n2 = l + G * e;
    // kept rows: ky = 0..Ky-1 at n2 < Ky, ky = -(Ky-1)..-1 at n2 > N2 - Ky
    int q = -1;
    if (n2 < g.Ky) q = n2;
    else if (n2 > N2 - g.Ky) q = n2 - (N2 - g.K2);
    x[e] = (act && q >= 0) ? src[q * g.K1 + j1] : make_float2(0.f, 0.f);
  }
  (void)lane;
  reg_fft<N2, true>(x, fbuf + (threadIdx.x / G) * BUF, a.tw, l);
  if (act) {
    float2* dst = a.mixin + ((size_t)(run * 4 + f) * g.N3 + j) * N2 * g.K1 + j1;
#pragma unroll
    for (int sl = 0; sl < E; sl++) dst[(size_t)reg_fft_out_index<N2>(l, sl) * g.K1] = x[sl];
  }
}

// The same for the field pairs of every run (blockIdx.z = 2 run + p; p = 0
// (u1, u3), p = 1 (b, u2)): each lane group transforms its column of both
// fields as one packed pair of transforms (sf_fft2.cuh), half the FP32
// instructions of two transforms, and stores them side by side, one 16-byte
// value per mode: four columns of a warp are 64 contiguous bytes of a row, not
// 32 of two rows. Bound by DRAM and by the L1's requests; 256x128x384: 63
// us with the fields apart, now 54.
template <int N2>
__global__ void __launch_bounds__(kYThreads) k_ifft_y2(StageArgs a) {
  using Y = YT2<N2>;
  constexpr int G = Y::G, E = Y::E;
  const Geo g = a.g;
  __shared__ float4 fbuf4[(kYThreads / G) * Y::BUF];
  __shared__ float4 tw4[Y::TWE];
  __shared__ __align__(16) float2 tw2[Y::TWE];
  const int grp = threadIdx.x / G, l = threadIdx.x % G;
  const int j1 = blockIdx.x * ycols<N2>() + grp;
  const int j = blockIdx.y + a.lvl0;
  const int run = blockIdx.z >> 1, p = blockIdx.z & 1;
  const bool act = j1 < g.K1;
  const float2* srcA = a.S + ((size_t)(run * 5 + (p ? 3 : 0)) * g.N3 + j) * g.Pp + j1;
  const float2* srcB = a.S + ((size_t)(run * 5 + (p ? 1 : 2)) * g.N3 + j) * g.Pp + j1;
  chain_begin();
  c2x x[E];
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int n2 = l + G * e;
    int q = -1;
    if (n2 < g.Ky) q = n2;
    else if (n2 > N2 - g.Ky) q = n2 - (N2 - g.K2);
    const bool in = act && q >= 0;
    const float2 A = in ? srcA[(size_t)q * g.K1] : make_float2(0.f, 0.f);
    const float2 B = in ? srcB[(size_t)q * g.K1] : make_float2(0.f, 0.f);
    x[e] = c2x{make_float2(A.x, B.x), make_float2(A.y, B.y)};
  }
  // the tables after this block's loads are on their way
  Y::fill(tw4, tw2, a.tw, threadIdx.x, kYThreads);
  __syncthreads();
  Y::template fft<true>(x, fbuf4 + grp * Y::BUF, tw4, tw2, l);
  if (act) {
    float4* dst = reinterpret_cast<float4*>(a.mixin) + ((size_t)(run * 2 + p) * g.N3 + j) * N2 * g.K1 + j1;
#pragma unroll
    for (int sl = 0; sl < E; sl++)
      dst[(size_t)Y::out(l, sl) * g.K1] = make_float4(x[sl].re.x, x[sl].im.x, x[sl].re.y, x[sl].im.y);
  }
}

// The combination pairs of two fields (blockIdx.z = 2 run + p; p = 0 the
// fields 1 and B, p = 1 the fields 2 and 3): r_f[q][j1] = Fy(C_f) + i ky
// Fy(C_fy). The pair of the C_fy is transformed first and waits, times i ky, in
// the registers; both are read as one 16-byte value per mode and row (see
// k_ifft_y2). 256x128x384: 127 us with every combination apart, now 108.
template <int N2>
__global__ void __launch_bounds__(kYThreads) k_fft_y(StageArgs a) {
  using Y = YT<N2>;
  constexpr int G = Y::G, E = Y::E;
  const Geo g = a.g;
  __shared__ float4 fbuf4[(kYThreads / G) * Y::BUF];
  __shared__ float4 tw4[Y::TWE];
  __shared__ __align__(16) float2 tw2[Y::TWE];
  const int grp = threadIdx.x / G, l = threadIdx.x % G;
  const int j1 = blockIdx.x * ypcols<N2>() + grp;
  const int j = blockIdx.y + a.lvl0;
  const int run = blockIdx.z >> 1, p = blockIdx.z & 1;
  const bool act = j1 < g.K1;
  const size_t ps = (size_t)g.N3 * N2 * g.K1;   // one pair's values
  const float4* src = reinterpret_cast<const float4*>(a.mixout) + (size_t)(run * 4 + 2 * p) * ps + (size_t)j * N2 * g.K1 + j1;
  float4* buf = fbuf4 + grp * Y::BUF;
  chain_begin();
  c2x y[E], x[E];
#pragma unroll
  for (int e = 0; e < E; e++) {
    const size_t o = (size_t)(l + G * e) * g.K1;
    const float4 v = act ? __ldcs(src + ps + o) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 w = act ? __ldcs(src + o) : make_float4(0.f, 0.f, 0.f, 0.f);
    y[e] = c2x{make_float2(v.x, v.z), make_float2(v.y, v.w)};
    x[e] = c2x{make_float2(w.x, w.z), make_float2(w.y, w.w)};
  }
  // the tables after this block's loads are on their way
  Y::fill(tw4, tw2, a.tw, threadIdx.x, kYThreads);
  __syncthreads();
  Y::template fft<false>(y, buf, tw4, tw2, l);
  Y::template fft<false>(x, buf, tw4, tw2, l);
  if (act) {
    float2* dA = a.rnl + ((size_t)(run * 4 + (p ? 1 : 0)) * g.N3 + j) * g.Pp + j1;
    float2* dB = a.rnl + ((size_t)(run * 4 + (p ? 2 : 3)) * g.N3 + j) * g.Pp + j1;
#pragma unroll
    for (int sl = 0; sl < E; sl++) {
      const int n2 = Y::out(l, sl);
      int q = -1;
      if (n2 < g.Ky) q = n2;
      else if (n2 > N2 - g.Ky) q = n2 - (N2 - g.K2);
      if (q >= 0) {
        const float2 ky = pk2(a.ky[q]);
        const float2 re = psub(x[sl].re, pmul(ky, y[sl].im)), im = pfma(ky, y[sl].re, x[sl].im);
        dA[(size_t)q * g.K1] = make_float2(re.x, im.x);
        dB[(size_t)q * g.K1] = make_float2(re.y, im.y);
      }
    }
  }
}

// ============================================================= x pass ====
// product ids (BuildRHS, IMEXRK.cpp:155-192; BuildRHSLinear, :212-257)
enum Prod { P_S1, P_SB1, P_P3, P_Q1, P_QB, P_P4, P_S12, P_S22, P_SB2, P_Q2, P_P3Y, P_COUNT };

constexpr int kXMaxThreads = 512;

// slots s = 0..S+1 hold level j0-1+s; product p is formed at slots
// [first, first+count)
__host__ __device__ __forceinline__ void prod_slots(int p, int S, int& first, int& count) {
  if (p == P_Q1 || p == P_QB || p == P_Q2) { first = 1; count = S + 1; }
  else if (p == P_P4) { first = 0; count = S + 1; }
  else { first = 1; count = S; }
}
__host__ __device__ inline int prod_rows(int nprod, int S) {
  int n = 0;
  for (int p = 0; p < nprod; p++) { int f, c; prod_slots(p, S, f, c); n += c; }
  return n;
}

// row of the transformed product p at slot s; p is a compile-time constant at
// every call, so the loop folds
__device__ __forceinline__ int hat_row(int p, int s, int S) {
  int base = 0;
#pragma unroll
  for (int q = 0; q < P_COUNT; q++) {
    if (q == p) break;
    int f, c;
    prod_slots(q, S, f, c);
    base += c;
  }
  int f, c;
  prod_slots(p, S, f, c);
  return base + s - f;
}

// products whose first slot repeats the last (Q products) or next-to-last
// (P4) slot of the slab below; a block that walks up through several slabs
// keeps those transformed rows instead of forming them again
__host__ __device__ __forceinline__ bool carried(int p) {
  return p == P_Q1 || p == P_QB || p == P_Q2 || p == P_P4;
}

// row stride (floats) of the nodal rows in shared memory: N1 padded by one
// lane group, so the lane groups of a warp, which read the same field at
// consecutive slots, fall on different banks
__host__ __device__ constexpr int nod_row(int N1) { return N1 + (N1 >= 256 ? 16 : (N1 >= 64 ? 8 : 4)); }

struct XLayout {  // shared-memory carve-up of k_xpass
  int nprod, nrows;
  size_t hat_off, stage_off, buf_off, nod_off, base_off, carry_off, bytes;
};

__host__ __device__ inline XLayout x_layout(int S, int N1, int K1, int dim3, int linear, int bufstride, int ngroups,
                                            int tlm, int prefetch) {
  XLayout L;
  L.nprod = dim3 ? P_COUNT : 6;
  L.nrows = prod_rows(L.nprod, S);
  size_t off = 0;
  // transformed products, one row of K1 per (product, slot), and the staged
  // input rows of phase A (4 x (S+2) x K1, twice that when the base rows of
  // a tangent-linear batch come along): their own bytes when a block loads
  // the next slab's rows during this slab's work, else the same bytes
  auto al16 = [](size_t b) { return (b + 15) & ~(size_t)15; };   // 16-byte aligned regions
  size_t hat = al16(sizeof(float2) * (size_t)L.nrows * K1),
         stage = al16(sizeof(float2) * (size_t)(tlm ? 8 : 4) * (S + 2) * K1);
  L.hat_off = off;
  if (prefetch) {
    off += hat;
    L.stage_off = off; off += stage;
  } else {
    L.stage_off = off; off += (hat > stage ? hat : stage);
  }
  L.buf_off = off;  off += sizeof(float2) * (size_t)ngroups * bufstride;
  L.nod_off = off;  off += sizeof(float) * (size_t)4 * (S + 2) * nod_row(N1);
  L.base_off = off; if (linear) off += sizeof(float) * (size_t)4 * (S + 2) * nod_row(N1);
  L.carry_off = off; off += sizeof(float2) * (size_t)4 * K1;   // transformed rows kept for the next slab
  L.bytes = off;
  return L;
}

// ---- BuildRHS / BuildRHSLinear products by pair ----
// Each forward transform carries two real products; a pair kind fixes which
// two, so the rows each lane reads and the arithmetic are compile-time
// constants and the two products of a pair share their loads. Products at
// slot i + 1 of a slab (i < S): (S1, SB1), (P3, P4), (S12, S22), (SB2, P3Y);
// the Q products at slot i + 2: (Q1, QB) and (Q2 at i + 2, Q2 at i + 3); the
// slab's first halo rows, (Q1, QB) at slot 1 and (P4 at slot 0, Q2 at slot 1),
// when no slab below handed them over.
enum PairKind { K_SSB1, K_P34, K_S122, K_SB2P, K_QQB, K_Q2Q2, K_HALO };

struct HalfC {  // one product at one slot: its rows and coefficients
  int s, sm, sp;
  float ub, ubm, tlo, tdi, hb, lof, top;
  bool live;
};

__device__ __forceinline__ HalfC half_coeffs(int s, int j0, int N3, const float* Ub, const float* zc) {
  HalfC c;
  const int t = j0 - 1 + s;
  c.live = t >= 0 && t < N3;
  const int tc = c.live ? t : 0;
  const bool lo = c.live && (t >= 1) && (s >= 1);
  c.s = s;
  c.sm = lo ? s - 1 : s;
  c.top = (t <= N3 - 2) ? 1.f : 0.f;
  c.sp = (t <= N3 - 2) ? s + 1 : s;
  c.lof = lo ? 1.f : 0.f;
  c.tlo = c.lof * zc[ZC_TILDE_LO * N3 + tc];
  c.tdi = c.lof * zc[ZC_TILDE_DI * N3 + tc];
  c.hb = 0.5f * c.lof;
  c.ub = Ub[tc];
  c.ubm = lo ? Ub[tc - 1] : 0.f;
  return c;
}

// product P of BuildRHS at point n (IMEXRK.cpp:155-192; the U1t*U1t product
// leaves out its x-independent U_^2 part, which ddx multiplies by zero)
template <int P, int N1>
__device__ __forceinline__ float prod_at(const float* nod, int NS, const HalfC& c, int n) {
  auto u = [&](int f, int slot) { return nod[(f * NS + slot) * nod_row(N1) + n]; };
  float v;
  if constexpr (P == P_S1) { const float a = u(0, c.s); v = a * (a + 2.f * c.ub); }
  else if constexpr (P == P_SB1) v = (u(0, c.s) + c.ub) * u(3, c.s);
  else if constexpr (P == P_P3)
    v = (c.tdi * u(0, c.s) + c.tlo * u(0, c.sm) + (c.tlo * c.ubm + c.tdi * c.ub)) * (c.lof * u(2, c.s));
  else if constexpr (P == P_Q1)
    v = (c.hb * u(0, c.s) + c.hb * u(0, c.sm) + (c.hb * c.ubm + c.hb * c.ub)) * (c.lof * u(2, c.s));
  else if constexpr (P == P_QB) v = (c.hb * u(3, c.s) + c.hb * u(3, c.sm)) * (c.lof * u(2, c.s));
  else if constexpr (P == P_P4) { const float d = 0.5f * u(2, c.s) + 0.5f * c.top * u(2, c.sp); v = d * d; }
  else if constexpr (P == P_S12) v = (u(0, c.s) + c.ub) * u(1, c.s);
  else if constexpr (P == P_S22) { const float a = u(1, c.s); v = a * a; }
  else if constexpr (P == P_SB2) v = u(1, c.s) * u(3, c.s);
  else if constexpr (P == P_Q2) v = (c.hb * u(1, c.s) + c.hb * u(1, c.sm)) * (c.lof * u(2, c.s));
  else v = (c.tdi * u(1, c.s) + c.tlo * u(1, c.sm)) * (c.lof * u(2, c.s));   // P_P3Y
  return c.live ? v : 0.f;
}

// product P of BuildRHSLinear at point n (IMEXRK.cpp:212-257): the
// derivative of BuildRHS's product about the base, whose rows `bas` hold
// U1b + U_, U2b, U3b, Bb (so the U_ terms come with the base's u1)
template <int P, int N1>
__device__ __forceinline__ float prod_at_lin(const float* nod, const float* bas, int NS, const HalfC& c, int n) {
  auto u = [&](int f, int slot) { return nod[(f * NS + slot) * nod_row(N1) + n]; };
  auto U = [&](int f, int slot) { return bas[(f * NS + slot) * nod_row(N1) + n]; };
  float v;
  if constexpr (P == P_S1) v = (2.f * u(0, c.s)) * U(0, c.s);
  else if constexpr (P == P_SB1) v = u(3, c.s) * U(0, c.s) + U(3, c.s) * u(0, c.s);
  else if constexpr (P == P_P3)
    v = (c.tdi * u(0, c.s) + c.tlo * u(0, c.sm)) * (c.lof * U(2, c.s)) +
        (c.tdi * U(0, c.s) + c.tlo * U(0, c.sm)) * (c.lof * u(2, c.s));
  else if constexpr (P == P_Q1)
    v = (c.hb * u(0, c.s) + c.hb * u(0, c.sm)) * (c.lof * U(2, c.s)) +
        (c.hb * U(0, c.s) + c.hb * U(0, c.sm)) * (c.lof * u(2, c.s));
  else if constexpr (P == P_QB)
    v = (c.hb * u(3, c.s) + c.hb * u(3, c.sm)) * (c.lof * U(2, c.s)) +
        (c.hb * U(3, c.s) + c.hb * U(3, c.sm)) * (c.lof * u(2, c.s));
  else if constexpr (P == P_P4)   // 2 Dir(u3) Dir(U3b)
    v = (u(2, c.s) + c.top * u(2, c.sp)) * (0.5f * U(2, c.s) + 0.5f * c.top * U(2, c.sp));
  else if constexpr (P == P_S12) v = u(0, c.s) * U(1, c.s) + U(0, c.s) * u(1, c.s);
  else if constexpr (P == P_S22) v = (2.f * u(1, c.s)) * U(1, c.s);
  else if constexpr (P == P_SB2) v = u(3, c.s) * U(1, c.s) + U(3, c.s) * u(1, c.s);
  else if constexpr (P == P_Q2)
    v = (c.hb * u(1, c.s) + c.hb * u(1, c.sm)) * (c.lof * U(2, c.s)) +
        (c.hb * U(1, c.s) + c.hb * U(1, c.sm)) * (c.lof * u(2, c.s));
  else   // P_P3Y
    v = (c.tdi * u(1, c.s) + c.tlo * u(1, c.sm)) * (c.lof * U(2, c.s)) +
        (c.tdi * U(1, c.s) + c.tlo * U(1, c.sm)) * (c.lof * u(2, c.s));
  return c.live ? v : 0.f;
}

template <int P0, int P1, int N1, int E, int G, bool LINEAR>
__device__ __forceinline__ void pair_eval(float2 (&x)[E], const float* nod, const float* bas, int NS, const HalfC& c0,
                                          const HalfC& c1, bool two, int l) {
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int n = l + G * e;
    if constexpr (LINEAR)
      x[e] = make_float2(prod_at_lin<P0, N1>(nod, bas, NS, c0, n), two ? prod_at_lin<P1, N1>(nod, bas, NS, c1, n) : 0.f);
    else
      x[e] = make_float2(prod_at<P0, N1>(nod, NS, c0, n), two ? prod_at<P1, N1>(nod, NS, c1, n) : 0.f);
  }
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::); }
// 16-byte asynchronous copy (both addresses 16-byte aligned)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}

// One block per (`iters` consecutive slabs of S output levels, y row, run).
// Lane groups of G lanes each run one transform at a time; all groups of the
// block step through their task lists in lockstep so every lane reaches
// every warp sync. Walking up from one slab to the next, the block keeps the
// two top nodal levels and the top transformed rows of the carried products
// (their z stencils reach one level across the slab boundary), so each level
// is transformed once rather than once per slab that touches it.
// The body of one x-pass block: (bx, by, bz) = (level column, y row, run)
// relative to a.xcol0 and a.run_offset, so that a kernel over many solvers'
// work items can run it for any block of any of them.
template <int N1, bool LINEAR>
__device__ __forceinline__ void xpass_body(const StageArgs& a, int S, int iters, int bx, int by, int bz) {
  constexpr int G = FFTShape<N1>::G, E = FFTShape<N1>::E, BUF = fft_buf_stride<N1>();
  const int NGB = blockDim.x / G;   // lane groups per block
  const Geo g = a.g;
  extern __shared__ __align__(16) unsigned char xsm[];
  const int tlm = LINEAR ? a.tlm : 0;   // base rows from a live run of this batch
  const XLayout L = x_layout(S, N1, g.K1, g.dim3, LINEAR, BUF, NGB, tlm, iters > 1);
  float2* hat = reinterpret_cast<float2*>(xsm + L.hat_off);
  float2* stg = reinterpret_cast<float2*>(xsm + L.stage_off);  // phase A input rows [4 or 8][S+2][K1]
  constexpr int NR = nod_row(N1);   // nodal row stride
  float* nod = reinterpret_cast<float*>(xsm + L.nod_off);      // [4][S+2][NR]: U1, U2, U3, B
  float* bnod = reinterpret_cast<float*>(xsm + L.base_off);    // [4][S+2][NR]: U1b+Ubar, U2b, U3b, Bb
  constexpr int K1 = N1 / 3;   // kept x modes (the solver's K1), a compile-time constant here
  const int N3 = g.N3;
  const int y = by;
  const int run = bz + a.run_offset;
  const int brun = tlm ? (run - tlm) % tlm : run;   // run that holds the base state
  const int gid = threadIdx.x / G, l = threadIdx.x % G;
  float2* buf = reinterpret_cast<float2*>(xsm + L.buf_off) + (size_t)gid * BUF;
  const float* Ub = a.Ubar + (size_t)run * N3;
  const float* zc = a.zc;
  const int NS = S + 2;
  const int nf = tlm ? 8 : 4;   // own u1,u2,u3,b (and the base run's)
  float2* carry = reinterpret_cast<float2*>(xsm + L.carry_off);   // [4][K1]: Q1, QB, Q2, P4
  // this lane's twiddles, held in registers for every transform of the block
  // (read from the table at each transform when E = 32 would not fit)
  constexpr bool kTwReg = E <= 16;
  float2 twl[kTwReg ? E : 1];
  if constexpr (kTwReg) lane_twiddles<N1>(twl, a.tw, l);
  auto fft_inv = [&](float2 (&v)[E]) {
    if constexpr (kTwReg) reg_fft_w<N1, true>(v, buf, twl, l);
    else reg_fft<N1, true>(v, buf, a.tw, l);
  };
  auto fft_fwd = [&](float2 (&v)[E]) {
    if constexpr (kTwReg) reg_fft_w<N1, false>(v, buf, twl, l);
    else reg_fft<N1, false>(v, buf, a.tw, l);
  };

  // stage the input rows u1, u2, u3, b (and the base run's) at slots s0..S+1
  // (levels jj0-1+s0 .. jj0+S) with asynchronous copies, one warp per row
  auto stage_rows = [&](int jj0, int s0) {
    const int NSn = NS - s0, nw = blockDim.x >> 5, lane = threadIdx.x & 31;
    for (int row = threadIdx.x >> 5; row < nf * NSn; row += nw) {
      const int fb = row / NSn, s = s0 + row - fb * NSn;
      const int f = fb & 3, rr = fb < 4 ? run : brun;
      const int t = jj0 - 1 + s;
      float2* d = stg + ((size_t)fb * NS + s) * K1;
      if (t < 0 || t >= N3 || (f == 1 && !g.dim3)) {
        for (int k = lane; k < K1; k += 32) d[k] = make_float2(0.f, 0.f);
      } else {
        const float2* src = g.dim3 ? a.mixin + mix_pair(g, rr * 2, mix_in_pair(f), mix_in_side(f), t, y)
                                   : a.S + ((size_t)(rr * 5 + f) * N3 + t) * g.Pp;
        const int ks = g.dim3 ? 2 : 1;   // two fields side by side
        for (int k = lane; k < K1; k += 32) cp_async8(d + k, src + ks * k);
      }
    }
  };
  const int col = bx + a.xcol0;   // level column of this block
  stage_rows(col * iters * S, 0);

  for (int it = 0; it < iters; it++) {
  const int j0 = (col * iters + it) * S;
  if (j0 >= N3) break;
  const int s0 = it == 0 ? 0 : 2;   // nodal slots 0, 1 come from the slab below
  const int NSn = NS - s0;

  if (LINEAR && !tlm) {  // frozen nodal base rows (IMEXRK.h:344-351), one warp per row
    const int nw = blockDim.x >> 5, lane = threadIdx.x & 31;
    for (int row = threadIdx.x >> 5; row < 4 * NS; row += nw) {
      const int f = row / NS, t = j0 - 1 + row - f * NS;
      float* d = bnod + (size_t)row * NR;
      if (t < 0 || t >= N3 || (f == 1 && !g.dim3)) {
        for (int x = lane; x < N1; x += 32) d[x] = 0.f;
      } else {
        const float* src = a.base + (((size_t)(run * 4 + f) * N3 + t) * g.N2 + y) * N1;
        for (int c = lane; c < N1 / 4; c += 32) cp_async16(d + 4 * c, src + 4 * c);
      }
    }
  }
  cp_async_wait_all();
  __syncthreads();
  if (LINEAR && !tlm) {   // U1b + U_ as nnTemp (phase A writes only the own rows meanwhile)
    for (int i = threadIdx.x; i < NS * N1; i += blockDim.x) {
      const int sl = i / N1, t = j0 - 1 + sl;
      if (t >= 0 && t < N3) bnod[sl * NR + (i - sl * N1)] += Ub[t];
    }
  }

  // ---- phase A: inverse transforms of (u1, u3) and (b, u2) (ToNodal) ----
  // (and of the base run's fields for a tangent-linear batch)
  const int ntA = NSn * (tlm ? 4 : 2);
  for (int base = 0; base < ntA; base += NGB) {
    const int task = base + gid;
    const bool valid = task < ntA;
    const int s = valid ? s0 + task % NSn : 0, pr4 = valid ? task / NSn : 0;
    const int pr = pr4 & 1, ofs = (pr4 >> 1) * 4;   // ofs 4: base rows
    const int fA = pr == 0 ? 0 : 3;       // u1 | b
    const int fB = pr == 0 ? 2 : 1;       // u3 | u2
    const float2* srcA = stg + ((size_t)(ofs + fA) * NS + s) * K1;
    const float2* srcB = stg + ((size_t)(ofs + fB) * NS + s) * K1;
    float2 x[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int n = l + G * e;
      float2 zz = make_float2(0.f, 0.f);
      if (n == 0) {
        zz = make_float2(srcA[0].x, srcB[0].x);   // c2r uses the real part of the k = 0 term
      } else if (n < K1) {
        const float2 A = srcA[n], B = srcB[n];
        zz = make_float2(A.x - B.y, A.y + B.x);            // A + iB
      } else if (n > N1 - K1) {
        const float2 A = srcA[N1 - n], B = srcB[N1 - n];
        zz = make_float2(A.x + B.y, B.x - A.y);            // conj(A) + i conj(B)
      }
      x[e] = zz;
    }
    fft_inv(x);
    if (valid) {
      float* rows = ofs ? bnod : nod;
      float* rA = rows + ((size_t)fA * NS + s) * NR;
      float* rB = rows + ((size_t)fB * NS + s) * NR;
      const int t = j0 - 1 + s;
      // the base's U1 row carries U_ (nnTemp = U1_tot + U_, IMEXRK.cpp:212)
      const float add = (ofs && fA == 0 && t >= 0 && t < N3) ? a.Ubar[(size_t)brun * N3 + t] : 0.f;
#pragma unroll
      for (int sl = 0; sl < E; sl++) {
        const int xo = reg_fft_out_index<N1>(l, sl);
        rA[xo] = x[sl].x + add;
        rB[xo] = x[sl].y;
      }
    }
  }
  __syncthreads();

  // the next slab's input rows load while this slab's products are formed
  if (it + 1 < iters && j0 + S < N3) stage_rows(j0 + S, 2);

  // rows carried over from the slab below
  if (it > 0)
    for (int i = threadIdx.x; i < 4 * K1; i += blockDim.x) {
      const int q = i / K1, k = i - q * K1;
      const int p = q == 0 ? P_Q1 : (q == 1 ? P_QB : (q == 2 ? P_Q2 : P_P4));
      if (p < L.nprod) hat[(size_t)hat_row(p, p == P_P4 ? 0 : 1, S) * K1 + k] = carry[i];
    }

  // ---- phase B/C: nodal products, forward transforms in pairs (ToModal) ----
  const int nprod = L.nprod;
  const float sc = 0.5f * g.inv_n12;
  const int NT = g.dim3 ? 5 : 3;   // pair kinds at every output level
  const int nmain = NT * S, nq2 = g.dim3 ? (S + 1) / 2 : 0, ntB = nmain + nq2 + (it == 0 ? 2 : 0);
  for (int base = 0; base < ntB; base += NGB) {
    const int task = base + gid;
    int kind = -1, i = 0;
    if (task < nmain) {
      const int q = task / S;
      kind = q < 2 ? q : (g.dim3 ? q : K_QQB);   // 2D: (S1, SB1), (P3, P4), (Q1, QB)
      i = task - q * S;
    } else if (task < nmain + nq2) {
      kind = K_Q2Q2;
      i = 2 * (task - nmain);
    } else if (task < ntB) {
      kind = task == nmain + nq2 ? K_QQB : K_HALO;
      i = -1;
    }
    int s0 = i + 1, s1 = i + 1, p0 = -1, p1 = -1;
    switch (kind) {
      case K_SSB1: p0 = P_S1; p1 = P_SB1; break;
      case K_P34: p0 = P_P3; p1 = P_P4; break;
      case K_S122: p0 = P_S12; p1 = P_S22; break;
      case K_SB2P: p0 = P_SB2; p1 = P_P3Y; break;
      case K_QQB: p0 = P_Q1; p1 = P_QB; s0 = s1 = i + 2; break;
      case K_Q2Q2: p0 = P_Q2; p1 = i + 1 < S ? P_Q2 : -1; s0 = i + 2; s1 = i + 3; break;
      case K_HALO: p0 = P_P4; p1 = g.dim3 ? P_Q2 : -1; s0 = 0; s1 = 1; break;
      default: break;
    }
    const HalfC c0 = half_coeffs(s0, j0, N3, Ub, zc), c1 = half_coeffs(s1, j0, N3, Ub, zc);
    const bool two = p1 >= 0;
    float2 x[E];
    switch (kind) {
      case K_SSB1: pair_eval<P_S1, P_SB1, N1, E, G, LINEAR>(x, nod, bnod, NS, c0, c1, true, l); break;
      case K_P34: pair_eval<P_P3, P_P4, N1, E, G, LINEAR>(x, nod, bnod, NS, c0, c1, true, l); break;
      case K_S122: pair_eval<P_S12, P_S22, N1, E, G, LINEAR>(x, nod, bnod, NS, c0, c1, true, l); break;
      case K_SB2P: pair_eval<P_SB2, P_P3Y, N1, E, G, LINEAR>(x, nod, bnod, NS, c0, c1, true, l); break;
      case K_QQB: pair_eval<P_Q1, P_QB, N1, E, G, LINEAR>(x, nod, bnod, NS, c0, c1, true, l); break;
      case K_Q2Q2: pair_eval<P_Q2, P_Q2, N1, E, G, LINEAR>(x, nod, bnod, NS, c0, c1, two, l); break;
      case K_HALO: pair_eval<P_P4, P_Q2, N1, E, G, LINEAR>(x, nod, bnod, NS, c0, c1, two, l); break;
      default:
#pragma unroll
        for (int e = 0; e < E; e++) x[e] = make_float2(0.f, 0.f);
    }
    fft_fwd(x);
#pragma unroll
    for (int sl = 0; sl < E; sl++) buf[reg_fft_out_index<N1>(l, sl)] = x[sl];
    __syncwarp();
    if (p0 >= 0) {
      float2* h0 = hat + (size_t)hat_row(p0, s0, S) * K1;
      float2* h1 = hat + (size_t)hat_row(two ? p1 : p0, s1, S) * K1;
#pragma unroll
      for (int q = 0; q < (K1 + G - 1) / G; q++) {
        const int k = l + q * G;
        if (k >= K1) break;
        const float2 zk = buf[k];
        const float2 zc2 = cconj(buf[(N1 - k) & (N1 - 1)]);
        h0[k] = make_float2((zk.x + zc2.x) * sc, (zk.y + zc2.y) * sc);          // (Zk + conj Z_{N-k}) / 2
        if (two) h1[k] = make_float2((zk.y - zc2.y) * sc, -(zk.x - zc2.x) * sc);  // (Zk - conj Z_{N-k}) / (2i)
      }
    }
    __syncwarp();
  }
  __syncthreads();

  // ---- phase D: z stencils of the products and x derivatives ----
  auto H = [&](int p, int s, int k) -> float2 { return hat[(size_t)hat_row(p, s, S) * K1 + k]; };
  for (int i = threadIdx.x; i < S * K1; i += blockDim.x) {
    const int si = i / K1, k = i - si * K1;
    const int t = j0 + si, s = si + 1;
    if (t >= N3) continue;
    const float kxv = a.kx[k];
    // ddz Dirichlet -> Neumann of a Q product (Differentiation.cpp:35-61)
    auto dzdn = [&](int p) -> float2 {
      if (t == 0) return make_float2(0.f, 0.f);
      float di = zc[ZC_DDN_DI * N3 + t];
      float2 v = cscale(H(p, s, k), di);
      if (t < N3 - 1) v = cadd(v, cscale(H(p, s + 1, k), zc[ZC_DDN_UP * N3 + t]));
      return v;
    };
    float2 dnd = make_float2(0.f, 0.f);  // ddz Neumann -> Dirichlet of P4
    if (t >= 2)
      dnd = cadd(cscale(H(P_P4, s - 1, k), zc[ZC_DND_LO * N3 + t]), cscale(H(P_P4, s, k), zc[ZC_DND_DI * N3 + t]));
    const float2 c1 = csub(cscale(cik(kxv, H(P_S1, s, k)), -1.f), dzdn(P_Q1));
    const float2 c3 = csub(cscale(cik(kxv, H(P_P3, s, k)), -1.f), dnd);
    const float2 cB = csub(cscale(cik(kxv, H(P_SB1, s, k)), -1.f), dzdn(P_QB));
    if (!g.dim3) {
      float2* r = a.rnl + (size_t)run * 4 * g.fblk + (size_t)t * g.Pp + k;
      r[0 * g.fblk] = c1;
      r[2 * g.fblk] = c3;
      r[3 * g.fblk] = cB;
    } else {
      const float2 c1y = cscale(H(P_S12, s, k), -1.f);
      const float2 c2 = csub(cscale(cik(kxv, H(P_S12, s, k)), -1.f), dzdn(P_Q2));
      const float2 c2y = cscale(H(P_S22, s, k), -1.f);
      const float2 c3y = cscale(H(P_P3Y, s, k), -1.f);
      const float2 cBy = cscale(H(P_SB2, s, k), -1.f);
      float4* m = reinterpret_cast<float4*>(a.mixout) + (((size_t)run * 4 * N3 + t) * g.N2 + y) * K1 + k;
      const size_t cs = g.mblk;
      m[0 * cs] = make_float4(c1.x, c1.y, cB.x, cB.y);
      m[1 * cs] = make_float4(c1y.x, c1y.y, cBy.x, cBy.y);
      m[2 * cs] = make_float4(c2.x, c2.y, c3.x, c3.y);
      m[3 * cs] = make_float4(c2y.x, c2y.y, c3y.x, c3y.y);
    }
  }

  // ---- keep what the next slab shares with this one ----
  if (it + 1 < iters) {
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * K1; i += blockDim.x) {
      const int q = i / K1, k = i - q * K1;
      const int p = q == 0 ? P_Q1 : (q == 1 ? P_QB : (q == 2 ? P_Q2 : P_P4));
      if (p < nprod) carry[i] = hat[(size_t)hat_row(p, p == P_P4 ? S : S + 1, S) * K1 + k];
    }
    for (int i = threadIdx.x; i < nf * 2 * N1; i += blockDim.x) {   // nodal slots S, S+1 -> 0, 1
      const int fb = i / (2 * N1), r = i - fb * 2 * N1, sl = r / N1, x = r - sl * N1;
      float* rows = fb < 4 ? nod : bnod;
      const int f = fb & 3;
      rows[((size_t)f * NS + sl) * NR + x] = rows[((size_t)f * NS + S + sl) * NR + x];
    }
    __syncthreads();
  }
  }   // slabs
}

template <int N1, bool LINEAR>
__global__ void __launch_bounds__(kXMaxThreads) k_xpass(StageArgs a, int S, int iters) {
  chain_begin();
  xpass_body<N1, LINEAR>(a, S, iters, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ============================================================ z pass ====
template <int ZW>
__global__ void __launch_bounds__(ZW * 32, ZW == 8 ? 3 : 1) k_z_proj_chunked(Geo g, float2* U, const float2* Psrc, float2* Pdst,
                                                           const float* zc, const float* fa, const float* fc,
                                                           const float* inv_den, const float* kx, const float* ky,
                                                           float pm) {
  z_proj_body<ZW>(g, U, Psrc, Pdst, zc, fa, fc, inv_den, kx, ky, pm, blockIdx.x, blockIdx.z);
}

template <int ZW, bool IC>
__global__ void __launch_bounds__(ZW * 32, ZW == 8 ? 3 : 1) k_z_step(StageArgs a) {
  z_step_body<ZW, IC>(a, blockIdx.x, blockIdx.z);
}


// ====================================================== factorisation ====
// Thomas factors of every (factor set, mode) in FP64 (Tridiagonal.h:14-27):
// inv_den_j = 1/(b_j - a_j C_{j-1}), stored as float. Rows follow
// UpdateForTimestep (IMEXRK.h:502-545) and the Laplacian of the constructor
// (IMEXRK.h:55-78) with Neumannify / Dirichlify (Differentiation.h:17-59).
__global__ void k_factor(Geo g, const double* __restrict__ bands, const double* __restrict__ kx,
                         const double* __restrict__ ky, double h0, double h1, double h2, double Re,
                         double Pr, float* inv_den) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int fs = blockIdx.y;
  const int N = g.N3;
  if (m >= g.Pp) return;
  float* out = inv_den + (size_t)fs * N * g.Pp + m;
  if (m >= g.P) {
    for (int j = 0; j < N; j++) out[(size_t)j * g.Pp] = 0.f;
    return;
  }
  const int q = m / g.K1, j1 = m - q * g.K1;
  const double kk = -(kx[j1] * kx[j1]) + -(ky[q] * ky[q]);
  const bool lap = (fs == kFS_Lap);
  const int fam = lap ? 0 : fs / 3, k = lap ? 0 : fs % 3;
  const bool dir = (fam == 2);
  const double h = k == 0 ? h0 : (k == 1 ? h1 : h2);
  const double s = 0.5 * h;
  const double den_re = (fam == 1) ? Re * Pr : Re;
  const double* lo = bands + (dir ? 3 : 0) * N;
  const double* di = bands + (dir ? 4 : 1) * N;
  const double* up = bands + (dir ? 5 : 2) * N;
  double Cprev = 0.0;
  for (int j = 0; j < N; j++) {
    double aj, bj, cj;
    if (lap) {
      aj = lo[j]; bj = di[j] + kk; cj = up[j];
    } else {
      aj = -(s * lo[j]) / den_re; bj = 1.0 - (s * (di[j] + kk)) / den_re; cj = -(s * up[j]) / den_re;
    }
    if (!dir) {   // Neumannify
      if (j == 0) { bj = 1; cj = 0; }
      if (j == 1) { aj = 0; bj = 1; cj = -1; }
      if (j == N - 2) { aj = 1; bj = -1; cj = 0; }
      if (j == N - 1) { aj = 0; bj = 1; cj = 0; }
      if (lap && m == 0 && j == 1) cj = 0;   // (0,0) mode pinned
    } else {      // Dirichlify
      if (j <= 2) { aj = 0; bj = 1; cj = 0; }
      if (j >= N - 2) { aj = 0; bj = 1; cj = 0; }
    }
    if (j == N - 1) cj = 0;
    double den = (j == 0) ? bj : bj - aj * Cprev;
    out[(size_t)j * g.Pp] = (float)(1.0 / den);
    Cprev = cj / den;
  }
}

// ============================================== layout transposes ====
// reference layout [N2][M1][N3] (z fastest) <-> kept layout [N3][Pp]
__global__ void k_gather_ref(Geo g, const float2* __restrict__ ref, float2* __restrict__ kept) {
  __shared__ float2 tile[32][33];
  const int M1 = g.N1 / 2 + 1;
  const int m0 = blockIdx.x * 32, jz0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int m = m0 + r, jz = jz0 + threadIdx.x;
    float2 v = make_float2(0.f, 0.f);
    if (m < g.P && jz < g.N3) {
      int q = m / g.K1, j1 = m - q * g.K1;
      int n2 = n2_of_q(q, g.Ky, g.K2, g.N2);
      v = ref[((size_t)M1 * n2 + j1) * g.N3 + jz];
    }
    tile[r][threadIdx.x] = v;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int jz = jz0 + r, m = m0 + threadIdx.x;
    if (jz < g.N3 && m < g.Pp) kept[(size_t)jz * g.Pp + m] = tile[threadIdx.x][r];
  }
}

__global__ void k_scatter_ref(Geo g, const float2* __restrict__ kept, float2* __restrict__ ref) {
  __shared__ float2 tile[32][33];
  const int M1 = g.N1 / 2 + 1;
  const int m0 = blockIdx.x * 32, jz0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int jz = jz0 + r, m = m0 + threadIdx.x;
    tile[threadIdx.x][r] = (jz < g.N3 && m < g.P) ? kept[(size_t)jz * g.Pp + m] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int m = m0 + r, jz = jz0 + threadIdx.x;
    if (m < g.P && jz < g.N3) {
      int q = m / g.K1, j1 = m - q * g.K1;
      int n2 = n2_of_q(q, g.Ky, g.K2, g.N2);
      ref[((size_t)M1 * n2 + j1) * g.N3 + jz] = tile[r][threadIdx.x];
    }
  }
}

// ============================================================ energies ====
// InnerProd (Integration.h:282-311) of each field pair in FP64: per level the
// sum over kept modes of w_m Re(a conj b) with w = 1 for (0,0) and 2 otherwise,
// then the vertical quadrature. out[pair*4 + f] accumulates field f
// (0 u1, 1 u2, 2 u3, 3 b).
__global__ void k_inner(Geo g, const float2* __restrict__ Sa, const float2* __restrict__ Sb,
                        const float* __restrict__ zc, double* out) {
  const int j = blockIdx.x;
  const int pair = blockIdx.y;
  const int f = blockIdx.z;
  const float2* a = Sa + ((size_t)(pair * 5 + f) * g.N3 + j) * g.Pp;
  const float2* b = Sb + ((size_t)(pair * 5 + f) * g.N3 + j) * g.Pp;
  double s = 0.0;
  for (int m = threadIdx.x; m < g.P; m += blockDim.x) {
    float2 x = a[m], y = b[m];
    double v = (double)x.x * y.x + (double)x.y * y.y;
    s += (m == 0) ? v : 2.0 * v;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    const float wz = zc[(f == 2 ? ZC_WZD : ZC_WZN) * g.N3 + j];
    if (wz != 0.f) atomicAdd(out + pair * 4 + f, t * (double)wz);
  }
}

// The squared-gradient integrals of the dissipation rates (sf_dissipation),
// InnerProd (Integration.h:282-311) of each gradient component at the
// location it lives on, in FP64: per level j the sum over kept modes of
// w_m [ (kx^2 + ky^2) |a_j|^2 wz(j) + |vertical difference|^2 / dz ], with
//   u1, u2, b (Neumann): ddz lands on Dirichlet rows, (a_j - a_{j-1}) / DY_j,
//                        integrated over rows 2..N3-2 with weights DY_j;
//   u3 (Dirichlet):      ddz lands on Neumann rows, (a_{j+1} - a_j) / DYF_j,
//                        integrated over rows 1..N3-2 with weights DYF_j
// (Differentiation.cpp:35-61, Integration.h:5-35). out[run*4 + f] accumulates.
__global__ void k_grad_sq(Geo g, const float2* __restrict__ S, const float* __restrict__ zc,
                          const double* __restrict__ kxd, const double* __restrict__ kyd, double* out) {
  const int j = blockIdx.x, run = blockIdx.y, f = blockIdx.z;
  const int N3 = g.N3;
  const bool dir = f == 2;
  const float2* a = S + ((size_t)(run * 5 + f) * N3 + j) * g.Pp;
  const double wz = (double)zc[(dir ? ZC_WZD : ZC_WZN) * N3 + j];
  int jn = -1;
  double iv = 0.0;
  if (!dir && j >= 2 && j <= N3 - 2) { jn = j - 1; iv = (double)zc[ZC_DND_DI * N3 + j]; }   // 1/DY_j
  if (dir && j >= 1 && j <= N3 - 2) { jn = j + 1; iv = (double)zc[ZC_DDN_UP * N3 + j]; }   // 1/DYF_j
  const float2* an = S + ((size_t)(run * 5 + f) * N3 + (jn >= 0 ? jn : j)) * g.Pp;
  double s = 0.0;
  for (int m = threadIdx.x; m < g.P; m += blockDim.x) {
    const int q = m / g.K1, j1 = m - q * g.K1;
    const double kk = kxd[j1] * kxd[j1] + (g.dim3 ? kyd[q] * kyd[q] : 0.0);
    const float2 x = a[m];
    double v = kk * ((double)x.x * x.x + (double)x.y * x.y) * wz;
    if (jn >= 0) {
      const float2 y = an[m];
      const double dx = (double)x.x - y.x, dy = (double)x.y - y.y;
      v += (dx * dx + dy * dy) * iv;
    }
    s += (m == 0) ? v : 2.0 * v;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    if (t != 0.0) atomicAdd(out + run * 4 + f, t);
  }
}

// ======================================================== launchers ====
static inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

struct XShape {
  int S, iters, threads;
  size_t bytes;
};

// launch shape of the x pass: slab height S, slabs per block, threads, bytes
template <int N1, bool LIN>
static XShape xpass_shape(const StageArgs& a, int nruns) {
  const Geo& g = a.g;
  const int tlm = LIN ? a.tlm : 0;
  constexpr int G = FFTShape<N1>::G, BUF = fft_buf_stride<N1>();
  const int nprod = g.dim3 ? P_COUNT : 6;
  // threads: enough lane groups for all phase-A transforms of a slab (one
  // round), at least two warps, at most kXMaxThreads
  auto threads = [&](int S) {
    int groups = a.xgroups > 0 ? a.xgroups : 2 * (S + 2);
    int t = ((groups * G + 31) / 32) * 32;
    return t < 64 ? 64 : (t > kXMaxThreads ? kXMaxThreads : t);
  };
  auto bytes = [&](int S, int pre) { return x_layout(S, N1, g.K1, g.dim3, LIN, BUF, threads(S) / G, tlm, pre).bytes; };
  (void)nprod;
  // largest slab whose shared memory lets two blocks share an SM, then
  // smaller slabs while the grid would leave SMs idle
  const int cand[] = {8, 6, 4, 3, 2};
  int S = 2;
  for (int c : cand)
    if (bytes(c, g.dim3) <= 112 * 1024) { S = c; break; }
  if (g.dim3 && S > 4) S = 4;
  for (int i = 0; i < 5; i++) {
    if (cand[i] >= S) continue;
    if ((long long)((g.N3 + S - 1) / S) * g.N2 * nruns >= 2 * 148) break;
    S = cand[i];
  }
  // slabs per block: in 3D as many as keep at least two waves of blocks, up
  // to 6 (measured at 256 x 128 x 384: 6 slabs 2.5% faster per step than 1,
  // 12 slower); in 2D one (carrying rows saves transforms but not lockstep
  // rounds there, and the extra barriers cost more)
  int iters = 1;
  while (g.dim3 && iters < 6 && S * (iters + 1) <= g.N3 &&
         (long long)cdiv(g.N3, S * (iters + 1)) * g.N2 * nruns >= 4 * 148)
    iters++;
  if (a.xslabs > 0) iters = std::min<int>(a.xslabs, (int)cdiv(g.N3, S));
  if (iters > 1 && bytes(S, 1) > 227 * 1024) iters = 1;   // no room for the prefetch buffer
  return XShape{S, iters, threads(S), bytes(S, iters > 1)};
}

// one launch over the level columns a.xcol0 .. a.xcol0 + a.xcols - 1 (all
// when a.xcols = 0); a column is the S * iters levels one block walks through
template <int N1, bool LIN>
static void xpass_launch(const StageArgs& a, int nruns, cudaStream_t st) {
  const Geo& g = a.g;
  const XShape x = xpass_shape<N1, LIN>(a, nruns);
  const int ncol = (int)cdiv(g.N3, x.S * x.iters);
  const int cols = a.xcols > 0 ? a.xcols : ncol - a.xcol0;
  dim3 grid(cols, g.N2, nruns);
  launch_chained(k_xpass<N1, LIN>, grid, x.threads, x.bytes, st, a.chained, a, x.S, x.iters);
}

template <int N1>
static int xpass_col_levels(const StageArgs& a, bool L, int nruns) {
  const XShape x = L ? xpass_shape<N1, true>(a, nruns) : xpass_shape<N1, false>(a, nruns);
  return x.S * x.iters;
}

static int xpass_column_levels(const StageArgs& a, bool L, int nruns) {
  switch (a.g.N1) {
    case 16: return xpass_col_levels<16>(a, L, nruns);
    case 32: return xpass_col_levels<32>(a, L, nruns);
    case 64: return xpass_col_levels<64>(a, L, nruns);
    case 128: return xpass_col_levels<128>(a, L, nruns);
    case 256: return xpass_col_levels<256>(a, L, nruns);
    default: return xpass_col_levels<512>(a, L, nruns);
  }
}

static void launch_xpass_runs(const StageArgs& a, bool L, int nruns, cudaStream_t st) {
  switch (a.g.N1) {
    case 16: L ? xpass_launch<16, true>(a, nruns, st) : xpass_launch<16, false>(a, nruns, st); break;
    case 32: L ? xpass_launch<32, true>(a, nruns, st) : xpass_launch<32, false>(a, nruns, st); break;
    case 64: L ? xpass_launch<64, true>(a, nruns, st) : xpass_launch<64, false>(a, nruns, st); break;
    case 128: L ? xpass_launch<128, true>(a, nruns, st) : xpass_launch<128, false>(a, nruns, st); break;
    case 256: L ? xpass_launch<256, true>(a, nruns, st) : xpass_launch<256, false>(a, nruns, st); break;
    case 512: L ? xpass_launch<512, true>(a, nruns, st) : xpass_launch<512, false>(a, nruns, st); break;
  }
}

// the x pass of runs run0 .. + nruns - 1, mode as launch_xmarch's: the level
// march where the setting and the grid take it, else the slab kernel
static void launch_xpass_mode(const StageArgs& a, int mode, int run0, int nruns, cudaStream_t st) {
  StageArgs b = a;
  b.run_offset = run0;
  // the base runs of a tangent-linear batch take the kernel that a plain batch
  // of its size takes, so that they stay bit for bit what they are there
  if (a.xkernel == 1 && xmarch_supported(a, mode, mode == 0 ? a.g.nrun : nruns)) {
    // the same level columns as the slab kernel's launch would cover
    int lo = 0, hi = a.g.N3;
    if (a.xcols > 0 || a.xcol0 > 0) {
      const int lv = xpass_column_levels(a, mode != 0, a.g.nrun);
      lo = a.xcol0 * lv;
      if (a.xcols > 0) hi = std::min(hi, (a.xcol0 + a.xcols) * lv);
    }
    launch_xmarch(b, mode, nruns, lo, hi, st);
    return;
  }
  launch_xpass_runs(b, mode != 0, nruns, st);
}

// the x pass of every run: one launch, or for a tangent-linear batch one
// nonlinear launch for the base runs and one linear launch for the rest
static int launch_xpass(const StageArgs& a, cudaStream_t st) {
  if (a.tlm > 0) {
    launch_xpass_mode(a, 0, 0, a.tlm, st);
    launch_xpass_mode(a, 2, a.tlm, a.g.nrun - a.tlm, st);
    return 2;
  }
  launch_xpass_mode(a, a.linear ? 1 : 0, 0, a.g.nrun, st);
  return 1;
}

// nz = runs x fields transformed (blockIdx.z = 4 run + field); a single
// field of a single run (nz = 1) reads and writes that field only
template <int N2>
static void ify_launch(const StageArgs& a, int nz, cudaStream_t st) {
  const int nl = a.nlvl > 0 ? a.nlvl : a.g.N3 - a.lvl0;
  if (nz % 4 == 0)   // whole runs: the fields in packed pairs
    launch_chained(k_ifft_y2<N2>, dim3(cdiv(a.g.K1, ycols<N2>()), nl, nz / 2), kYThreads, 0, st, a.chained, a);
  else
    k_ifft_y<N2><<<dim3(cdiv(a.g.K1, ycols<N2>()), nl, nz), kYThreads, 0, st>>>(a);
}
template <int N2>
static void fy_launch(const StageArgs& a, cudaStream_t st) {
  const int nl = a.nlvl > 0 ? a.nlvl : a.g.N3 - a.lvl0;
  launch_chained(k_fft_y<N2>, dim3(cdiv(a.g.K1, ypcols<N2>()), nl, a.g.nrun * 2), kYThreads, 0, st, a.chained, a);
}
static void launch_ifft_y_z(const StageArgs& a, int nz, cudaStream_t st) {
  switch (a.g.N2) {
    case 16: ify_launch<16>(a, nz, st); break;
    case 32: ify_launch<32>(a, nz, st); break;
    case 64: ify_launch<64>(a, nz, st); break;
    case 128: ify_launch<128>(a, nz, st); break;
    case 256: ify_launch<256>(a, nz, st); break;
  }
}
static void launch_ifft_y(const StageArgs& a, int nrun, cudaStream_t st) { launch_ifft_y_z(a, nrun * 4, st); }
static void launch_fft_y(const StageArgs& a, cudaStream_t st) {
  switch (a.g.N2) {
    case 16: fy_launch<16>(a, st); break;
    case 32: fy_launch<32>(a, st); break;
    case 64: fy_launch<64>(a, st); break;
    case 128: fy_launch<128>(a, st); break;
    case 256: fy_launch<256>(a, st); break;
  }
}
int launch_fft_y_combos(const StageArgs& a, cudaStream_t st) {
  launch_fft_y(a, st);
  return 1;
}

// opt-in shared-memory limits of every kernel, set once per process before
// any launch (and outside stream capture)
int prepare_kernels() {
  const int lim = 227 * 1024;
  cudaError_t e = cudaSuccess;
#define ATTR(K) if (e == cudaSuccess) e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  ATTR((k_xpass<16, false>)) ATTR((k_xpass<32, false>)) ATTR((k_xpass<64, false>))
  ATTR((k_xpass<128, false>)) ATTR((k_xpass<256, false>)) ATTR((k_xpass<512, false>))
  ATTR((k_xpass<16, true>)) ATTR((k_xpass<32, true>)) ATTR((k_xpass<64, true>))
  ATTR((k_xpass<128, true>)) ATTR((k_xpass<256, true>)) ATTR((k_xpass<512, true>))
  ATTR(k_z_proj_chunked<8>) ATTR(k_z_proj_chunked<16>)
  ATTR((k_z_step<8, false>)) ATTR((k_z_step<8, true>)) ATTR((k_z_step<16, false>)) ATTR((k_z_step<16, true>))
#undef ATTR
  if (e == cudaSuccess && prepare_xmarch_kernels() != 0) return -1;
  if (e == cudaSuccess && prepare_zstep_tma_kernels() != 0) return -1;
  if (e == cudaSuccess && prepare_zstep_c_kernels() != 0) return -1;
  if (e == cudaSuccess && prepare_zstep_f_kernels() != 0) return -1;
  return e == cudaSuccess ? 0 : -1;
}

static size_t zchunk_smem(const Geo& g, int zw) { return sizeof(float) * ((size_t)g.N3 * 32 + 3 * zw * 32); }

// z chunks per block: 16 (shorter serial sweeps, one 16-warp block per SM)
// when the grid leaves SMs without a block, else 8 (three blocks per SM)
static int z_chunks(const Geo& g, int fields) {
  return (long long)cdiv(g.P, 16) * fields * g.nrun < 148 ? 16 : 8;
}

int launch_project(const StageArgs& a, cudaStream_t st) {
  const Geo& g = a.g;
  const dim3 grid(cdiv(g.P, 16), 1, g.nrun);
  if ((a.zchunks ? a.zchunks : z_chunks(g, 1)) == 16)
    k_z_proj_chunked<16><<<grid, 16 * 32, zchunk_smem(g, 16), st>>>(g, a.Sn, a.S, a.Sn, a.zc, a.fa, a.fc,
                                                                      a.inv_den, a.kx, a.ky, a.pm);
  else
    k_z_proj_chunked<8><<<grid, 8 * 32, zchunk_smem(g, 8), st>>>(g, a.Sn, a.S, a.Sn, a.zc, a.fa, a.fc, a.inv_den,
                                                                   a.kx, a.ky, a.pm);
  return 1;
}

// the merged z pass (CN solves of every field, then the projection): one
// block per 16 modes, so the chunk count follows from the mode groups alone;
// chunks of 48 levels or more take the variant with end-test-free interior
// sweeps (measured 7% faster at 384 levels in 8 chunks, and slower with
// 32-level chunks, where it is not used)
// the z pass as k_z_step_tma: where the solver asks for it, has its tensor
// maps, and the launch takes 8 chunks
bool z_step_takes_tma(const StageArgs& a) {
  const int zw = a.zchunks ? a.zchunks : z_chunks(a.g, 1);
  return a.zkernel == 1 && a.zmaps && zw == 8 && zstep_tma_supported(a.g);
}

// the z pass as k_z_step_f, or as k_z_step_c on grids too tall for its shared
// memory: where the solver asks for it and the grid has the levels for
// k_z_step_c's 16 chunks (the chunk count is the kernel's own)
bool z_step_takes_c(const StageArgs& a) { return a.zkernel == 2 && zstep_c_supported(a.g); }

static void launch_z_step(const StageArgs& a, cudaStream_t st) {
  const Geo& g = a.g;
  const dim3 zgrid(cdiv(g.P, 16), 1, g.nrun);
  const int zw = a.zchunks ? a.zchunks : z_chunks(g, 1);
  if (z_step_takes_c(a)) {
    zstep_f_supported(g) ? launch_z_step_f(a, st) : launch_z_step_c(a, st);
    return;
  }
  if (z_step_takes_tma(a) && launch_z_step_tma(a, st)) return;
  const bool ic = cdiv(g.N3, zw) >= 48;
  if (zw == 16) {
    if (ic) k_z_step<16, true><<<zgrid, 16 * 32, zchunk_smem(g, 16), st>>>(a);
    else k_z_step<16, false><<<zgrid, 16 * 32, zchunk_smem(g, 16), st>>>(a);
  } else {
    if (ic) k_z_step<8, true><<<zgrid, 8 * 32, zchunk_smem(g, 8), st>>>(a);
    else k_z_step<8, false><<<zgrid, 8 * 32, zchunk_smem(g, 8), st>>>(a);
  }
}

const char* stage_kernel_name(const Geo& g, int i) {
  static const char* n3[] = {"k_ifft_y", "k_xpass", "k_fft_y", "k_z_step"};
  static const char* n2[] = {"k_xpass", "k_z_step"};
  return g.dim3 ? n3[i] : n2[i];
}
int stage_kernel_count(const Geo& g) { return g.dim3 ? 4 : 2; }

// The 3D x-y pass in level bands: band b's inverse y transforms (stream y1,
// all bands back to back), x pass (the stage's stream, after the inverse
// transforms of its own band and of the band above, whose lowest level its
// z stencils read) and forward y transforms (stream y2, after that band's x
// pass). The memory-bound y transforms of the other bands then run beside the
// compute-bound x pass instead of before and after it. Bands follow the x
// pass's block columns, so no block straddles two bands.
static int launch_xy_banded(const StageArgs& a, cudaStream_t st, const XYAux& aux) {
  const Geo& g = a.g;
  const int lv = xpass_column_levels(a, a.linear != 0, g.nrun);
  const int ncol = (int)cdiv(g.N3, lv);
  const int B = std::min(std::min(aux.bands, kMaxBands), ncol);
  auto c0 = [&](int b) { return (int)((long long)ncol * b / B); };
  auto band = [&](int b) {
    StageArgs y = a;
    y.lvl0 = c0(b) * lv;
    y.nlvl = std::min(g.N3, c0(b + 1) * lv) - y.lvl0;
    return y;
  };
  cudaEventRecord(aux.fork, st);
  cudaStreamWaitEvent(aux.y1, aux.fork, 0);
  cudaStreamWaitEvent(aux.y2, aux.fork, 0);
  for (int b = 0; b < B; b++) {
    launch_ifft_y(band(b), g.nrun, aux.y1);
    cudaEventRecord(aux.ev_ify[b], aux.y1);
  }
  for (int b = 0; b < B; b++) {
    cudaStreamWaitEvent(st, aux.ev_ify[std::min(b + 1, B - 1)], 0);
    StageArgs x = a;
    x.xcol0 = c0(b);
    x.xcols = c0(b + 1) - c0(b);
    launch_xpass(x, st);
    cudaEventRecord(aux.ev_x[b], st);
  }
  for (int b = 0; b < B; b++) {
    cudaStreamWaitEvent(aux.y2, aux.ev_x[b], 0);
    launch_fft_y(band(b), aux.y2);
  }
  cudaEventRecord(aux.join, aux.y2);
  cudaStreamWaitEvent(st, aux.join, 0);
  return 3 * B;
}

int launch_stage(const StageArgs& args, cudaStream_t st, cudaEvent_t* ev, const XYAux* aux) {
  StageArgs a = args;
  const Geo& g = a.g;
  if (g.dim3 && aux && aux->bands > 1 && !ev && !a.tlm) {
    const int n = launch_xy_banded(a, st, *aux);
    launch_z_step(a, st);
    return n + 1;
  }
  // in 2D only before k_z_step_f: an x pass chained alone, between two ordinary launches of another z
  // kernel, costs 1 us a step (64x20: 76.7, 75.8 without; 256x28 x 4: 81.0, 80.4)
  a.chained = !ev && (g.dim3 || (z_step_takes_c(a) && zstep_f_supported(g)));
  int n = 0;
  auto mark = [&]() {
    if (ev) cudaEventRecord(ev[n], st);
    n++;
  };
  if (g.dim3) {
    launch_ifft_y(a, g.nrun, st);
    mark();
  }
  const int extra = launch_xpass(a, st) - 1;   // a tangent-linear batch launches the x pass twice
  mark();
  if (g.dim3) {
    launch_fft_y(a, st);
    mark();
  }
  launch_z_step(a, st);
  mark();
  return n + extra;
}

int launch_z_solves(const StageArgs& a, cudaStream_t st) {
  launch_z_step(a, st);
  return 1;
}

int launch_factor(const Geo& g, const double* bands, const double* kx, const double* ky, double h0, double h1,
                  double h2, double Re, double Pr, float* inv_den, cudaStream_t st) {
  k_factor<<<dim3(cdiv(g.Pp, 128), kNumFS), 128, 0, st>>>(g, bands, kx, ky, h0, h1, h2, Re, Pr, inv_den);
  return 1;
}

int launch_gather_ref(const Geo& g, const float2* ref, float2* kept, cudaStream_t st) {
  k_gather_ref<<<dim3(cdiv(g.Pp, 32), cdiv(g.N3, 32)), dim3(32, 8), 0, st>>>(g, ref, kept);
  return 1;
}

int launch_scatter_ref(const Geo& g, const float2* kept, float2* ref, cudaStream_t st) {
  k_scatter_ref<<<dim3(cdiv(g.P, 32), cdiv(g.N3, 32)), dim3(32, 8), 0, st>>>(g, kept, ref);
  return 1;
}

int launch_grad_sq(const Geo& g, const float2* S, int nruns, const float* zc, const double* kxd, const double* kyd,
                   double* out, cudaStream_t st) {
  k_grad_sq<<<dim3(g.N3, nruns, 4), 256, 0, st>>>(g, S, zc, kxd, kyd, out);
  return 1;
}

int launch_energy(const Geo& g, const float2* Sa, const float2* Sb, int npairs, const float* zc, const float* Ri,
                  double* out, cudaStream_t st) {
  (void)Ri;
  k_inner<<<dim3(g.N3, npairs, 4), 256, 0, st>>>(g, Sa, Sb, zc, out);
  return 1;
}

// nodal field of one modal field (kept layout, one run) -> base [N3][N2][N1]
// via the same transforms as the x pass: used once per set_base.
__global__ void k_base_x(Geo g, const float2* __restrict__ rows, long long row_stride_level,
                         long long row_stride_y, float* __restrict__ out, const float2* __restrict__ tw) {
  extern __shared__ float2 wsm[];
  const int t = blockIdx.x, y = blockIdx.y;
  const int lane = threadIdx.x;
  float2* wk = wsm;
  const float2* src = rows + (size_t)t * row_stride_level + (size_t)y * row_stride_y;
  for (int x = lane; x < g.N1; x += 32) wk[x] = make_float2(0.f, 0.f);
  __syncwarp();
  for (int k = lane; k < g.K1; k += 32) {
    float2 A = src[k];
    if (k == 0) wk[0] = make_float2(A.x, 0.f);
    else { wk[k] = A; wk[g.N1 - k] = cconj(A); }
  }
  __syncwarp();
  warp_fft(wk, g.N1, g.logN1, tw, true, lane);
  float* o = out + ((size_t)t * g.N2 + y) * g.N1;
  for (int x = lane; x < g.N1; x += 32) o[x] = wk[x].x;
}

int launch_base_nodal(const Geo& g, const float2* kept_modal, int field, float* base_out, const float2* tw,
                      float* scratch_mixed, cudaStream_t st) {
  (void)field;
  if (!g.dim3) {
    k_base_x<<<dim3(g.N3, 1), 32, sizeof(float2) * g.N1, st>>>(g, kept_modal, g.Pp, 0, base_out, tw);
    return 1;
  }
  // 3D: inverse y transform into scratch [N3][N2][K1], then x
  StageArgs a = {};
  a.g = g;
  a.g.nrun = 1;
  a.S = kept_modal;   // treated as field 0 of a one-run state
  a.mixin = reinterpret_cast<float2*>(scratch_mixed);
  a.tw = tw;
  launch_ifft_y_z(a, 1, st);   // that field only: the input and the scratch hold one field
  k_base_x<<<dim3(g.N3, g.N2), 32, sizeof(float2) * g.N1, st>>>(g, a.mixin, (long long)g.N2 * g.K1, g.K1,
                                                                base_out, tw);
  return 2;
}

}  // namespace sf
