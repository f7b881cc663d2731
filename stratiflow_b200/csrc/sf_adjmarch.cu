// The adjoint x pass (BuildRHSAdjoint, IMEXRK.cpp:260-379, with the forcing of
// UpdateAdjointVariables, IMEXRK.h:461-500) as level-marching lane groups, in
// the manner of k_xmarch (sf_xmarch.cu): a lane group owns a row and walks up
// a range of levels; every transform is one of a packed pair; a lane's points
// are its own from the inverse transforms to the products, so nothing is
// exchanged but the transforms' transposes.
//
// Per level, the inverse transforms (each line a packed pair)
//   U1 + i U3,    B + i U2        the adjoint fields
//   U1T + i U3T,  BT + i U2T      the direct totals (U_ in U1T)
//   d1U1T + i d1U3T, d1BT + i d1U2T   their x derivatives (i kx on the rows)
//   d2U1T + i d2U3T, d2BT + i d2U2T   their y derivatives (3D)
// and the forward ones
//   F1 + i F2,    F3 + i FB       the forcings of level t-1
//   Q1 + i QB,    Q2 + i D        Bar(U1) U3T, Bar(B) U3T, Bar(U2) U3T; Dir(U3) Dir(U3T) of level t-1
//   U1 U1T + i B U1T,  U2 U1T + i Tilde(U1T) U3      (times i kx)
//   U1 U2T + i U2 U2T, Tilde(U2T) U3 + i B U2T       (3D: the C_fy of the forward pass)
// The z derivatives of the direct totals are taken on the nodal values, from
// the levels a lane holds, instead of being transformed as four more rows.
// The terms that need the level above (Dir of a product, ddz of U3T) wait one
// step in the lane's registers.
//
// The slab form (k_xpass_adj3: 20 rows and 16 products of unpacked transforms,
// one block per SM, products chosen by a switch at every point) took 574 us a
// launch at 128x64x128; this 60 us. The whole adjoint step (us): 128x64x128
// 1774 -> 362, 256x64x128 3829 -> 605, 256x1x256 222 -> 137, 64x1x64 134 -> 93.
#include "sf_xmt.cuh"

namespace sf {

template <int N1, bool D3>
struct AMShape : XMT<N1> {
  using T = XMT<N1>;
  static constexpr int ROWS = D3 ? 12 : 6;   // staged input rows
  // shared memory of one row: two levels of the adjoint and of the direct
  // nodal values, the transpose buffer, the carried combinations and the
  // staged rows of the next level
  static constexpr size_t group_bytes =
      (sizeof(float4) * (size_t)(4 * N1 + T::TB + 2 * T::NKS * T::G) + sizeof(float2) * ROWS * T::K1 + 15) / 16 * 16;
  static constexpr size_t table_bytes = (sizeof(float4) + sizeof(float2)) * (size_t)T::TWE;
  static constexpr int fit = (int)((227 * 1024 - table_bytes) / (T::W * group_bytes));
  static constexpr int WARPS = fit > 8 ? 8 : fit;   // 8: 255 registers
  static constexpr size_t smem(int warps) { return table_bytes + (size_t)warps * T::W * group_bytes; }
  static_assert(WARPS >= 1, "one warp fits an SM");
};

// every level of every row of every run; 3D: the units (run, block of W y
// rows, level) split evenly over the launch's warps; 2D: segments of seg
// levels, one per lane group
template <int N1, bool D3>
__global__ void __launch_bounds__(AMShape<N1, D3>::WARPS * 32, 1) k_adjmarch(const __grid_constant__ StageArgs a, int seg) {
  using X = AMShape<N1, D3>;
  using T = XMT<N1>;
  constexpr int G = T::G, E = T::E, K1 = T::K1, W = T::W, NKS = T::NKS, ROWS = X::ROWS, H = ROWS / 2 - (D3 ? 2 : 0);
  const Geo& g = a.g;
  const int N3 = g.N3, N2 = D3 ? g.N2 : 1;
  extern __shared__ __align__(16) unsigned char xsm[];
  float4* tw4 = reinterpret_cast<float4*>(xsm);
  float2* tw2 = reinterpret_cast<float2*>(xsm + sizeof(float4) * T::TWE);
  T::fill(tw4, tw2, a.tw, threadIdx.x, blockDim.x);
  chain_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int gw = lane / G, l = lane - gw * G;
  __builtin_assume(l >= 0 && l < G);
  unsigned char* gb = xsm + X::table_bytes + (size_t)(warp * W + gw) * X::group_bytes;
  float4* ring = reinterpret_cast<float4*>(gb);     // [2 levels][E slots][G lanes]: U1, B, U3, U2
  float4* dring = ring + 2 * N1;                    // U1T, BT, U3T, U2T
  float4* tbuf = dring + 2 * N1;
  float4* cbuf = tbuf + T::TB;                      // [2][NKS][G]: (c1, cB), (c2, c3) awaiting their z terms
  float2* stg = reinterpret_cast<float2*>(cbuf + 2 * NKS * G);   // 3D [6][K1] pairs, 2D [6][K1]
  __syncthreads();
  const int partner_lane = (lane & ~(G - 1)) | ((G - l) & (G - 1));
  float4 w1[8];
#pragma unroll
  for (int k = 0; k < 8; k++)
    w1[k] = (N1 == 256 || N1 == 128) ? tw4[(k * G + l) % T::TWE] : make_float4(0.f, 0.f, 0.f, 0.f);
  // zero, but not known to the compiler: an order between the batches (sf_xmarch.cu)
  const int rz = (int)(gridDim.x >> 30);
  int tok = 0;
  const float* __restrict__ zc = a.zc;
  const float sc = 0.5f * g.inv_n12;
  const float2 SC = make_float2(sc, sc);
  const float iK = a.adj_invK;

  const long long NW = (long long)gridDim.x * nwarps;
  const long long wid = (long long)blockIdx.x * nwarps + warp;
  const long long NYB = D3 ? N2 / W : (N3 + seg - 1) / seg;
  const long long U = D3 ? (long long)g.nrun * NYB * N3 : ((long long)g.nrun * NYB + W - 1) / W;
  long long u = U * wid / NW;
  const long long uend = U * (wid + 1) / NW;

  while (u < uend) {
    int run, y = 0, ta, n;   // n levels from ta; every group of the warp has the same n
    if (D3) {
      const long long rb = u / N3;
      ta = (int)(u - rb * N3);
      n = (int)std::min<long long>(N3 - ta, uend - u);
      u += n;
      run = (int)(rb / NYB);
      y = (int)(rb % NYB) * W + gw;
    } else {
      const long long sg = u * W + gw;
      u++;
      const bool act = sg < g.nrun * NYB;
      run = act ? (int)(sg / NYB) : 0;
      ta = act ? (int)(sg % NYB) * seg : N3 + 2;   // an idle group marches through levels that do not exist
      n = seg;
    }
    const float Ri = a.Ri[run];
    const size_t tstride = D3 ? (size_t)N2 * K1 : (size_t)g.Pp, fstride = (size_t)N3 * tstride;
    float2* __restrict__ dst = D3 ? a.mixout + 2 * ((size_t)run * 4 * fstride + (size_t)y * K1) : a.rnl + (size_t)run * 4 * fstride;
    const float2* __restrict__ mean = a.adir + (size_t)run * 4 * N3 * g.Pp;   // (0,0) modes of the direct totals

    // the input rows of level t: the adjoint fields, the direct ones, (their y
    // derivatives); 3D as the pairs (u1, u3), (b, u2), 2D as rows u1, u3, b
    auto prefetch = [&](int t) {
      if (t < 0 || t >= N3) return;
#pragma unroll
      for (int i = 0; i < 6; i++) {
        if (D3) {
          const float2* src = a.amix + 2 * ((size_t)(run * 6 + i) * fstride + (size_t)y * K1 + (size_t)t * tstride + l);
#pragma unroll
          for (int j = 0; j < (K1 + G - 1) / G; j++)
            if (l + G * j < K1) xm_cp16(stg + 2 * (i * K1 + l + G * j), src + 2 * G * j);
        } else {
          const int r = i % 3, f = r == 0 ? 0 : r + 1;
          const float2* src = (i < 3 ? a.S + (size_t)(run * 5 + f) * fstride : a.adir + (size_t)(run * 4 + f) * fstride);
          src += (size_t)t * tstride + l;
#pragma unroll
          for (int j = 0; j < (K1 + G - 1) / G; j++)
            if (l + G * j < K1) xm_cp8(stg + i * K1 + l + G * j, src + G * j);
        }
      }
    };
    auto kk = [&](int i) { return T::kmode(l, i); };
    auto Ca = [&](int i) -> float4& { return cbuf[i * G + l]; };
    auto Cb = [&](int i) -> float4& { return cbuf[(NKS + i) * G + l]; };
    // 3D: the pair p of combinations; 2D: field f (r1, r3, rB) alone
    auto store2 = [&](int p, int lvl, int i, float2 v, float2 w) {
      reinterpret_cast<float4*>(dst)[(size_t)p * fstride + (size_t)lvl * tstride + kk(i)] = make_float4(v.x, v.y, w.x, w.y);
    };
    auto store = [&](int f, int lvl, int i, float2 v) {
      if (lvl >= 0 && lvl < N3) dst[(size_t)f * fstride + (size_t)lvl * tstride + kk(i)] = v;
    };
    auto ikx = [&](float k, float2 v) { return make_float2(-k * v.y, k * v.x); };

    // this lane's points: what waits for the level above
    float g1[E], g2[D3 ? E : 1], dzp[E], f3a[E];
#pragma unroll
    for (int s = 0; s < E; s++) {
      g1[s] = dzp[s] = f3a[s] = 0.f;
      if (D3) g2[s] = 0.f;
    }
    prefetch(ta - 1);
    // step k, level t = ta - 1 + k: k = 0 only transforms the level's fields;
    // 1 <= k <= n forms its products and those of level t-1 that waited for
    // it; k = n + 1 only the latter
#pragma unroll 1
    for (int k = 0; k <= n + 1; k++) {
      const int t = ta - 1 + k, tm = t - 1;
      const bool lv = t >= 0 && t < N3, lvm = tm >= 0 && tm < N3;
      float4 *cur = ring + (size_t)(k & 1) * N1, *dcur = dring + (size_t)(k & 1) * N1;
      const float4 *prev = ring + (size_t)((k - 1) & 1) * N1, *dprev = dring + (size_t)((k - 1) & 1) * N1;
      // the c2r input of the pair (u1 + i u3, b + i u2) of the rows at st, times i kx with DX
      auto rows = [&](c2x (&x)[E], const float2* st, bool DX) {
#pragma unroll
        for (int e = 0; e < E; e++) {
          x[e] = c2x{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          if (G * e >= K1 && G * e + G - 1 <= N1 - K1) continue;   // zero at every lane
          const int n = l + G * e;
          const bool dir = n < K1, cnj = n > N1 - K1;
          const int m0 = dir ? n : (cnj ? N1 - n : 0), m = m0 + tok;
          const float on = (dir || cnj) ? 1.f : 0.f;
          const float sg = dir ? -1.f : 1.f;
          const float im0 = (n == 0) ? 0.f : on;             // k = 0: real parts only
          float2 A, B, C_, D = make_float2(0.f, 0.f);
          if (D3) {
            const float4 p = reinterpret_cast<const float4*>(st)[m], q = reinterpret_cast<const float4*>(st)[K1 + m];
            A = make_float2(p.x, p.y);
            B = make_float2(p.z, p.w);
            C_ = make_float2(q.x, q.y);
            D = make_float2(q.z, q.w);
          } else {
            A = st[m];
            B = st[K1 + m];
            C_ = st[2 * K1 + m];
          }
          if (DX) {
            const float kx = __ldg(a.kx + m0);
            A = ikx(kx, A);
            B = ikx(kx, B);
            C_ = ikx(kx, C_);
            D = ikx(kx, D);
          }
          if (lv)
            x[e] = c2x{make_float2(on * A.x + (sg * im0) * B.y, on * C_.x + (sg * im0) * D.y),
                       make_float2(on * B.x - (sg * im0) * A.y, on * D.x - (sg * im0) * C_.y)};
        }
      };
      xm_cp_wait();
      __syncwarp();
      {
        c2x x[E];
        rows(x, stg, false);
        T::template fft<true>(x, tbuf, tw4, tw2, l, w1);
#pragma unroll
        for (int s = 0; s < E; s++) cur[s * G + l] = c2x_f4(x[s]);
        tok = __float_as_int(x[0].re.x) & rz;
      }
      {
        c2x x[E];
        rows(x, stg + H * K1, false);
        T::template fft<true>(x, tbuf, tw4, tw2, l, w1);
#pragma unroll
        for (int s = 0; s < E; s++) dcur[s * G + l] = c2x_f4(x[s]);
        tok = __float_as_int(x[0].re.x) & rz;
      }
      if (k == 0) {
        __syncwarp();
        prefetch(t + 1);
        continue;
      }
      const bool fin = k >= 2;   // level t-1 belongs to this segment: finish it
      const float topm = (lvm && tm <= N3 - 2) ? 1.f : 0.f;   // Dir of level t-1 reaches level t
      // F1, F2 of level t-1: -(d U1T U1 + d U2T U2 + Dir(d U3T U3) + d BT B), d = ddx, ddy
      float F1[E], F2[D3 ? E : 1];
      auto forcing = [&](const c2x (&x)[E], float (&gp)[E], float (&F)[E]) {
#pragma unroll
        for (int s = 0; s < E; s++) {
          const float4 v = cur[s * G + l + tok];   // U1, B, U3, U2
          const float h = 0.5f * (x[s].im.x * v.z);
          F[s] = -(gp[s] + topm * h);
          gp[s] = x[s].re.x * v.x + (D3 ? x[s].im.y * v.w : 0.f) + h + x[s].re.y * v.y;
        }
      };
      {
        c2x x[E];
        rows(x, stg + H * K1, true);
        if (!D3) {
          __syncwarp();   // the staged rows are read: the next level's copies may start
          if (k <= n) prefetch(t + 1);
        }
        T::template fft<true>(x, tbuf, tw4, tw2, l, w1);
        forcing(x, g1, F1);
        tok = __float_as_int(x[0].re.x) & rz;
      }
      if constexpr (D3) {
        c2x x[E];
        rows(x, stg + 2 * H * K1, false);
        __syncwarp();
        if (k <= n) prefetch(t + 1);
        T::template fft<true>(x, tbuf, tw4, tw2, l, w1);
        forcing(x, g2, F2);
        tok = __float_as_int(x[0].re.x) & rz;
      }

      // ---- coefficients of level t and of level t-1 ----
      const bool lo = lv && t >= 1, lom = lvm && tm >= 1;
      const float lof = lo ? 1.f : 0.f, hb = 0.5f * lof, lm = lvm ? 1.f : 0.f;
      const float tlo = lo ? zc[ZC_TILDE_LO * N3 + t] : 0.f, tdi = lo ? zc[ZC_TILDE_DI * N3 + t] : 0.f;
      const float flo = lo ? zc[ZC_FULL_LO * N3 + t] : 0.f, fdi = lo ? zc[ZC_FULL_DI * N3 + t] : 0.f;
      const float flm = lom ? zc[ZC_FULL_LO * N3 + tm] : 0.f, fdm = lom ? zc[ZC_FULL_DI * N3 + tm] : 0.f;
      const float ndl = (lv && t >= 2) ? zc[ZC_DND_LO * N3 + t] : 0.f, ndd = (lv && t >= 2) ? zc[ZC_DND_DI * N3 + t] : 0.f;
      const float dnm = lom ? zc[ZC_DDN_DI * N3 + tm] : 0.f, dum = (lom && tm < N3 - 1) ? zc[ZC_DDN_UP * N3 + tm] : 0.f;
      const float avB = lv ? mean[((size_t)3 * N3 + t) * g.Pp].x : 0.f, avW = lvm ? mean[((size_t)2 * N3 + tm) * g.Pp].x : 0.f;
      const float fu = fin ? dum : 0.f;
      const float fd = (fin && lvm && tm >= 2) ? zc[ZC_DND_DI * N3 + tm] : 0.f;
      const float sd = lo ? zc[ZC_DDN_DI * N3 + t] : 0.f;
      const float lvf = lv ? 1.f : 0.f;

      // the forward transform pairs, one batch at a time: b = 0 the forcings of
      // level t-1 (fin), 1 Q and D, 2 the i kx products, 3 (3D) the C_fy ones (k <= n)
      const int nb = k <= n ? (D3 ? 4 : 3) : 2;
#pragma unroll 1
      for (int b = 0; b < nb; b++) {
        c2x z[E];
        if (b == 0) {
#pragma unroll
          for (int s = 0; s < E; s++) {
            const float4 v = cur[s * G + l + tok], p = prev[s * G + l + tok];
            const float4 d = dcur[s * G + l + tok], q = dprev[s * G + l + tok];
            // F3 of level t-1 = f3a - Full(ddz U3T) U3, ddz U3T of level t-1 from U3T of both
            const float dz = dnm * q.z + dum * d.z;
            const float F3 = f3a[s] - (flm * dzp[s] + fdm * dz) * p.z;
            dzp[s] = dz;
            // FB of level t-1 = (U3T - <u3T>)/K + Ri Dir(U3)
            const float FB = iK * (q.z - avW) + Ri * (0.5f * p.z + 0.5f * topm * v.z);
            // level t's (BT - <bT>)/K - (ddz(u1T) Full(U1) + ddz(u2T) Full(U2) + ddz(bT) Full(B))
            float w = (ndl * q.x + ndd * d.x) * (flo * p.x + fdi * v.x) + (ndl * q.y + ndd * d.y) * (flo * p.y + fdi * v.y);
            if (D3) w += (ndl * q.w + ndd * d.w) * (flo * p.w + fdi * v.w);
            f3a[s] = lvf * (iK * (d.y - avB)) - w;
            z[T::pos(s)] = c2x{make_float2(lm * F1[s], lm * F3), make_float2(D3 ? lm * F2[D3 ? s : 0] : 0.f, lm * FB)};
          }
          if (!fin) continue;
        } else if (b == 1) {
#pragma unroll
          for (int s = 0; s < E; s++) {
            const float4 v = cur[s * G + l + tok], p = prev[s * G + l + tok];
            const float4 d = dcur[s * G + l + tok], q = dprev[s * G + l + tok];
            const float D = lm * ((0.5f * p.z + 0.5f * topm * v.z) * (0.5f * q.z + 0.5f * topm * d.z));
            const float q1 = hb * (v.x + p.x) * d.z, qb = hb * (v.y + p.y) * d.z;
            z[T::pos(s)] = D3 ? c2x{make_float2(q1, hb * (v.w + p.w) * d.z), make_float2(qb, D)}
                              : c2x{make_float2(q1, D), make_float2(qb, 0.f)};
          }
        } else if (b == 2) {
#pragma unroll
          for (int s = 0; s < E; s++) {
            const float4 v = cur[s * G + l + tok], d = dcur[s * G + l + tok], q = dprev[s * G + l + tok];
            const float c3 = (tdi * d.x + tlo * q.x) * v.z;
            z[T::pos(s)] = D3 ? c2x{make_float2(v.x * d.x, v.w * d.x), make_float2(v.y * d.x, c3)}
                              : c2x{make_float2(v.x * d.x, c3), make_float2(v.y * d.x, 0.f)};
          }
        } else {
#pragma unroll
          for (int s = 0; s < E; s++) {
            const float4 v = cur[s * G + l + tok], d = dcur[s * G + l + tok], q = dprev[s * G + l + tok];
            z[T::pos(s)] = c2x{make_float2(v.x * d.w, (tdi * d.w + tlo * q.w) * v.z), make_float2(v.w * d.w, v.y * d.w)};
          }
        }
        T::template fft<false>(z, tbuf, tw4, tw2, l, w1);
#pragma unroll
        for (int i = 0; i < NKS; i++) {
          const int s = T::kslot(i);
          const c2x zs = z[s];
          const c2x po = z[T::partner(i, false)];
          c2x p;
          p.re.x = __shfl_sync(0xffffffffu, po.re.x, partner_lane);
          p.re.y = __shfl_sync(0xffffffffu, po.re.y, partner_lane);
          p.im.x = __shfl_sync(0xffffffffu, po.im.x, partner_lane);
          p.im.y = __shfl_sync(0xffffffffu, po.im.y, partner_lane);
          if (l == 0) p = z[T::partner(i, true)];
          if (kk(i) >= K1) continue;
          const float2 SR = pmul(padd(zs.re, p.re), SC), DI = pmul(psub(zs.im, p.im), SC);
          const float2 SI = pmul(padd(zs.im, p.im), SC), DR = pmul(psub(p.re, zs.re), SC);
          const float2 A1 = make_float2(SR.x, DI.x), A2 = make_float2(SI.x, DR.x);   // transform A's products
          const float2 B1 = make_float2(SR.y, DI.y), B2 = make_float2(SI.y, DR.y);   // transform B's
          if (b == 0) {   // F1, F2, F3, FB of level t-1 join what it carries
            const float4 ca = Ca(i), cb = Cb(i);
            Ca(i) = make_float4(ca.x + A1.x, ca.y + A1.y, ca.z + B2.x, ca.w + B2.y);
            Cb(i) = make_float4(cb.x + A2.x, cb.y + A2.y, cb.z + B1.x, cb.w + B1.y);
          } else if (b == 1) {   // Q1, QB; 3D Q2, D; 2D D
            const float2 Dp = D3 ? B2 : B1;
            if (fin) {
              const float4 ca = Ca(i), cb = Cb(i);
              const float2 c1 = make_float2(ca.x + fu * A1.x, ca.y + fu * A1.y);
              const float2 cB = make_float2(ca.z + fu * A2.x, ca.w + fu * A2.y);
              const float2 c3 = make_float2(cb.z + fd * Dp.x, cb.w + fd * Dp.y);
              if (D3) {
                store2(0, tm, i, c1, cB);
                store2(2, tm, i, make_float2(cb.x + fu * B1.x, cb.y + fu * B1.y), c3);
              } else {
                store(0, tm, i, c1);
                store(2, tm, i, c3);
                store(3, tm, i, cB);
              }
            }
            Ca(i) = make_float4(sd * A1.x, sd * A1.y, sd * A2.x, sd * A2.y);
            Cb(i) = D3 ? make_float4(sd * B1.x, sd * B1.y, ndl * Dp.x, ndl * Dp.y)
                       : make_float4(0.f, 0.f, ndl * Dp.x, ndl * Dp.y);
          } else if (b == 2) {   // U1 U1T, B U1T; 3D U2 U1T, Tilde(U1T) U3; 2D Tilde(U1T) U3
            const float kx = __ldg(a.kx + kk(i));
            const float2 a1 = ikx(kx, A1), aB = ikx(kx, A2), b1 = ikx(kx, B1), b2 = ikx(kx, B2);
            const float4 ca = Ca(i), cb = Cb(i);
            Ca(i) = make_float4(ca.x + a1.x, ca.y + a1.y, ca.z + aB.x, ca.w + aB.y);
            Cb(i) = D3 ? make_float4(cb.x + b1.x, cb.y + b1.y, cb.z + b2.x, cb.w + b2.y)
                       : make_float4(0.f, 0.f, cb.z + b1.x, cb.w + b1.y);
          } else {   // U1 U2T, U2 U2T, Tilde(U2T) U3, B U2T
            store2(1, t, i, A1, B2);
            store2(3, t, i, A2, B1);
          }
        }
        tok = __float_as_int(z[0].re.x) & rz;
      }
    }
  }
}

template <int N1, bool D3>
static void adjmarch_launch(const StageArgs& a, cudaStream_t st) {
  using X = AMShape<N1, D3>;
  const Geo& g = a.g;
  const int nsm = sm_count();
  if (D3) {
    launch_chained(k_adjmarch<N1, D3>, dim3(nsm), X::WARPS * 32, X::smem(X::WARPS), st, a.chained, a, 0);
    return;
  }
  const long long room = (long long)nsm * X::WARPS * X::W;   // 2D: as k_xmarch's segments
  const int seg = (int)(((long long)g.nrun * g.N3 + room - 1) / room);
  const long long warps = ((long long)g.nrun * ((g.N3 + seg - 1) / seg) + X::W - 1) / X::W;
  const int wb = (int)std::min<long long>(X::WARPS, (warps + nsm - 1) / nsm);
  launch_chained(k_adjmarch<N1, D3>, dim3((unsigned)((warps + wb - 1) / wb)), wb * 32, X::smem(wb), st, a.chained, a, seg);
}

// the grids whose rows have a march layout of 8 points per lane
bool adjmarch_supported(const Geo& g) {
  if (g.dim3) return (g.N1 == 64 || g.N1 == 128 || g.N1 == 256) && g.N2 % 4 == 0;
  return g.N1 >= 32 && g.N1 <= 256;
}

int launch_adjmarch(const StageArgs& a, cudaStream_t st) {
  const bool d3 = a.g.dim3 != 0;
  switch (a.g.N1) {
    case 32: adjmarch_launch<32, false>(a, st); break;
    case 64: d3 ? adjmarch_launch<64, true>(a, st) : adjmarch_launch<64, false>(a, st); break;
    case 128: d3 ? adjmarch_launch<128, true>(a, st) : adjmarch_launch<128, false>(a, st); break;
    case 256: d3 ? adjmarch_launch<256, true>(a, st) : adjmarch_launch<256, false>(a, st); break;
    default: return 0;
  }
  return 1;
}

template <int N1, bool D3>
static cudaError_t adjmarch_attr() {
  return cudaFuncSetAttribute(k_adjmarch<N1, D3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)AMShape<N1, D3>::smem(AMShape<N1, D3>::WARPS));
}
int prepare_adjmarch_kernels() {
  for (cudaError_t e : {adjmarch_attr<64, true>(), adjmarch_attr<128, true>(), adjmarch_attr<256, true>(),
                        adjmarch_attr<32, false>(), adjmarch_attr<64, false>(), adjmarch_attr<128, false>(),
                        adjmarch_attr<256, false>()})
    if (e != cudaSuccess) return -1;
  return 0;
}

}  // namespace sf
