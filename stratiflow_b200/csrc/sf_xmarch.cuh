// The marching x pass' device code (sf_xmarch.cu describes it), shared by
// k_xmarch and the ensembles' stage kernel (sf_ens.cu).
#pragma once
#include "sf_xmt.cuh"

namespace sf {

// D3: 3D rows (else 2D); MODE 0: BuildRHS; 1: BuildRHSLinear about the frozen
// nodal base; 2: about the live state of the base run
// CR: the carried combinations in registers instead of shared memory (where
// a warp has 168 registers and needs no more; the ensembles' kernel, which
// holds its z items too, spills: a stage of 64 members 159 us without, 164 with)
template <int N1, bool D3, int MODE, bool CR = (XMT<N1>::NKS <= 3 && MODE == 0)>
struct XMShape : XMT<N1> {
  using T = XMT<N1>;
  // shared memory of one row: two levels of nodal values (float4 per x
  // point, a ring: this level and the one below), those of the base (MODE 1,
  // 2), the transpose buffer, the carried combinations ((c1, cB), (c2, c3) per
  // kept slot and lane; 2D: c3 alone in the second) and the staged input rows
  // of the next level (2 rows of pairs or 3 rows x K1, and the base run's)
  static constexpr int ROWS = D3 ? 4 : 3;
  static constexpr size_t group_bytes =
      (sizeof(float4) * (size_t)((MODE ? 4 : 2) * N1 + T::TB + (CR ? 0 : 2 * T::NKS * T::G)) +
       sizeof(float2) * (MODE == 2 ? 2 : 1) * ROWS * T::K1 + 15) / 16 * 16;
  static constexpr size_t table_bytes = (sizeof(float4) + sizeof(float2)) * (size_t)T::TWE;
  // warps of a block, one block per SM: as many as the shared memory takes,
  // 12 at most (168 registers)
  static constexpr int fit = (int)((227 * 1024 - table_bytes) / (T::W * group_bytes));
  static constexpr int WARPS = fit > 12 ? 12 : fit;
  static constexpr size_t smem(int warps) { return table_bytes + (size_t)warps * T::W * group_bytes; }
  static_assert(table_bytes % 16 == 0, "16-byte aligned regions");
  static_assert(WARPS >= 1, "one warp fits an SM");
};

// the transform tables of one grid width at the start of the block's shared memory
template <int N1>
__device__ __forceinline__ void xmarch_tables(unsigned char* xsm, const float2* tw) {
  using T = XMT<N1>;
  T::fill(reinterpret_cast<float4*>(xsm), reinterpret_cast<float2*>(xsm + sizeof(float4) * T::TWE), tw, threadIdx.x,
          blockDim.x);
}

// Units u .. uend - 1 by the calling warp, of levels t_lo .. t_hi - 1 of every
// row of runs a.run_offset .. + nruns - 1. 3D: units (run, block of W y rows,
// level). 2D: a unit is W segments of seg levels, one per lane group (the
// groups of a warp march in step, each on its own segment). The block has
// filled the tables (and waited); each warp has its own part of xsm.
template <int N1, bool D3, int MODE, bool CR = (XMT<N1>::NKS <= 3 && MODE == 0)>
__device__ __forceinline__ void xmarch_rows(const StageArgs& a, unsigned char* xsm, int nruns, int t_lo, int t_hi, int seg,
                                            long long u, const long long uend) {
  using X = XMShape<N1, D3, MODE, CR>;
  using T = XMT<N1>;
  constexpr int G = T::G, E = T::E, K1 = T::K1, W = T::W, NKS = T::NKS, ROWS = X::ROWS;
  const Geo& g = a.g;
  const int N3 = g.N3, N2 = D3 ? g.N2 : 1;
  const float4* tw4 = reinterpret_cast<const float4*>(xsm);
  const float2* tw2 = reinterpret_cast<const float2*>(xsm + sizeof(float4) * T::TWE);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gw = lane / G, l = lane - gw * G;
  __builtin_assume(l >= 0 && l < G);
  unsigned char* gb = xsm + X::table_bytes + (size_t)(warp * W + gw) * X::group_bytes;
  float4* ring = reinterpret_cast<float4*>(gb);     // [2 levels][E slots][G lanes]: u1, b, u3, u2
  float4* bring = ring + 2 * N1;                    // MODE 1, 2: the base's (U_ in u1)
  float4* tbuf = ring + (MODE ? 4 : 2) * N1;        // transpose buffer
  float4* cbuf = tbuf + T::TB;                      // [2][NKS][G]: (c1, cB), (c2, c3) awaiting their z terms
  float2* stg = reinterpret_cast<float2*>(cbuf + (CR ? 0 : 2 * NKS * G));   // 3D [2][K1] pairs (u1, u3), (b, u2) of the next level, 2D [3][K1] u1, u3, b; then the base run's
  const int partner_lane = (lane & ~(G - 1)) | ((G - l) & (G - 1));
  // the first-stage twiddles of the 128- and 256-point transforms, held in registers
  float4 w1[8];
#pragma unroll
  for (int k = 0; k < 8; k++)
    w1[k] = (N1 == 256 || N1 == 128) ? tw4[(k * G + l) % T::TWE] : make_float4(0.f, 0.f, 0.f, 0.f);
  // zero, but not known to the compiler: a batch's shared-memory reads take
  // (bits of the last batch's result) & rz as an offset, a true dependency
  // that keeps the compiler from starting one batch's products and
  // transform under the last one's, which would need both register sets
  const int rz = (int)(gridDim.x >> 30);
  int tok = 0;
  const float* __restrict__ zc = a.zc;
  const float sc = 0.5f * g.inv_n12;
  const float2 SC = make_float2(sc, sc);

  const int L = t_hi - t_lo;
  // 3D: units of one level; 2D: segments, W side by side
  const long long NYB = D3 ? N2 / W : (L + seg - 1) / seg;

  while (u < uend) {
    int run, y = 0, ta, n;   // n levels from ta; every group of the warp has the same n
    bool act = true;
    if (D3) {
      const long long rb = u / L;
      ta = t_lo + (int)(u - rb * L);
      n = (int)std::min<long long>(t_hi - ta, uend - u);
      u += n;
      run = (int)(rb / NYB);
      y = (int)(rb % NYB) * W + gw;
    } else {
      const long long sg = u * W + gw;
      u++;
      act = sg < nruns * NYB;
      run = act ? (int)(sg / NYB) : 0;
      ta = act ? t_lo + (int)(sg % NYB) * seg : N3 + 2;   // an idle group marches through levels that do not exist
      n = seg;
    }
    run += a.run_offset;
    const int brun = MODE == 2 ? (run - a.tlm) % a.tlm : run;
    const float* __restrict__ Ub = a.Ubar + (size_t)run * N3;
    const float* __restrict__ UbB = a.Ubar + (size_t)brun * N3;
    const size_t tstride = D3 ? (size_t)N2 * K1 : (size_t)g.Pp, fstride = (size_t)N3 * tstride;
    // 3D: rows of pairs at src + 2 (pair * fstride + t * tstride); 2D: rows at src + field * fstride + t * tstride
    const float2* __restrict__ src = D3 ? a.mixin + 2 * ((size_t)run * 2 * fstride + (size_t)y * K1) : a.S + (size_t)run * 5 * fstride;
    const float2* __restrict__ bsrc =
        D3 ? a.mixin + 2 * ((size_t)brun * 2 * fstride + (size_t)y * K1) : a.S + (size_t)brun * 5 * fstride;
    float2* __restrict__ dst = D3 ? a.mixout + 2 * ((size_t)run * 4 * fstride + (size_t)y * K1) : a.rnl + (size_t)run * 4 * fstride;
    const float* __restrict__ bnod = MODE == 1 ? a.base + ((size_t)run * 4 * N3 * N2 + y) * N1 : nullptr;

    // the input rows of level t into the stage by asynchronous copies (16
    // bytes for a pair, 8 in 2D, where a row of K1 complex values is not
    // 16-byte aligned in general)
    auto prefetch = [&](int t) {
      if (t < 0 || t >= N3) return;
      constexpr int R = D3 ? 2 : 3;
#pragma unroll
      for (int i = 0; i < (MODE == 2 ? 2 : 1) * R; i++) {
        const int r = i % R;
        const float2* sf = (i < R ? src : bsrc);
        if (D3) {
          sf += 2 * (r * fstride + (size_t)t * tstride + l);
#pragma unroll
          for (int j = 0; j < (K1 + G - 1) / G; j++)
            if (l + G * j < K1) xm_cp16(stg + 2 * (i * K1 + l + G * j), sf + 2 * G * j);
        } else {
          sf += (r == 0 ? 0 : r + 1) * fstride + (size_t)t * tstride + l;
#pragma unroll
          for (int j = 0; j < (K1 + G - 1) / G; j++)
            if (l + G * j < K1) xm_cp8(stg + i * K1 + l + G * j, sf + G * j);
        }
      }
    };
    // this lane's kept mode in kept slot i
    auto kk = [&](int i) { return T::kmode(l, i); };
    // c1, cB and c2, c3 of the last level, awaiting their z terms, per kept slot
    float4 ca_[CR ? NKS : 1], cb_[CR ? NKS : 1];
    auto Ca = [&](int i) -> float4& { return CR ? ca_[CR ? i : 0] : cbuf[i * G + l]; };
    auto Cb = [&](int i) -> float4& { return CR ? cb_[CR ? i : 0] : cbuf[(NKS + i) * G + l]; };
    // 3D: the pair p of combinations; 2D: field f (r1, r3, rB) alone
    auto store2 = [&](int p, int lvl, int i, float2 v, float2 w) {
      reinterpret_cast<float4*>(dst)[(size_t)p * fstride + (size_t)lvl * tstride + kk(i)] = make_float4(v.x, v.y, w.x, w.y);
    };
    auto store = [&](int f, int lvl, int i, float2 v) {
      if (lvl < t_hi && lvl >= t_lo) dst[(size_t)f * fstride + (size_t)lvl * tstride + kk(i)] = v;
    };
    auto mikx = [&](float k, float2 v) { return make_float2(k * v.y, -k * v.x); };   // -(i k) v

    prefetch(ta - 1);
    // step k, level t = ta - 1 + k: the inverse transform of level t, then (1
    // <= k <= n) every product of level t and P4 of level t-1, or (k = n + 1)
    // only Q1, QB, Q2 of level t and P4 of level t-1 (k = 0 only transforms)
#pragma unroll 1
    for (int k = 0; k <= n + 1; k++) {
      const int t = ta - 1 + k;
      const bool lv = t >= 0 && t < N3;
      const bool flow = !D3 || lv;   // the same for every group of the warp
      // c2r input of the pair (u1 + i u3, b + i u2) at n = l + G e: A + iB
      // at n < K1 (real parts only at n = 0), conj(A) + i conj(B) of mode
      // N1 - n at n > N1 - K1, zero between; one load per field from the
      // mode index and a sign, so no position loads two rows
      auto rows = [&](c2x (&x)[E], const float2* st) {
#pragma unroll
        for (int e = 0; e < E; e++) {
          if (G * e >= K1 && G * e + G - 1 <= N1 - K1) {   // zero at every lane
            x[e] = c2x{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            continue;
          }
          const int n = l + G * e;
          const bool dir = n < K1, cnj = n > N1 - K1;
          const int m = (dir ? n : (cnj ? N1 - n : 0)) + tok;
          const float on = (dir || cnj) ? 1.f : 0.f;
          const float sg = dir ? -1.f : 1.f;                 // A.x + sg B.y, B.x - sg A.y
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
          const float2 re = make_float2(on * A.x + (sg * im0) * B.y, on * C_.x + (sg * im0) * D.y);
          const float2 im = make_float2(on * B.x - (sg * im0) * A.y, on * D.x - (sg * im0) * C_.y);
          x[e] = c2x{re, im};
          if (!D3 && !lv) x[e] = c2x{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        }
      };
      float4* curl = ring + (size_t)(k & 1) * N1;
      const float4* prev = ring + (size_t)((k - 1) & 1) * N1;
      float4* bcur = bring + (size_t)(k & 1) * N1;
      const float4* bprev = bring + (size_t)((k - 1) & 1) * N1;
      // MODE 1: the base's nodal values, on their way while the level is transformed
      float bv[MODE == 1 ? E : 1][4];
      if (MODE == 1) {
#pragma unroll
        for (int s = 0; s < E; s++)
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const int f = c == 0 ? 0 : (c == 1 ? 3 : (c == 2 ? 2 : 1));
            bv[s][c] = (lv && (D3 || f != 1)) ? __ldcs(bnod + ((size_t)f * N3 + t) * N2 * N1 + T::pos(s) * G + l) : 0.f;
          }
      }
      // level t into its ring slot (u1, b, u3, u2 per x point; zero outside 0..N3-1)
      c2x x[E];   // MODE 0: and kept for the first batch
      if (flow) {
        xm_cp_wait();
        __syncwarp();
        rows(x, stg);
        if (MODE != 2) {
          __syncwarp();   // the staged rows are read: the next level's copies may start
          if (k <= n) prefetch(t + 1);
        }
        T::template fft<true>(x, tbuf, tw4, tw2, l, w1);
#pragma unroll
        for (int s = 0; s < E; s++) curl[s * G + l] = c2x_f4(x[s]);
        tok = __float_as_int(x[0].re.x) & rz;
        if (MODE == 2) {
          rows(x, stg + ROWS * K1);
          __syncwarp();
          if (k <= n) prefetch(t + 1);
          T::template fft<true>(x, tbuf, tw4, tw2, l, w1);
          const float ub = lv ? UbB[t] : 0.f;
#pragma unroll
          for (int s = 0; s < E; s++) {
            float4 v = c2x_f4(x[s]);
            v.x += ub;
            bcur[s * G + l] = v;
          }
          tok = __float_as_int(x[0].re.x) & rz;
        }
      } else {
        __syncwarp();
        if (k <= n) prefetch(t + 1);
#pragma unroll
        for (int s = 0; s < E; s++) {
          x[s] = c2x{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          curl[s * G + l] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (MODE == 2) {
#pragma unroll
          for (int s = 0; s < E; s++) bcur[s * G + l] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      if (MODE == 1) {
        const float ub = lv ? Ub[t] : 0.f;
#pragma unroll
        for (int s = 0; s < E; s++) bcur[s * G + l] = make_float4(bv[s][0] + ub, bv[s][1], bv[s][2], bv[s][3]);
      }
      if (k == 0) continue;

      // ---- coefficients of level t (products) and of the combinations ----
      const bool lo = lv && t >= 1, lvm = t >= 1 && t - 1 < N3;
      const float lof = lo ? 1.f : 0.f, hb = 0.5f * lof, lm = lvm ? 1.f : 0.f;
      const float ub = lv ? Ub[t] : 0.f, ubm = lo ? Ub[t - 1] : 0.f;
      const float tlo = lo ? zc[ZC_TILDE_LO * N3 + t] : 0.f, tdi = lo ? zc[ZC_TILDE_DI * N3 + t] : 0.f;
      const float topm = (t - 1 <= N3 - 2) ? 1.f : 0.f;   // Dir(u3) of level t-1 reaches level t
      const int tm = t - 1;
      const bool fin = k >= 2;   // level t-1 belongs to this segment: finish it
      const float fu = (fin && tm >= 1 && tm < N3 - 1) ? zc[ZC_DDN_UP * N3 + tm] : 0.f;
      const float fd = (fin && tm >= 2 && tm < N3) ? zc[ZC_DND_DI * N3 + tm] : 0.f;
      const float sd = (lv && t >= 1) ? zc[ZC_DDN_DI * N3 + t] : 0.f;
      const float sl = (lv && t >= 2) ? zc[ZC_DND_LO * N3 + t] : 0.f;

      // the forward transform pairs of the step, one batch at a time:
      //   3D b = 0: Q1 + i QB, Q2 + i P4 (level t-1)   [1 <= k <= n + 1]
      //      b = 1: S1 + i SB1, S12 + i SB2            [k <= n]
      //      b = 2: P3 + i P3Y, S22                    [k <= n]
      //   2D b = 0: Q1 + i QB, P4 (level t-1)
      //      b = 1: S1 + i SB1, P3
      const int nb = k <= n ? (D3 ? 3 : 2) : 1;
      auto batch = [&](int b, auto first) __attribute__((always_inline)) {
        constexpr bool F0 = decltype(first)::value;   // b = 0
        c2x z[E];
        // the value of a product of two linear forms: x y, or its derivative
        // about the base, x Y + X y
        auto pr = [&](float x, float y, float X, float Y) { return MODE ? x * Y + X * y : x * y; };
        if (F0) {
#pragma unroll
          for (int s = 0; s < E; s++) {
            const float4 pv = prev[s * G + l + tok], cv = MODE == 0 ? c2x_f4(x[s]) : curl[s * G + l + tok];   // u1, b, u3, u2 of t-1, t
            const float U1 = cv.x, Bv = cv.y, U3 = cv.z, U2 = cv.w;
            const float w3 = lof * U3;
            float q1 = hb * U1 + hb * pv.x, qb = hb * Bv + hb * pv.y, q2 = hb * U2 + hb * pv.w, p4;
            if (MODE == 0) {
              q1 = (q1 + (hb * ubm + hb * ub)) * w3;
              qb *= w3;
              q2 *= w3;
              const float d = 0.5f * pv.z + 0.5f * topm * U3;
              p4 = d * d;
            } else {
              const float4 bp = bprev[s * G + l + tok], bc = bcur[s * G + l + tok];
              const float W3 = lof * bc.z;
              q1 = pr(q1, w3, hb * bc.x + hb * bp.x, W3);
              qb = pr(qb, w3, hb * bc.y + hb * bp.y, W3);
              q2 = pr(q2, w3, hb * bc.w + hb * bp.w, W3);
              p4 = (pv.z + topm * U3) * (0.5f * bp.z + 0.5f * topm * bc.z);
            }
            z[T::pos(s)] = D3 ? c2x{make_float2(q1, q2), make_float2(qb, lm * p4)}
                              : c2x{make_float2(q1, lm * p4), make_float2(qb, 0.f)};
          }
        } else if (b == 1) {
#pragma unroll
          for (int s = 0; s < E; s++) {
            const float4 cv = curl[s * G + l + tok];
            const float U1 = cv.x, Bv = cv.y, U2 = cv.w;
            float s1, sb1, s12, sb2;
            float4 bc;
            if (MODE == 0) {
              const float u1t = U1 + ub;
              s1 = U1 * (U1 + 2.f * ub);
              sb1 = u1t * Bv;
              s12 = u1t * U2;
              sb2 = U2 * Bv;
            } else {
              bc = bcur[s * G + l + tok];
              s1 = (2.f * U1) * bc.x;
              sb1 = Bv * bc.x + bc.y * U1;
              s12 = U1 * bc.w + bc.x * U2;
              sb2 = Bv * bc.w + bc.y * U2;
            }
            if (D3) {
              z[T::pos(s)] = c2x{make_float2(s1, s12), make_float2(sb1, sb2)};
            } else {
              const float4 pv = prev[s * G + l + tok];
              const float w3 = lof * cv.z;
              float p3 = tdi * U1 + tlo * pv.x;
              if (MODE == 0) {
                p3 = (p3 + (tlo * ubm + tdi * ub)) * w3;
              } else {
                const float4 bp = bprev[s * G + l + tok];
                p3 = pr(p3, w3, tdi * bc.x + tlo * bp.x, lof * bc.z);
              }
              z[T::pos(s)] = c2x{make_float2(s1, p3), make_float2(sb1, 0.f)};
            }
          }
        } else {
#pragma unroll
          for (int s = 0; s < E; s++) {
            const float4 pv = prev[s * G + l + tok], cv = curl[s * G + l + tok];
            const float U1 = cv.x, U3 = cv.z, U2 = cv.w;
            const float w3 = lof * U3;
            float p3 = tdi * U1 + tlo * pv.x, p3y = tdi * U2 + tlo * pv.w, s22;
            if (MODE == 0) {
              p3 = (p3 + (tlo * ubm + tdi * ub)) * w3;
              p3y *= w3;
              s22 = U2 * U2;
            } else {
              const float4 bp = bprev[s * G + l + tok], bc = bcur[s * G + l + tok];
              const float W3 = lof * bc.z;
              p3 = pr(p3, w3, tdi * bc.x + tlo * bp.x, W3);
              p3y = pr(p3y, w3, tdi * bc.w + tlo * bp.w, W3);
              s22 = (2.f * U2) * bc.w;
            }
            z[T::pos(s)] = c2x{make_float2(p3, s22), make_float2(p3y, 0.f)};
          }
        }
        T::template fft<false>(z, tbuf, tw4, tw2, l, w1);
        // split each transform of the pair into its two real products at
        // the kept modes: (Z_k + conj Z_{N-k}) / 2 and (Z_k - conj Z_{N-k}) / (2i),
        // times 1/(N1 N2)
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
          if (F0) {   // A1 = Q1, A2 = QB; 3D B1 = Q2, B2 = P4 of level t-1; 2D B1 = P4
            const float2 P4 = D3 ? B2 : B1;
            if (fin) {
              const float4 ca = Ca(i), cb = Cb(i);
              const float2 c1 = make_float2(ca.x - fu * A1.x, ca.y - fu * A1.y);
              const float2 cB = make_float2(ca.z - fu * A2.x, ca.w - fu * A2.y);
              const float2 c3 = make_float2(cb.z - fd * P4.x, cb.w - fd * P4.y);
              if (D3) {
                store2(0, tm, i, c1, cB);
                store2(2, tm, i, make_float2(cb.x - fu * B1.x, cb.y - fu * B1.y), c3);
              } else {
                store(0, tm, i, c1);
                store(2, tm, i, c3);
                store(3, tm, i, cB);
              }
            }
            Ca(i) = make_float4(-sd * A1.x, -sd * A1.y, -sd * A2.x, -sd * A2.y);
            Cb(i) = make_float4(-sd * B1.x, -sd * B1.y, -sl * P4.x, -sl * P4.y);
          } else if (b == 1) {   // 3D S1, SB1, S12, SB2; 2D S1, SB1, P3
            const float k = __ldg(a.kx + kk(i));
            const float2 a1 = mikx(k, A1), aB = mikx(k, A2), a2 = mikx(k, B1);
            const float4 ca = Ca(i), cb = Cb(i);
            Ca(i) = make_float4(a1.x + ca.x, a1.y + ca.y, aB.x + ca.z, aB.y + ca.w);
            if (D3) {
              Cb(i) = make_float4(a2.x + cb.x, a2.y + cb.y, cb.z, cb.w);
              store2(1, t, i, make_float2(-B1.x, -B1.y), make_float2(-B2.x, -B2.y));
            } else {
              Cb(i) = make_float4(0.f, 0.f, cb.z + a2.x, cb.w + a2.y);
            }
          } else {   // P3, P3Y, S22
            const float2 a3 = mikx(__ldg(a.kx + kk(i)), A1);
            const float4 cb = Cb(i);
            Cb(i) = make_float4(cb.x, cb.y, cb.z + a3.x, cb.w + a3.y);
            store2(3, t, i, make_float2(-B1.x, -B1.y), make_float2(-A2.x, -A2.y));
          }
        }
        tok = __float_as_int(z[0].re.x) & rz;
      };
      batch(0, std::true_type{});
#pragma unroll 1
      for (int b = 1; b < nb; b++) batch(b, std::false_type{});
    }
  }
}

}  // namespace sf
