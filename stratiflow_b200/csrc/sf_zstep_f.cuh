// The z pass of a stage (ExplicitRK, FinishRHS, CrankNicolson and the Thomas
// solves of every field, IMEXRK.cpp:75-134, then RemoveDivergence,
// IMEXRK.cpp:43-73) with all fields of a mode group solved at once.
//
// What bounds k_z_step_c (sf_zstep_c.cuh), which solves a group's fields one
// after the other, is the latency of its serial chain: 4 or 5 systems, each
// three sweeps and two block-wide scans, and the new velocities go through
// global memory between the solves and the projection. The Crank-Nicolson
// systems do not depend on one another, so here a block owns 8 modes and its
// warps take (field, four z-chunks): every field's solve runs at the same
// time, the solutions stay in shared memory, and the projection, shared by
// all the warps in chunks NF times shorter, reads them there and writes each
// velocity once. Two scans for the solves, two for the projection, one barrier
// each. A warp's four chunks are composed by shuffles, the warps' maps by
// every lane for itself.
//
// 8 modes are 64 bytes of a level's row (two whole sectors); twice as many
// blocks as with 16 modes leave fewer SMs idle and a last wave half as long.
// Chunks of up to L = 4 or 8 levels live in registers (every input loaded at once,
// be_j and the pivots never reloaded); longer ones keep be_j / D_j in the
// block's shared rows and load the pivots again in each sweep, L = 0. What
// remains is the latency of those loads, about 1900 cycles under load at
// 256x128x384: fewer, larger batches are worth more than more warps (two
// blocks of 16 warps there take 243-290 us, one with twice the levels in
// flight 170).
//
// r_old: the buffers of r take turns over a step's stages, so nothing is copied
// for the next stage's zeta term (its own buffer was written each stage: 4 of
// 24 field-sized transfers); u3's and b's r are completed in place by the
// linear buoyancy terms, in the stages that another follows.
//
// The arithmetic of every term is k_z_step_c's, in the same order; the chunks
// are others, so the two agree to rounding.
#pragma once
#include "sf_zstep_c.cuh"

namespace sf {

constexpr int kFM = 8;   // modes per block
constexpr int kFI = 8;   // levels of pivots loaded ahead in a long chunk's later sweeps

constexpr int kFTabFloats = 21;   // floats per level of the tables in shared memory

// one launch's shape: NF fields, CQ warps per field of four chunks each
template <int NF, int CQ>
struct ZfShape {
  static constexpr int NW = NF * CQ, THREADS = 32 * NW, CC = 4 * CQ, CP = 4 * NW;
  // rows of the solutions (X), then two buffers of the warps' chunk maps
  // and, for long chunks, the coefficient tables, with the columns of p, u3 and b
  __host__ __device__ static size_t smem(int N3, bool tables, bool cols) {
    return sizeof(float2) * ((size_t)(NF + (cols ? 3 : 0)) * N3 * kFM + 2 * NW * kFM) + sizeof(float) * 2 * NW * kFM +
           (tables ? sizeof(float) * kFTabFloats * N3 : 0);
  }
};

// The per-level coefficients a block reads: the packed rows of the solver's
// tables (StageArgs::zt1, zt2, ztq, zac, dBdz), from shared memory when the
// chunks are long (SM; L1 beside two blocks' rows is too small to hold them,
// and an L2 latency per level is what each sweep would wait for), else from
// global memory, where a chunk's few rows are loaded with its inputs.
template <bool SM>
struct ZfTab {
  const float4 *n, *d, *t2, *q;   // d2z (Neumann) and u's a_j; d2z (Dirichlet) and u3's a_j; zt2; ztq
  const float4* c;                // b's a_j, the c_j of u, b, u3   (SM)
  const float4* nb;               // as n with b's a_j (global)
  const float* dB;
};

struct ZfMap {   // v -> A v + B
  float A;
  float2 B;
};

// The value entering this lane's chunk: the maps of the chunks below it (UP)
// or above it applied to 0. The lane's own map is m; the warp's four chunks
// are 8 lanes apart; wi of nw warps share the system, whose maps lie at
// WA / WB[k * kFM + ml], k < nw. Every thread of the block comes here.
template <bool UP>
__device__ __forceinline__ float2 zf_scan(ZfMap m, float* WA, float2* WB, int wi, int nw, int ml, int cs) {
  const unsigned full = 0xffffffffu;
#pragma unroll
  for (int d = 1; d < 4; d <<= 1) {
    const float A = UP ? __shfl_up_sync(full, m.A, 8 * d) : __shfl_down_sync(full, m.A, 8 * d);
    float2 B;
    B.x = UP ? __shfl_up_sync(full, m.B.x, 8 * d) : __shfl_down_sync(full, m.B.x, 8 * d);
    B.y = UP ? __shfl_up_sync(full, m.B.y, 8 * d) : __shfl_down_sync(full, m.B.y, 8 * d);
    if (UP ? cs >= d : cs + d < 4) {   // this map after the others'
      m.B = cfma(m.A, B, m.B);
      m.A *= A;
    }
  }
  if (cs == (UP ? 3 : 0)) {
    WA[wi * kFM + ml] = m.A;
    WB[wi * kFM + ml] = m.B;
  }
  ZfMap e;   // the warp's chunks before this one
  e.A = UP ? __shfl_up_sync(full, m.A, 8) : __shfl_down_sync(full, m.A, 8);
  e.B.x = UP ? __shfl_up_sync(full, m.B.x, 8) : __shfl_down_sync(full, m.B.x, 8);
  e.B.y = UP ? __shfl_up_sync(full, m.B.y, 8) : __shfl_down_sync(full, m.B.y, 8);
  if (cs == (UP ? 0 : 3)) e = ZfMap{1.f, cz()};
  __syncthreads();
  float2 v = cz();
  if (UP) {
#pragma unroll 4
    for (int k = 0; k < wi; k++) v = cfma(WA[k * kFM + ml], v, WB[k * kFM + ml]);
  } else {
#pragma unroll 4
    for (int k = nw - 1; k > wi; k--) v = cfma(WA[k * kFM + ml], v, WB[k * kFM + ml]);
  }
  return cfma(e.A, v, e.B);
}

// what a lane knows of its mode and its chunk of one field's system
struct ZfLane {
  int ml, cs, m, run, N3, Pp, js, je;
  bool act;
  float kxv, kyv;
};

__device__ __forceinline__ void zf_cp16(void* smem, const void* gmem) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem));
}
__device__ __forceinline__ void zf_cp_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// levels per chunk: odd where that fits, so that the four chunks of a warp
// read their rows and coefficients from different shared-memory banks
template <int L>
__host__ __device__ constexpr int zf_chunk(int c) {
  return (L == 0 || (c | 1) <= L) ? c | 1 : c;
}

// pass 1 of the Crank-Nicolson solve of field F (0, 1: u1, u2; 2: u3,
// Dirichlet; 3: b): the right-hand side, be_j = R_j / den_j (into be[] or the
// shared rows X) and the chunk's upward map. Every global array is read at
// one 32-bit offset from a base that is the same for the whole block. A batch
// of U levels is straight-line code: levels past the chunk's end repeat its
// last one and leave the map and memory alone, so that the compiler may move
// every load of a batch ahead of its arithmetic. Long chunks load the next
// batch while they work on this one.
template <int F, int L, int U, bool SM, bool COL, bool PIPE>
__device__ __forceinline__ ZfMap zf_rhs(const StageArgs& a, const ZfLane& t, const ZfTab<SM>& tab, float2* X,
                                        const float2* Pc, const float2* Wc, const float2* Bc,
                                        float2 (&be_)[L ? L : 1], float (&bi_)[L ? L : 1]) {
  constexpr int FAM = F == 3 ? 2 : (F == 2 ? 1 : 0);
  constexpr bool dir = FAM == 1;
  const int N3 = t.N3, js = t.js, je = t.je;
  const unsigned Pp = t.Pp, m = t.m;
  const int fs = (FAM == 2 ? 1 : (dir ? 2 : 0)) * 3 + a.stage;   // factor sets: velocity, buoyancy, u3
  const size_t FB = (size_t)N3 * Pp;
  const float* __restrict__ iden = a.inv_den + fs * FB;
  const float d1 = -(t.kxv * t.kxv), d2 = -(t.kyv * t.kyv);
  const float cco = (FAM == 2) ? a.cb : a.cv;
  // no buoyancy force on the (0,0) mode (IMEXRK.cpp:141-143) or in the adjoint step
  const bool lin = !a.adjoint && !(FAM == 1 && m == 0);
  const float Ri = FAM == 1 ? a.Ri[t.run] : 0.f;
  const float2* __restrict__ Sr = a.S + (size_t)t.run * 5 * FB;
  const float2* __restrict__ uc = Sr + F * FB;
  const float2* __restrict__ xc = Sr + (FAM == 2 ? 2 : 3) * FB;   // b for u3, u3 for b
  const float2* __restrict__ pc = Sr + 4 * FB;
  float2* rc = a.rnl + (size_t)(t.run * 4 + F) * FB;
  const float2* __restrict__ rold = a.rold + (size_t)(t.run * 4 + F) * FB;
  const bool use_rold = (a.hz != 0.f);
  // the next stage reads this stage's explicit terms from where they lie (the
  // solver's two buffers take turns); only those of u3 and b are not yet whole
  const bool keep = F >= 2 && a.stage < 2 && !a.adjoint;
  const float kgrad = (F == 0) ? t.kxv : t.kyv;
  const float2 *Uc = F == 2 ? Wc : Bc, *Xc = F == 2 ? Bc : Wc;   // COL: this field's column, and the other's
  constexpr bool UC = COL && F >= 2;
  ZfMap map{1.f, cz()};
  const int jl = je > js ? je - 1 : min(js, N3 - 1);   // the chunk's last level (an empty chunk: some level)
  const int jf = min(js, N3 - 1), jm = max(jf - 1, 0);
  float2 um = UC ? Uc[jm * kFM] : uc[jm * Pp + m];
  float2 u0 = UC ? Uc[jf * kFM] : uc[jf * Pp + m];
  float2 pm1 = cz(), xm = cz();
  if (FAM == 1) {
    pm1 = COL ? Pc[jm * kFM] : pc[jm * Pp + m];
    xm = COL ? Xc[jm * kFM] : xc[jm * Pp + m];
  }
  if (FAM == 2) xm = COL ? Xc[jf * kFM] : xc[jf * Pp + m];
  struct In {
    float2 u, r, o, p, x;
    float bi;
  };
  auto load = [&](In (&v)[U], int j0) {
#pragma unroll
    for (int i = 0; i < U; i++) {
      const int j = min(j0 + i, jl), jn = min(j + 1, N3 - 1);
      const unsigned o = j * Pp + m, on = jn * Pp + m;
      if (!UC) v[i].u = __ldcg(uc + on);
      if (!COL) v[i].r = __ldcg(rc + o);
      if (use_rold) v[i].o = __ldcg(rold + o);
      v[i].bi = __ldcg(iden + o);
      if (!COL && FAM != 2) v[i].p = __ldcg(pc + o);
      if (!COL && FAM == 1) v[i].x = __ldcg(xc + o);
      if (!COL && FAM == 2) v[i].x = __ldcg(xc + on);
    }
  };
  auto work = [&](In (&v)[U], int j0) {
#pragma unroll
    for (int i = 0; i < U; i++) {
      const bool in = j0 + i < je;
      const int j = min(j0 + i, jl), jn = min(j + 1, N3 - 1);
      const float2 up = UC ? Uc[jn * kFM] : v[i].u;
      const float2 p = FAM == 2 ? cz() : (COL ? Pc[j * kFM] : v[i].p);
      const float2 x = FAM == 0 ? cz() : (COL ? Xc[(FAM == 2 ? jn : j) * kFM] : v[i].x);
      const float4 z1 = dir ? tab.d[j] : ((FAM == 2 && !SM) ? tab.nb[j] : tab.n[j]);   // d2z lower, diagonal, upper; a_j
      const float aj = (FAM == 2 && SM) ? tab.c[j].x : z1.w;
      float2 rt = COL ? X[j * kFM] : v[i].r, gp;
      if (FAM == 0) {
        gp = czik(kgrad, p);   // i k p
      } else if (FAM == 1) {
        const float4 z2 = tab.t2[j];
        gp = cfma(z2.x, pm1, cmul(z2.y, p));
        pm1 = p;
        const float2 rb = cfma(Ri, cfma(z2.z, xm, cmul(z2.w, x)), rt);   // r3 += Ri Full(b - <b>)
        if (lin) rt = rb;
        xm = x;
      } else {
        // rB -= dB/dz ReinterpolateDirichlet(u3), whose top row has no level above
        const float2 dw = cfma(0.5f, xm, j + 1 < N3 ? cmul(0.5f, x) : cz());
        if (lin) rt = cfma(-tab.dB[j], dw, rt);
        xm = x;
      }
      float2 R = u0;
      if (use_rold) R = cfma(a.hz, v[i].o, R);
      if (FAM != 2) R = cfma(-a.h, gp, R);
      R = cfma(a.hb, rt, R);
      const float2 d2u = cfma(z1.z, up, cfma(z1.y, u0, cmul(z1.x, um)));
      R = cfma(cco, padd(cfma(d2, u0, cmul(d1, u0)), d2u), R);
      // ZeroEnds (Field.h:475-486): the first two (Dirichlet: three) levels and the last two
      if ((unsigned)(j - (dir ? 3 : 2)) >= (unsigned)(N3 - (dir ? 5 : 4))) R = cz();
      const float2 be = cmul(v[i].bi, R);
      const float al = -aj * v[i].bi;
      if (L) {
        be_[i] = be;
        bi_[i] = v[i].bi;
      } else if (in) {
        X[j * kFM] = be;
      }
      if (keep && in && t.act) rc[j * Pp + m] = rt;
      const float2 B = cfma(al, map.B, be);
      map.A = in ? map.A * al : map.A;
      map.B = in ? B : map.B;
      um = u0;
      u0 = up;
    }
  };
  In v[U];
  load(v, js);
  if (L) {
    static_assert(L == 0 || L == U, "a short chunk is one batch");
    work(v, js);
  } else if (!PIPE) {
    for (int j0 = js; j0 < je; j0 += U) {
      if (j0 > js) load(v, j0);
      work(v, j0);
    }
  } else {
    In w[U];
    for (int j0 = js; j0 < je; j0 += 2 * U) {
      load(w, j0 + U);
      work(v, j0);
      load(v, j0 + 2 * U);
      work(w, j0 + U);
    }
  }
  return map;
}

// pass 2, D_j = al_j D_{j-1} + be_j from the value D entering the chunk, and
// the chunk's map of the downward sweep x_j = D_j - C_j x_{j+1}. AC(j) gives
// (a_j, c_j); PIN: the (0,0) mode's C_1 is 0 (IMEXRK.h:68-74).
template <int L, bool PIN, class ACF>
__device__ __forceinline__ ZfMap zf_mid(const ZfLane& t, ACF AC, const float* __restrict__ iden, float2 D, float2* X,
                                        float2 (&be)[L ? L : 1], float (&bi)[L ? L : 1]) {
  ZfMap b{1.f, cz()};
  const int jl = t.je > t.js ? t.je - 1 : min(t.js, t.N3 - 1);
  auto level = [&](int j, bool in, float bij, float2 bej) {
    const float2 q = AC(j);
    D = cfma(-q.x * bij, D, bej);
    const float2 B = cfma(b.A, D, b.B);
    const float A = -b.A * ((PIN && t.m == 0 && j == 1) ? 0.f : q.y * bij);
    b.A = in ? A : b.A;
    b.B = in ? B : b.B;
    return D;
  };
  if (L) {
#pragma unroll
    for (int i = 0; i < L; i++) be[i] = level(min(t.js + i, jl), t.js + i < t.je, bi[i], be[i]);
  } else {
    for (int j0 = t.js; j0 < t.je; j0 += kFI) {
      float bj[kFI];
      float2 ej[kFI];
#pragma unroll
      for (int i = 0; i < kFI; i++) {
        const int j = min(j0 + i, jl);
        bj[i] = __ldcg(iden + (unsigned)(j * t.Pp + t.m));
        ej[i] = X[j * kFM];
      }
#pragma unroll
      for (int i = 0; i < kFI; i++) {
        const bool in = j0 + i < t.je;
        const float2 d = level(min(j0 + i, jl), in, bj[i], ej[i]);
        if (in) X[(j0 + i) * kFM] = d;
      }
    }
  }
  return b;
}

// The whole z pass of a stage for the 8 modes of block coordinate bx of run
// bz, by NF * CQ warps: L levels at most per chunk of the solves (0: any
// number) and PL per chunk of the projection, whose D_j stay in registers.
// After the solves X holds the new velocities.
template <int NF, int CQ, int L, int PL, int U, bool SM, bool COL, bool PIPE>
__device__ __forceinline__ void z_step_f_body(const StageArgs& a, const int bx, const int bz) {
  using Z = ZfShape<NF, CQ>;
  const Geo& g = a.g;
  extern __shared__ __align__(16) float zfsm[];
  const int N3 = g.N3, Pp = g.Pp;
  float2* X = reinterpret_cast<float2*>(zfsm);
  float2* WB = X + (size_t)NF * N3 * kFM;
  float* WA = reinterpret_cast<float*>(WB + 2 * Z::NW * kFM);
  ZfTab<SM> tab;
  float2 *Pc = nullptr, *Wc = nullptr, *Bc = nullptr;
  if (SM) {
    float4* T = reinterpret_cast<float4*>(WA + 2 * Z::NW * kFM);
    float* dB = reinterpret_cast<float*>(T + 5 * N3);
    if (COL) {
      // the columns of r (into X) and of p, u3, b, 64 bytes a level, all in
      // flight at once
      Pc = reinterpret_cast<float2*>(dB + N3);
      Wc = Pc + (size_t)N3 * kFM;
      Bc = Wc + (size_t)N3 * kFM;
      const float2* S0 = a.S + (size_t)bz * 5 * N3 * Pp + bx * kFM;
      const float2* r0 = a.rnl + (size_t)bz * 4 * N3 * Pp + bx * kFM;
      for (int i = threadIdx.x; i < N3 * 4; i += Z::THREADS) {
        const int j = i >> 2, c = 2 * (i & 3);
        const unsigned o = j * Pp + c;
        const int d = j * kFM + c;
        const size_t FB = (size_t)N3 * Pp;
        zf_cp16(Pc + d, S0 + 4 * FB + o);
        zf_cp16(Wc + d, S0 + 2 * FB + o);
        zf_cp16(Bc + d, S0 + 3 * FB + o);
#pragma unroll
        for (int k = 0; k < NF; k++) zf_cp16(X + (size_t)k * N3 * kFM + d, r0 + (NF == 4 || k == 0 ? k : k + 1) * FB + o);
      }
      Pc += threadIdx.x & 7;
      Wc += threadIdx.x & 7;
      Bc += threadIdx.x & 7;
    }
    for (int j = threadIdx.x; j < N3; j += Z::THREADS) {
      const float4 *z1 = a.zt1 + a.stage * N3 + j, zu = z1[0], zd = z1[6 * N3];
      const float2 *ac = a.zac + a.stage * N3 + j;
      T[j] = zu;
      T[N3 + j] = zd;
      T[2 * N3 + j] = a.zt2[j];
      T[3 * N3 + j] = a.ztq[j];
      T[4 * N3 + j] = make_float4(z1[3 * N3].w, ac[0].y, ac[3 * N3].y, ac[6 * N3].y);
      dB[j] = a.dBdz[(size_t)bz * N3 + j];
    }
    tab.n = T;
    tab.d = T + N3;
    tab.t2 = T + 2 * N3;
    tab.q = T + 3 * N3;
    tab.c = T + 4 * N3;
    tab.dB = dB;
    if (COL) zf_cp_wait();
    else chain_begin();
    __syncthreads();
  } else {
    tab.n = a.zt1 + a.stage * N3;
    tab.nb = tab.n + 3 * N3;
    tab.d = tab.n + 6 * N3;
    tab.t2 = a.zt2;
    tab.q = a.ztq;
    tab.dB = a.dBdz + (size_t)bz * N3;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  ZfLane t;
  t.ml = lane & 7;
  t.cs = lane >> 3;
  const int m0 = bx * kFM + t.ml;
  t.act = m0 < g.P;
  t.m = t.act ? m0 : 0;
  t.run = bz;
  t.N3 = N3;
  t.Pp = Pp;
  const int q = t.m / g.K1;
  t.kxv = a.kx[t.m - q * g.K1];
  t.kyv = NF == 4 ? a.ky[q] : 0.f;
  const int slot = w / CQ, wf = w - slot * CQ;        // this warp's field and its place in it
  const int f = NF == 4 ? slot : (slot == 0 ? 0 : slot + 1);
  {
    const int chunk = zf_chunk<L>((N3 + Z::CC - 1) / Z::CC), c = 4 * wf + t.cs;
    t.js = min(N3, c * chunk);
    t.je = min(N3, t.js + chunk);
  }
  float2* Xf = X + (size_t)slot * N3 * kFM + t.ml;
  {
    float2 be[L ? L : 1];
    float bi[L ? L : 1];
    ZfMap mp;
    if (f == 3) mp = zf_rhs<3, L, U, SM, COL, PIPE>(a, t, tab, Xf, Pc, Wc, Bc, be, bi);
    else if (f == 2) mp = zf_rhs<2, L, U, SM, COL, PIPE>(a, t, tab, Xf, Pc, Wc, Bc, be, bi);
    else if (NF == 4 && f == 1) mp = zf_rhs<1, L, U, SM, COL, PIPE>(a, t, tab, Xf, Pc, Wc, Bc, be, bi);
    else mp = zf_rhs<0, L, U, SM, COL, PIPE>(a, t, tab, Xf, Pc, Wc, Bc, be, bi);
    const int fam = f == 3 ? 1 : (f == 2 ? 2 : 0);
    const float* __restrict__ iden = a.inv_den + (size_t)(fam * 3 + a.stage) * N3 * Pp;
    // (a_j, c_j) of this field's systems: the a_j of its d2z row (b's beside
    // the c_j), floats 3 or 0 of a float4
    const float* ta = SM ? reinterpret_cast<const float*>(fam == 1 ? tab.c : (fam == 2 ? tab.d : tab.n)) + (fam == 1 ? 0 : 3) : nullptr;
    const float* tc = SM ? reinterpret_cast<const float*>(tab.c) + 1 + fam : nullptr;
    const float2* __restrict__ acg = a.zac + (fam * 3 + a.stage) * N3;
    auto AC = [&](int j) { return SM ? make_float2(ta[4 * j], tc[4 * j]) : acg[j]; };
    const float2 Din = zf_scan<true>(mp, WA + slot * CQ * kFM, WB + slot * CQ * kFM, wf, CQ, t.ml, t.cs);
    mp = zf_mid<L, false>(t, AC, iden, Din, Xf, be, bi);
    float2 x = zf_scan<false>(mp, WA + (Z::NW + slot * CQ) * kFM, WB + (Z::NW + slot * CQ) * kFM, wf, CQ, t.ml, t.cs);
    // ---- x_j = D_j - C_j x_{j+1}: the velocities stay here, b is finished ----
    float2* out = a.Sn + (size_t)(t.run * 5 + 3) * N3 * Pp;
    auto put = [&](int j, bool in, float bij, float2 D) {
      x = cfma(-(AC(j).y * bij), x, D);
      if (in) {
        if (f != 3) Xf[j * kFM] = x;
        else if (t.act) out[(unsigned)(j * Pp + t.m)] = x;
      }
    };
    if (L) {
      // from the chunk's last level: the slots above it are skipped, so that
      // x_je meets the right level
#pragma unroll
      for (int i = L - 1; i >= 0; i--)
        if (t.js + i < t.je) put(t.js + i, true, bi[i], be[i]);
    } else {
      for (int j0 = t.je - 1; j0 >= t.js; j0 -= kFI) {
        float bj[kFI];
        float2 Dj[kFI];
#pragma unroll
        for (int i = 0; i < kFI; i++) {
          const int j = max(j0 - i, t.js);
          bj[i] = __ldcg(iden + (unsigned)(j * Pp + t.m));
          Dj[i] = Xf[j * kFM];
        }
#pragma unroll
        for (int i = 0; i < kFI; i++) put(max(j0 - i, t.js), j0 - i >= t.js, bj[i], Dj[i]);
      }
    }
  }
  // ---- RemoveDivergence: all warps, chunks of the whole column ----
  {
    const int chunk = zf_chunk<PL>((N3 + Z::CP - 1) / Z::CP), c = 4 * w + t.cs;
    t.js = min(N3, c * chunk);
    t.je = min(N3, t.js + chunk);
  }
  const float2* X1 = X + t.ml;
  const float2* X2 = X + (size_t)N3 * kFM + t.ml;               // 3D only
  const float2* X3 = X + (size_t)(NF - 2) * N3 * kFM + t.ml;
  const float* __restrict__ iden = a.inv_den + (size_t)kFS_Lap * N3 * Pp;
  auto AC = [&](int j) {
    const float4 z = tab.q[j];   // ddz (D -> N) diagonal and upper, the Laplacian's a_j and c_j
    return make_float2(z.z, z.w);
  };
  const size_t FB = (size_t)N3 * Pp;
  const float2* __restrict__ ps = a.S + (size_t)(t.run * 5 + 4) * FB;
  float2* on = a.Sn + (size_t)t.run * 5 * FB;                   // u1
  const int jl = t.je > t.js ? t.je - 1 : min(t.js, N3 - 1);
  float2 be[PL], pv[PL];
  float bi[PL];
  // the pivots and p, loaded while the slower fields' warps finish
#pragma unroll
  for (int i = 0; i < PL; i++) {
    const int j = min(t.js + i, jl);
    const unsigned o = j * Pp + t.m;
    bi[i] = __ldcg(iden + o);
    pv[i] = COL ? Pc[j * kFM] : __ldcg(ps + o);
  }
  __syncthreads();
  ZfMap mp{1.f, cz()};
#pragma unroll
  for (int i = 0; i < PL; i++) {
    const bool in = t.js + i < t.je;
    const int j = min(t.js + i, jl);
    const float4 z = tab.q[j];
    float2 s = cmul(t.kxv, X1[j * kFM]);
    if (NF == 4) s = cfma(t.kyv, X2[j * kFM], s);   // kx u1 + ky u2
    float2 dv = padd(make_float2(-s.y, s.x), cfma(z.y, X3[min(j + 1, N3 - 1) * kFM], cmul(z.x, X3[j * kFM])));
    if ((unsigned)(j - 2) >= (unsigned)(N3 - 4)) dv = cz();
    be[i] = cmul(bi[i], dv);
    const float al = -z.z * bi[i];
    const float2 B = cfma(al, mp.B, be[i]);
    mp.A = in ? mp.A * al : mp.A;
    mp.B = in ? B : mp.B;
  }
  const float2 Din = zf_scan<true>(mp, WA, WB, w, Z::NW, t.ml, t.cs);
  mp = zf_mid<PL, true>(t, AC, iden, Din, nullptr, be, bi);
  float2 qn = zf_scan<false>(mp, WA + Z::NW * kFM, WB + Z::NW * kFM, w, Z::NW, t.ml, t.cs);   // q at level je
  // ---- q_j = D_j - C_j q_{j+1}; u -= grad q, p += pm q ----
#pragma unroll
  for (int i = PL - 1; i >= 0; i--) {
    const int j = t.js + i;
    if (j >= t.je) continue;
    const float C = (t.m == 0 && j == 1) ? 0.f : tab.q[j].w * bi[i];
    const float2 qj = cfma(-C, qn, be[i]);
    if (t.act) {
      const unsigned o = j * Pp + t.m;
      on[o] = psub(X1[j * kFM], czik(t.kxv, qj));
      if (NF == 4) on[FB + o] = psub(X2[j * kFM], czik(t.kyv, qj));
      on[4 * FB + o] = cfma(a.pm, qj, pv[i]);
      const int jj = j + 1;   // u3_{j+1} -= ddz(q)_{j+1}: zero coefficients in rows below 2
      if (jj < N3) {
        const float4 z2 = tab.t2[jj];
        on[2 * FB + o + Pp] = psub(X3[jj * kFM], cfma(z2.x, qj, cmul(z2.y, qn)));
      }
      if (j == 0) on[2 * FB + o] = X3[0];
    }
    qn = qj;
  }
}

}  // namespace sf
