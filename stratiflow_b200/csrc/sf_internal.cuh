// Internal declarations shared by the kernels and the C-ABI layer.
//
// Device data layout (all complex values are float2):
//   state   S[2]    [nrun][5][N3][Pp]   u1,u2,u3,b,p per run; two copies,
//                                       stage k reads one and writes the other
//   rold            [nrun][4][N3][Pp]   explicit terms r1,r2,r3,rB of the last
//                                       stage (the zeta term of ExplicitRK)
//   rnl             [nrun][4][N3][Pp]   nonlinear terms of this stage (with
//                                       k_z_step_f the two take turns)
//   qbuf            [nrun][N3][Pp]      forward-sweep scratch of the pressure solve
//   mixin  (3D)     [nrun][2][N3][N2][K1][2]  fields after the inverse y
//                   transform, two side by side: (u1, u3), (b, u2)
//   mixout (3D)     [nrun][4][N3][N2][K1][2]  x-transformed product
//                   combinations: (C_1, C_B), (C_1y, C_By), (C_2, C_3), (C_2y, C_3y)
//   base            [nrun][4][N3][N2][N1]  frozen nodal base of the linear step
// Pp = roundup(K1*K2, 16) is the plane stride of one level; mode m = q*K1+j1.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sf {

constexpr int kMaxN = 512;        // largest N1 / N2 of the FFTs
constexpr int kNumFS = 10;        // factor sets: 3 families x 3 stages + Laplacian
constexpr int kFS_Lap = 9;

// per-level coefficient arrays in `zc`, each N3 floats
enum ZC {
  ZC_D2N_LO, ZC_D2N_DI, ZC_D2N_UP,
  ZC_D2D_LO, ZC_D2D_DI, ZC_D2D_UP,
  ZC_DND_LO, ZC_DND_DI,       // ddz Neumann -> Dirichlet (rows 2..N-1)
  ZC_DDN_DI, ZC_DDN_UP,       // ddz Dirichlet -> Neumann (rows 1..N-1)
  ZC_FULL_LO, ZC_FULL_DI,     // ReinterpolateFull
  ZC_TILDE_LO, ZC_TILDE_DI,   // ReinterpolateTilde
  ZC_WZN, ZC_WZD,             // vertical quadrature weights (Integration.h:5-35)
  ZC_COUNT
};

struct Geo {
  int N1, N2, N3;
  int K1, K2, Ky;   // kept x modes, kept y modes, non-negative kept y modes
  int P, Pp;        // kept modes per level, padded plane stride
  int logN1, logN2;
  int nrun;
  int dim3;
  float inv_n12;    // 1/(N1*N2), the ToModal scaling (Field.h:759)
  long long fblk;   // complex elements of one field block: N3*Pp
  long long mblk;   // complex elements of one mixed block: N3*N2*K1
};

struct StageArgs {
  Geo g;
  const float2* S;      // current state [nrun][5][N3][Pp]
  float2* Sn;           // next state
  float2* rold;
  float2* rnl;
  float2* qbuf;
  float2* mixin;
  float2* mixout;
  const float* zc;      // ZC_COUNT x N3
  const float* fa;      // kNumFS x N3 sub-diagonals a_j
  const float* fc;      // kNumFS x N3 super-diagonals c_j
  // the same rows packed for k_z_step_f, one vector load per level:
  const float4* zt1;    // 9 x N3 per Crank-Nicolson factor set: d2z lower, diagonal, upper; a_j
  const float4* zt2;    // N3: ddz (N -> D) lower, diagonal; ReinterpolateFull lower, diagonal
  const float4* ztq;    // N3: ddz (D -> N) diagonal, upper; the Laplacian's a_j, c_j
  const float2* zac;    // kNumFS x N3: a_j, c_j
  const float* inv_den; // kNumFS x N3 x Pp, 1/(b_j - a_j C_{j-1}) (FP64-factorised)
  const float* kx;      // K1
  const float* ky;      // K2
  const float* Ri;      // nrun
  const float* Ubar;    // nrun x N3
  const float* dBdz;    // nrun x N3
  const float2* tw;     // kMaxN twiddles e^{-2 pi i k/kMaxN}, the full circle
  const float* base;    // nrun x 4 x N3 x N2 x N1 (linear step only)
  int stage;
  int linear;
  int tlm;          // tangent-linear batch: runs < tlm are nonlinear bases, run r >= tlm
                    // is linearised about the current state of run (r - tlm) % tlm
  int run_offset;   // first run of this launch (x pass)
  int xslabs;       // slabs per x-pass block (0: chosen by the launcher)
  int adjoint;      // adjoint step: no linear buoyancy terms in the z solve
  const float2* adir;   // adjoint step: the direct total state of the substep [nrun][4][N3][Pp]
  float2* amix;         // 3D adjoint step: 12 y-transformed fields [nrun][6][N3][N2][K1][2], paired as mixin
  float adj_invK;       // adjoint step: 1/K of the mixing objective (IMEXRK.h:487)
  float h, hz, hb, cv, cb, pm;
  // level band of one launch of the y transforms (levels lvl0 .. lvl0+nlvl-1;
  // nlvl = 0: all) and level columns of one x-pass launch (xcol0 .. +xcols-1;
  // xcols = 0: all), for the banded 3D x-y pass
  int lvl0, nlvl, xcol0, xcols;
  int zchunks;      // z chunks per block of the z solves (8 or 16; 0: chosen by the launcher)
  int xgroups;      // lane groups per x-pass block (0: chosen by the launcher)
  int xkernel;      // x pass: 1 level-marching lane groups (k_xmarch) where they pay, 0 slab blocks (k_xpass)
  int zkernel;      // z pass: 0 k_z_step, 1 k_z_step_tma (inputs by the tensor-memory accelerator),
                    // 2 k_z_step_f (every field of a mode group at once)
  const void* zmaps;   // host ZMaps of the solver (k_z_step_tma), or null
  int* zerr;           // device word set by a k_z_step_tma wait that ran out
  int chained;         // the stage's kernels follow one another in one stream with nothing between (launch_chained)
};

// A stage's kernels are launched while the one before them runs out: their
// blocks are on the SMs when its last block ends, the tables that were there
// before it are filled, and they wait (chain_begin) until its results are
// visible. Hides the kernels' launch latency where it counts: 64x32x64, four
// steps 275 -> 264 us; adjoint step at 128x64x128 389 -> 368; 64x64 in 2D 46 ->
// 44; larger grids do not notice. Letting the next kernel's blocks in earlier,
// while the last wave still runs, costs more than it gives (302 us, and 1690
// for 1564 at 256x128x384): they hold places that work would be spread over. In
// a kernel that was launched in the ordinary way chain_begin does nothing.
template <class... P>
inline void launch_chained(void (*fn)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool chained, P... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&c, fn, args...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void chain_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

// the tensor maps of k_z_step_tma's inputs (each the bytes of one
// CUtensorMap), encoded once per solver, and the state buffers they view
struct alignas(64) ZMap {
  unsigned char bytes[128];
};
struct ZMaps {
  ZMap s[2], rnl, rold, iden;
  const void* sbase[2];
  const void* rbase[3];   // rnl, rold, inv_den
};

// side streams and events of the banded 3D x-y pass: the inverse y
// transforms of every band run on y1, the x passes on the stage's stream, the
// forward y transforms on y2, each band waiting only for what it reads
constexpr int kMaxBands = 8;
struct XYAux {
  cudaStream_t y1, y2;
  cudaEvent_t fork, join;
  cudaEvent_t ev_ify[kMaxBands], ev_x[kMaxBands];
  int bands;
};

// one block's work in an ensemble launch: member solver `run`; x pass: units x
// .. x + iters - 1 (one per warp) of segments of S levels; z: mode group x
struct EnsItem {
  int run, x, S, iters;
};
constexpr int kEnsThreads = 384;
constexpr int kEnsFusedN3 = 484;   // the tallest column of a z item in k_z_step_f's shape of 12 warps

// launchers (sf_kernels.cu); each returns the number of kernels launched
int prepare_kernels();
// the z pass with TMA-fed first sweeps (sf_zstep.cu)
bool zstep_tma_supported(const Geo& g);
int zstep_tma_maps(const Geo& g, const float2* S0, const float2* S1, const float2* rnl, const float2* rold,
                   const float* inv_den, ZMaps* out);
int launch_z_step_tma(const StageArgs& a, cudaStream_t st);
bool z_step_takes_tma(const StageArgs& a);
// the z pass with one lane per complex mode (sf_zstep2.cu)
bool zstep_c_supported(const Geo& g);
int launch_z_step_c(const StageArgs& a, cudaStream_t st);
int prepare_zstep_c_kernels();
bool z_step_takes_c(const StageArgs& a);
int prepare_zstep_tma_kernels();
// the z pass with all fields of a mode group at once (sf_zstep3.cu)
bool zstep_f_supported(const Geo& g);
int launch_z_step_f(const StageArgs& a, cudaStream_t st);
int prepare_zstep_f_kernels();
// the x pass as level-marching lane groups (sf_xmarch.cu): levels t_lo ..
// t_hi - 1 of every y row of runs a.run_offset .. + nruns - 1; mode 0
// BuildRHS, 1 BuildRHSLinear about the frozen base, 2 about the live base run
bool xmarch_supported(const StageArgs& a, int mode, int nruns);
int launch_xmarch(const StageArgs& a, int mode, int nruns, int t_lo, int t_hi, cudaStream_t st);
int prepare_xmarch_kernels();
// the adjoint x pass in the same manner (sf_adjmarch.cu): every level of every run
bool adjmarch_supported(const Geo& g);
int launch_adjmarch(const StageArgs& a, cudaStream_t st);
int prepare_adjmarch_kernels();
// one stage; if ev != nullptr, ev[i] is recorded after the i-th kernel
int launch_stage(const StageArgs& a, cudaStream_t st, cudaEvent_t* ev = nullptr, const XYAux* aux = nullptr);
int stage_kernel_count(const Geo& g);
const char* stage_kernel_name(const Geo& g, int i);
int launch_project(const StageArgs& a, cudaStream_t st);  // RemoveDivergence only
int launch_z_solves(const StageArgs& a, cudaStream_t st);   // CN solve + RemoveDivergence
int launch_fft_y_combos(const StageArgs& a, cudaStream_t st);   // 3D: mixout's 8 combinations -> rnl
// TimeStepAdjoint's stage (sf_adjoint.cu): the direct state of the substep
// into a.adir, then the adjoint x pass and the z solves; 2D
int launch_stage_adjoint(StageArgs a, const float2* below, const float2* above, float frac, float2* adir,
                         cudaStream_t st);
size_t adjoint_smem_needed(const Geo& g);
int prepare_adjoint_kernels();
int launch_factor(const Geo& g, const double* bands, const double* kx, const double* ky,
                  double h0, double h1, double h2, double Re, double Pr, float* inv_den,
                  cudaStream_t st);
int launch_gather_ref(const Geo& g, const float2* ref, float2* kept, cudaStream_t st);
int launch_scatter_ref(const Geo& g, const float2* kept, float2* ref, cudaStream_t st);
int launch_energy(const Geo& g, const float2* Sa, const float2* Sb, int nrun_pairs,
                  const float* zc, const float* Ri, double* out, cudaStream_t st);
// ensembles of 2D solvers of different grids (sf_ens.cu): one stage of every
// member in one launch of `blocks` persistent blocks over work-item counters
// (counters[0] the next item, counters[1 + r] member r's finished x items;
// cleared before each step); args holds one StageArgs per member
int ensemble_z_modes(int N3);
int ensemble_x_warps(int N1);
int ensemble_x_rows(int N1);
size_t ensemble_smem(int N1, int N3);
int prepare_ensemble_kernels();
int launch_ens_stage(const StageArgs* args, const EnsItem* xitems, int nx, const EnsItem* zitems, int nz,
                     int* counters, const int* xneed, int* err, int blocks, size_t smem, cudaStream_t st);
int ensemble_stage_blocks();
int launch_grad_sq(const Geo& g, const float2* S, int nruns, const float* zc, const double* kxd, const double* kyd,
                   double* out, cudaStream_t st);
int launch_base_nodal(const Geo& g, const float2* kept_modal, int field, float* base_out,
                      const float2* tw, float* scratch_mixed, cudaStream_t st);

// ------------------------------------------------------- device helpers ----
#ifdef __CUDACC__
// where field f of mixin's pairs lies, and the first element of row (t, y) of
// pair p after pair0, on its side
__device__ __forceinline__ int mix_in_pair(int f) { return f == 0 || f == 2 ? 0 : 1; }
__device__ __forceinline__ int mix_in_side(int f) { return f == 2 || f == 1 ? 1 : 0; }
__device__ __forceinline__ size_t mix_pair(const Geo& g, int pair0, int p, int side, int t, int y) {
  return ((((size_t)(pair0 + p) * g.N3 + t) * g.N2 + y) * g.K1) * 2 + side;
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// (i*k) * a
__device__ __forceinline__ float2 cik(float k, float2 a) { return make_float2(-k * a.y, k * a.x); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

// In-place radix-2 decimation-in-time FFT of n = 2^logn points held in shared
// memory at a[0..n), executed by one warp. Unnormalised; sign -1 (forward)
// or +1 (inverse). tw holds e^{-2 pi i k/kMaxN}, k < kMaxN (only k < kMaxN/2 used here).
__device__ __forceinline__ void warp_fft(float2* a, int n, int logn, const float2* __restrict__ tw,
                                         bool inverse, int lane) {
  const int shift = 32 - logn;
  for (int i = lane; i < n; i += 32) {
    int r = (int)(__brev((unsigned)i) >> shift);
    if (i < r) {
      float2 t = a[i];
      a[i] = a[r];
      a[r] = t;
    }
  }
  __syncwarp();
  const int half_n = n >> 1;
  for (int s = 1; s <= logn; s++) {
    const int half = 1 << (s - 1);
    const int twstep = kMaxN >> s;   // e^{-2 pi i pos/(2 half)} = tw[pos * kMaxN/(2 half)]
    for (int bt = lane; bt < half_n; bt += 32) {
      int pos = bt & (half - 1);
      int i0 = ((bt >> (s - 1)) << s) + pos;
      int i1 = i0 + half;
      float2 w = tw[pos * twstep];
      if (inverse) w.y = -w.y;
      float2 x0 = a[i0];
      float2 x1 = cmul(a[i1], w);
      a[i0] = cadd(x0, x1);
      a[i1] = csub(x0, x1);
    }
    __syncwarp();
  }
}
#endif

}  // namespace sf
