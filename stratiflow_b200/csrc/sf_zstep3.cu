// k_z_step_f: the z pass with all fields of 8 modes solved at once (the
// device code is in sf_zstep_f.cuh), its shapes and the rule between them.
#include "sf_zstep_f.cuh"

namespace sf {

// NF fields, CQ warps per field, chunks of the solves in registers (L levels
// at most; 0: in shared memory), PL levels per chunk of the projection, U
// levels loaded ahead, SM the coefficient tables in shared memory, COL the
// columns of r, p, u3, b too, PIPE the next batch loaded under this one, NB
// blocks per SM that the registers are held to
template <int NF, int CQ, int L, int PL, int U, bool SM, bool COL, bool PIPE, int NB>
__global__ void __launch_bounds__(ZfShape<NF, CQ>::THREADS, NB) k_z_step_f(StageArgs a) {
  if (!SM || COL) chain_begin();   // else when the tables are filled
  z_step_f_body<NF, CQ, L, PL, U, SM, COL, PIPE>(a, blockIdx.x, blockIdx.z);
}

namespace {

struct ZfKernel {
  void (*fn)(StageArgs);
  size_t (*smem)(int);
  int threads, cc, cp, L, PL;   // chunks of the solves and of the projection, and the levels they may have
};
template <int NF, int CQ, int L, int PL, int U, bool SM, bool COL, bool PIPE, int NB>
constexpr ZfKernel zf_kernel() {
  using Z = ZfShape<NF, CQ>;
  return ZfKernel{k_z_step_f<NF, CQ, L, PL, U, SM, COL, PIPE, NB>, [](int N3) { return Z::smem(N3, SM, COL); },
                  Z::THREADS, Z::CC, Z::CP, L, PL};
}

// Measured per launch (us), k_z_step_c in brackets; "many" has more blocks
// of 8 modes than the GPU has SMs:
//   3D  short4   64x32x64        10.5 (29.7)
//       short8   64x32x96        12.8 (34.8), one 16.3;    128x64x96 19.1, two 22.0
//       mid      64x32x128       15.1, one 20.8;           3 x 64x64x128 32.2, two 37.1; 256x128x128 72, two 67
//       one      32x16x332       27.8 (63.7), two 44.4;    256x128x384 174 (180), two 211 (two blocks do not fit one SM)
//       two      2 x 128x64x180  46 (84.5), one 55.4;      256x128x128 67 (72.7), one 89.4
//   2D  short4   64x1x64         10.2 (26.1)
//       short8   128x1x128       12.4 (32.7), one 16.7;    32 x 128x1x128 19.8 (32.7), many 26.3
//       one      6 x 512x1x388   26.9 (61.5), many 43.5, tall 27.4;  1 x 256x1x260 23.5, tall 25.5
//       many     64 x 256x1x256  89.3 (101), one 99.8;     8 x 512x1x256 32.5 (40.5), one 36.3
//       tall     as "one" where its columns do not fit. Over several waves of blocks of 384 levels
//                and more it would be the faster: 64 x 256x1x384 127, one 135 (143); 32 x 256x1x484
//                93, one 98; 16 x 256x1x388 49, one 48
// Two blocks of an SM only pay where the SM's L1 keeps some of its room and
// the second block has something to do; with one block each lane may hold
// more levels' loads in flight.
constexpr ZfKernel k3short4 = zf_kernel<4, 4, 4, 1, 4, false, false, false, 1>();
constexpr ZfKernel k3short8 = zf_kernel<4, 3, 8, 2, 8, false, false, false, 1>();
constexpr ZfKernel k3mid = zf_kernel<4, 4, 8, 2, 8, false, false, false, 1>();
constexpr ZfKernel k3one = zf_kernel<4, 4, 0, 12, 4, true, false, false, 1>();
constexpr ZfKernel k3two = zf_kernel<4, 3, 0, 8, 3, true, false, false, 2>();
constexpr ZfKernel k2short4 = zf_kernel<3, 4, 4, 2, 4, false, false, false, 1>();
constexpr ZfKernel k2short8 = zf_kernel<3, 4, 8, 3, 8, false, false, false, 1>();
constexpr ZfKernel k2one = zf_kernel<3, 4, 0, 12, 4, true, true, true, 1>();
constexpr ZfKernel k2many = zf_kernel<3, 4, 0, 8, 2, true, false, false, 2>();
constexpr ZfKernel k2tall = zf_kernel<3, 8, 0, 9, 2, true, false, false, 1>();

constexpr size_t kSmem1 = 227 * 1024;          // a block's shared memory
constexpr size_t kSmem2 = (228 / 2 - 1) * 1024;   // so that two blocks share an SM
constexpr size_t kSmem3 = (228 / 3 - 1) * 1024;

// the chunks hold N3 levels and the rows fit `room` bytes
bool zf_takes(const ZfKernel& k, int N3, size_t room = kSmem1) {
  return (k.L == 0 || (N3 + k.cc - 1) / k.cc <= k.L) && (N3 + k.cp - 1) / k.cp <= k.PL && k.smem(N3) <= room;
}

// the shape for a grid; null: too tall for every shape (k_z_step_c runs). The
// z-chunk setting's 8 and 16 ask for more and for fewer blocks per SM
const ZfKernel* zf_pick(const Geo& g, int zchunks) {
  const long long blocks = (long long)((g.P + kFM - 1) / kFM) * g.nrun;
  const bool many = zchunks ? zchunks == 8 : blocks > 148;
  const int N3 = g.N3;
  if (g.dim3) {
    if (zf_takes(k3short4, N3)) return &k3short4;
    if (zf_takes(k3short8, N3)) return &k3short8;
    if (blocks <= 4 * 148 && zf_takes(k3mid, N3)) return &k3mid;
    if (many && zf_takes(k3two, N3, kSmem2)) return &k3two;
    return zf_takes(k3one, N3) ? &k3one : nullptr;
  }
  if (zf_takes(k2short4, N3)) return &k2short4;
  if (zf_takes(k2short8, N3)) return &k2short8;
  if (many && zf_takes(k2many, N3, kSmem3)) return &k2many;
  if (zf_takes(k2one, N3)) return &k2one;
  return zf_takes(k2tall, N3) ? &k2tall : nullptr;
}

}  // namespace

bool zstep_f_supported(const Geo& g) { return zf_pick(g, 0) && zf_pick(g, 16); }

int launch_z_step_f(const StageArgs& a, cudaStream_t st) {
  const ZfKernel& k = *zf_pick(a.g, a.zchunks);
  launch_chained(k.fn, dim3((a.g.P + kFM - 1) / kFM, 1, a.g.nrun), k.threads, k.smem(a.g.N3), st, a.chained, a);
  return 1;
}

int prepare_zstep_f_kernels() {
  for (const ZfKernel* k : {&k3short4, &k3short8, &k3mid, &k3one, &k3two, &k2short4, &k2short8, &k2one, &k2many, &k2tall})
    if (cudaFuncSetAttribute(k->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem1) != cudaSuccess) return -1;
  return 0;
}

}  // namespace sf
