// Device-resident state vectors: the algebra of the reference's StateVector
// (StateVector.h:40-149, 415-421) on states in the kept layout, with FP64
// reductions. Used by the Newton-Krylov, Arnoldi and continuation drivers,
// whose Krylov bases live on the device.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/stratiflow_b200.h"
#include "sf_internal.cuh"

using namespace sf;

extern void sf_set_error_message(const std::string& msg);
// geometry and coefficient access of a solver (sf_solver.cu)
extern const Geo& sf_solver_geo(const sf_solver* s);
extern const float* sf_solver_zc(const sf_solver* s);
extern float2* sf_solver_state(sf_solver* s, int run);
extern cudaStream_t sf_solver_stream(const sf_solver* s);
extern const std::vector<double>& sf_solver_z(const sf_solver* s, int which);

struct sf_vecs {
  Geo g{};
  int nvec = 0;
  float2* d = nullptr;      // [nvec][5][N3][Pp]
  double* red = nullptr;    // reduction scratch
  int cap_red = 0;
  float* coef = nullptr;    // block-update coefficients
  size_t cap_coef = 0;
  const float* zc = nullptr;
  cudaStream_t st = nullptr;
  std::vector<double> z, zf;
};

namespace {

int vfail(int code, const std::string& m) {
  sf_set_error_message(m);
  return code;
}
#define VCK(call)                                                                              \
  do {                                                                                         \
    cudaError_t e__ = (call);                                                                  \
    if (e__ != cudaSuccess) return vfail(SF_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e__)); \
  } while (0)

inline size_t vstride(const Geo& g) { return (size_t)5 * g.fblk; }   // complex elements per vector

// y += alpha x over u1,u2,u3,b of `count` consecutive vectors
// (StateVector::MulAdd, StateVector.h:67-78); f4 = 4 fields, vs = vector stride
__global__ void k_axpy(float2* __restrict__ y, const float2* __restrict__ x, float alpha, size_t f4, size_t vs,
                       int count) {
  const size_t n = f4 * count;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t o = (i / f4) * vs + (i % f4);
    float2 a = x[o], b = y[o];
    y[o] = make_float2(b.x + alpha * a.x, b.y + alpha * a.y);
  }
}
// y = a y + b x over all five fields
__global__ void k_lincomb(float2* __restrict__ y, const float2* __restrict__ x, float a, float b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float2 u = y[i], v = x[i];
    y[i] = make_float2(a * u.x + b * v.x, a * u.y + b * v.y);
  }
}

// out[k] = sum over fields f of w_f * InnerProd(v_k.f, x_k'.f) (Integration.h:282-311)
// for k < count; v_k at base + k*stride, x_k' = x + k*xstride (xstride 0:
// every v_k against one x). With `sum`, all k accumulate into out[0].
// Block (level, k, field).
__global__ void k_dots(Geo g, const float2* __restrict__ base, size_t stride, const float2* __restrict__ x,
                       size_t xstride, const float* __restrict__ zc, double wb, double* out, int sum) {
  const int j = blockIdx.x, k = blockIdx.y, f = blockIdx.z;
  if (f == 1 && !g.dim3) return;
  const float2* a = base + k * stride + ((size_t)f * g.N3 + j) * g.Pp;
  const float2* b = x + k * xstride + ((size_t)f * g.N3 + j) * g.Pp;
  double s = 0.0;
  for (int m = threadIdx.x; m < g.P; m += blockDim.x) {
    float2 u = a[m], v = b[m];
    double t = (double)u.x * v.x + (double)u.y * v.y;
    s += (m == 0) ? t : 2.0 * t;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    const double wz = zc[(f == 2 ? ZC_WZD : ZC_WZN) * g.N3 + j];
    const double wf = (f == 3) ? wb : 1.0;
    if (wz != 0.0) atomicAdd(out + (sum ? 0 : k), t * wz * wf);
  }
}

// Block Gram matrix: part[c][i][k] = the share of chunk c (kGramLevels levels
// of one field) of Dot(V_i, W_k), i < nv, k < nw <= kMaxBlock, FP64.
//
// A contraction over the modes and levels, on the FP64 tensor instruction
// (m8n8k4): a warp keeps MA x NA tiles of 8 x 8 sums. The order of the k
// within a sum is free, so a lane loads four consecutive floats of its row of
// V (and of W) with one 16-byte load and feeds one of them to each of four
// instructions; nothing goes through shared memory. The four warps of a block
// take the levels of its chunk in turn and add their sums at the end. Bound
// by the FP64 rate (1.3 GFLOP for 320 x 16 vectors of 256x1x256, 37 us) and
// the one reading of V (29 us); with one dot product per lane and pair, each
// converting its two floats and reading W through the L1, 413 us; now 64.
constexpr int kGramLevels = 8;
constexpr int kMaxBlock = 32;

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int MA, int NA>
__global__ void __launch_bounds__(128) k_gram(Geo g, const float2* __restrict__ V, int nv,
                                               const float2* __restrict__ W, int nw, size_t stride,
                                               const float* __restrict__ zc, double Ri, double* __restrict__ part) {
  const int nch = (g.N3 + kGramLevels - 1) / kGramLevels;
  const int fi = blockIdx.x / nch, chunk = blockIdx.x - fi * nch;
  const int f = g.dim3 || fi == 0 ? fi : fi + 1;   // 2D: u1, u3, b
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  const int i0 = blockIdx.y * 8 * MA;
  double acc[MA][NA][2] = {};
  const int steps = (2 * g.P + 15) / 16;   // of 16 floats of a level's row
  for (int j = chunk * kGramLevels + warp; j < min(g.N3, (chunk + 1) * kGramLevels); j += 4) {
    const double wz = (double)zc[(f == 2 ? ZC_WZD : ZC_WZN) * g.N3 + j] * (f == 3 ? Ri : 1.0);
    if (wz == 0.0) continue;
    const size_t row = ((size_t)f * g.N3 + j) * g.Pp;
    // rows past the end repeat the last one: their sums are not written
    const float4 *av[MA], *bv[NA];
#pragma unroll
    for (int t = 0; t < MA; t++)
      av[t] = reinterpret_cast<const float4*>(V + (size_t)min(i0 + 8 * t + r, nv - 1) * stride + row) + q;
#pragma unroll
    for (int t = 0; t < NA; t++)
      bv[t] = reinterpret_cast<const float4*>(W + (size_t)min(8 * t + r, nw - 1) * stride + row) + q;
    // the loads of the next step go ahead of this step's arithmetic
    float4 na[MA], nb[NA];
#pragma unroll
    for (int t = 0; t < MA; t++) na[t] = av[t][0];
#pragma unroll
    for (int t = 0; t < NA; t++) nb[t] = bv[t][0];
    for (int s = 0; s < steps; s++) {
      float a[MA][4], b[NA][4];
      const int left = 2 * g.P - (16 * s + 4 * q);   // floats of kept modes from this lane's on
#pragma unroll
      for (int t = 0; t < MA; t++) {
        const float4 x = na[t];
        a[t][0] = left > 0 ? x.x : 0.f;
        a[t][1] = left > 1 ? x.y : 0.f;
        a[t][2] = left > 2 ? x.z : 0.f;
        a[t][3] = left > 3 ? x.w : 0.f;
      }
#pragma unroll
      for (int t = 0; t < NA; t++) {
        const float4 x = nb[t];
        b[t][0] = left > 0 ? x.x : 0.f;
        b[t][1] = left > 1 ? x.y : 0.f;
        b[t][2] = left > 2 ? x.z : 0.f;
        b[t][3] = left > 3 ? x.w : 0.f;
      }
      const int n = min(s + 1, steps - 1);
#pragma unroll
      for (int t = 0; t < MA; t++) na[t] = av[t][4 * n];
#pragma unroll
      for (int t = 0; t < NA; t++) nb[t] = bv[t][4 * n];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        // the (0,0) mode counts once, the others twice (Integration.h:282-311)
        const double w = (s == 0 && q == 0 && e < 2) ? wz : 2.0 * wz;
        double bd[NA];
#pragma unroll
        for (int t = 0; t < NA; t++) bd[t] = w * (double)b[t][e];
#pragma unroll
        for (int u = 0; u < MA; u++) {
          const double ad = (double)a[u][e];
#pragma unroll
          for (int t = 0; t < NA; t++) mma_f64(acc[u][t], ad, bd[t]);
        }
      }
    }
  }
  // the warps' sums: element (row r, columns 2q, 2q + 1) of each 8 x 8 tile
  __shared__ double sum[3][MA * NA * 2][32];
  if (warp > 0) {
#pragma unroll
    for (int u = 0; u < MA; u++)
#pragma unroll
      for (int t = 0; t < NA; t++)
#pragma unroll
        for (int e = 0; e < 2; e++) sum[warp - 1][(u * NA + t) * 2 + e][lane] = acc[u][t][e];
  }
  __syncthreads();
  if (warp > 0) return;
#pragma unroll
  for (int u = 0; u < MA; u++)
#pragma unroll
    for (int t = 0; t < NA; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int k = (u * NA + t) * 2 + e, i = i0 + 8 * u + r, c = 8 * t + 2 * q + e;
        if (i < nv && c < nw)
          part[((size_t)blockIdx.x * nv + i) * nw + c] = acc[u][t][e] + sum[0][k][lane] + sum[1][k][lane] + sum[2][k][lane];
      }
}

// out[e] = the sum over the partials, in a fixed order: a block takes 32
// entries, eight threads each
__global__ void __launch_bounds__(256) k_gram_sum(const double* __restrict__ part, int nparts, int nvw,
                                                  double* __restrict__ out) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (e < nvw)
    for (int c = w; c < nparts; c += 8) s += part[(size_t)c * nvw + e];
  red[w][lane] = s;
  __syncthreads();
  if (w > 0 || e >= nvw) return;
  for (int k = 1; k < 8; k++) s += red[k][lane];
  out[e] = s;
}

// W_k += sum_i coef[i][k] V_i over u1,u2,u3,b, k < nw <= NW; coef holds NW
// floats per i (alpha included, zeros past nw). Each warp of a block sums
// every eighth V_i of the same 64 values of all NW results, two values per
// lane, the results in packed pairs of k; the warps' sums are added in shared
// memory. Bound by the one reading of V (320 vectors of 256x1x256: 252 MB, 39
// us) and the FMAs (28 us); with the coefficients converted from FP64 by
// every thread 347 us, now 98.
template <int NW>
__global__ void __launch_bounds__(256) k_update(Geo g, float2* __restrict__ W, int nw, const float2* __restrict__ V,
                                                int nv, size_t stride, const float* __restrict__ coef) {
  __shared__ float4 red[4][NW][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t n = (size_t)4 * g.fblk;                      // a multiple of 64: Pp is one of 16, N3 of 4
  const size_t e = (size_t)blockIdx.x * 64 + 2 * lane;      // this lane's two values
  constexpr int H = (NW + 1) / 2;
  float2 acc[4][H];   // re, im, re, im; (k, k + 1)
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int h = 0; h < H; h++) acc[c][h] = make_float2(0.f, 0.f);
  if (e < n) {
#pragma unroll 4
    for (int i = warp; i < nv; i += 8) {
      const float4 v = *reinterpret_cast<const float4*>(V + (size_t)i * stride + e);
      float2 c[H];
      if (NW == 1) {
        c[0] = make_float2(coef[i], 0.f);
      } else {
#pragma unroll
        for (int h = 0; h < H; h += 2) {
          const float4 x = __ldg(reinterpret_cast<const float4*>(coef + (size_t)i * NW) + h / 2);
          c[h] = make_float2(x.x, x.y);
          c[h + 1 < H ? h + 1 : h] = make_float2(x.z, x.w);
        }
      }
#pragma unroll
      for (int h = 0; h < H; h++) {
        acc[0][h] = __ffma2_rn(c[h], make_float2(v.x, v.x), acc[0][h]);
        acc[1][h] = __ffma2_rn(c[h], make_float2(v.y, v.y), acc[1][h]);
        acc[2][h] = __ffma2_rn(c[h], make_float2(v.z, v.z), acc[2][h]);
        acc[3][h] = __ffma2_rn(c[h], make_float2(v.w, v.w), acc[3][h]);
      }
    }
  }
  // the upper four warps' sums to the lower four, then those to the results
  for (int half = 1; half >= 0; half--) {
    if ((warp >> 2) == half) {
#pragma unroll
      for (int k = 0; k < NW; k++) {
        float4& r = red[warp & 3][k][lane];
        const int h = k / 2;
        const float4 x = k % 2 == 0 ? make_float4(acc[0][h].x, acc[1][h].x, acc[2][h].x, acc[3][h].x)
                                    : make_float4(acc[0][h].y, acc[1][h].y, acc[2][h].y, acc[3][h].y);
        r = half ? x : make_float4(r.x + x.x, r.y + x.y, r.z + x.z, r.w + x.w);
      }
    }
    __syncthreads();
  }
  if (e >= n) return;
  for (int k = warp; k < nw; k += 8) {
    float4 s = red[0][k][lane];
#pragma unroll
    for (int w = 1; w < 4; w++) {
      const float4 x = red[w][k][lane];
      s = make_float4(s.x + x.x, s.y + x.y, s.z + x.z, s.w + x.w);
    }
    float4* w = reinterpret_cast<float4*>(W + (size_t)k * stride + e);
    const float4 o = *w;
    *w = make_float4(o.x + s.x, o.y + s.y, o.z + s.z, o.w + s.w);
  }
}

// keep field f of mode m only if bit f of fieldmask is set and lo <= j1 < hi;
// p is zeroed
__global__ void k_band(Geo g, float2* v, int fieldmask, int lo, int hi) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= g.Pp) return;
  const int j1 = m % g.K1;
  for (int f = 0; f < 5; f++) {
    const bool keep = f < 4 && ((fieldmask >> f) & 1) && j1 >= lo && j1 < hi && m < g.P;
    if (keep) continue;
    for (int j = 0; j < g.N3; j++) v[((size_t)f * g.N3 + j) * g.Pp + m] = make_float2(0.f, 0.f);
  }
}

// StateVector::EnforceBCs (StateVector.h:415-421): u3 ZeroEnds, u1,u2,b
// NeumannEnds, on the kept modes
__global__ void k_enforce_bcs(Geo g, float2* v) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= g.P) return;
  const int N3 = g.N3;
  auto at = [&](int f, int j) -> float2& { return v[((size_t)f * N3 + j) * g.Pp + m]; };
  const float2 z = make_float2(0.f, 0.f);
  at(2, 0) = z; at(2, 1) = z; at(2, 2) = z; at(2, N3 - 2) = z; at(2, N3 - 1) = z;
  for (int f : {0, 1, 3}) {
    at(f, 0) = at(f, 1);
    at(f, N3 - 1) = at(f, N3 - 2);
  }
}

// ModalField::PhaseShift (Field.h:1168-1174) on u1,u2,u3,b: mode j1 times e^{i j1 shift}
__global__ void k_phase(Geo g, float2* v, double shift) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= g.P) return;
  const int j1 = m % g.K1;
  double sn, cs;
  sincos(j1 * shift, &sn, &cs);
  const float c = (float)cs, s = (float)sn;
  for (int f = 0; f < 4; f++)
    for (int j = 0; j < g.N3; j++) {
      float2& a = v[((size_t)f * g.N3 + j) * g.Pp + m];
      const float2 b = a;
      a = make_float2(b.x * c - b.y * s, b.x * s + b.y * c);
    }
}

// subtract a real constant from the (0,0) mode of one field (RemoveAverage)
__global__ void k_sub_mean(Geo g, float2* v, int f, float value) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.N3) return;
  v[((size_t)f * g.N3 + j) * g.Pp].x -= value;
}

inline unsigned nb(size_t n, int t) {
  size_t b = (n + t - 1) / t;
  return (unsigned)(b > 4096 ? 4096 : b);
}

}  // namespace

extern "C" {

int sf_vecs_create(sf_solver* like, int nvec, sf_vecs** out) {
  if (!like || nvec < 1 || !out) return vfail(SF_EINVAL, "bad argument");
  sf_vecs* v = new sf_vecs();
  v->g = sf_solver_geo(like);
  v->nvec = nvec;
  v->zc = sf_solver_zc(like);
  v->st = sf_solver_stream(like);
  v->z = sf_solver_z(like, 0);
  v->zf = sf_solver_z(like, 1);
  cudaError_t e = cudaMalloc(&v->d, sizeof(float2) * vstride(v->g) * nvec);
  if (e == cudaSuccess) e = cudaMemsetAsync(v->d, 0, sizeof(float2) * vstride(v->g) * nvec, v->st);
  v->cap_red = nvec;
  if (e == cudaSuccess) e = cudaMalloc(&v->red, sizeof(double) * v->cap_red);
  if (e != cudaSuccess) {
    if (v->d) cudaFree(v->d);
    if (v->red) cudaFree(v->red);
    delete v;
    return vfail(e == cudaErrorMemoryAllocation ? SF_ENOMEM : SF_ECUDA, cudaGetErrorString(e));
  }
  *out = v;
  return SF_OK;
}

int sf_vecs_destroy(sf_vecs* v) {
  if (!v) return SF_OK;
  // no use of the solver's stream here: the solver may be gone already;
  // cudaFree waits for the device work that may still read the memory
  cudaFree(v->d);
  cudaFree(v->red);
  cudaFree(v->coef);
  delete v;
  return SF_OK;
}

int sf_vecs_count(sf_vecs* v, int* n) {
  if (!v || !n) return vfail(SF_EINVAL, "bad argument");
  *n = v->nvec;
  return SF_OK;
}

int sf_vecs_device(sf_vecs* v, int i, void** ptr) {
  if (!v || i < 0 || i >= v->nvec || !ptr) return vfail(SF_EINVAL, "bad argument");
  *ptr = v->d + (size_t)i * vstride(v->g);
  return SF_OK;
}

int sf_vecs_from_run(sf_vecs* v, int i, sf_solver* s, int run, int count) {
  if (!v || !s || count < 1 || i < 0 || i + count > v->nvec || run < 0 || run + count > sf_solver_geo(s).nrun)
    return vfail(SF_EINVAL, "bad argument");
  VCK(cudaStreamSynchronize(sf_solver_stream(s)));
  VCK(cudaMemcpyAsync(v->d + (size_t)i * vstride(v->g), sf_solver_state(s, run),
                      sizeof(float2) * vstride(v->g) * count, cudaMemcpyDeviceToDevice, v->st));
  return SF_OK;
}

int sf_vecs_to_run(sf_vecs* v, int i, sf_solver* s, int run, int count) {
  if (!v || !s || count < 1 || i < 0 || i + count > v->nvec || run < 0 || run + count > sf_solver_geo(s).nrun)
    return vfail(SF_EINVAL, "bad argument");
  VCK(cudaStreamSynchronize(v->st));
  VCK(cudaMemcpyAsync(sf_solver_state(s, run), v->d + (size_t)i * vstride(v->g),
                      sizeof(float2) * vstride(v->g) * count, cudaMemcpyDeviceToDevice, sf_solver_stream(s)));
  VCK(cudaStreamSynchronize(sf_solver_stream(s)));
  return SF_OK;
}

int sf_vecs_copy(sf_vecs* v, int dst, sf_vecs* w, int src) {
  if (!v || !w || dst < 0 || dst >= v->nvec || src < 0 || src >= w->nvec) return vfail(SF_EINVAL, "bad argument");
  VCK(cudaMemcpyAsync(v->d + (size_t)dst * vstride(v->g), w->d + (size_t)src * vstride(w->g),
                      sizeof(float2) * vstride(v->g), cudaMemcpyDeviceToDevice, v->st));
  return SF_OK;
}

int sf_vecs_set_host(sf_vecs* v, int i, const float* host) {
  if (!v || !host || i < 0 || i >= v->nvec) return vfail(SF_EINVAL, "bad argument");
  VCK(cudaMemcpyAsync(v->d + (size_t)i * vstride(v->g), host, sizeof(float2) * vstride(v->g), cudaMemcpyHostToDevice,
                      v->st));
  VCK(cudaStreamSynchronize(v->st));
  return SF_OK;
}

int sf_vecs_get_host(sf_vecs* v, int i, float* host) {
  if (!v || !host || i < 0 || i >= v->nvec) return vfail(SF_EINVAL, "bad argument");
  VCK(cudaMemcpyAsync(host, v->d + (size_t)i * vstride(v->g), sizeof(float2) * vstride(v->g), cudaMemcpyDeviceToHost,
                      v->st));
  VCK(cudaStreamSynchronize(v->st));
  return SF_OK;
}

// v[y+k] += alpha w[x+k] on u1,u2,u3,b for k < count (MulAdd)
int sf_vecs_axpy(sf_vecs* v, int y, double alpha, sf_vecs* w, int x, int count) {
  if (!v || !w || count < 1 || y < 0 || y + count > v->nvec || x < 0 || x + count > w->nvec)
    return vfail(SF_EINVAL, "bad argument");
  const size_t f4 = (size_t)4 * v->g.fblk, vs = vstride(v->g);
  k_axpy<<<nb(f4 * count, 256), 256, 0, v->st>>>(v->d + (size_t)y * vs, w->d + (size_t)x * vs, (float)alpha, f4, vs,
                                                  count);
  VCK(cudaGetLastError());
  return SF_OK;
}

// v[y+k] = a v[y+k] + b w[x+k] on all five fields, k < count
int sf_vecs_lincomb(sf_vecs* v, int y, double a, double b, sf_vecs* w, int x, int count) {
  if (!v || !w || count < 1 || y < 0 || y + count > v->nvec || x < 0 || x + count > w->nvec)
    return vfail(SF_EINVAL, "bad argument");
  size_t n = vstride(v->g) * count;
  k_lincomb<<<nb(n, 256), 256, 0, v->st>>>(v->d + (size_t)y * vstride(v->g), w->d + (size_t)x * vstride(v->g),
                                            (float)a, (float)b, n);
  VCK(cudaGetLastError());
  return SF_OK;
}

int sf_vecs_scale(sf_vecs* v, int i, double alpha, int count) {
  if (!v || count < 1 || i < 0 || i + count > v->nvec) return vfail(SF_EINVAL, "bad argument");
  return sf_vecs_lincomb(v, i, alpha, 0.0, v, i, count);
}

static int ensure_red(sf_vecs* v, int count) {
  if (count > v->cap_red) {
    cudaFree(v->red);
    v->cap_red = count;
    VCK(cudaMalloc(&v->red, sizeof(double) * count));
  }
  return SF_OK;
}

// out[k] = StateVector::Dot(v[first + k], w[x]) for k < count, FP64
int sf_vecs_dots(sf_vecs* v, int first, int count, sf_vecs* w, int x, double Ri, double* out) {
  if (!v || !w || !out || first < 0 || count < 1 || first + count > v->nvec || x < 0 || x >= w->nvec)
    return vfail(SF_EINVAL, "bad argument");
  int rc = ensure_red(v, count);
  if (rc) return rc;
  VCK(cudaMemsetAsync(v->red, 0, sizeof(double) * count, v->st));
  k_dots<<<dim3(v->g.N3, count, 4), 256, 0, v->st>>>(v->g, v->d + (size_t)first * vstride(v->g), vstride(v->g),
                                                     w->d + (size_t)x * vstride(w->g), 0, v->zc, Ri, v->red, 0);
  VCK(cudaGetLastError());
  VCK(cudaMemcpyAsync(out, v->red, sizeof(double) * count, cudaMemcpyDeviceToHost, v->st));
  VCK(cudaStreamSynchronize(v->st));
  return SF_OK;
}

// *out = sum_k Dot(v[a + k], w[b + k]) for k < count, FP64
int sf_vecs_dot_sum(sf_vecs* v, int a, sf_vecs* w, int b, int count, double Ri, double* out) {
  if (!v || !w || !out || count < 1 || a < 0 || a + count > v->nvec || b < 0 || b + count > w->nvec)
    return vfail(SF_EINVAL, "bad argument");
  int rc = ensure_red(v, 1);
  if (rc) return rc;
  VCK(cudaMemsetAsync(v->red, 0, sizeof(double), v->st));
  k_dots<<<dim3(v->g.N3, count, 4), 256, 0, v->st>>>(v->g, v->d + (size_t)a * vstride(v->g), vstride(v->g),
                                                     w->d + (size_t)b * vstride(w->g), vstride(w->g), v->zc, Ri,
                                                     v->red, 1);
  VCK(cudaGetLastError());
  VCK(cudaMemcpyAsync(out, v->red, sizeof(double), cudaMemcpyDeviceToHost, v->st));
  VCK(cudaStreamSynchronize(v->st));
  return SF_OK;
}

int sf_vecs_enforce_bcs(sf_vecs* v, int i, int count) {
  if (!v || count < 1 || i < 0 || i + count > v->nvec) return vfail(SF_EINVAL, "bad argument");
  for (int k = 0; k < count; k++)
    k_enforce_bcs<<<(v->g.P + 127) / 128, 128, 0, v->st>>>(v->g, v->d + (size_t)(i + k) * vstride(v->g));
  VCK(cudaGetLastError());
  return SF_OK;
}

// StateVector::RemovePhaseShift (StateVector.h:103-120): shift = pi/2 -
// arg(u1(1,0,N3/2)) unless `shift` is given (use_given != 0); returns it
int sf_vecs_phase_shift(sf_vecs* v, int i, int use_given, double* shift) {
  if (!v || !shift || i < 0 || i >= v->nvec) return vfail(SF_EINVAL, "bad argument");
  if (!use_given) {
    float2 h;
    const float2* p = v->d + (size_t)i * vstride(v->g) + (size_t)(v->g.N3 / 2) * v->g.Pp + 1;   // u1, j1=1, j2=0
    VCK(cudaMemcpyAsync(&h, p, sizeof(float2), cudaMemcpyDeviceToHost, v->st));
    VCK(cudaStreamSynchronize(v->st));
    *shift = -std::atan2((double)h.y, (double)h.x) + 3.141592653589793238462 / 2;
  }
  k_phase<<<(v->g.P + 127) / 128, 128, 0, v->st>>>(v->g, v->d + (size_t)i * vstride(v->g), *shift);
  VCK(cudaGetLastError());
  return SF_OK;
}

// RemoveAverage(field, L3) (Integration.h:236-240) for field 0 (u1) or 3 (b):
// subtract IntegrateVertically(real (0,0) stack)/(2 L3) from the (0,0) stack
int sf_vecs_remove_average(sf_vecs* v, int i, int field, double L3) {
  if (!v || i < 0 || i >= v->nvec || (field != 0 && field != 3)) return vfail(SF_EINVAL, "bad argument");
  const Geo& g = v->g;
  std::vector<float2> col(g.N3);
  const float2* base = v->d + (size_t)i * vstride(g) + (size_t)field * g.fblk;
  VCK(cudaMemcpy2DAsync(col.data(), sizeof(float2), base, sizeof(float2) * g.Pp, sizeof(float2), g.N3,
                        cudaMemcpyDeviceToHost, v->st));
  VCK(cudaStreamSynchronize(v->st));
  double integ = 0.0;   // Neumann quadrature (Integration.h:8-21)
  for (int k = 1; k < g.N3 - 1; k++) integ += (v->z[k + 1] - v->z[k]) * (double)col[k].x;
  const float value = (float)(integ / L3 / 2);
  k_sub_mean<<<(g.N3 + 127) / 128, 128, 0, v->st>>>(g, v->d + (size_t)i * vstride(g), field, value);
  VCK(cudaGetLastError());
  return SF_OK;
}

// out[i * nb + k] = Dot(v[a + i], w[b + k]) (StateVector::Dot, FP64)
int sf_vecs_gram(sf_vecs* v, int a, int na, sf_vecs* w, int b, int nb, double Ri, double* out) {
  if (!v || !w || !out || na < 1 || nb < 1 || nb > kMaxBlock || a < 0 || a + na > v->nvec || b < 0 ||
      b + nb > w->nvec)
    return vfail(SF_EINVAL, "bad argument (1 <= nb <= 32)");
  const Geo& g = v->g;
  const int nch = (g.N3 + kGramLevels - 1) / kGramLevels;
  const size_t nvw = (size_t)na * nb, parts = (size_t)(g.dim3 ? 4 : 3) * nch;
  int rc = ensure_red(v, (int)(nvw * (parts + 1)));
  if (rc) return rc;
  double* part = v->red + nvw;
  auto* wd = w->d + (size_t)b * vstride(w->g);
  auto* vd = v->d + (size_t)a * vstride(g);
  const size_t vs = vstride(g);
  // 32 vectors of V per warp; 16 where there are no more, or where a block of 32 has twice the sums
  auto launch = [&](auto* k, int ma) {
    k<<<dim3((unsigned)parts, (na + 8 * ma - 1) / (8 * ma)), 128, 0, v->st>>>(g, vd, na, wd, nb, vs, v->zc, Ri, part);
  };
  if (nb <= 8) na <= 16 ? launch(k_gram<2, 1>, 2) : launch(k_gram<4, 1>, 4);
  else if (nb <= 16) na <= 16 ? launch(k_gram<2, 2>, 2) : launch(k_gram<4, 2>, 4);
  else launch(k_gram<2, 4>, 2);
  VCK(cudaGetLastError());
  k_gram_sum<<<(unsigned)((nvw + 31) / 32), 256, 0, v->st>>>(part, (int)parts, (int)nvw, v->red);
  VCK(cudaGetLastError());
  VCK(cudaMemcpyAsync(out, v->red, sizeof(double) * nvw, cudaMemcpyDeviceToHost, v->st));
  VCK(cudaStreamSynchronize(v->st));
  return SF_OK;
}

// w[b + k] += alpha sum_i coef[i * nb + k] v[a + i] on u1..b (v and w ranges
// must not overlap)
int sf_vecs_update(sf_vecs* w, int b, int nb, double alpha, sf_vecs* v, int a, int na, const double* coef) {
  if (!v || !w || !coef || na < 1 || nb < 1 || nb > kMaxBlock || a < 0 || a + na > v->nvec || b < 0 ||
      b + nb > w->nvec)
    return vfail(SF_EINVAL, "bad argument (1 <= nb <= 32)");
  if (v == w && a < b + nb && b < a + na) return vfail(SF_EINVAL, "overlapping ranges");
  // two launches above 16 vectors, whose sums would not fit the registers
  for (int k0 = 0; k0 < nb; k0 += 16) {
    const int k = std::min(16, nb - k0), NW = k <= 1 ? 1 : (k <= 4 ? 4 : (k <= 8 ? 8 : 16));
    const size_t nc = (size_t)na * NW;
    if (nc > w->cap_coef) {
      cudaFree(w->coef);
      w->coef = nullptr;
      w->cap_coef = 0;
      VCK(cudaMalloc(&w->coef, sizeof(float) * nc));
      w->cap_coef = nc;
    }
    std::vector<float> c(nc, 0.f);
    for (int i = 0; i < na; i++)
      for (int j = 0; j < k; j++) c[(size_t)i * NW + j] = (float)(alpha * coef[(size_t)i * nb + k0 + j]);
    // from pageable memory: c has been read when the call returns
    VCK(cudaMemcpyAsync(w->coef, c.data(), sizeof(float) * nc, cudaMemcpyHostToDevice, w->st));
    const Geo& g = w->g;
    const unsigned blocks = (unsigned)(((size_t)4 * g.fblk + 63) / 64);
    const size_t vs = vstride(g);
    float2* wd = w->d + (size_t)(b + k0) * vs;
    const float2* vd = v->d + (size_t)a * vs;
    if (NW == 1) k_update<1><<<blocks, 256, 0, w->st>>>(g, wd, k, vd, na, vs, w->coef);
    else if (NW == 4) k_update<4><<<blocks, 256, 0, w->st>>>(g, wd, k, vd, na, vs, w->coef);
    else if (NW == 8) k_update<8><<<blocks, 256, 0, w->st>>>(g, wd, k, vd, na, vs, w->coef);
    else k_update<16><<<blocks, 256, 0, w->st>>>(g, wd, k, vd, na, vs, w->coef);
    VCK(cudaGetLastError());
  }
  return SF_OK;
}

// keep only the fields in field_mask (bit f: u1, u2, u3, b) and the modes
// with j1_lo <= j1 < j1_hi of vector i; p is zeroed
int sf_vecs_band(sf_vecs* v, int i, int field_mask, int j1_lo, int j1_hi) {
  if (!v || i < 0 || i >= v->nvec) return vfail(SF_EINVAL, "bad argument");
  k_band<<<(v->g.Pp + 127) / 128, 128, 0, v->st>>>(v->g, v->d + (size_t)i * vstride(v->g), field_mask, j1_lo, j1_hi);
  VCK(cudaGetLastError());
  return SF_OK;
}

// copy the z column of one mode of one field of vector i (N3 complex values)
// to the host (write = 0) or from it (write = 1)
int sf_vecs_column(sf_vecs* v, int i, int field, int mode, float* host, int write) {
  if (!v || !host || i < 0 || i >= v->nvec || field < 0 || field > 4 || mode < 0 || mode >= v->g.P)
    return vfail(SF_EINVAL, "bad argument");
  float2* col = v->d + (size_t)i * vstride(v->g) + (size_t)field * v->g.fblk + mode;
  const size_t pitch = sizeof(float2) * v->g.Pp;
  if (write) {
    VCK(cudaMemcpy2DAsync(col, pitch, host, sizeof(float2), sizeof(float2), v->g.N3, cudaMemcpyHostToDevice, v->st));
  } else {
    VCK(cudaMemcpy2DAsync(host, sizeof(float2), col, pitch, sizeof(float2), v->g.N3, cudaMemcpyDeviceToHost, v->st));
  }
  VCK(cudaStreamSynchronize(v->st));
  return SF_OK;
}

// zero the p field of vectors i..i+count-1
int sf_vecs_zero_pressure(sf_vecs* v, int i, int count) {
  if (!v || count < 1 || i < 0 || i + count > v->nvec) return vfail(SF_EINVAL, "bad argument");
  for (int k = 0; k < count; k++)
    VCK(cudaMemsetAsync(v->d + (size_t)(i + k) * vstride(v->g) + (size_t)4 * v->g.fblk, 0,
                        sizeof(float2) * v->g.fblk, v->st));
  return SF_OK;
}

int sf_vecs_synchronize(sf_vecs* v) {
  if (!v) return vfail(SF_EINVAL, "bad argument");
  VCK(cudaStreamSynchronize(v->st));
  return SF_OK;
}

}  // extern "C"
