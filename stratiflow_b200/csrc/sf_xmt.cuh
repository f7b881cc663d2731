// Lane layouts of the level-marching x passes (sf_xmarch.cu, sf_adjmarch.cu).
#pragma once
#include <algorithm>
#include "sf_internal.cuh"
#include "sf_fft2.cuh"

namespace sf {

// Lane layout of the march for one grid width N1: G lanes per y row, E x
// points per lane (x = l + G e), W rows per warp, the output slots that hold
// the kept modes, and the packed transform pair.
template <int N1>
struct XMT {   // N1 = 32, 64: two-stage transforms over FFTShape<N1>::G lanes
  static constexpr int G = FFTShape<N1>::G, E = FFTShape<N1>::E, H = E / G, K1 = N1 / 3;
  static constexpr int W = 32 / G;                  // rows per warp
  static constexpr int NK2 = (K1 - 1) / E + 1;
  static constexpr int NKS = H * NK2;               // output slots holding a kept mode for some lane
  static constexpr int TB = fft2_buf_elems<N1>();   // float4 per transpose buffer
  static constexpr int TWE = E * G;                 // twiddle table entries
  // output slot of the i-th kept candidate; slot h*G + k2 holds mode l + h*G + E*k2
  __host__ __device__ static constexpr int kslot(int i) { return (i / NK2) * G + i % NK2; }
  __device__ __forceinline__ static int kmode(int l, int i) { return l + (kslot(i) / G) * G + E * (kslot(i) % G); }
  // x position index e (x = l + G e) of inverse output slot s
  __host__ __device__ static constexpr int pos(int s) { return s / G + H * (s % G); }
  // slot holding mode N1 - k at lane G - l (l >= 1) or at lane 0 (l = 0)
  __host__ __device__ static constexpr int partner(int i, bool lane0) {
    const int s = kslot(i), h = s / G, k2 = s % G;
    const int q = lane0 ? (E - h - H * k2) % E : E - 1 - h - H * k2;
    return (q % H) * G + q / H;
  }
  __device__ __forceinline__ static void fill(float4* tw4, float2* tw2, const float2* tw, int tid, int nthr) {
    fill_tw2<N1>(tw4, tw2, tw, tid, nthr);
  }
  template <bool INV>
  __device__ __forceinline__ static void fft(c2x (&x)[E], float4* buf, const float4* tw4, const float2* tw2, int l,
                             const float4 (&)[8]) {
    reg_fft2<N1, INV>(x, buf, tw4, tw2, l);
  }
};
template <>
struct XMT<128> {   // 16 lanes per row: three stages, 8 x 4 x 4 (reg_fft2_128h)
  static constexpr int G = 16, E = 8, K1 = 42, W = 2;
  static constexpr int NKS = 3;                     // modes l, l + 16, l + 32
  static constexpr int TB = 8 * 17, TWE = 8 * 16;
  // slot of out[l + 16 j]: j = i + 2 q in slot i*4 + q
  __host__ __device__ static constexpr int jslot(int j) { return (j % 2) * 4 + j / 2; }
  __host__ __device__ static constexpr int kslot(int i) { return jslot(i); }
  __device__ __forceinline__ static int kmode(int l, int i) { return l + 16 * i; }
  __host__ __device__ static constexpr int pos(int s) { return s / 4 + 2 * (s % 4); }
  __host__ __device__ static constexpr int partner(int i, bool lane0) { return jslot(lane0 ? (8 - i) % 8 : 7 - i); }
  __device__ __forceinline__ static void fill(float4* tw4, float2* tw2, const float2* tw, int tid, int nthr) {
    fill_tw2_128h(tw4, tw2, tw, tid, nthr);
  }
  template <bool INV>
  __device__ __forceinline__ static void fft(c2x (&x)[E], float4* buf, const float4*, const float2* tw2, int l, const float4 (&w1)[8]) {
    reg_fft2_128h<INV>(x, buf, tw2, l, w1);
  }
};
template <>
struct XMT<256> {   // a whole warp per row: three stages, 8 x 8 x 4 (reg_fft2_256w)
  static constexpr int G = 32, E = 8, K1 = 85, W = 1;
  static constexpr int NKS = 3;                     // modes l, l + 32, l + 64
  static constexpr int TB = 8 * 33, TWE = 8 * 32;
  // slot of out[l + 32 j]: j = h + 2 q in slot h*4 + q
  __host__ __device__ static constexpr int jslot(int j) { return (j % 2) * 4 + j / 2; }
  __host__ __device__ static constexpr int kslot(int i) { return jslot(i); }
  __device__ __forceinline__ static int kmode(int l, int i) { return l + 32 * i; }
  __host__ __device__ static constexpr int pos(int s) { return s / 4 + 2 * (s % 4); }
  __host__ __device__ static constexpr int partner(int i, bool lane0) { return jslot(lane0 ? (8 - i) % 8 : 7 - i); }
  __device__ __forceinline__ static void fill(float4* tw4, float2* tw2, const float2* tw, int tid, int nthr) {
    fill_tw2_256w(tw4, tw2, tw, tid, nthr);
  }
  template <bool INV>
  __device__ __forceinline__ static void fft(c2x (&x)[E], float4* buf, const float4* tw4, const float2* tw2, int l,
                             const float4 (&w1)[8]) {
    reg_fft2_256w<INV>(x, buf, tw4, tw2, l, w1);
  }
};

template <>
struct XMT<512> {   // a whole warp per row: 16 points per lane (reg_fft2_512w)
  static constexpr int G = 32, E = 16, K1 = 170, W = 1;
  static constexpr int NKS = 6;                     // modes l + 32 j, j < 6
  static constexpr int TB = 16 * 33, TWE = 16 * 32;
  // slot of out[l + 32 j]: j = i + 4 q in slot i*4 + q
  __host__ __device__ static constexpr int jslot(int j) { return (j % 4) * 4 + j / 4; }
  __host__ __device__ static constexpr int kslot(int i) { return jslot(i); }
  __device__ __forceinline__ static int kmode(int l, int i) { return l + 32 * i; }
  __host__ __device__ static constexpr int pos(int s) { return s / 4 + 4 * (s % 4); }
  __host__ __device__ static constexpr int partner(int i, bool lane0) { return jslot(lane0 ? (16 - i) % 16 : 15 - i); }
  __device__ __forceinline__ static void fill(float4* tw4, float2* tw2, const float2* tw, int tid, int nthr) {
    fill_tw2_512w(tw4, tw2, tw, tid, nthr);
  }
  template <bool INV>
  __device__ __forceinline__ static void fft(c2x (&x)[E], float4* buf, const float4* tw4, const float2* tw2, int l,
                             const float4 (&)[8]) {
    reg_fft2_512w<INV>(x, buf, tw4, tw2, l);
  }
};

__device__ __forceinline__ void xm_cp8(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void xm_cp16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void xm_cp_wait() { asm volatile("cp.async.wait_all;\n" ::); }

__device__ __forceinline__ float4 c2x_f4(const c2x& v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }

inline int sm_count() {
  static const int n = [] {
    int dev = 0, k = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&k, cudaDevAttrMultiProcessorCount, dev);
    return k;
  }();
  return n;
}

}  // namespace sf
