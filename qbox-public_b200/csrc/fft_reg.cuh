// Complex arithmetic and the short prime DFTs in registers (2, 3, 4, 5, 7,
// 11 points) that the register transforms of fft_lane.cuh are built from.
//
// Sign convention: DIR = +1 computes out[k] = sum_j in[j] exp(+2 pi i jk/N)
// (the reference's backward transform, unscaled), DIR = -1 the forward one.
// The small DFTs use the cosines and sines of 2 pi j/R as literal constants.
#pragma once

#include <cuda_runtime.h>

namespace qbx {
namespace reg {

template <typename T> struct CT;
template <> struct CT<float> { using c = float2; };
template <> struct CT<double> { using c = double2; };

// cos(2 pi j/R), sin(2 pi j/R) for 1 <= j <= (R-1)/2
__host__ __device__ constexpr double rcos(int R, int j) {
  return R == 3 ? -0.5
       : R == 5 ? (j == 1 ? 0.30901699437494745 : -0.8090169943749475)
       : R == 7 ? (j == 1 ? 0.6234898018587335 : j == 2 ? -0.2225209339563144 : -0.9009688679024191)
       : (j == 1 ? 0.8412535328311812 : j == 2 ? 0.41541501300188644
          : j == 3 ? -0.14231483827328514 : j == 4 ? -0.6548607339452851 : -0.9594929736144974);
}
__host__ __device__ constexpr double rsin(int R, int j) {
  return R == 3 ? 0.8660254037844386
       : R == 5 ? (j == 1 ? 0.9510565162951535 : 0.5877852522924731)
       : R == 7 ? (j == 1 ? 0.7818314824680298 : j == 2 ? 0.9749279121818236 : 0.4338837391175581)
       : (j == 1 ? 0.5406408174555976 : j == 2 ? 0.9096319953545183
          : j == 3 ? 0.9898214418809327 : j == 4 ? 0.7557495743542583 : 0.28173255684142967);
}

// ------------------------------------------------------------ arithmetic
template <typename C> __device__ __forceinline__ C cmk(double x, double y) {
  C r; r.x = x; r.y = y; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) {
  C r; r.x = a.x + b.x; r.y = a.y + b.y; return r;
}
template <typename C> __device__ __forceinline__ C csub(C a, C b) {
  C r; r.x = a.x - b.x; r.y = a.y - b.y; return r;
}
// a s + b for a real s
template <typename C, typename Real> __device__ __forceinline__ C cfma(C a, Real s, C b) {
  C r; r.x = a.x * s + b.x; r.y = a.y * s + b.y; return r;
}
// FP32: both parts in one instruction (sm_100 f32x2 arithmetic, the same
// roundings).  These kernels are bound by issue: at 140^3, 512 band pairs, xd
// 2.37 -> 2.22 ms and xv 4.45 -> 4.06; at 72 x 40 x 112 xv 0.070 -> 0.066.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 p, q, s;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\t"
      "add.rn.f32x2 s, p, q;\n\tmov.b64 {%0, %1}, s;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 p, q, s;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\t"
      "sub.rn.f32x2 s, p, q;\n\tmov.b64 {%0, %1}, s;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 cfma(float2 a, float s, float2 b) {
  float2 r;
  asm("{.reg .b64 p, q, t, u;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\t"
      "mov.b64 t, {%5, %6};\n\tfma.rn.f32x2 u, p, q, t;\n\tmov.b64 {%0, %1}, u;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(s), "f"(b.x), "f"(b.y));
  return r;
}
// a s for a real s
__device__ __forceinline__ float2 cscale(float2 a, float s) {
  float2 r;
  asm("{.reg .b64 p, q, u;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\t"
      "mul.rn.f32x2 u, p, q;\n\tmov.b64 {%0, %1}, u;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(s));
  return r;
}
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
// a * conj(b)
template <typename C> __device__ __forceinline__ C cmulc(C a, C b) {
  C r; r.x = a.x * b.x + a.y * b.y; r.y = a.y * b.x - a.x * b.y; return r;
}
// DIR * i * a
template <int DIR, typename C> __device__ __forceinline__ C cmuli(C a) {
  C r;
  if (DIR > 0) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; }
  return r;
}

// R-point DFT in registers: v[k] <- sum_q v[q] exp(DIR 2 pi i qk/R)
template <int R, int DIR, typename C>
__device__ __forceinline__ void dft(C (&v)[R]) {
  if constexpr (R == 2) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const C a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
    const C c = cadd(v[1], v[3]), d = cmuli<DIR>(csub(v[1], v[3]));
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = cadd(b, d);
    v[3] = csub(b, d);
  } else {
    // odd prime R: pair q with R-q,
    //   out_k = v0 + sum_m (v_m + v_{R-m}) cos(2 pi mk/R)
    //              + DIR i sum_m (v_m - v_{R-m}) sin(2 pi mk/R)
    using Real = decltype(v[0].x);
    constexpr int H = (R - 1) / 2;
    C a[H + 1], b[H + 1];
    C s0 = v[0];
#pragma unroll
    for (int m = 1; m <= H; ++m) {
      a[m] = cadd(v[m], v[R - m]);
      b[m] = cmuli<DIR>(csub(v[m], v[R - m]));   // the factor DIR i once per pair
      s0 = cadd(s0, a[m]);
    }
    C out[R];
    out[0] = s0;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      C r = v[0], i = cmk<C>(0, 0);
#pragma unroll
      for (int m = 1; m <= H; ++m) {
        const int j = (m * k) % R;
        r = cfma(a[m], (Real)rcos(R, j <= H ? j : R - j), r);
        i = cfma(b[m], (Real)(j <= H ? rsin(R, j) : -rsin(R, R - j)), i);
      }
      out[k] = cadd(r, i);
      out[R - k] = csub(r, i);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = out[k];
  }
}

}  // namespace reg
}  // namespace qbx
