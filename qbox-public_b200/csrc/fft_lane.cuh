// Register DFTs of composite length for the FFT kernels (fft_pencil.cuh): a
// compile-time mixed-radix Cooley-Tukey recursion over the short DFTs of
// fft_reg.cuh, its twiddles compile-time constants computed by a constexpr
// cosine/sine below.
#pragma once

#include <cuda_runtime.h>

#include "fft_reg.cuh"

namespace qbx {
namespace lane {

using reg::cadd;
using reg::cmk;
using reg::cmul;
using reg::cmulc;
using reg::csub;

// ------------------------------------------------------------ constexpr trig
// cos and sin of 2 pi p / q for integers 0 <= p < q, by Taylor series after
// reduction to |angle| <= pi/4 (the octant symmetries of the circle); the
// series is summed to double precision.
__host__ __device__ constexpr double cx_pi() { return 3.14159265358979323846264338327950288; }
__host__ __device__ constexpr double taylor_sin(double a) {
  double term = a, sum = a;
  for (int n = 1; n < 14; ++n) {
    term *= -a * a / ((2.0 * n) * (2.0 * n + 1.0));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double taylor_cos(double a) {
  double term = 1.0, sum = 1.0;
  for (int n = 1; n < 14; ++n) {
    term *= -a * a / ((2.0 * n - 1.0) * (2.0 * n));
    sum += term;
  }
  return sum;
}
// angle 2 pi p / q = (pi/4) * (8 p / q): octant o and remainder r in [0, 1)
__host__ __device__ constexpr void cx_cossin(long p, long q, double& c, double& s) {
  p %= q;
  if (p < 0) p += q;
  const long num = 8 * p;
  const long o = num / q;                         // octant 0..7
  const double r = (double)(num - o * q) / (double)q;   // fraction of the octant
  const double a = r * cx_pi() / 4.0;            // in [0, pi/4)
  const double b = (1.0 - r) * cx_pi() / 4.0;    // pi/4 - a
  double cc = 0, ss = 0;
  switch (o) {
    case 0: cc = taylor_cos(a); ss = taylor_sin(a); break;
    case 1: cc = taylor_sin(b); ss = taylor_cos(b); break;
    case 2: cc = -taylor_sin(a); ss = taylor_cos(a); break;
    case 3: cc = -taylor_cos(b); ss = taylor_sin(b); break;
    case 4: cc = -taylor_cos(a); ss = -taylor_sin(a); break;
    case 5: cc = -taylor_sin(b); ss = -taylor_cos(b); break;
    case 6: cc = taylor_sin(a); ss = -taylor_cos(a); break;
    default: cc = taylor_cos(b); ss = -taylor_sin(b); break;
  }
  c = cc;
  s = ss;
}
__host__ __device__ constexpr double cx_cos(long p, long q) {
  double c = 0, s = 0;
  cx_cossin(p, q, c, s);
  return c;
}
__host__ __device__ constexpr double cx_sin(long p, long q) {
  double c = 0, s = 0;
  cx_cossin(p, q, c, s);
  return s;
}

// ------------------------------------------------------------ register DFT
__host__ __device__ constexpr int first_radix(int m) {
  return m % 4 == 0 && m != 8 ? 4 : m % 2 == 0 ? 2 : m % 3 == 0 ? 3 : m % 5 == 0 ? 5
       : m % 7 == 0 ? 7 : m % 11 == 0 ? 11 : 0;
}
__host__ __device__ constexpr bool reg_ok(int m) {
  while (m > 1) {
    const int r = first_radix(m);
    if (r == 0) return false;
    m /= r;
  }
  return true;
}

// v[k] <- sum_j v[j] exp(DIR 2 pi i jk/M), all in registers (M <= ~36)
template <int M, int DIR, typename C>
__device__ __forceinline__ void dft_reg(C (&v)[M]) {
  if constexpr (M == 1) {
    return;
  } else if constexpr (M == 2 || M == 3 || M == 4 || M == 5 || M == 7 || M == 11) {
    reg::dft<M, DIR>(v);
  } else {
    // M = R Q: R interleaved sub-sequences of length Q, then R-point DFTs
    constexpr int R = first_radix(M);
    constexpr int Q = M / R;
    static_assert(R > 0, "register DFT length must factor into 2, 3, 5, 7, 11");
    using Real = decltype(v[0].x);
    C sub[R][Q];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int k = 0; k < Q; ++k) sub[r][k] = v[r + R * k];
#pragma unroll
    for (int r = 0; r < R; ++r) dft_reg<Q, DIR>(sub[r]);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      C w[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r == 0 || q == 0) {
          w[r] = sub[r][q];
        } else {
          const Real c = (Real)cx_cos((long)r * q, M);
          const Real s = (Real)(DIR * cx_sin((long)r * q, M));
          const C x = sub[r][q];
          w[r] = cmk<C>(x.x * c - x.y * s, x.x * s + x.y * c);
        }
      }
      reg::dft<R, DIR>(w);
#pragma unroll
      for (int s2 = 0; s2 < R; ++s2) v[q + Q * s2] = w[s2];
    }
  }
}

}  // namespace lane
}  // namespace qbx
