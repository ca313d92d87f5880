// Staged 3-D FFTs of the electronic step as three kernels of line transforms
// (z sticks, y columns, x rows) for any grid whose lengths are compiled here,
// cubic or not, band pairs at Gamma or single bands at a k point, FP32 or
// FP64.
//
// Layout.  Between the passes z is the fastest index,
//
//   sticks [slot][stick][z]    tile [slot][column][y][z]    rho, V [x][y][z]
//
// so a line along y or x is one of many neighbouring lines in memory: the
// lanes of a warp work on lines that differ in z (or in (y, z) flattened), and
// every load and store of the y and x passes is coalesced without a
// transposition.  A slot is a band pair (Gamma) or a band (k points).
//
// Line transform.  A line of N = R1 R2 points (R1 >= R2, both at most 20) is
// held by the threads of one CTA, R1 or R2 values each:
//
//   X[k + R1 m] = sum_j W_R2^{jm} ( W_N^{jk} sum_q x[j + R2 q] W_R1^{qk} )
//
// R2 items do an R1-point DFT in registers (inputs straight from global
// memory), twiddle and write shared memory; R1 items read R2 values each, do
// the second DFT and hand the results on (to global memory, to the density
// sum, or times V(r) into the opposite transform, which starts from this
// distribution and ends in the first one).  One exchange through shared memory
// per transform is all the traffic a line causes on chip; with the line index
// fastest in shared memory it has no bank conflicts.
//
// The wavefunction sphere fills at most the points within prune_width(N) of
// zero on each axis (the grid Qbox builds is at least 4 hmax + 1 long), so the
// R1-point DFTs load, or store, only the q that reach such points.
//
// What they replace: plane kernels that held a whole z plane in shared memory
// (one or two CTAs per SM, latency bound, cubic grids of 18 lengths only) and,
// for every other grid and for k points, runtime-radix kernels.  What bounds
// them now is HBM for the y passes (80 % of the measured copy rate at 140^3)
// and FP32 issue with the shared-memory exchange for xv.  Per step, density +
// H psi, before and after (ms): 512 atoms 140^3 FP32 15.5 -> 10.8, FP64 94.7 ->
// 21.1; 64 atoms 84^3 FP32 0.70 -> 0.40, FP64 2.24 -> 0.67; 112 x 72 x 40 FP32
// 1.09 -> 0.23; two k points 84^3 FP64 13.4 -> 2.4.
#pragma once

#include <cuda_runtime.h>

#include "fft_lane.cuh"
#include "fft_reg.cuh"
#include "qbx_internal.h"

namespace qbx {
namespace pen {

using reg::cmk;
using reg::cmul;
using reg::cmulc;
using reg::CT;

// N = R1 R2 with R1 >= R2 as close to square as the register DFTs allow
struct Fac { int r1, r2; };
__host__ __device__ constexpr Fac fac(int n) {
  int r2 = 1;
  for (int r = 2; r * r <= n; ++r)
    if (n % r == 0 && n / r <= 20 && lane::reg_ok(r) && lane::reg_ok(n / r)) r2 = r;
  return Fac{n / r2, r2};
}
// inputs j + q R2 of some item j lie within the sphere
// (the factors are template constants: evaluated in the kernels they cost
// ten times the transform)
template <int N> struct Keep {
  static constexpr int r1 = fac(N).r1, r2 = fac(N).r2, pw = prune_width(N);
  template <bool ALL = false> __host__ __device__ static constexpr bool q(int i) {
    return ALL || i * r2 <= pw || i * r2 + r2 - 1 >= N - pw;
  }
  template <bool ALL> static constexpr unsigned mask() {
    unsigned m = 0;
    for (int i = 0; i < r1; ++i) m |= (q<ALL>(i) ? 1u : 0u) << i;
    return m;
  }
};

// Lines per CTA: 16 (eight neighbouring FP64 lines already fill 128-byte
// segments), fewer where 16 lines would not fit in 48 KB of shared memory.
template <typename T, int N> __host__ __device__ constexpr int lines() {
  const int per = 2 * (int)sizeof(T) * (N + 2 * fac(N).r1 + 2);
  return 16 * per + 2 * (int)sizeof(T) * N <= 48 * 1024 ? 16 : 8;
}
// Of V(r) in FP32, two floats a point, xv holds in shared memory both (unless its
// first DFT is of 14 points), or the second, or the second of the later points:
// what fits in 48 KB.  lows: the second floats of a thread in registers.
template <int N> __host__ __device__ constexpr bool v_shared() {
  return fac(N).r1 != 14 && lines<float, N>() * (8 + 8) * N + 8 * N <= 48 * 1024;
}
template <int N> __host__ __device__ constexpr int v_lows() {
  return lines<float, N>() * (8 + 4) * N + 8 * N <= 48 * 1024 ? 0 : fac(N).r2 / 2;
}

// CTAs per SM that the register file should hold.  The R1-point DFT sets what
// a thread needs: with 14 points and more the y and x kernels want 72 registers
// in FP32 and 128 in FP64, shorter ones 56 and 96; the z kernels, which wait on
// their gathers, run faster with more CTAs (140 points, 512 band pairs, FP64:
// zb 2.2 -> 1.6 ms at 96 registers, yb 3.2 -> 3.6 ms).
enum Kind { KZ, KXY, KXV };
template <typename T, int N, int KIND> __host__ __device__ constexpr int min_ctas() {
  const int threads = lines<T, N>() * fac(N).r1;
  const bool lng = fac(N).r1 >= 14;
  const int want = sizeof(T) == 4 ? (KIND != KZ && lng ? 72 : 56)
                                  : (KIND == KXV || (KIND == KXY && lng) ? 128 : 96);
  const int b = 65536 / (((threads + 31) / 32) * 32 * want);
  return b < 1 ? 1 : b > 8 ? 8 : b;
}

enum Op { ZB, ZF, ZBK, ZFK, YB, YF, XD, XV, GZB, GZF, GYB, GYF, GXR, GXG };

struct Args {
  DeviceSticks g;
  const double2* tw[3];          // exp(+2 pi i k/n) of the x, y, z lengths
  int op = 0;
  const double2* c = nullptr;    // coefficients, band-major, ngw per band
  double2* hc = nullptr;
  const double* g2 = nullptr;
  double scale = 0;
  int ngw = 0, nst = 0, first = 0;   // first: band pair (or band) of slot 0
  void* sticks = nullptr;
  void* tile = nullptr;
  int nslots = 0;
  int chunks = 1;                // CTAs that share the slots of one set of lines
  const void* v = nullptr;       // V(r), [x][y][z]; FP32 passes: float2, the value rounded
                                 // to FP32 and the rest
  double* rho = nullptr;         // density, [x][y][z]
  const double* w = nullptr;     // weights, two per slot (band n at w[n])
  int nw = 0;                    // weights in all; beyond: zero
  double wout = 1;               // the sums are added to rho times this
  bool rho_set = false;          // store the density instead of adding (chunks == 1)
  // real fields on a whole grid (the density basis, G* passes): two coefficient
  // arrays and two fields per slot, the second of each may be null
  double2* gc[4] = {nullptr, nullptr, nullptr, nullptr};
  double* gf[4] = {nullptr, nullptr, nullptr, nullptr};
  const double* fadd = nullptr;  // GXR: field 0 = Re + fadd; GXG: the fields times fmul
  const double* fmul = nullptr;
  bool chain = false;            // GXR: field 1 = Im + the new field 0
  cudaStream_t stream = nullptr;
};

// the twiddles W_N^{jk} as [k][j]: a thread's j or k is fixed, so every twiddle
// it reads lies at a constant offset from its first (with the x passes' column
// offsets kept as products: xv at 140^3 FP32 4.06 -> 3.57 ms, FP64 8.5 -> 7.5)
template <typename C, int N>
__device__ __forceinline__ void load_tw(C* tw, const double2* src) {
  constexpr int R2 = fac(N).r2;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const double2 w = __ldg(src + (i / R2) * (i % R2));
    tw[i] = cmk<C>(w.x, w.y);
  }
}

// first half of a transform: R1-point DFT of item j and its twiddles, into
// shared memory at [k][j] (strides sk, sj)
template <int N, int DIR, bool ALL = false, typename C>
__device__ __forceinline__ void first_half(C (&v)[fac(N).r1], int j, const C* tw, C* s, int sk) {
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2;
  constexpr unsigned MASK = Keep<N>::template mask<ALL>();
  lane::dft_reg_in<R1, DIR, MASK>(v);
  s[0] = v[0];
  tw += j;
#pragma unroll
  for (int k = 1; k < R1; ++k) {
    const C w = tw[k * R2];
    s[k * sk] = DIR > 0 ? cmul(v[k], w) : cmulc(v[k], w);
  }
}

// the opposite order: R2-point DFT of item k, twiddled, into [k][j]
template <int N, int DIR, typename C>
__device__ __forceinline__ void first_half_rev(C (&u)[fac(N).r2], int k, const C* tw, C* s, int sj) {
  constexpr int R2 = fac(N).r2;
  lane::dft_reg<R2, DIR>(u);
  s[0] = u[0];
  tw += k * R2;
#pragma unroll
  for (int j = 1; j < R2; ++j) {
    const C w = tw[j];
    s[j * sj] = DIR > 0 ? cmul(u[j], w) : cmulc(u[j], w);
  }
}

// ------------------------------------------------------------------ z sticks
// Shared layout of the z kernels: [line][k][j], rows of an odd pitch.
template <int N> struct ZS {
  static constexpr int R1 = fac(N).r1, R2 = fac(N).r2;
  static constexpr int PJ = R2 | 1;
  static constexpr int LINE = R1 * PJ | 1;
};

// Coefficients to sticks.  One CTA takes kLines sticks of a slot; K: one
// complex band per slot and one stick per rod, else two real bands and the
// +G and -G sticks of each rod (stick 0 holds both halves of rod 0).  G: one
// or two real fields on the density sphere, which fills the whole line.
template <typename T, int N, bool K, bool G = false>
__global__ void __launch_bounds__((lines<T, N>()) * fac(N).r1, (min_ctas<T, N, KZ>()))
zb(Args a) {
  using C = typename CT<T>::c;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<T, N>();
  __shared__ C tw[N];
  __shared__ C sm[kLines * ZS<N>::LINE];
  const DeviceSticks& g = a.g;
  const int s0 = blockIdx.x * kLines;
  const int slot = blockIdx.y;
  const int b1 = K ? a.first + slot : 2 * (a.first + slot);
  const double2* c1 = G ? a.gc[2 * slot] : a.c + (size_t)b1 * a.ngw;
  const double2* c2 = G ? a.gc[2 * slot + 1] : (!K && b1 + 1 < a.nst) ? c1 + a.ngw : nullptr;
  {
    const int j = threadIdx.x % R2, line = threadIdx.x / R2, s = s0 + line;
    const bool on = line < kLines && s < g.nvec;
    C v[R1];
    if (on) {
      const int r = K ? s : (s + 1) >> 1;
      const int lmin = g.rod_lmin[r], size = g.rod_size[r], first = g.rod_first[r];
      const bool mstick = !K && s > 0 && (s & 1) == 0;
#pragma unroll
      for (int q = 0; q < R1; ++q) {
        v[q] = cmk<C>(0, 0);
        if (Keep<N>::template q<G>(q)) {
          const int z = j + q * R2;
          const int lz = z < (N + 1) / 2 ? z : z - N;
          const bool minus = mstick || (!K && s == 0 && lz <= 0);
          const int i = (minus ? -lz : lz) - lmin;
          if (i >= 0 && i < size) {
            const double2 p = c1[first + i];
            if (K) {
              v[q] = cmk<C>(p.x, p.y);
            } else {
              const double2 d = c2 ? c2[first + i] : make_double2(0.0, 0.0);
              // +G: c1 + i c2 ; -G: conj(c1) + i conj(c2)
              v[q] = minus ? cmk<C>(p.x + d.y, d.x - p.y) : cmk<C>(p.x - d.y, p.y + d.x);
            }
          }
        }
      }
    }
    load_tw<C, N>(tw, a.tw[2]);        // while the coefficients arrive
    __syncthreads();
    if (on) first_half<N, +1, G>(v, j, tw, sm + line * ZS<N>::LINE + j, ZS<N>::PJ);
  }
  __syncthreads();
  const int k = threadIdx.x % R1, line = threadIdx.x / R1, s = s0 + line;
  if (line < kLines && s < g.nvec) {
    const C* row = sm + line * ZS<N>::LINE + k * ZS<N>::PJ;
    C u[R2];
#pragma unroll
    for (int j = 0; j < R2; ++j) u[j] = row[j];
    lane::dft_reg<R2, +1>(u);
    C* out = (C*)a.sticks + ((size_t)slot * g.nvec + s) * N + k;
#pragma unroll
    for (int m = 0; m < R2; ++m) out[m * R1] = u[m];
  }
}

// Sticks to coefficients: hc = 1/2 g2 c + Z(G) scale, the two bands of a
// slot unpacked at Gamma (G: no kinetic term).  One CTA takes the sticks of kLines/2 rods (K:
// kLines rods).
template <typename T, int N, bool K, bool G = false>
__global__ void __launch_bounds__((lines<T, N>()) * fac(N).r1, (min_ctas<T, N, KZ>()))
zf(Args a) {
  using C = typename CT<T>::c;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<T, N>();
  constexpr int RODS = K ? kLines : kLines / 2;
  __shared__ C tw[N];
  __shared__ C sm[kLines * ZS<N>::LINE];
  const DeviceSticks& g = a.g;
  const int r0 = blockIdx.x * RODS, r1 = min(g.nrods, r0 + RODS);
  const int s0 = K ? r0 : (r0 == 0 ? 0 : 2 * r0 - 1);
  const int nl = (K ? r1 : 2 * r1 - 1) - s0;
  const int slot = blockIdx.y;
  {
    const int k = threadIdx.x % R1, line = threadIdx.x / R1;
    C u[R2];
    if (line < nl) {
      const C* in = (const C*)a.sticks + ((size_t)slot * g.nvec + s0 + line) * N + k;
#pragma unroll
      for (int m = 0; m < R2; ++m) u[m] = in[m * R1];
    }
    load_tw<C, N>(tw, a.tw[2]);        // while the sticks arrive
    __syncthreads();
    if (line < nl)
      first_half_rev<N, -1>(u, k, tw, sm + line * ZS<N>::LINE + k * ZS<N>::PJ, 1);
  }
  __syncthreads();
  {
    const int j = threadIdx.x % R2, line = threadIdx.x / R2;
    C v[R1];
    if (line < nl) {
      const C* col = sm + line * ZS<N>::LINE + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) v[k] = col[k * ZS<N>::PJ];
      lane::dft_reg<R1, -1>(v);
    }
    __syncthreads();
    if (line < nl) {
      C* row = sm + line * ZS<N>::LINE + j;
#pragma unroll
      for (int q = 0; q < R1; ++q)
        if (Keep<N>::template q<G>(q)) row[q * R2] = v[q];
    }
  }
  __syncthreads();
  const int ig0 = g.rod_first[r0];
  const int ig1 = g.rod_first[r1 - 1] + g.rod_size[r1 - 1];
  const int b1 = K ? a.first + slot : 2 * (a.first + slot);
  const bool two = !K && b1 + 1 < a.nst;
  for (int ig = ig0 + threadIdx.x; ig < ig1; ig += blockDim.x) {
    int r = r0;
    while (r + 1 < r1 && g.rod_first[r + 1] <= ig) ++r;
    const int l = g.rod_lmin[r] + (ig - g.rod_first[r]);
    const int zp = l < 0 ? l + N : l;
    const double kin = G ? 0.0 : 0.5 * a.g2[ig];
    const size_t i1 = (size_t)b1 * a.ngw + ig;
    const double2 x = G ? make_double2(0.0, 0.0) : a.c[i1];
    if (K) {
      const C p = sm[(r - r0) * ZS<N>::LINE + zp];
      a.hc[i1] = make_double2(kin * x.x + p.x * a.scale, kin * x.y + p.y * a.scale);
    } else {
      const int zm = l > 0 ? N - l : -l;
      const int sp = (r == 0) ? 0 : 2 * r - 1 - s0;
      const int sn = (r == 0) ? 0 : 2 * r - s0;
      const C P = sm[sp * ZS<N>::LINE + zp];
      const C M = sm[sn * ZS<N>::LINE + zm];
      // c1 = (Z(G) + conj Z(-G))/2, c2 = -i (Z(G) - conj Z(-G))/2
      const double px = P.x, py = P.y, mx = M.x, my = M.y;
      const double2 u = make_double2(0.5 * (px + mx) * a.scale, 0.5 * (py - my) * a.scale);
      const double2 w = make_double2(0.5 * (py + my) * a.scale, 0.5 * (mx - px) * a.scale);
      if (G) {
        a.gc[2 * slot][ig] = u;
        if (a.gc[2 * slot + 1]) a.gc[2 * slot + 1][ig] = w;
      } else {
        a.hc[i1] = make_double2(kin * x.x + u.x, kin * x.y + u.y);
        if (two) {
          const size_t i2 = i1 + a.ngw;
          const double2 y = a.c[i2];
          a.hc[i2] = make_double2(kin * y.x + w.x, kin * y.y + w.y);
        }
      }
    }
  }
}

// -------------------------------------------------------------- y columns
// Lines (column, z) flattened; the sticks of a column through the column map.
template <typename T, int N, bool G = false>
__global__ void __launch_bounds__((lines<T, N>()) * fac(N).r1, (min_ctas<T, N, KXY>()))
yb(Args a) {
  using C = typename CT<T>::c;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<T, N>();
  __shared__ C tw[N];
  __shared__ C sm[N * kLines];
  const DeviceSticks& g = a.g;
  const int lane = threadIdx.x % kLines, item = threadIdx.x / kLines;
  const int line = blockIdx.x * kLines + lane;
  const bool on = line < g.ncol * g.n2;
  const int col = on ? line / g.n2 : 0, z = line - col * g.n2;
  load_tw<C, N>(tw, a.tw[1]);
  int off[R1];
  if (item < R2 && on) {
#pragma unroll
    for (int q = 0; q < R1; ++q)
      if (Keep<N>::template q<G>(q)) {
        const int s = g.colmap[col * N + item + q * R2];
        off[q] = s < 0 ? -1 : s * g.n2 + z;
      }
  }
  const size_t zs = (size_t)g.nvec * g.n2, ts = (size_t)g.ncol * N * g.n2;
  const int per = (a.nslots + gridDim.y - 1) / gridDim.y;
  const int e = min(a.nslots, (int)(blockIdx.y + 1) * per);
  const bool load = item < R2 && on;
  C v[R1];
  auto fetch = [&](int slot) {
    const C* in = (const C*)a.sticks + slot * zs;
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      v[q] = cmk<C>(0, 0);
      if (Keep<N>::template q<G>(q) && off[q] >= 0) v[q] = in[off[q]];
    }
  };
  int slot = blockIdx.y * per;
  if (load && slot < e) fetch(slot);
  for (; slot < e; ++slot) {
    __syncthreads();
    if (load) {
      first_half<N, +1, G>(v, item, tw, sm + item * kLines + lane, R2 * kLines);
      if (slot + 1 < e) fetch(slot + 1);   // in flight over the second half
    }
    __syncthreads();
    if (on) {
      C u[R2];
#pragma unroll
      for (int j = 0; j < R2; ++j) u[j] = sm[(item * R2 + j) * kLines + lane];
      lane::dft_reg<R2, +1>(u);
      C* out = (C*)a.tile + slot * ts + ((size_t)col * N + item) * g.n2 + z;
#pragma unroll
      for (int m = 0; m < R2; ++m) out[(size_t)m * R1 * g.n2] = u[m];
    }
  }
}

template <typename T, int N, bool G = false>
__global__ void __launch_bounds__((lines<T, N>()) * fac(N).r1, (min_ctas<T, N, KXY>()))
yf(Args a) {
  using C = typename CT<T>::c;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<T, N>();
  __shared__ C tw[N];
  __shared__ C sm[N * kLines];
  const DeviceSticks& g = a.g;
  const int lane = threadIdx.x % kLines, item = threadIdx.x / kLines;
  const int line = blockIdx.x * kLines + lane;
  const bool on = line < g.ncol * g.n2;
  const int col = on ? line / g.n2 : 0, z = line - col * g.n2;
  load_tw<C, N>(tw, a.tw[1]);
  int off[R1];
  if (item < R2 && on) {
#pragma unroll
    for (int q = 0; q < R1; ++q)
      if (Keep<N>::template q<G>(q)) {
        const int s = g.colmap[col * N + item + q * R2];
        off[q] = s < 0 ? -1 : s * g.n2 + z;
      }
  }
  const size_t zs = (size_t)g.nvec * g.n2, ts = (size_t)g.ncol * N * g.n2;
  const int per = (a.nslots + gridDim.y - 1) / gridDim.y;
  const int e = min(a.nslots, (int)(blockIdx.y + 1) * per);
  C u[R2];
  auto fetch = [&](int slot) {
    const C* in = (const C*)a.tile + slot * ts + ((size_t)col * N + item) * g.n2 + z;
#pragma unroll
    for (int m = 0; m < R2; ++m) u[m] = in[(size_t)m * R1 * g.n2];
  };
  int slot = blockIdx.y * per;
  if (on && slot < e) fetch(slot);
  for (; slot < e; ++slot) {
    __syncthreads();
    if (on) {
      first_half_rev<N, -1>(u, item, tw, sm + item * R2 * kLines + lane, kLines);
      if (slot + 1 < e) fetch(slot + 1);   // in flight over the second half
    }
    __syncthreads();
    if (item < R2 && on) {
      C v[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) v[k] = sm[(k * R2 + item) * kLines + lane];
      lane::dft_reg<R1, -1>(v);
      C* out = (C*)a.sticks + slot * zs;
#pragma unroll
      for (int q = 0; q < R1; ++q)
        if (Keep<N>::template q<G>(q) && off[q] >= 0) out[off[q]] = v[q];
    }
  }
}

// ----------------------------------------------------------------- x rows
// Lines (y, z) flattened, from the occupied columns of the tile.  A CTA keeps
// its lines over all slots of its chunk, so the density of a point stays in
// a register until the chunk ends, and V(r) is read once.  The next slot's
// loads are in flight over the second half.  The density's weights, products and
// sums are FP64 in both precisions; with FP32 ones and these xd<float> takes (us) 72
// and 73 at 84^3 (64 band pairs), 478 and 511 at 112^3 (216), 2140 and 2150 at 140^3
// (512).
template <int N>
__device__ __forceinline__ void x_columns(const DeviceSticks& g, int item, int nl,
                                          int (&off)[fac(N).r1]) {
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2;
#pragma unroll
  for (int q = 0; q < R1; ++q)
    if (Keep<N>::q(q)) {
      const int col = g.xcol[item + q * R2];
      off[q] = col < 0 ? -1 : col * nl;
    }
}

template <typename T, int N>
__global__ void __launch_bounds__((lines<T, N>()) * fac(N).r1, (min_ctas<T, N, KXY>()))
xd(Args a) {
  using C = typename CT<T>::c;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<T, N>();
  __shared__ C tw[N];
  __shared__ C sm[N * kLines];
  const DeviceSticks& g = a.g;
  const int lane = threadIdx.x % kLines, item = threadIdx.x / kLines;
  const int line = blockIdx.x * kLines + lane;
  const int nl = g.n1 * g.n2;
  const bool on = line < nl;
  load_tw<C, N>(tw, a.tw[0]);
  int off[R1];
  if (item < R2) x_columns<N>(g, item, nl, off);
  double acc[R2];
#pragma unroll
  for (int m = 0; m < R2; ++m) acc[m] = 0;
  const size_t ts = (size_t)g.ncol * nl;
  const int per = (a.nslots + gridDim.y - 1) / gridDim.y;
  const int e = min(a.nslots, (int)(blockIdx.y + 1) * per);
  const bool load = item < R2 && on;
  C v[R1];
  auto fetch = [&](int slot) {
    const C* in = (const C*)a.tile + slot * ts + line;
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      v[q] = cmk<C>(0, 0);
      if (Keep<N>::q(q) && off[q] >= 0) v[q] = in[off[q]];
    }
  };
  int slot = blockIdx.y * per;
  if (load && slot < e) fetch(slot);
  for (; slot < e; ++slot) {
    __syncthreads();
    if (load) {
      first_half<N, +1>(v, item, tw, sm + item * kLines + lane, R2 * kLines);
      if (slot + 1 < e) fetch(slot + 1);   // in flight over the second half
    }
    const int n1 = 2 * (a.first + slot);
    const double w1 = n1 < a.nw ? a.w[n1] : 0.0;
    const double w2 = n1 + 1 < a.nw ? a.w[n1 + 1] : 0.0;
    __syncthreads();
    if (on) {
      C u[R2];
#pragma unroll
      for (int j = 0; j < R2; ++j) u[j] = sm[(item * R2 + j) * kLines + lane];
      lane::dft_reg<R2, +1>(u);
#pragma unroll
      for (int m = 0; m < R2; ++m) {
        const double p = u[m].x, q = u[m].y;
        acc[m] = fma(w1 * p, p, fma(w2 * q, q, acc[m]));
      }
    }
  }
  if (on) {
    double* rho = a.rho + (size_t)item * nl + line;
#pragma unroll
    for (int m = 0; m < R2; ++m) {
      double* p = rho + (size_t)m * R1 * nl;
      const double x = a.wout * acc[m];
      if (gridDim.y > 1) atomicAdd(p, x);
      else *p = a.rho_set ? x : *p + x;
    }
  }
}

// The tile in place: x transform to psi(r), times V(r), transform back.  A
// thread's second-half reads and its writes of the way back are the same
// places in shared memory, and so are its last reads and the next slot's first
// writes: two barriers per slot.
//   FP32: the product with V(r) is that with the FP64 value but for its own
// rounding: V(r) is a float and the rest of it another, both in shared memory, two
// packed instructions where V(r) rounded to FP32 in registers takes two scalar
// ones (us of 64 slots of N x 96 x 96 points, V(r) rounded and whole: 64 82 and 85, 84
// 132 and 132, 96 133 and 134, 128 207 and 214, 144 221 and 214).  With the 14-point
// DFT, and where the room is short, only the rest is there (112 171 -> 185, both in
// shared memory 190; 140 218 -> 236, both 245; 224 337 -> 362; all in registers spills:
// 140 240, 224 380).
//   FP32 also loads the next slot's points before the last half, which hides their
// latency (without and with: 60 112 -> 102, 84 151 -> 140, 96 153 -> 142, 140 248 ->
// 235, 192 335 -> 309, 240 427 -> 404; equal within 2 % at 126 and 144, and 82 -> 87 at
// 56, 153 -> 157 at 90).  In FP64 (7510 -> 7730 us at 140^3, 512 band pairs) the compiler
// spills, and the points are loaded at the start of their slot.
template <typename T, int N>
__global__ void __launch_bounds__((lines<T, N>()) * fac(N).r1, (min_ctas<T, N, KXV>()))
xv(Args a) {
  using C = typename CT<T>::c;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<T, N>();
  constexpr bool kFloat = sizeof(T) == 4, kAhead = kFloat, kBoth = kFloat && v_shared<N>();
  constexpr int kLows = kFloat ? v_lows<N>() : 0, kRest = R2 - kLows;
  __shared__ C tw[N];
  __shared__ C sm[N * kLines];
  // [k][j] as sm; an entry is its thread's own
  __shared__ float2 vall[kBoth ? N * kLines : 1];
  __shared__ float vrest[kFloat && !kBoth ? R1 * kRest * kLines : 1];
  const DeviceSticks& g = a.g;
  const int lane = threadIdx.x % kLines, item = threadIdx.x / kLines;
  const int line = blockIdx.x * kLines + lane;
  const int nl = g.n1 * g.n2;
  const bool on = line < nl, load = item < R2 && on;
  load_tw<C, N>(tw, a.tw[0]);
  int off[R1];
  if (item < R2) x_columns<N>(g, item, nl, off);
  T vr[kBoth ? 1 : R2], vlow[kLows ? kLows : 1];
  if (on) {
    const size_t p = (size_t)item * nl + line;
#pragma unroll
    for (int m = 0; m < R2; ++m) {
      if constexpr (kFloat) {
        const float2 v = ((const float2*)a.v)[p + (size_t)m * R1 * nl];
        if constexpr (kBoth) {
          vall[(item * R2 + m) * kLines + lane] = v;
        } else {
          vr[m] = v.x;
          if (m < kLows) vlow[m < kLows ? m : 0] = v.y;
          else vrest[(item * kRest + m - kLows) * kLines + lane] = v.y;
        }
      } else {
        vr[m] = ((const double*)a.v)[p + (size_t)m * R1 * nl];
      }
    }
  }
  const size_t ts = (size_t)g.ncol * nl;
  const int per = (a.nslots + gridDim.y - 1) / gridDim.y;
  const int e = min(a.nslots, (int)(blockIdx.y + 1) * per);
  C v[R1], next[kAhead ? R1 : 1];
  auto fetch = [&](int slot, C (&x)[R1]) {
    const C* in = (const C*)a.tile + slot * ts + line;
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      x[q] = cmk<C>(0, 0);
      if (Keep<N>::q(q) && off[q] >= 0) x[q] = in[off[q]];
    }
  };
  int slot = blockIdx.y * per;
  if constexpr (kAhead)
    if (load && slot < e) fetch(slot, next);
  __syncthreads();
  for (; slot < e; ++slot) {
    C* tile = (C*)a.tile + slot * ts + line;
    if (load) {
      if constexpr (kAhead) {
#pragma unroll
        for (int q = 0; q < R1; ++q) v[q] = next[q];
      } else {
        fetch(slot, v);
      }
      first_half<N, +1>(v, item, tw, sm + item * kLines + lane, R2 * kLines);
    }
    __syncthreads();
    if (on) {
      C u[R2];
#pragma unroll
      for (int j = 0; j < R2; ++j) u[j] = sm[(item * R2 + j) * kLines + lane];
      lane::dft_reg<R2, +1>(u);
#pragma unroll
      for (int m = 0; m < R2; ++m) {
        if constexpr (kFloat) {
          float2 v;
          if constexpr (kBoth) v = vall[(item * R2 + m) * kLines + lane];
          else v = make_float2(vr[m], m < kLows ? vlow[m < kLows ? m : 0]
                                      : vrest[(item * kRest + m - kLows) * kLines + lane]);
          u[m] = reg::cfma(u[m], v.x, reg::cscale(u[m], v.y));
        } else {
          u[m].x *= vr[m];
          u[m].y *= vr[m];
        }
      }
      first_half_rev<N, -1>(u, item, tw, sm + item * R2 * kLines + lane, kLines);
    }
    if constexpr (kAhead)
      if (load && slot + 1 < e) fetch(slot + 1, next);
    __syncthreads();
    if (load) {
#pragma unroll
      for (int k = 0; k < R1; ++k) v[k] = sm[(k * R2 + item) * kLines + lane];
      lane::dft_reg<R1, -1>(v);
#pragma unroll
      for (int q = 0; q < R1; ++q)
        if (Keep<N>::q(q) && off[q] >= 0) tile[off[q]] = v[q];
    }
  }
}

// One complex transform of real fields on the whole grid per slot: the tile to
// the slot's fields 0 (and 1), or back from them.  The pointwise work next to it
// rides along: field 0 takes fadd (v_xc += ...), field 1 the new field 0 (V =
// V_local + v_xc), the fields to be transformed are multiplied by fmul.
template <int N>
__global__ void __launch_bounds__((lines<double, N>()) * fac(N).r1, (min_ctas<double, N, KXY>()))
xr(Args a) {
  using C = double2;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<double, N>();
  __shared__ C tw[N];
  __shared__ C sm[N * kLines];
  const DeviceSticks& g = a.g;
  const int lane = threadIdx.x % kLines, item = threadIdx.x / kLines;
  const int line = blockIdx.x * kLines + lane;
  const int nl = g.n1 * g.n2;
  const bool on = line < nl;
  load_tw<C, N>(tw, a.tw[0]);
  C v[R1];
  if (item < R2 && on) {
    const C* in = (const C*)a.tile + (size_t)blockIdx.y * g.ncol * nl + line;
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      const int col = g.xcol[item + q * R2];
      v[q] = col >= 0 ? in[(size_t)col * nl] : make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  if (item < R2 && on) first_half<N, +1, true>(v, item, tw, sm + item * kLines + lane, R2 * kLines);
  __syncthreads();
  if (!on) return;
  C u[R2];
#pragma unroll
  for (int j = 0; j < R2; ++j) u[j] = sm[(item * R2 + j) * kLines + lane];
  lane::dft_reg<R2, +1>(u);
  double *f0 = a.gf[2 * blockIdx.y], *f1 = a.gf[2 * blockIdx.y + 1];
#pragma unroll
  for (int m = 0; m < R2; ++m) {
    const size_t p = (size_t)(item + m * R1) * nl + line;
    const double f = a.fadd ? u[m].x + a.fadd[p] : u[m].x;
    f0[p] = f;
    if (f1) f1[p] = a.chain ? u[m].y + f : u[m].y;
  }
}

template <int N>
__global__ void __launch_bounds__((lines<double, N>()) * fac(N).r1, (min_ctas<double, N, KXY>()))
xg(Args a) {
  using C = double2;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<double, N>();
  __shared__ C tw[N];
  __shared__ C sm[N * kLines];
  const DeviceSticks& g = a.g;
  const int lane = threadIdx.x % kLines, item = threadIdx.x / kLines;
  const int line = blockIdx.x * kLines + lane;
  const int nl = g.n1 * g.n2;
  const bool on = line < nl;
  load_tw<C, N>(tw, a.tw[0]);
  C u[R2];
  if (on) {
    const double *f0 = a.gf[2 * blockIdx.y], *f1 = a.gf[2 * blockIdx.y + 1];
#pragma unroll
    for (int m = 0; m < R2; ++m) {
      const size_t p = (size_t)(item + m * R1) * nl + line;
      const double w = a.fmul ? a.fmul[p] : 1.0;
      u[m] = make_double2(f0[p] * w, f1 ? f1[p] * w : 0.0);
    }
  }
  __syncthreads();
  if (on) first_half_rev<N, -1>(u, item, tw, sm + item * R2 * kLines + lane, kLines);
  __syncthreads();
  if (item < R2 && on) {
    C v[R1];
#pragma unroll
    for (int k = 0; k < R1; ++k) v[k] = sm[(k * R2 + item) * kLines + lane];
    lane::dft_reg<R1, -1>(v);
    C* out = (C*)a.tile + (size_t)blockIdx.y * g.ncol * nl + line;
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      const int col = g.xcol[item + q * R2];
      if (col >= 0) out[(size_t)col * nl] = v[q];
    }
  }
}

// -------------------------------------------------- lines of a whole grid
// In place, FP64, every line along one axis of an x-fastest grid.  Along y and
// z the neighbouring lines are neighbours in memory (inner of them, then the
// next N inner elements), as in the passes above; along x (gc) the line itself
// is contiguous and is exchanged as a z stick.
template <int N, int DIR>
__global__ void __launch_bounds__((lines<double, N>()) * fac(N).r1, (min_ctas<double, N, KXY>()))
gs(double2* __restrict__ grid, const double2* __restrict__ tw_g, int inner, int nlines) {
  using C = double2;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<double, N>();
  __shared__ C tw[N];
  __shared__ C sm[N * kLines];
  const int lane = threadIdx.x % kLines, item = threadIdx.x / kLines;
  const int line = blockIdx.x * kLines + lane;
  const bool on = line < nlines;
  const int o = on ? line / inner : 0;
  C* base = grid + (size_t)o * inner * N + (line - o * inner);
  load_tw<C, N>(tw, tw_g);
  C v[R1];
  if (item < R2 && on) {
#pragma unroll
    for (int q = 0; q < R1; ++q) v[q] = base[(size_t)(item + q * R2) * inner];
  }
  __syncthreads();
  if (item < R2 && on)
    first_half<N, DIR, true>(v, item, tw, sm + item * kLines + lane, R2 * kLines);
  __syncthreads();
  if (on) {
    C u[R2];
#pragma unroll
    for (int j = 0; j < R2; ++j) u[j] = sm[(item * R2 + j) * kLines + lane];
    lane::dft_reg<R2, DIR>(u);
#pragma unroll
    for (int m = 0; m < R2; ++m) base[(size_t)(item + m * R1) * inner] = u[m];
  }
}

template <int N, int DIR>
__global__ void __launch_bounds__((lines<double, N>()) * fac(N).r1, (min_ctas<double, N, KZ>()))
gc(double2* __restrict__ grid, const double2* __restrict__ tw_g, int nlines) {
  using C = double2;
  constexpr int R1 = fac(N).r1, R2 = fac(N).r2, kLines = lines<double, N>();
  __shared__ C tw[N];
  __shared__ C sm[kLines * ZS<N>::LINE];
  const int l0 = blockIdx.x * kLines;
  load_tw<C, N>(tw, tw_g);
  C v[R1];
  const int j = threadIdx.x % R2, lj = threadIdx.x / R2;
  const bool on = lj < kLines && l0 + lj < nlines;
  if (on) {
    const C* in = grid + (size_t)(l0 + lj) * N + j;
#pragma unroll
    for (int q = 0; q < R1; ++q) v[q] = in[q * R2];
  }
  __syncthreads();
  if (on) first_half<N, DIR, true>(v, j, tw, sm + lj * ZS<N>::LINE + j, ZS<N>::PJ);
  __syncthreads();
  const int k = threadIdx.x % R1, line = threadIdx.x / R1;
  if (line < kLines && l0 + line < nlines) {
    const C* row = sm + line * ZS<N>::LINE + k * ZS<N>::PJ;
    C u[R2];
#pragma unroll
    for (int i = 0; i < R2; ++i) u[i] = row[i];
    lane::dft_reg<R2, DIR>(u);
    C* out = grid + (size_t)(l0 + line) * N + k;
#pragma unroll
    for (int m = 0; m < R2; ++m) out[m * R1] = u[m];
  }
}

// ---------------------------------------------------------------- launches
template <int N>
void run_grid(Context& ctx, double2* grid, const double2* tw, int inner, int nlines, int dir) {
  constexpr int kLines = lines<double, N>();
  const int nb = (nlines + kLines - 1) / kLines, th = kLines * fac(N).r1;
  cudaStream_t st = ctx.stream;
  if (inner > 1) {
    if (dir > 0) gs<N, +1><<<nb, th, 0, st>>>(grid, tw, inner, nlines);
    else gs<N, -1><<<nb, th, 0, st>>>(grid, tw, inner, nlines);
  } else {
    if (dir > 0) gc<N, +1><<<nb, th, 0, st>>>(grid, tw, nlines);
    else gc<N, -1><<<nb, th, 0, st>>>(grid, tw, nlines);
  }
  QBX_LAUNCHED(ctx);
}

template <typename T, int N>
void run(Context& ctx, const Args& a) {
  constexpr int R1 = fac(N).r1, kLines = lines<T, N>();
  static_assert(R1 <= 20 && fac(N).r2 > 1, "no factorisation into two register DFTs");
  const DeviceSticks& g = a.g;
  const int th = kLines * R1;
  auto cdiv = [](int x, int y) { return (x + y - 1) / y; };
  const dim3 gy(cdiv(g.ncol * g.n2, kLines), a.chunks), gx(cdiv(g.n1 * g.n2, kLines), a.chunks);
  cudaStream_t st = a.stream;
  switch (a.op) {
    case ZB: zb<T, N, false><<<dim3(cdiv(g.nvec, kLines), a.nslots), th, 0, st>>>(a); break;
    case ZF: zf<T, N, false><<<dim3(cdiv(g.nrods, kLines / 2), a.nslots), th, 0, st>>>(a); break;
    case YB: yb<T, N><<<gy, th, 0, st>>>(a); break;
    case YF: yf<T, N><<<gy, th, 0, st>>>(a); break;
    case XD: xd<T, N><<<gx, th, 0, st>>>(a); break;
    case XV: xv<T, N><<<gx, th, 0, st>>>(a); break;
    default:
      if constexpr (sizeof(T) == 8) {
        const dim3 gzb(cdiv(g.nvec, kLines), a.nslots);
        if (a.op == ZBK) zb<T, N, true><<<gzb, th, 0, st>>>(a);
        else if (a.op == ZFK) zf<T, N, true><<<dim3(cdiv(g.nrods, kLines), a.nslots), th, 0, st>>>(a);
        else if (a.op == GZB) zb<T, N, false, true><<<gzb, th, 0, st>>>(a);
        else if (a.op == GZF) zf<T, N, false, true><<<dim3(cdiv(g.nrods, kLines / 2), a.nslots), th, 0, st>>>(a);
        else if (a.op == GYB) yb<T, N, true><<<gy, th, 0, st>>>(a);
        else if (a.op == GYF) yf<T, N, true><<<gy, th, 0, st>>>(a);
        else if (a.op == GXR) xr<N><<<gx, th, 0, st>>>(a);
        else xg<N><<<gx, th, 0, st>>>(a);
      }
  }
  QBX_LAUNCHED(ctx);
}

}  // namespace pen

// One pass over lines of length n in the context type T, and the transform
// of nlines lines of a whole FP64 grid (inner neighbouring lines contiguous;
// inner = 1: the lines themselves are); false when no kernel of that length
// is compiled.  Each fft_pencil_*.cu holds some lengths.
#define QBX_PENCIL_DECLARE(I)                                                        \
  template <typename T> bool pencil_##I(Context& ctx, int n, const pen::Args& a);    \
  bool pencil_grid_##I(Context& ctx, int n, double2* grid, const double2* tw, int inner, \
                       int nlines, int dir);
QBX_PENCIL_DECLARE(0)
QBX_PENCIL_DECLARE(1)
QBX_PENCIL_DECLARE(2)
QBX_PENCIL_DECLARE(3)
QBX_PENCIL_DECLARE(4)
QBX_PENCIL_DECLARE(5)
QBX_PENCIL_DECLARE(6)
QBX_PENCIL_DECLARE(7)
#undef QBX_PENCIL_DECLARE

// Mean of |X|^2/(N |x|^2) over the kept points x of a length-n transform whose
// roots are rounded to FP32 (its arithmetic aside): one plus some 1e-8.  The
// transform is otherwise unbiased, so a density or an H psi divided by the
// gains of its three axes carries no systematic charge or energy error.
double pencil_gain_fp32(int n);

// The lengths an FFT grid can have from 16 to 256: even 2^a 3^{0..2} 5^{0,1}
// 7^{0,1} 11^{0,1}.
inline bool pencil_length(int n) {
  for (int x : {16, 18, 20, 22, 24, 28, 30, 32, 36, 40, 42, 44, 48, 56, 60, 64, 66, 70, 72, 80,
                84, 88, 90, 96, 110, 112, 120, 126, 128, 132, 140, 144, 154, 160, 168, 176, 180,
                192, 198, 210, 220, 224, 240, 252, 256})
    if (n == x) return true;
  return false;
}

}  // namespace qbx

// The functions of one fft_pencil_*.cu: LENGTHS(X) lists X(n) for its lengths.
#define QBX_PENCIL_CASE(N) \
  case N: pen::run<T, N>(ctx, a); return true;
#define QBX_PENCIL_GRID_CASE(N) \
  case N: pen::run_grid<N>(ctx, grid, tw, inner, nlines, dir); return true;
#define QBX_PENCIL_FUNCTIONS(I, LENGTHS)                                                  \
  namespace qbx {                                                                         \
  template <typename T> bool pencil_##I(Context& ctx, int n, const pen::Args& a) {        \
    switch (n) { LENGTHS(QBX_PENCIL_CASE) }                                               \
    return false;                                                                         \
  }                                                                                       \
  template bool pencil_##I<float>(Context&, int, const pen::Args&);                       \
  template bool pencil_##I<double>(Context&, int, const pen::Args&);                      \
  bool pencil_grid_##I(Context& ctx, int n, double2* grid, const double2* tw, int inner,  \
                       int nlines, int dir) {                                             \
    switch (n) { LENGTHS(QBX_PENCIL_GRID_CASE) }                                          \
    return false;                                                                         \
  }                                                                                       \
  }
