// Staged 3-D FFTs of the electronic step on sm_100a.
//
// Wavefunction transforms (the hot path) never build the full 3-D grid in HBM.  A
// band pair psi_1 + i psi_2 (the reference's two-real-functions packing,
// src/BasisMapping.cpp:667-750), or a band at a k point, goes through z sticks,
// y columns and x rows; the density sum and the product with V(r) happen in the
// x pass.  The kernels are the line passes of fft_pencil.cuh; this file holds their
// launches (pencil_pass), the density-basis transforms on the same kernels
// (field_passes), and the runtime-radix kernels for what those do not take:
//
//   k_zfft_bwd, k_xy, k_zfft_fwd : one CTA per z plane, mixed-radix (2, 3, 4, 5, 7,
//                11) self-sorting Stockham passes over shared memory with a twiddle
//                table exp(+2 pi i k/n) built in FP64: grids with a length below 16 or
//                above 256, spheres wider than prune_width (some k points), a slot
//                larger than the stick buffer, QBX_FAST_FFT=0, qbx_density_static
//   k_line_fft : the lines of a whole grid, the same passes
#include <algorithm>
#include <complex>
#include <cstdio>
#include <type_traits>
#include <vector>

#include "fft_pencil.cuh"
#include "qbx_internal.h"

namespace qbx {

template <typename T> struct Cplx;
template <> struct Cplx<float> { using t = float2; };
template <> struct Cplx<double> { using t = double2; };

template <typename C> __device__ __forceinline__ C mk(double x, double y) {
  C r; r.x = x; r.y = y; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) {
  C r; r.x = a.x + b.x; r.y = a.y + b.y; return r;
}
template <typename C> __device__ __forceinline__ C csub(C a, C b) {
  C r; r.x = a.x - b.x; r.y = a.y - b.y; return r;
}
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
// multiply by DIR * i
template <int DIR, typename C> __device__ __forceinline__ C muli(C a) {
  C r;
  if (DIR > 0) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; }
  return r;
}
template <int DIR, typename C> __device__ __forceinline__ C twid(const C* tw, int k) {
  C w = tw[k];
  if (DIR < 0) w.y = -w.y;
  return w;
}

// R-point DFT, out[k] = sum_q v[q] exp(DIR 2 pi i q k / R); roots from the
// length-n table at stride n/R.
template <int R, int DIR, typename C>
__device__ __forceinline__ void small_dft(C* v, const C* tw, int rs) {
  if (R == 2) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if (R == 4) {
    const C a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
    const C c = cadd(v[1], v[3]), d = muli<DIR>(csub(v[1], v[3]));
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = cadd(b, d);
    v[3] = csub(b, d);
  } else {
    C out[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      C acc = v[0];
#pragma unroll
      for (int q = 1; q < R; ++q) acc = cadd(acc, cmul(v[q], twid<DIR>(tw, ((q * k) % R) * rs)));
      out[k] = acc;
    }
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = out[k];
  }
}

// One Stockham pass over nlines contiguous lines of length n (line stride ls).
template <int R, int DIR, typename C>
__device__ __forceinline__ void stockham_pass(const C* __restrict__ src, C* __restrict__ dst,
                                              int n, int nlines, int ls, int Ns, const C* tw) {
  const int nb = n / R;
  const int total = nlines * nb;
  const int tws = n / (Ns * R);
  const int rs = n / R;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int line = t / nb;
    const int i = t - line * nb;
    const C* s = src + line * ls;
    C* d = dst + line * ls;
    const int j = i % Ns;
    C v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = s[i + q * nb];
    if (Ns > 1) {
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = cmul(v[q], twid<DIR>(tw, q * j * tws));
    }
    small_dft<R, DIR>(v, tw, rs);
    const int base = (i / Ns) * Ns * R + j;
#pragma unroll
    for (int q = 0; q < R; ++q) d[base + q * Ns] = v[q];
  }
}

// FFT of nlines lines held in a (ping) with b as the pong buffer; every
// thread of the CTA participates.  Returns the buffer holding the result.
template <int DIR, typename C>
__device__ C* fft_lines(C* a, C* b, int nlines, int ls, const RadixPlan& p, const C* tw) {
  int Ns = 1;
  for (int s = 0; s < p.nstage; ++s) {
    const int r = p.radix[s];
    switch (r) {
      case 2: stockham_pass<2, DIR>(a, b, p.n, nlines, ls, Ns, tw); break;
      case 3: stockham_pass<3, DIR>(a, b, p.n, nlines, ls, Ns, tw); break;
      case 4: stockham_pass<4, DIR>(a, b, p.n, nlines, ls, Ns, tw); break;
      case 5: stockham_pass<5, DIR>(a, b, p.n, nlines, ls, Ns, tw); break;
      case 7: stockham_pass<7, DIR>(a, b, p.n, nlines, ls, Ns, tw); break;
      default: stockham_pass<11, DIR>(a, b, p.n, nlines, ls, Ns, tw); break;
    }
    __syncthreads();
    C* t = a; a = b; b = t;
    Ns *= r;
  }
  return a;
}

template <typename C>
__device__ __forceinline__ void load_twiddles(C* dst, const double2* src, int n) {
  for (int k = threadIdx.x; k < n; k += blockDim.x) dst[k] = mk<C>(src[k].x, src[k].y);
}

// --------------------------------------------------------- z backward
// zbuf layout: [pair][z][stick], stick fastest.
template <typename T>
__global__ void __launch_bounds__(256)
k_zfft_bwd(const double2* __restrict__ c, int ngw, int nst, int pair0,
           DeviceSticks g, const double2* __restrict__ twz,
           typename Cplx<T>::t* __restrict__ zbuf, int rods_per_cta) {
  using C = typename Cplx<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tw = reinterpret_cast<C*>(smem_raw);
  const int n2 = g.n2;
  C* A = tw + n2;
  C* B = A + 2 * rods_per_cta * n2;
  const int r0 = blockIdx.x * rods_per_cta;
  const int r1 = min(g.nrods, r0 + rods_per_cta);
  const int s0 = (r0 == 0) ? 0 : 2 * r0 - 1;
  const int nl = (2 * r1 - 1) - s0;
  const int pl = blockIdx.y;
  const int b1 = 2 * (pair0 + pl);
  const double2* c1 = c + (size_t)b1 * ngw;
  const double2* c2 = (b1 + 1 < nst) ? c + (size_t)(b1 + 1) * ngw : nullptr;
  load_twiddles(tw, twz, n2);
  const int half = (n2 + 1) / 2;
  for (int t = threadIdx.x; t < nl * n2; t += blockDim.x) {
    const int line = t / n2, z = t - line * n2;
    const int s = s0 + line;
    const int r = (s + 1) >> 1;
    const int lz = z < half ? z : z - n2;
    bool minus;
    int l;
    if (r == 0) { minus = (lz <= 0); l = minus ? -lz : lz; }
    else { minus = ((s & 1) == 0); l = minus ? -lz : lz; }
    const int lmin = g.rod_lmin[r];
    double vx = 0.0, vy = 0.0;
    if (l >= lmin && l < lmin + g.rod_size[r]) {
      const int ig = g.rod_first[r] + (l - lmin);
      const double2 p = c1[ig];
      const double2 q = c2 ? c2[ig] : make_double2(0.0, 0.0);
      // +G: c1 + i c2 ; -G: conj(c1) + i conj(c2)
      if (!minus) { vx = p.x - q.y; vy = p.y + q.x; }
      else        { vx = p.x + q.y; vy = q.x - p.y; }
    }
    A[line * n2 + z] = mk<C>(vx, vy);
  }
  __syncthreads();
  C* res = fft_lines<+1>(A, B, nl, n2, g.pz, tw);
  C* out = zbuf + (size_t)pl * n2 * g.nvec;
  for (int t = threadIdx.x; t < nl * n2; t += blockDim.x) {
    const int line = t % nl, z = t / nl;
    out[(size_t)z * g.nvec + s0 + line] = res[line * n2 + z];
  }
}

// --------------------------------------------------------- z forward
template <typename T>
__global__ void __launch_bounds__(256)
k_zfft_fwd(const typename Cplx<T>::t* __restrict__ zbuf, int ngw, int nst, int pair0,
           DeviceSticks g, const double2* __restrict__ twz, double scale,
           const double2* __restrict__ c, const double* __restrict__ g2,
           double2* __restrict__ hc, int rods_per_cta) {
  using C = typename Cplx<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tw = reinterpret_cast<C*>(smem_raw);
  const int n2 = g.n2;
  C* A = tw + n2;
  C* B = A + 2 * rods_per_cta * n2;
  const int r0 = blockIdx.x * rods_per_cta;
  const int r1 = min(g.nrods, r0 + rods_per_cta);
  const int s0 = (r0 == 0) ? 0 : 2 * r0 - 1;
  const int nl = (2 * r1 - 1) - s0;
  const int pl = blockIdx.y;
  const int b1 = 2 * (pair0 + pl);
  const bool two = (b1 + 1 < nst);
  load_twiddles(tw, twz, n2);
  const C* in = zbuf + (size_t)pl * n2 * g.nvec;
  for (int t = threadIdx.x; t < nl * n2; t += blockDim.x) {
    const int line = t % nl, z = t / nl;
    A[line * n2 + z] = in[(size_t)z * g.nvec + s0 + line];
  }
  __syncthreads();
  C* res = fft_lines<-1>(A, B, nl, n2, g.pz, tw);
  const int ig0 = g.rod_first[r0];
  const int ig1 = g.rod_first[r1 - 1] + g.rod_size[r1 - 1];
  for (int ig = ig0 + threadIdx.x; ig < ig1; ig += blockDim.x) {
    int r = r0;
    while (r + 1 < r1 && g.rod_first[r + 1] <= ig) ++r;
    const int l = g.rod_lmin[r] + (ig - g.rod_first[r]);
    const int zp = ((l % n2) + n2) % n2;
    const int zm = ((-l % n2) + n2) % n2;
    const int sp = (r == 0) ? 0 : 2 * r - 1 - s0;
    const int sm = (r == 0) ? 0 : 2 * r - s0;
    const C P = res[sp * n2 + zp];
    const C M = res[sm * n2 + zm];
    // c1 = (Z(G) + conj Z(-G))/2, c2 = -i (Z(G) - conj Z(-G))/2
    const double px = P.x, py = P.y, mx = M.x, my = M.y;
    const double c1x = 0.5 * (px + mx) * scale, c1y = 0.5 * (py - my) * scale;
    const double c2x = 0.5 * (py + my) * scale, c2y = 0.5 * (mx - px) * scale;
    const double kin = 0.5 * g2[ig];
    const size_t i1 = (size_t)b1 * ngw + ig;
    const double2 a = c[i1];
    hc[i1] = make_double2(kin * a.x + c1x, kin * a.y + c1y);
    if (two) {
      const size_t i2 = i1 + ngw;
      const double2 b = c[i2];
      hc[i2] = make_double2(kin * b.x + c2x, kin * b.y + c2y);
    }
  }
}

// ------------------------------------------------------------ xy plane
enum { OP_DENSITY = 0, OP_VPSI = 1 };

template <int DIR, typename C>
__device__ void y_pass(C* P, C* S, int ncol, int n1, int cc, const RadixPlan& py, const C* twy) {
  for (int c0 = 0; c0 < ncol; c0 += cc) {
    const int nc = min(cc, ncol - c0);
    C* blk = P + c0 * n1;
    C* res = fft_lines<DIR>(blk, S, nc, n1, py, twy);
    if (res != blk) {
      for (int t = threadIdx.x; t < nc * n1; t += blockDim.x) blk[t] = res[t];
      __syncthreads();
    }
  }
}

template <typename T, int OP>
__global__ void __launch_bounds__(512)
k_xy(typename Cplx<T>::t* __restrict__ zbuf, int npairs, int pairs_per_cta,
     DeviceSticks g, const double2* __restrict__ twx, const double2* __restrict__ twy,
     const double* __restrict__ v, double* __restrict__ rho,
     const double* __restrict__ w, int pair0, int nst, int cc, int rr) {
  using C = typename Cplx<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n0 = g.n0, n1 = g.n1, ncol = g.ncol, nvec = g.nvec;
  C* tx = reinterpret_cast<C*>(smem_raw);
  C* ty = tx + n0;
  C* P = ty + n1;
  C* S = P + ncol * n1;
  const int z = blockIdx.x;
  load_twiddles(tx, twx, n0);
  load_twiddles(ty, twy, n1);
  const int pbeg = blockIdx.y * pairs_per_cta;
  const int pend = min(npairs, pbeg + pairs_per_cta);
  for (int pl = pbeg; pl < pend; ++pl) {
    C* zp = zbuf + ((size_t)pl * g.n2 + z) * nvec;
    for (int t = threadIdx.x; t < ncol * n1; t += blockDim.x) P[t] = mk<C>(0.0, 0.0);
    __syncthreads();
    for (int s = threadIdx.x; s < nvec; s += blockDim.x)
      P[g.stick_col[s] * n1 + g.stick_y[s]] = zp[s];
    __syncthreads();
    y_pass<+1>(P, S, ncol, n1, cc, g.py, ty);
    double w1 = 0.0, w2 = 0.0;
    if (OP == OP_DENSITY) {
      const int b1 = 2 * (pair0 + pl);
      w1 = w[b1];
      w2 = (b1 + 1 < nst) ? w[b1 + 1] : 0.0;
    }
    for (int y0 = 0; y0 < n1; y0 += rr) {
      const int nr = min(rr, n1 - y0);
      C* R1 = S;
      C* R2 = S + rr * n0;
      for (int t = threadIdx.x; t < nr * n0; t += blockDim.x) R1[t] = mk<C>(0.0, 0.0);
      __syncthreads();
      for (int t = threadIdx.x; t < nr * ncol; t += blockDim.x) {
        const int r = t / ncol, cidx = t - r * ncol;
        R1[r * n0 + g.col_x[cidx]] = P[cidx * n1 + y0 + r];
      }
      __syncthreads();
      C* res = fft_lines<+1>(R1, R2, nr, n0, g.px, tx);
      const size_t rowbase = ((size_t)z * n1 + y0) * n0;
      if (OP == OP_DENSITY) {
        for (int t = threadIdx.x; t < nr * n0; t += blockDim.x) {
          const C val = res[t];
          const double a = val.x, b = val.y;
          atomicAdd(&rho[rowbase + t], w1 * a * a + w2 * b * b);
        }
        __syncthreads();
      } else {
        for (int t = threadIdx.x; t < nr * n0; t += blockDim.x) {
          const double vv = v[rowbase + t];
          C val = res[t];
          val.x *= vv; val.y *= vv;
          res[t] = val;
        }
        __syncthreads();
        C* other = (res == R1) ? R2 : R1;
        C* res2 = fft_lines<-1>(res, other, nr, n0, g.px, tx);
        for (int t = threadIdx.x; t < nr * ncol; t += blockDim.x) {
          const int r = t / ncol, cidx = t - r * ncol;
          P[cidx * n1 + y0 + r] = res2[r * n0 + g.col_x[cidx]];
        }
        __syncthreads();
      }
    }
    if (OP == OP_VPSI) {
      y_pass<-1>(P, S, ncol, n1, cc, g.py, ty);
      for (int s = threadIdx.x; s < nvec; s += blockDim.x)
        zp[s] = P[g.stick_col[s] * n1 + g.stick_y[s]];
      __syncthreads();
    }
  }
}

// ------------------------------------------------ full-grid line passes
// In-place FFT of all lines along one axis of an n0 x n1 x n2 grid (x
// fastest).  A CTA takes L lines; for the y and z axes these are L adjacent
// x so that global accesses stay coalesced.
template <int DIR>
__global__ void __launch_bounds__(256)
k_line_fft(double2* __restrict__ grid, int n0, int n1, int n2, int axis, RadixPlan p,
           const double2* __restrict__ tw_g, int L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* tw = reinterpret_cast<double2*>(smem_raw);
  const int n = p.n;
  double2* A = tw + n;
  double2* B = A + L * n;
  load_twiddles(tw, tw_g, n);
  // line set of this CTA
  size_t base;
  size_t estride, lstride;
  int nl;
  if (axis == 0) {
    const int nlines = n1 * n2;
    const int l0 = blockIdx.x * L;
    nl = min(L, nlines - l0);
    base = (size_t)l0 * n0;
    estride = 1; lstride = n0;
  } else if (axis == 1) {
    const int xt = (n0 + L - 1) / L;
    const int zb = blockIdx.x / xt, x0 = (blockIdx.x % xt) * L;
    nl = min(L, n0 - x0);
    base = (size_t)x0 + (size_t)n0 * n1 * zb;
    estride = n0; lstride = 1;
  } else {
    const int xt = (n0 + L - 1) / L;
    const int yb = blockIdx.x / xt, x0 = (blockIdx.x % xt) * L;
    nl = min(L, n0 - x0);
    base = (size_t)x0 + (size_t)n0 * yb;
    estride = (size_t)n0 * n1; lstride = 1;
  }
  for (int t = threadIdx.x; t < nl * n; t += blockDim.x) {
    int line, e;
    if (axis == 0) { line = t / n; e = t - line * n; }
    else { line = t % nl; e = t / nl; }
    A[line * n + e] = grid[base + e * estride + line * lstride];
  }
  __syncthreads();
  double2* res = fft_lines<DIR>(A, B, nl, n, p, tw);
  for (int t = threadIdx.x; t < nl * n; t += blockDim.x) {
    int line, e;
    if (axis == 0) { line = t / n; e = t - line * n; }
    else { line = t % nl; e = t / nl; }
    grid[base + e * estride + line * lstride] = res[line * n + e];
  }
}

__global__ void k_scatter_sphere(const double2* __restrict__ c, const int* __restrict__ ip,
                                 const int* __restrict__ im, int ng, double2* __restrict__ grid) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ng; i += gridDim.x * blockDim.x) {
    const double2 v = c[i];
    grid[ip[i]] = v;
    grid[im[i]] = make_double2(v.x, -v.y);
  }
}

__global__ void k_scatter_pair(const double2* __restrict__ c1, const double2* __restrict__ c2,
                               const int* __restrict__ ip, const int* __restrict__ im, int ng,
                               double2* __restrict__ grid) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ng; i += gridDim.x * blockDim.x) {
    const double2 p = c1[i];
    const double2 q = c2 ? c2[i] : make_double2(0.0, 0.0);
    grid[ip[i]] = make_double2(p.x - q.y, p.y + q.x);
    grid[im[i]] = make_double2(p.x + q.y, q.x - p.y);
  }
}

__global__ void k_gather_sphere(const double2* __restrict__ grid, const int* __restrict__ ip,
                                int ng, double scale, double2* __restrict__ c) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ng; i += gridDim.x * blockDim.x) {
    const double2 v = grid[ip[i]];
    c[i] = make_double2(v.x * scale, v.y * scale);
  }
}

// complex basis: only +G is stored (BasisMapping::vector_to_zvec,
// src/BasisMapping.cpp:655-663)
__global__ void k_scatter_plus(const double2* __restrict__ c, const int* __restrict__ ip, int ng,
                               double2* __restrict__ grid) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ng; i += gridDim.x * blockDim.x)
    grid[ip[i]] = c[i];
}

// two real functions out of one complex transform
// (BasisMapping::zvec_to_doublevector, src/BasisMapping.cpp:716-750), with
// the forward transform's 1/N applied to the grid values
__global__ void k_gather_pair(const double2* __restrict__ grid, const int* __restrict__ ip,
                              const int* __restrict__ im, int ng, double scale,
                              double2* __restrict__ c1, double2* __restrict__ c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ng; i += gridDim.x * blockDim.x) {
    const double2 p = grid[ip[i]], m = grid[im[i]];
    const double a = p.x * scale, b = p.y * scale, c = m.x * scale, d = m.y * scale;
    c1[i] = make_double2(0.5 * (a + c), 0.5 * (b - d));
    c2[i] = make_double2(0.5 * (b + d), 0.5 * (c - a));
  }
}

__global__ void k_real_to_grid(const double* __restrict__ f, double scale, size_t n,
                               double2* __restrict__ grid) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    grid[i] = make_double2(f[i] * scale, 0.0);
}

__global__ void k_grid_real(const double2* __restrict__ grid, size_t n, double* __restrict__ f) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    f[i] = grid[i].x;
}

// both parts of a grid of two packed real fields
__global__ void k_grid_split(const double2* __restrict__ grid, size_t n, double* __restrict__ f0,
                             double* __restrict__ f1) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double2 v = grid[i];
    f0[i] = v.x;
    f1[i] = v.y;
  }
}

// grid = f0 w + i f1 w (f1 may be null)
__global__ void k_real2_mul_to_grid(const double* __restrict__ f0, const double* __restrict__ f1,
                                    const double* __restrict__ w, size_t n,
                                    double2* __restrict__ grid) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double x = w[i];
    grid[i] = make_double2(f0[i] * x, f1 ? f1[i] * x : 0.0);
  }
}

// ------------------------------------------------------------ launchers
static std::vector<double2> twiddle_table(int n) {
  std::vector<double2> t(n);
  for (int k = 0; k < n; k++) {
    const double a = 2.0 * M_PI * (double)k / (double)n;
    t[k] = make_double2(cos(a), sin(a));
  }
  return t;
}

// the twiddle table of one axis of a context's grid
static const double2* twiddles(const Context& ctx, int axis) { return ctx.dws.tw[axis]; }

void upload_sticks(DeviceSticks& d, const Basis& b) {
  free_sticks(d);
  d.n0 = b.n0; d.n1 = b.n1; d.n2 = b.n2;
  d.nrods = b.nrods; d.nvec = b.nvec; d.ncol = b.ncol;
  d.rod_first = dupload(b.rod_first);
  d.rod_lmin = dupload(b.rod_lmin);
  d.rod_size = dupload(b.rod_size);
  d.stick_y = dupload(b.stick_y);
  d.stick_col = dupload(b.stick_col);
  d.col_x = dupload(b.col_x);
  {
    std::vector<int> xc(b.n0, -1);
    for (int i = 0; i < b.ncol; i++) xc[b.col_x[i]] = i;
    d.xcol = dupload(xc);
  }
  d.ip = dupload(b.ip);
  d.im = dupload(b.im);
  {
    std::vector<int> cm((size_t)b.ncol * b.n1, -1);
    for (int s = 0; s < b.nvec; s++) cm[(size_t)b.stick_col[s] * b.n1 + b.stick_y[s]] = s;
    d.colmap = dupload(cm);
  }
  auto dist = [](int x, int n) { x = ((x % n) + n) % n; return std::min(x, n - x); };
  d.xw = d.yw = d.zw = 0;
  for (int x : b.col_x) d.xw = std::max(d.xw, dist(x, b.n0));
  for (int y : b.stick_y) d.yw = std::max(d.yw, dist(y, b.n1));
  for (int r = 0; r < b.nrods; r++)
    d.zw = std::max({d.zw, std::abs(b.rod_lmin[r]), std::abs(b.rod_lmin[r] + b.rod_size[r] - 1)});
  d.px = make_plan(b.n0);
  d.py = make_plan(b.n1);
  d.pz = make_plan(b.n2);
  d.gain32 = 1.0;
  double gain = 1.0;
  for (int i = 0; i < 3; i++) {
    const int n3[3] = {b.n0, b.n1, b.n2};
    if (i == 0 || n3[i] != n3[i - 1]) gain = pencil_length(n3[i]) ? pencil_gain_fp32(n3[i]) : 1.0;
    d.gain32 *= gain;
  }
  const int n[3] = {b.n0, b.n1, b.n2};
  for (int a = 0; a < 3; a++) {
    std::vector<double2> t = twiddle_table(n[a]);
    d.tw[a] = dalloc<double2>(n[a]);
    h2d_sync(d.tw[a], t.data(), n[a] * sizeof(double2));
  }
}

void free_sticks(DeviceSticks& d) {
  for (int a = 0; a < 3; a++) dfree(d.tw[a]);
  dfree(d.rod_first); dfree(d.rod_lmin); dfree(d.rod_size);
  dfree(d.stick_y); dfree(d.stick_col); dfree(d.col_x); dfree(d.xcol);
  dfree(d.ip); dfree(d.im);
  dfree(d.colmap);
}

static const int kRodsPerCta = 8;

template <typename T>
static size_t zsmem(int n2) {
  return sizeof(typename Cplx<T>::t) * (size_t)n2 * (1 + 4 * kRodsPerCta);
}

template <typename T>
struct XYConfig {
  size_t smem;
  int cc, rr;
};

static int max_smem_optin(int dev) {
  int v = 0;
  QBX_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  return v;
}

template <typename T>
static XYConfig<T> xy_config(const DeviceSticks& g, int dev) {
  using C = typename Cplx<T>::t;
  const size_t fixed = sizeof(C) * ((size_t)g.n0 + g.n1 + (size_t)g.ncol * g.n1);
  const size_t limit = (size_t)max_smem_optin(dev);
  // FP32 tiles leave room for two CTAs per SM
  size_t budget = sizeof(T) == 4 ? std::min(limit, (size_t)112 * 1024) : limit;
  if (budget < fixed + sizeof(C) * 2 * g.n0) budget = limit;
  QBX_REQUIRE(budget >= fixed + sizeof(C) * 2 * g.n0, 20,
              "FFT plane tile does not fit in shared memory");
  const size_t scratch = budget - fixed;
  XYConfig<T> c;
  c.cc = (int)std::min<size_t>(g.ncol, scratch / (sizeof(C) * g.n1));
  c.rr = (int)std::min<size_t>(g.n1, scratch / (sizeof(C) * 2 * g.n0));
  const size_t need = std::max(sizeof(C) * (size_t)c.cc * g.n1, sizeof(C) * 2 * (size_t)c.rr * g.n0);
  c.smem = fixed + need;
  QBX_REQUIRE(c.cc >= 1 && c.rr >= 1, 20, "FFT plane tile does not fit in shared memory");
  return c;
}

template <typename T>
static void staged_batch(Context& ctx, int op, const double* c, const double* v, double* rho,
                         const double* w, double* hc, int pair0, int npairs) {
  using C = typename Cplx<T>::t;
  const DeviceSticks& g = ctx.dws;
  cudaStream_t st = ctx.stream;
  C* zbuf = (C*)ctx.d_zbuf;
  const double2* twz = twiddles(ctx, 2);
  const double2* twx = twiddles(ctx, 0);
  const double2* twy = twiddles(ctx, 1);
  const int ngw = ctx.wb.ng;
  dim3 zgrid((g.nrods + kRodsPerCta - 1) / kRodsPerCta, npairs);
  const size_t zs = zsmem<T>(g.n2);
  allow_smem(k_zfft_bwd<T>, zs);
  {
    ProfScope ps(ctx, "zfft_bwd");
    k_zfft_bwd<T><<<zgrid, 256, zs, st>>>((const double2*)c, ngw, ctx.nst, pair0, g, twz, zbuf,
                                           kRodsPerCta);
    QBX_LAUNCHED(ctx);
  }
  XYConfig<T> xc = xy_config<T>(g, ctx.device);
  int sms = 0;
  QBX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
  // enough (plane, pair-chunk) CTAs to cover every SM a couple of times
  int chunks = std::max(1, (3 * sms + g.n2 - 1) / g.n2);
  chunks = std::min(chunks, npairs);
  const int ppc = (npairs + chunks - 1) / chunks;
  chunks = (npairs + ppc - 1) / ppc;
  dim3 xgrid(g.n2, chunks);
  if (op == OP_DENSITY) {
    allow_smem(k_xy<T, OP_DENSITY>, xc.smem);
    ProfScope ps(ctx, "xy_density");
    k_xy<T, OP_DENSITY><<<xgrid, 512, xc.smem, st>>>(zbuf, npairs, ppc, g, twx, twy, nullptr, rho, w,
                                                   pair0, ctx.nst, xc.cc, xc.rr);
    QBX_LAUNCHED(ctx);
  } else {
    allow_smem(k_xy<T, OP_VPSI>, xc.smem);
    {
      ProfScope ps(ctx, "xy_vpsi");
      k_xy<T, OP_VPSI><<<xgrid, 512, xc.smem, st>>>(zbuf, npairs, ppc, g, twx, twy, v, nullptr,
                                                  nullptr, pair0, ctx.nst, xc.cc, xc.rr);
      QBX_LAUNCHED(ctx);
    }
    allow_smem(k_zfft_fwd<T>, zs);
    const double scale = 1.0 / ((double)g.n0 * g.n1 * g.n2);
    ProfScope ps(ctx, "zfft_fwd");
    k_zfft_fwd<T><<<zgrid, 256, zs, st>>>(zbuf, ngw, ctx.nst, pair0, g, twz, scale,
                                           (const double2*)c, ctx.d_g2_w, (double2*)hc, kRodsPerCta);
    QBX_LAUNCHED(ctx);
  }
}

// ------------------------------------------------ complex basis (k != 0)
// One band per stick line: the basis at k has one rod per (h,k) column and
// no -G half to fill (BasisMapping::vector_to_zvec and zvec_to_vector of a
// complex basis, src/BasisMapping.cpp:585-627, 703-750).  zbuf holds band
// `band0 + slot` in slot, [slot][z][stick] as for band pairs, so the plane
// kernels run unchanged on the complex sticks.
__global__ void __launch_bounds__(256)
k_zfft_bwd_k(const double2* __restrict__ c, int ngw, int band0, DeviceSticks g,
             const double2* __restrict__ twz, double2* __restrict__ zbuf, int rods_per_cta) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tw = reinterpret_cast<C*>(smem_raw);
  const int n2 = g.n2;
  C* A = tw + n2;
  C* B = A + rods_per_cta * n2;
  const int r0 = blockIdx.x * rods_per_cta;
  const int r1 = min(g.nrods, r0 + rods_per_cta);
  const int nl = r1 - r0;
  const int pl = blockIdx.y;
  const double2* cb = c + (size_t)(band0 + pl) * ngw;
  load_twiddles(tw, twz, n2);
  const int half = (n2 + 1) / 2;
  for (int t = threadIdx.x; t < nl * n2; t += blockDim.x) {
    const int line = t / n2, z = t - line * n2;
    const int r = r0 + line;
    const int l = z < half ? z : z - n2;
    const int lmin = g.rod_lmin[r];
    C v = make_double2(0.0, 0.0);
    if (l >= lmin && l < lmin + g.rod_size[r]) v = cb[g.rod_first[r] + (l - lmin)];
    A[line * n2 + z] = v;
  }
  __syncthreads();
  C* res = fft_lines<+1>(A, B, nl, n2, g.pz, tw);
  C* out = zbuf + (size_t)pl * n2 * g.nvec;
  for (int t = threadIdx.x; t < nl * n2; t += blockDim.x) {
    const int line = t % nl, z = t / nl;
    out[(size_t)z * g.nvec + r0 + line] = res[line * n2 + z];
  }
}

// z transform back and hc = 1/2 |k+G|^2 c + (V psi)(G) / N
__global__ void __launch_bounds__(256)
k_zfft_fwd_k(const double2* __restrict__ zbuf, int ngw, int band0, DeviceSticks g,
             const double2* __restrict__ twz, double scale, const double2* __restrict__ c,
             const double* __restrict__ g2, double2* __restrict__ hc, int rods_per_cta) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tw = reinterpret_cast<C*>(smem_raw);
  const int n2 = g.n2;
  C* A = tw + n2;
  C* B = A + rods_per_cta * n2;
  const int r0 = blockIdx.x * rods_per_cta;
  const int r1 = min(g.nrods, r0 + rods_per_cta);
  const int nl = r1 - r0;
  const int pl = blockIdx.y;
  load_twiddles(tw, twz, n2);
  const C* in = zbuf + (size_t)pl * n2 * g.nvec;
  for (int t = threadIdx.x; t < nl * n2; t += blockDim.x) {
    const int line = t % nl, z = t / nl;
    A[line * n2 + z] = in[(size_t)z * g.nvec + r0 + line];
  }
  __syncthreads();
  C* res = fft_lines<-1>(A, B, nl, n2, g.pz, tw);
  const int ig0 = g.rod_first[r0];
  const int ig1 = g.rod_first[r1 - 1] + g.rod_size[r1 - 1];
  const size_t boff = (size_t)(band0 + pl) * ngw;
  for (int ig = ig0 + threadIdx.x; ig < ig1; ig += blockDim.x) {
    int r = r0;
    while (r + 1 < r1 && g.rod_first[r + 1] <= ig) ++r;
    const int l = g.rod_lmin[r] + (ig - g.rod_first[r]);
    const int z = ((l % n2) + n2) % n2;
    const C p = res[(r - r0) * n2 + z];
    const double kin = 0.5 * g2[ig];
    const double2 a = c[boff + ig];
    hc[boff + ig] = make_double2(kin * a.x + p.x * scale, kin * a.y + p.y * scale);
  }
}

// ------------------------------------------------------- line-pass FFTs
// (fft_pencil.cuh) The grids of the plane-free passes: z fastest.
// a grid value as the passes read it: FP64, or the value rounded to FP32 and the
// rest (none where the rounded value is not finite)
template <typename B> __device__ __forceinline__ B grid_value(double x);
template <> __device__ __forceinline__ double grid_value<double>(double x) { return x; }
template <> __device__ __forceinline__ float2 grid_value<float2>(double x) {
  const float hi = (float)x;
  return make_float2(hi, isfinite(hi) ? (float)(x - (double)hi) : 0.f);
}

// x-fastest grid <-> [x][y][z], 32 x 32 tiles of (x, z) at each y
template <typename A, typename B, bool ADD>
__global__ void __launch_bounds__(256)
k_grid_to_zfast(const A* __restrict__ in, int n0, int n1, int n2, bool to_zfast,
                B* __restrict__ out) {
  __shared__ B t[32][33];
  const int x0 = blockIdx.x * 32, z0 = blockIdx.y * 32, y = blockIdx.z;
  const int a = threadIdx.x & 31, b = threadIdx.x >> 5;
  for (int i = b; i < 32; i += 8) {
    const int x = to_zfast ? x0 + a : x0 + i, z = to_zfast ? z0 + i : z0 + a;
    if (x < n0 && z < n2)
      t[i][a] = grid_value<B>(in[to_zfast ? ((size_t)z * n1 + y) * n0 + x : ((size_t)x * n1 + y) * n2 + z]);
  }
  __syncthreads();
  for (int i = b; i < 32; i += 8) {
    const int x = to_zfast ? x0 + i : x0 + a, z = to_zfast ? z0 + a : z0 + i;
    if (x < n0 && z < n2) {
      B* o = out + (to_zfast ? ((size_t)x * n1 + y) * n2 + z : ((size_t)z * n1 + y) * n0 + x);
      if constexpr (ADD) *o += t[a][i];
      else *o = t[a][i];
    }
  }
}

static int nblk(size_t n);
static bool pencil_ok(const Context& ctx, const DeviceSticks& g, bool fp32);

__global__ void k_to_floats(const double* __restrict__ x, size_t n, float2* __restrict__ y) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    y[i] = grid_value<float2>(x[i]);
}

// The context's real-space grids (density, potentials, gradients) are kept z
// fastest when both of its bases go through the line passes, which then read
// and write them directly; callers of the library always see x fastest.
bool grid_zfast_possible(const Context& ctx) {
  const DeviceSticks& g = ctx.dvs;
  return pencil_ok(ctx, ctx.dws, false) && ctx.zfast_bytes >=
         sizeof(double2) * (size_t)g.n2 * ((size_t)g.nvec + (size_t)g.ncol * g.n1);
}

// The runtime-radix kernels' stick buffer (up to 4 GB), for contexts whose
// Gamma sphere or one of whose k points is not the line passes'; the precision
// sets its size.
void ensure_radix_buffer(Context& ctx) {
  bool radix = !pencil_ok(ctx, ctx.dws, ctx.precision == MIXED);
  for (const KPointSet& kp : ctx.kpts) radix = radix || !pencil_ok(ctx, kp.dks, false);
  const size_t need = density_stick_bytes_per_pair(ctx) * ctx.pair_batch;
  if (!radix || ctx.zbuf_bytes == need) return;
  if (ctx.d_zbuf) cudaFree(ctx.d_zbuf);
  ctx.d_zbuf = nullptr;
  ctx.zbuf_bytes = 0;
  QBX_CUDA(cudaMalloc(&ctx.d_zbuf, need));
  ctx.zbuf_bytes = need;
}

// f as callers see it (x fastest), in `out`; and the opposite
void grid_to_caller(Context& ctx, const double* f, double* out) {
  const DeviceSticks& g = ctx.dvs;
  const dim3 tg((g.n0 + 31) / 32, (g.n2 + 31) / 32, g.n1);
  k_grid_to_zfast<double, double, false><<<tg, 256, 0, ctx.stream>>>(f, g.n0, g.n1, g.n2, false,
                                                                     out);
  QBX_LAUNCHED(ctx);
}
void grid_from_caller(Context& ctx, const double* f, double* out) {
  const DeviceSticks& g = ctx.dvs;
  const dim3 tg((g.n0 + 31) / 32, (g.n2 + 31) / 32, g.n1);
  k_grid_to_zfast<double, double, false><<<tg, 256, 0, ctx.stream>>>(f, g.n0, g.n1, g.n2, true,
                                                                     out);
  QBX_LAUNCHED(ctx);
}

// With k points the grids are z fastest only if every k point's sphere runs
// through the line passes; every field that the context holds moves to the new
// order (a stress without a new step combines them point by point).
void kpoints_grid_order(Context& ctx) {
  ensure_radix_buffer(ctx);
  bool z = grid_zfast_possible(ctx);
  for (const KPointSet& kp : ctx.kpts) z = z && pencil_ok(ctx, kp.dks, false);
  if (z == ctx.grid_zfast) return;
  const size_t N = ctx.N();
  for (double* f : {ctx.d_rhor, ctx.d_vr, ctx.d_vxc, ctx.d_exc, ctx.d_vx2, ctx.d_grad,
                    ctx.d_grad + N, ctx.d_grad + 2 * N}) {
    if (z) grid_from_caller(ctx, f, (double*)ctx.d_grid);
    else grid_to_caller(ctx, f, (double*)ctx.d_grid);
    QBX_CUDA(cudaMemcpyAsync(f, ctx.d_grid, N * sizeof(double), cudaMemcpyDeviceToDevice,
                             ctx.stream));
  }
  ctx.grid_zfast = z;
}

template <typename T>
static bool pencil_run(Context& ctx, int n, const pen::Args& a) {
  return pencil_0<T>(ctx, n, a) || pencil_1<T>(ctx, n, a) || pencil_2<T>(ctx, n, a) ||
         pencil_3<T>(ctx, n, a) || pencil_4<T>(ctx, n, a) || pencil_5<T>(ctx, n, a) ||
         pencil_6<T>(ctx, n, a) || pencil_7<T>(ctx, n, a);
}

// matrix of the FP32 register DFT of m points (row-major, the roots as the
// kernels round them)
using zmat = std::vector<std::complex<double>>;
static zmat roots_fp32(int n) {
  zmat r(n);
  for (int k = 0; k < n; k++)
    r[k] = {(double)(float)lane::cx_cos(k, n), (double)(float)lane::cx_sin(k, n)};
  return r;
}
static zmat dft_fp32(int m) {
  zmat f((size_t)m * m);
  const zmat w = roots_fp32(m);
  const int r1 = lane::first_radix(m);
  if (m == r1) {
    for (int k = 0; k < m; k++)
      for (int j = 0; j < m; j++) f[(size_t)k * m + j] = w[(j * k) % m];
    return f;
  }
  const int q1 = m / r1;
  const zmat a = dft_fp32(q1), b = dft_fp32(r1);
  for (int s = 0; s < r1; s++)
    for (int q = 0; q < q1; q++)
      for (int r = 0; r < r1; r++)
        for (int k = 0; k < q1; k++)
          f[(size_t)(q + q1 * s) * m + r + r1 * k] =
              b[(size_t)s * r1 + r] * w[r * q] * a[(size_t)q * q1 + k];
  return f;
}

double pencil_gain_fp32(int n) {
  const int r1 = pen::fac(n).r1, r2 = pen::fac(n).r2, pw = prune_width(n);
  const zmat a = dft_fp32(r1), b = dft_fp32(r2), w = roots_fp32(n);
  zmat bn(r2, 0.0);                        // column norms of the second DFT
  for (int j = 0; j < r2; j++)
    for (int m = 0; m < r2; m++) bn[j] += std::norm(b[(size_t)m * r2 + j]);
  double sum = 0.0;
  int count = 0;
  for (int x = 0; x < n; x++) {
    if (x > pw && x < n - pw) continue;
    const int j = x % r2, q = x / r2;
    for (int k = 0; k < r1; k++)
      sum += bn[j].real() * std::norm(w[j * k]) * std::norm(a[(size_t)k * r1 + q]);
    count++;
  }
  return sum / ((double)count * n);
}

// bytes of one slot's sticks and of its tile
static size_t pencil_stick_bytes(const DeviceSticks& g, bool fp32) {
  return (fp32 ? sizeof(float2) : sizeof(double2)) * (size_t)g.n2 * g.nvec;
}
static size_t pencil_tile_bytes(const DeviceSticks& g, bool fp32) {
  return (fp32 ? sizeof(float2) : sizeof(double2)) * (size_t)g.n2 * g.ncol * g.n1;
}

// The line passes take every grid whose lengths are compiled, whose sphere
// lies within prune_width on each axis and whose slot fits the stick buffer;
// the rest runs the runtime-radix kernels above.
static bool pencil_ok(const Context& ctx, const DeviceSticks& g, bool fp32) {
  return ctx.fast_fft && ctx.d_zfast && pencil_length(g.n0) && pencil_length(g.n1) &&
         pencil_length(g.n2) && g.xw <= prune_width(g.n0) && g.yw <= prune_width(g.n1) &&
         g.zw <= prune_width(g.n2) &&
         pencil_stick_bytes(g, fp32) + pencil_tile_bytes(g, fp32) <= ctx.zfast_bytes;
}

// The buffer that keeps every slot's tile (`need` bytes): allocated, outside
// stream capture, when `keep` asks for it and the device has room; without
// `keep` only a buffer that is there already.  Null: no such buffer, and the
// tiles go through the stick buffer in batches.  Room is twice the buffer and 4 GB,
// since a context works without it: as much again is left to the contexts that a
// program makes after this one's first step.
static void* tile_area(Context& ctx, size_t need, bool keep) {
  if (ctx.d_wtile && ctx.wtile_bytes >= need) return ctx.d_wtile;
  if (!keep || ctx.wtile_mode == 0 || ctx.capturing) return nullptr;
  size_t freeb = 0, total = 0;
  QBX_CUDA(cudaMemGetInfo(&freeb, &total));
  if (freeb >= 2 * need + ((size_t)4 << 30)) {
    if (ctx.d_wtile) cudaFree(ctx.d_wtile);
    ctx.d_wtile = nullptr;
    const cudaError_t e = cudaMalloc(&ctx.d_wtile, need);
    if (e == cudaSuccess) {
      ctx.wtile_bytes = need;
      return ctx.d_wtile;
    }
    ctx.d_wtile = nullptr;
    if (e != cudaErrorMemoryAllocation) QBX_CUDA(e);
    cudaGetLastError();   // taken by another context or process since
  }
  if (ctx.wtile_mode < 0) ctx.wtile_mode = 0;   // no room: transform twice for this cell
  return nullptr;
}

// Slots first ... first + nslots of one wavefunction block (band pairs, or
// bands of a k point with `complex_basis`) through the line passes.  Density:
// added into rho (x fastest; `add`) or stored there.  H psi: hc = 1/2 g2 c + V
// psi.  area: room for the tiles of all these slots (then the x pass is one
// launch, and with `have` the tiles are those of the density pass), or null:
// sticks and tiles in batches through the stick buffer.
template <typename T>
static void pencil_pass(Context& ctx, const DeviceSticks& g, bool complex_basis, int op,
                        const double* c, int ngw, const double* g2, const double* v, double* rho,
                        bool add, const double* w, int nw, double* hc, void* area, bool have,
                        int first, int nslots) {
  using C = typename Cplx<T>::t;
  const size_t N = ctx.N();
  const dim3 tg((g.n0 + 31) / 32, (g.n2 + 31) / 32, g.n1);
  pen::Args a;
  a.g = g;
  for (int i = 0; i < 3; i++) a.tw[i] = g.tw[i];
  a.c = (const double2*)c;
  a.hc = (double2*)hc;
  a.g2 = g2;
  // FP32: the gain of the rounded roots taken out (as 1 in FP64)
  const double gain = sizeof(T) == 4 ? g.gain32 : 1.0;
  a.scale = 1.0 / ((double)N * gain);
  a.wout = 1.0 / gain;
  a.ngw = ngw;
  a.nst = ctx.nst;
  a.w = w;
  a.nw = nw;
  // density and V(r), z fastest: the context's own grids where they are kept
  // so (grid_zfast), else transposed through d_grid
  const bool zfast = ctx.grid_zfast;
  a.rho = zfast ? rho : (double*)ctx.d_grid;
  using V = std::conditional_t<sizeof(T) == 4, float2, double>;
  V* vt = (V*)((double*)ctx.d_grid + N);
  a.v = vt;
  a.stream = ctx.stream;
  if (op == OP_VPSI) {
    if (zfast && sizeof(T) == 8) {
      a.v = v;
    } else {
      if (zfast) k_to_floats<<<nblk(N), 256, 0, ctx.stream>>>(v, N, (float2*)vt);
      else k_grid_to_zfast<double, V, false><<<tg, 256, 0, ctx.stream>>>(v, g.n0, g.n1, g.n2, true,
                                                                        vt);
      QBX_LAUNCHED(ctx);
    }
  }
  const size_t sb = pencil_stick_bytes(g, sizeof(T) == 4), tb = pencil_tile_bytes(g, sizeof(T) == 4);
  const int batch = (int)std::min<size_t>(nslots, ctx.zfast_bytes / (area ? sb : sb + tb));
  const int xcta = (g.n1 * g.n2 + 15) / 16, ycta = (g.ncol * g.n2 + 15) / 16;
  auto pass = [&](int n, int what, int chunks, const char* name) {
    ProfScope ps(ctx, name);
    a.op = what;
    a.chunks = chunks;
    QBX_REQUIRE(pencil_run<T>(ctx, n, a), 21, "no line kernel of this length");
  };
  auto slots = [&](int s0, int ns) {
    a.first = first + s0;
    a.nslots = ns;
    a.sticks = ctx.d_zfast;
    a.tile = area ? (void*)((C*)area + s0 * (tb / sizeof(C)))
                  : (void*)((C*)ctx.d_zfast + batch * (sb / sizeof(C)));
  };
  // CTAs per set of lines: enough for several per SM.  A CTA of the y passes
  // takes up to 4 slots, one of the x passes up to 16
  auto chunks = [&](int ns, int cta, int most) {
    return std::min(ns, std::max((ns + most - 1) / most, (1184 + cta - 1) / cta));
  };
  auto back = [&](int s0, int ns) {
    slots(s0, ns);
    pass(g.n2, complex_basis ? pen::ZBK : pen::ZB, 1, "zfft_bwd");
    pass(g.n1, pen::YB, chunks(ns, ycta, 4), "y_bwd");
  };
  auto forth = [&](int s0, int ns) {
    slots(s0, ns);
    pass(g.n1, pen::YF, chunks(ns, ycta, 4), "y_fwd");
    pass(g.n2, complex_basis ? pen::ZFK : pen::ZF, 1, "zfft_fwd");
  };
  auto x = [&](int s0, int ns) {
    slots(s0, ns);
    const int ch = chunks(ns, xcta, 16);
    if (op == OP_DENSITY) {
      a.rho_set = s0 == 0 && ch == 1 && !(zfast && add);
      if (s0 == 0 && !a.rho_set && !(zfast && add))
        QBX_CUDA(cudaMemsetAsync(a.rho, 0, N * sizeof(double), ctx.stream));
      pass(g.n0, pen::XD, ch, "xy_density");
    } else {
      pass(g.n0, pen::XV, ch, "xy_vpsi");
    }
  };
  for (int s0 = 0; s0 < nslots; s0 += batch) {
    const int ns = std::min(batch, nslots - s0);
    if (!have) back(s0, ns);
    if (area) continue;
    x(s0, ns);
    if (op == OP_VPSI) forth(s0, ns);
  }
  if (area) {
    x(0, nslots);
    for (int s0 = 0; op == OP_VPSI && s0 < nslots; s0 += batch)
      forth(s0, std::min(batch, nslots - s0));
  }
  if (op == OP_DENSITY && !zfast) {
    if (add)
      k_grid_to_zfast<double, double, true><<<tg, 256, 0, ctx.stream>>>(a.rho, g.n0, g.n1, g.n2,
                                                                        false, rho);
    else
      k_grid_to_zfast<double, double, false><<<tg, 256, 0, ctx.stream>>>(a.rho, g.n0, g.n1, g.n2,
                                                                         false, rho);
    QBX_LAUNCHED(ctx);
  }
}

static constexpr int kRodsPerCtaK = 2 * kRodsPerCta;   // one line per rod

// bands of a k point per pass through the context's stick buffer
static int kbands_per_batch(const Context& ctx, const KPointSet& kp) {
  const size_t per_band = (size_t)kp.dks.n2 * kp.dks.nvec * sizeof(double2);
  const int nb = (int)std::min<size_t>((size_t)ctx.nst, ctx.zbuf_bytes / per_band);
  QBX_REQUIRE(nb >= 1, 20, "stick buffer too small for one band of this k point");
  return nb;
}

static void staged_k(Context& ctx, KPointSet& kp, int op, const double* v, double* rho) {
  const DeviceSticks& g = kp.dks;
  if (pencil_ok(ctx, g, false)) {
    // tiles of all k points one after the other
    size_t off = 0, need = 0;
    bool all = true;
    for (KPointSet& q : ctx.kpts) {
      if (&q == &kp) off = need;
      need += pencil_tile_bytes(q.dks, false) * ctx.nst;
      all = all && pencil_ok(ctx, q.dks, false);
    }
    char* area = all ? (char*)tile_area(ctx, need, op == OP_DENSITY && ctx.tile_store) : nullptr;
    const bool have = op == OP_VPSI && area && ctx.tile_use && kp.tile_valid;
    // the weights are two per band, both the band's
    pencil_pass<double>(ctx, g, true, op, kp.d_c, kp.kb.ng, kp.d_g2, v, rho, true, kp.d_w2,
                        2 * ctx.nst, kp.d_hc, area ? area + off : nullptr, have, 0, ctx.nst);
    kp.tile_valid = op == OP_DENSITY && area && ctx.tile_store;
    return;
  }
  QBX_REQUIRE(!ctx.grid_zfast, 21, "this k point's sphere does not fit the line passes");
  cudaStream_t st = ctx.stream;
  double2* zbuf = (double2*)ctx.d_zbuf;
  const int ngw = kp.kb.ng;
  const size_t zs = zsmem<double>(g.n2);
  allow_smem(k_zfft_bwd_k, zs);
  allow_smem(k_zfft_fwd_k, zs);
  XYConfig<double> xc = xy_config<double>(g, ctx.device);
  allow_smem(k_xy<double, OP_DENSITY>, xc.smem);
  allow_smem(k_xy<double, OP_VPSI>, xc.smem);
  int sms = 0;
  QBX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
  const int nbmax = kbands_per_batch(ctx, kp);
  for (int b0 = 0; b0 < ctx.nst; b0 += nbmax) {
    const int nb = std::min(nbmax, ctx.nst - b0);
    dim3 zgrid((g.nrods + kRodsPerCtaK - 1) / kRodsPerCtaK, nb);
    k_zfft_bwd_k<<<zgrid, 256, zs, st>>>((const double2*)kp.d_c, ngw, b0, g, g.tw[2], zbuf,
                                         kRodsPerCtaK);
    QBX_LAUNCHED(ctx);
    int chunks = std::max(1, (3 * sms + g.n2 - 1) / g.n2);
    chunks = std::min(chunks, nb);
    const int ppc = (nb + chunks - 1) / chunks;
    chunks = (nb + ppc - 1) / ppc;
    dim3 xgrid(g.n2, chunks);
    if (op == OP_DENSITY) {
      // the pair kernel's weights w[2 slot], w[2 slot + 1] are both the band's
      k_xy<double, OP_DENSITY><<<xgrid, 512, xc.smem, st>>>(zbuf, nb, ppc, g, g.tw[0], g.tw[1],
                                                           nullptr, rho, kp.d_w2, b0, 2 * ctx.nst,
                                                           xc.cc, xc.rr);
      QBX_LAUNCHED(ctx);
    } else {
      k_xy<double, OP_VPSI><<<xgrid, 512, xc.smem, st>>>(zbuf, nb, ppc, g, g.tw[0], g.tw[1], v,
                                                        nullptr, nullptr, b0, 2 * ctx.nst, xc.cc,
                                                        xc.rr);
      QBX_LAUNCHED(ctx);
      const double scale = 1.0 / ((double)g.n0 * g.n1 * g.n2);
      k_zfft_fwd_k<<<zgrid, 256, zs, st>>>(zbuf, ngw, b0, g, g.tw[2], scale,
                                           (const double2*)kp.d_c, kp.d_g2, (double2*)kp.d_hc,
                                           kRodsPerCtaK);
      QBX_LAUNCHED(ctx);
    }
  }
}

// rho += sum_n weight occ_n / Omega |psi_nk|^2 (SlaterDet::compute_density,
// complex branch, src/SlaterDet.cpp:280-298)
void launch_density_k(Context& ctx, KPointSet& kp, double* rho) {
  ProfScope ps(ctx, "density_k");
  staged_k(ctx, kp, OP_DENSITY, nullptr, rho);
}

// hc = 1/2 |k+G|^2 c + FFT_fwd(v FFT_bwd(c)) (SlaterDet::rs_mul_add, complex
// branch, src/SlaterDet.cpp:458-475, with the kinetic term of
// EnergyFunctional::energy, src/EnergyFunctional.cpp:789-839)
void launch_vpsi_k(Context& ctx, KPointSet& kp, const double* v) {
  ProfScope ps(ctx, "vpsi_k");
  staged_k(ctx, kp, OP_VPSI, v, nullptr);
}

static int nblk(size_t n);

// This GPU's band pairs of c through the line passes; false when the grid is
// not theirs.  The tiles of a density pass are kept for the H psi pass of the
// same step where the step functions ask for it (tile_store, tile_use).
static bool staged_pencil(Context& ctx, int op, const double* c, const double* v, double* rho,
                          const double* w, double* hc) {
  const bool fp32 = ctx.precision == MIXED;
  const DeviceSticks& g = ctx.dws;
  if (!pencil_ok(ctx, g, fp32)) return false;
  int plo = 0, phi = 0;
  shard_pairs(ctx, plo, phi);
  const bool keep = op == OP_DENSITY && ctx.tile_store;
  const bool have = op == OP_VPSI && ctx.tile_use && ctx.tile_valid && ctx.tile_src == c;
  ctx.tile_valid = false;
  if (phi <= plo) {
    if (op == OP_DENSITY)
      QBX_CUDA(cudaMemsetAsync(rho, 0, ctx.N() * sizeof(double), ctx.stream));
    return true;
  }
  void* area = tile_area(ctx, pencil_tile_bytes(g, fp32) * (phi - plo), keep);
  auto run = [&](auto t) {
    pencil_pass<decltype(t)>(ctx, g, false, op, c, ctx.wb.ng, ctx.d_g2_w, v, rho, false, w,
                             ctx.nst, hc, area, have, plo, phi - plo);
  };
  if (fp32) run(0.f);
  else run(0.0);
  if (keep && area) {
    ctx.tile_valid = true;
    ctx.tile_src = c;
  }
  return true;
}

static void staged(Context& ctx, int op, const double* c, const double* v, double* rho,
                   const double* w, double* hc) {
  if (staged_pencil(ctx, op, c, v, rho, w, hc)) return;
  if (op == OP_DENSITY)
    QBX_CUDA(cudaMemsetAsync(rho, 0, ctx.N() * sizeof(double), ctx.stream));
  int plo = 0, phi = 0;
  shard_pairs(ctx, plo, phi);
  for (int p0 = plo; p0 < phi; p0 += ctx.pair_batch) {
    const int np = std::min(ctx.pair_batch, phi - p0);
    if (ctx.precision == MIXED)
      staged_batch<float>(ctx, op, c, v, rho, w, hc, p0, np);
    else
      staged_batch<double>(ctx, op, c, v, rho, w, hc, p0, np);
  }
}

// With the band pairs split over GPUs (qbx_set_band_shard) each GPU
// transforms its own pairs; the density is then summed over the GPUs and
// the H*psi blocks gathered, so every GPU continues with the whole of both.
void launch_density(Context& ctx, const double* c, double* rho) {
  staged(ctx, OP_DENSITY, c, nullptr, rho, density_weights(ctx), nullptr);
  if (ctx.shard_comm) shard_sum(ctx, rho, ctx.N());
}

void launch_vpsi(Context& ctx, const double* c, const double* v, double* hc) {
  staged(ctx, OP_VPSI, c, v, nullptr, nullptr, hc);
  if (ctx.shard_comm) shard_gather_bands(ctx, hc);
}

static bool pencil_grid(Context& ctx, int n, double2* grid, const double2* tw, int inner,
                        int nlines, int dir) {
  return pencil_grid_0(ctx, n, grid, tw, inner, nlines, dir) ||
         pencil_grid_1(ctx, n, grid, tw, inner, nlines, dir) ||
         pencil_grid_2(ctx, n, grid, tw, inner, nlines, dir) ||
         pencil_grid_3(ctx, n, grid, tw, inner, nlines, dir) ||
         pencil_grid_4(ctx, n, grid, tw, inner, nlines, dir) ||
         pencil_grid_5(ctx, n, grid, tw, inner, nlines, dir) ||
         pencil_grid_6(ctx, n, grid, tw, inner, nlines, dir) ||
         pencil_grid_7(ctx, n, grid, tw, inner, nlines, dir);
}

// full-grid transform of `grid` on the geometry of d (sizes, twiddles)
static void grid_fft_on(Context& ctx, const DeviceSticks& b, double2* grid, int dir) {
  ProfScope ps(ctx, "grid_fft");
  const int n[3] = {b.n0, b.n1, b.n2};
  const int L = 16;
  for (int axis = 0; axis < 3; axis++) {
    const double2* tw = b.tw[axis];
    // compiled lengths: register lines (fft_pencil.cuh)
    const int inner = axis == 0 ? 1 : axis == 1 ? b.n0 : b.n0 * b.n1;
    const int nlines = axis == 0 ? b.n1 * b.n2 : axis == 1 ? b.n0 * b.n2 : b.n0 * b.n1;
    if (ctx.fast_fft && pencil_grid(ctx, n[axis], grid, tw, inner, nlines, dir)) continue;
    const RadixPlan p = make_plan(n[axis]);
    int nblocks;
    if (axis == 0) nblocks = (b.n1 * b.n2 + L - 1) / L;
    else if (axis == 1) nblocks = ((b.n0 + L - 1) / L) * b.n2;
    else nblocks = ((b.n0 + L - 1) / L) * b.n1;
    const size_t smem = sizeof(double2) * (size_t)n[axis] * (1 + 2 * L);
    if (dir > 0) {
      allow_smem(k_line_fft<+1>, smem);
      k_line_fft<+1><<<nblocks, 256, smem, ctx.stream>>>(grid, b.n0, b.n1, b.n2, axis, p, tw, L);
    } else {
      allow_smem(k_line_fft<-1>, smem);
      k_line_fft<-1><<<nblocks, 256, smem, ctx.stream>>>(grid, b.n0, b.n1, b.n2, axis, p, tw, L);
    }
    QBX_LAUNCHED(ctx);
  }
}

// full-grid transform of the density-basis grid held in ctx.d_grid
static void grid_fft(Context& ctx, int dir) { grid_fft_on(ctx, ctx.dvs, (double2*)ctx.d_grid, dir); }

// One band c (ng coefficients of the half sphere) to its real values on the
// grid of d (FourierTransform::backward, one band), x fastest, into f.
void wfgrid_backward(Context& ctx, const DeviceSticks& d, int ng, const double* c, double* f) {
  const size_t N = (size_t)d.n0 * d.n1 * d.n2;
  QBX_REQUIRE(N <= ctx.N(), 1, "grid larger than the density grid's workspace");
  QBX_CUDA(cudaMemsetAsync(ctx.d_grid, 0, N * sizeof(double2), ctx.stream));
  k_scatter_sphere<<<nblk(ng), 256, 0, ctx.stream>>>((const double2*)c, d.ip, d.im, ng,
                                                     (double2*)ctx.d_grid);
  QBX_LAUNCHED(ctx);
  grid_fft_on(ctx, d, (double2*)ctx.d_grid, +1);
  k_grid_real<<<nblk(N), 256, 0, ctx.stream>>>((const double2*)ctx.d_grid, N, f);
  QBX_LAUNCHED(ctx);
}

// The inverse: real values f on the grid of d to the band's coefficients
// (FourierTransform::forward with its 1/N, then the half sphere).
void wfgrid_forward(Context& ctx, const DeviceSticks& d, int ng, const double* f, double* c) {
  const size_t N = (size_t)d.n0 * d.n1 * d.n2;
  QBX_REQUIRE(N <= ctx.N(), 1, "grid larger than the density grid's workspace");
  k_real_to_grid<<<nblk(N), 256, 0, ctx.stream>>>(f, 1.0, N, (double2*)ctx.d_grid);
  QBX_LAUNCHED(ctx);
  grid_fft_on(ctx, d, (double2*)ctx.d_grid, -1);
  k_gather_sphere<<<nblk(ng), 256, 0, ctx.stream>>>((const double2*)ctx.d_grid, d.ip, ng,
                                                    1.0 / (double)N, (double2*)c);
  QBX_LAUNCHED(ctx);
}

static int nblk(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 148 * 16); }

// z = x + y (z may be either)
__global__ void k_add(const double* x, const double* y, size_t n, double* z) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    z[i] = x[i] + y[i];
}

// ----------------------------------------------- a caller's basis and grid
// The grid of a FourierTransform built on any basis (its Miller indices in
// the caller's order): sizes, twiddle tables, radix plans and the grid
// index of +G and (real basis) -G of each coefficient.  The transforms are
// full-grid line passes; the staged z-stick kernels serve the contexts'
// own bases.
void upload_grid_map(DeviceSticks& d, int n0, int n1, int n2, const std::vector<int>& ip,
                     const std::vector<int>& im) {
  free_sticks(d);
  d = DeviceSticks{};
  d.n0 = n0; d.n1 = n1; d.n2 = n2;
  d.ip = dupload(ip);
  if (!im.empty()) d.im = dupload(im);
  d.px = make_plan(n0);
  d.py = make_plan(n1);
  d.pz = make_plan(n2);
  const int n[3] = {n0, n1, n2};
  for (int a = 0; a < 3; a++) {
    std::vector<double2> t = twiddle_table(n[a]);
    d.tw[a] = dalloc<double2>(n[a]);
    h2d_sync(d.tw[a], t.data(), n[a] * sizeof(double2));
  }
}

// FourierTransform::backward (src/FourierTransform.cpp:159-200): one band
// (c2 == nullptr) or the pair c1 + i c2 (real basis) from the basis to the
// complex grid, unscaled synthesis
void basis_ft_backward(Context& ctx, const DeviceSticks& d, int ng, bool real_basis,
                       const double* c1, const double* c2, double* grid) {
  const size_t N = (size_t)d.n0 * d.n1 * d.n2;
  QBX_CUDA(cudaMemsetAsync(grid, 0, N * sizeof(double2), ctx.stream));
  if (!real_basis) {
    k_scatter_plus<<<nblk(ng), 256, 0, ctx.stream>>>((const double2*)c1, d.ip, ng,
                                                     (double2*)grid);
  } else if (c2) {
    k_scatter_pair<<<nblk(ng), 256, 0, ctx.stream>>>((const double2*)c1, (const double2*)c2, d.ip,
                                                     d.im, ng, (double2*)grid);
  } else {
    k_scatter_sphere<<<nblk(ng), 256, 0, ctx.stream>>>((const double2*)c1, d.ip, d.im, ng,
                                                       (double2*)grid);
  }
  QBX_LAUNCHED(ctx);
  grid_fft_on(ctx, d, (double2*)grid, +1);
}

// FourierTransform::forward (src/FourierTransform.cpp:147-196): the grid is
// transformed in place (the reference also overwrites f), scaled by 1/N and
// gathered onto the basis; with c2 the two real functions are unpacked
void basis_ft_forward(Context& ctx, const DeviceSticks& d, int ng, bool real_basis, double* grid,
                      double* c1, double* c2) {
  const size_t N = (size_t)d.n0 * d.n1 * d.n2;
  grid_fft_on(ctx, d, (double2*)grid, -1);
  const double scale = 1.0 / (double)N;
  if (c2) {
    QBX_REQUIRE(real_basis, 1, "the two-band forward transform needs a real basis");
    k_gather_pair<<<nblk(ng), 256, 0, ctx.stream>>>((const double2*)grid, d.ip, d.im, ng, scale,
                                                    (double2*)c1, (double2*)c2);
  } else {
    k_gather_sphere<<<nblk(ng), 256, 0, ctx.stream>>>((const double2*)grid, d.ip, ng, scale,
                                                      (double2*)c1);
  }
  QBX_LAUNCHED(ctx);
}

// ------------------------------------------- transforms of the density basis
// One complex FP64 transform of one or two real fields between the density
// sphere and the context's grids.  Kept z fastest, they run as the line
// passes of fft_pencil.cuh on the density sphere's sticks: three kernels that
// read the coefficients and write the fields, in place of a cleared grid, a
// scatter, three in-place passes over the whole grid and an extraction.  With
// the GGA's last two fields packed into one transform, update_vhxc takes (ms)
// 0.45 -> 0.22 at 84^3 and 1.24 -> 0.57 at 140^3, PBE; what is left there is
// the latency of some twenty short kernels, and at 140^3 HBM.
// Two transforms (the GGA's three gradient components) go through as two slots of
// the same launches.
static void field_passes(Context& ctx, pen::Args& a, int nslots, bool back) {
  ProfScope ps(ctx, "grid_fft");
  const DeviceSticks& g = ctx.dvs;
  a.g = g;
  for (int i = 0; i < 3; i++) a.tw[i] = g.tw[i];
  a.ngw = ctx.vb.ng;
  a.nslots = a.chunks = nslots;
  a.sticks = ctx.d_zfast;
  a.tile = (double2*)ctx.d_zfast + (size_t)nslots * g.nvec * g.n2;
  a.stream = ctx.stream;
  const int order[3] = {back ? pen::GZB : pen::GXG, back ? pen::GYB : pen::GYF,
                        back ? pen::GXR : pen::GZF};
  const int n[3] = {back ? g.n2 : g.n0, g.n1, back ? g.n0 : g.n2};
  for (int i = 0; i < 3; i++) {
    a.op = order[i];
    QBX_REQUIRE(pencil_run<double>(ctx, n[i], a), 21, "no line kernel of this length");
  }
}
// f0 = Re (+ add), f1 = Im (+ the new f0 with `chain`) of the transform of
// c0 + i c1 (c1, f1 may be null)
static void fields_backward(Context& ctx, const double* c0, const double* c1, double* f0,
                            double* f1, const double* add, bool chain) {
  pen::Args a;
  a.gc[0] = (double2*)c0;
  a.gc[1] = (double2*)c1;
  a.gf[0] = f0;
  a.gf[1] = f1;
  a.fadd = add;
  a.chain = chain;
  field_passes(ctx, a, 1, true);
}
static void fields_forward(Context& ctx, const double* f0, const double* f1, const double* mul,
                           double scale, double* c0, double* c1) {
  pen::Args a;
  a.gf[0] = (double*)f0;
  a.gf[1] = (double*)f1;
  a.fmul = mul;
  a.scale = scale / (double)ctx.N();
  a.gc[0] = (double2*)c0;
  a.gc[1] = (double2*)c1;
  field_passes(ctx, a, 1, false);
}

void vb_backward(Context& ctx, const double* coef, double* real_out) {
  if (ctx.grid_zfast) return fields_backward(ctx, coef, nullptr, real_out, nullptr, nullptr, false);
  const size_t N = ctx.N();
  QBX_CUDA(cudaMemsetAsync(ctx.d_grid, 0, N * sizeof(double2), ctx.stream));
  k_scatter_sphere<<<nblk(ctx.vb.ng), 256, 0, ctx.stream>>>((const double2*)coef, ctx.dvs.ip,
                                                            ctx.dvs.im, ctx.vb.ng, (double2*)ctx.d_grid);
  QBX_LAUNCHED(ctx);
  grid_fft(ctx, +1);
  k_grid_real<<<nblk(N), 256, 0, ctx.stream>>>((const double2*)ctx.d_grid, N, real_out);
  QBX_LAUNCHED(ctx);
}

void vb_backward_pair(Context& ctx, const double* a, const double* b, double* out0, double* out1) {
  if (ctx.grid_zfast) return fields_backward(ctx, a, b, out0, out1, nullptr, false);
  const size_t N = ctx.N();
  QBX_CUDA(cudaMemsetAsync(ctx.d_grid, 0, N * sizeof(double2), ctx.stream));
  k_scatter_pair<<<nblk(ctx.vb.ng), 256, 0, ctx.stream>>>((const double2*)a, (const double2*)b,
                                                          ctx.dvs.ip, ctx.dvs.im, ctx.vb.ng,
                                                          (double2*)ctx.d_grid);
  QBX_LAUNCHED(ctx);
  grid_fft(ctx, +1);
  k_grid_split<<<nblk(N), 256, 0, ctx.stream>>>((const double2*)ctx.d_grid, N, out0, out1);
  QBX_LAUNCHED(ctx);
}

void vb_forward_real_pair(Context& ctx, const double* f0, const double* f1, const double* w,
                          double* c0, double* c1) {
  if (ctx.grid_zfast) return fields_forward(ctx, f0, f1, w, 1.0, c0, c1);
  const size_t N = ctx.N();
  k_real2_mul_to_grid<<<nblk(N), 256, 0, ctx.stream>>>(f0, f1, w, N, (double2*)ctx.d_grid);
  QBX_LAUNCHED(ctx);
  grid_fft(ctx, -1);
  if (f1) {
    k_gather_pair<<<nblk(ctx.vb.ng), 256, 0, ctx.stream>>>((const double2*)ctx.d_grid, ctx.dvs.ip,
                                                           ctx.dvs.im, ctx.vb.ng, 1.0 / (double)N,
                                                           (double2*)c0, (double2*)c1);
  } else {
    k_gather_sphere<<<nblk(ctx.vb.ng), 256, 0, ctx.stream>>>((const double2*)ctx.d_grid, ctx.dvs.ip,
                                                             ctx.vb.ng, 1.0 / (double)N,
                                                             (double2*)c0);
  }
  QBX_LAUNCHED(ctx);
}

void vb_forward_real(Context& ctx, const double* f, double scale, double* coef) {
  if (ctx.grid_zfast) return fields_forward(ctx, f, nullptr, nullptr, scale, coef, nullptr);
  const size_t N = ctx.N();
  k_real_to_grid<<<nblk(N), 256, 0, ctx.stream>>>(f, scale, N, (double2*)ctx.d_grid);
  QBX_LAUNCHED(ctx);
  grid_fft(ctx, -1);
  k_gather_sphere<<<nblk(ctx.vb.ng), 256, 0, ctx.stream>>>((const double2*)ctx.d_grid, ctx.dvs.ip,
                                                           ctx.vb.ng, 1.0 / (double)N, (double2*)coef);
  QBX_LAUNCHED(ctx);
}

// two slots of the density basis fit the stick buffer
static bool two_field_slots(const Context& ctx) {
  const DeviceSticks& g = ctx.dvs;
  return ctx.grid_zfast && ctx.zfast_bytes >= 2 * sizeof(double2) * (size_t)g.n2 *
                                                  ((size_t)g.nvec + (size_t)g.ncol * g.n1);
}
// three real fields f, f + N, f + 2 N of the coefficients c[0], c[1], c[2], and
// the coefficients of the three fields times w
void vb_backward3(Context& ctx, double* const c[3], double* f) {
  const size_t N = ctx.N();
  if (!two_field_slots(ctx)) {
    vb_backward_pair(ctx, c[0], c[1], f, f + N);
    vb_backward(ctx, c[2], f + 2 * N);
    return;
  }
  pen::Args a;
  for (int j = 0; j < 3; j++) {
    a.gc[j] = (double2*)c[j];
    a.gf[j] = f + j * N;
  }
  field_passes(ctx, a, 2, true);
}
void vb_forward_real3(Context& ctx, const double* f, const double* w, double* const c[3]) {
  const size_t N = ctx.N();
  if (!two_field_slots(ctx)) {
    vb_forward_real_pair(ctx, f, f + N, w, c[0], c[1]);
    vb_forward_real_pair(ctx, f + 2 * N, nullptr, w, c[2], nullptr);
    return;
  }
  pen::Args a;
  for (int j = 0; j < 3; j++) {
    a.gc[j] = (double2*)c[j];
    a.gf[j] = (double*)f + j * N;
  }
  a.fmul = w;
  a.scale = 1.0 / (double)N;
  field_passes(ctx, a, 2, false);
}

// out0 = add + back(a) and, with b, out1 = out0 + back(b): the sums over the
// grid that follow a transform, in its last pass where the line passes run.
// Without b, out0 is not add and d_exc keeps its contents (the LDA's energy
// density, which the stress reads later); with b, d_exc is scratch.
void vb_backward_add(Context& ctx, const double* a, const double* b, const double* add,
                     double* out0, double* out1) {
  if (ctx.grid_zfast) return fields_backward(ctx, a, b, out0, out1, add, b != nullptr);
  const size_t N = ctx.N();
  if (!b) {
    vb_backward(ctx, a, out0);
    k_add<<<nblk(N), 256, 0, ctx.stream>>>(add, out0, N, out0);
    QBX_LAUNCHED(ctx);
    return;
  }
  vb_backward_pair(ctx, a, b, ctx.d_exc, out1);
  k_add<<<nblk(N), 256, 0, ctx.stream>>>(add, ctx.d_exc, N, out0);
  QBX_LAUNCHED(ctx);
  k_add<<<nblk(N), 256, 0, ctx.stream>>>(out0, out1, N, out1);
  QBX_LAUNCHED(ctx);
}

void wb_backward_pair(Context& ctx, const double* c1, const double* c2, double* grid_out) {
  const size_t N = ctx.N();
  QBX_CUDA(cudaMemsetAsync(ctx.d_grid, 0, N * sizeof(double2), ctx.stream));
  k_scatter_pair<<<nblk(ctx.wb.ng), 256, 0, ctx.stream>>>((const double2*)c1, (const double2*)c2,
                                                          ctx.dws.ip, ctx.dws.im, ctx.wb.ng,
                                                          (double2*)ctx.d_grid);
  QBX_LAUNCHED(ctx);
  grid_fft(ctx, +1);
  QBX_CUDA(cudaMemcpyAsync(grid_out, ctx.d_grid, N * sizeof(double2), cudaMemcpyDeviceToDevice,
                           ctx.stream));
}

}  // namespace qbx

namespace qbx {

// Density of nst bands of c (device, default order) added into rho, with the
// stick buffer and the three twiddle tables supplied by the caller instead
// of the context's own.  Batches of band pairs are sized to zbuf_bytes.
template <typename T>
static void density_buffers_t(Context& ctx, const double* c, int nst, const double* w,
                              double* rho, void* zbuf, size_t zbuf_bytes, const double2* twx,
                              const double2* twy, const double2* twz) {
  using C = typename Cplx<T>::t;
  const DeviceSticks& g = ctx.dws;
  cudaStream_t st = ctx.stream;
  const size_t per_pair = sizeof(C) * (size_t)g.n2 * g.nvec;
  const int npairs_all = (nst + 1) / 2;
  const int batch = (int)std::min<size_t>(npairs_all, zbuf_bytes / per_pair);
  QBX_REQUIRE(batch >= 1, 60, "stick buffer smaller than one band pair");
  const size_t zs = zsmem<T>(g.n2);
  allow_smem(k_zfft_bwd<T>, zs);
  XYConfig<T> xc = xy_config<T>(g, ctx.device);
  allow_smem(k_xy<T, OP_DENSITY>, xc.smem);
  int sms = 0;
  QBX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
  for (int p0 = 0; p0 < npairs_all; p0 += batch) {
    const int npairs = std::min(batch, npairs_all - p0);
    dim3 zgrid((g.nrods + kRodsPerCta - 1) / kRodsPerCta, npairs);
    k_zfft_bwd<T><<<zgrid, 256, zs, st>>>((const double2*)c, ctx.wb.ng, nst, p0, g, twz, (C*)zbuf,
                                           kRodsPerCta);
    QBX_LAUNCHED(ctx);
    int chunks = std::max(1, (3 * sms + g.n2 - 1) / g.n2);
    chunks = std::min(chunks, npairs);
    const int ppc = (npairs + chunks - 1) / chunks;
    chunks = (npairs + ppc - 1) / ppc;
    dim3 xgrid(g.n2, chunks);
    k_xy<T, OP_DENSITY><<<xgrid, 512, xc.smem, st>>>((C*)zbuf, npairs, ppc, g, twx, twy, nullptr,
                                                     rho, w, p0, nst, xc.cc, xc.rr);
    QBX_LAUNCHED(ctx);
  }
}

size_t density_stick_bytes_per_pair(const Context& ctx) {
  const size_t e = ctx.precision == MIXED ? sizeof(float2) : sizeof(double2);
  return e * (size_t)ctx.dws.n2 * ctx.dws.nvec;
}

void density_with_buffers(Context& ctx, const double* c, int nst, const double* w, double* rho,
                          void* zbuf, size_t zbuf_bytes, const double2* twx, const double2* twy,
                          const double2* twz) {
  if (ctx.precision == MIXED)
    density_buffers_t<float>(ctx, c, nst, w, rho, zbuf, zbuf_bytes, twx, twy, twz);
  else
    density_buffers_t<double>(ctx, c, nst, w, rho, zbuf, zbuf_bytes, twx, twy, twz);
}

}  // namespace qbx

namespace qbx {

// ------------------------------------------------------------ autotuner
// Times H psi and the density of this context's wavefunctions and names the
// kernels that run them: the line passes (fft_pencil.cuh), whose shapes are
// fixed per length at compile time, or the runtime-radix kernels on grids of
// other lengths (the passes were the faster on every grid that has both).
// The timings are appended to `log`.
std::string autotune_fft(Context& ctx, std::vector<std::pair<std::string, double>>* log) {
  QBX_REQUIRE(ctx.have_cell && ctx.d_zfast, 7, "autotune needs a cell");
  double* rho_tmp = dalloc<double>(ctx.N());
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  auto release = [&]() {
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
    dfree(rho_tmp);
  };
  try {
    for (cudaEvent_t& e : ev) QBX_CUDA(cudaEventCreate(&e));
    float ms[2] = {0.f, 0.f};
    for (int rep = 0; rep < 2; rep++) {   // the first pass warms up
      QBX_CUDA(cudaEventRecord(ev[0], ctx.stream));
      launch_vpsi(ctx, ctx.d_c, ctx.d_vr, ctx.d_ctmp);
      QBX_CUDA(cudaEventRecord(ev[1], ctx.stream));
      launch_density(ctx, ctx.d_c, rho_tmp);
      QBX_CUDA(cudaEventRecord(ev[2], ctx.stream));
      QBX_CUDA(cudaEventSynchronize(ev[2]));
      for (int i = 0; i < 2; i++) QBX_CUDA(cudaEventElapsedTime(&ms[i], ev[i], ev[i + 1]));
    }
    if (log) {
      log->push_back({"H psi", ms[0]});
      log->push_back({"density", ms[1]});
    }
  } catch (...) {
    release();
    throw;
  }
  release();
  return pencil_ok(ctx, ctx.dws, ctx.precision == MIXED) ? "line passes" : "runtime-radix kernels";
}

}  // namespace qbx
