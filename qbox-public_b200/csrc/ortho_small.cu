// The n x n algebra of SlaterDet::ortho_align and DoubleMatrix::polar for up to
// 128 bands as one kernel on one cluster of CTAs.
//
// At these sizes the Cholesky factor, its inverse, the polar iteration and the
// products around them are a chain of some forty library and pointwise kernels
// of 3 to 70 us each, all latency (cuSOLVER's potrf takes 16 us at n = 16 and
// 70 us at 128, each polar iteration some ten launches inside a conditional
// graph node).  Here a cluster of ceil(n/16) CTAs (at most 8, one column panel
// of 16 each) runs the whole chain: every matrix product is one pass of FP64
// tensor-core MMAs (m8n8k4) with the left operand in shared memory, the results
// go through L2, and a cluster barrier separates the steps.  Cholesky factor and
// inverse are computed by every CTA for itself in shared memory, so that they
// need no barrier.  Everything is FP64.
//
//   ortho:  S = L L^T (lower triangle given), T = L^-1 B, T <- polar(T),
//           X = L^-T T, and I - X for the mixed path's rotation
//   polar:  X <- polar(X)
//
// What bounds it: the serial chain of pivots in the Cholesky factor (one warp per
// 16 x 16 diagonal block, its rows in registers: 95 of 155 us at 128 bands before
// every index of them was a compile-time one), then the latency of a product's
// operand copy from L2 and of the cluster barriers.  16 bands 22 us, 128 bands 109
// us; psda_update of the eager step (ms) at 16 bands FP64 0.38 -> 0.13, 97 bands
// mixed 0.60 -> 0.30, 128 bands mixed 0.63 -> 0.38 (FP64 with the whole-product
// overlap 0.92 -> 0.40).  The limit of 128 is one matrix in a CTA's shared
// memory and eight panels in a portable cluster.
#include <cstdint>
#include <type_traits>

#include "qbx_internal.h"

namespace qbx {

namespace {

constexpr int kMax = 128;          // bands
constexpr int P = 132;             // pitch of a column in shared memory: = 4 mod 16, so
                                   // that the MMA fragments read without bank conflicts
constexpr int kThreads = 256;      // 8 warps, 16 rows of a product each
constexpr int kMat = P * kMax;     // one matrix
constexpr int kPanel = P * 16;     // one column panel
constexpr size_t kSmem = sizeof(double) * (kMat + 2 * kPanel + 16 * 20 + 64);

struct SmallArgs {
  int n = 0;
  const double* S = nullptr;     // overlap, lower triangle (ortho)
  const double* B = nullptr;     // C^T C_last (ortho) or x (polar)
  double* X = nullptr;           // result
  double* IX = nullptr;          // I - X (may be null)
  double* work = nullptr;        // ortho_small_elems(n)
  double tol = 0;
  int maxiter = 0;
  bool ortho = false;
  bool chol_higham = false;      // Higham step from the Cholesky factor of x^T x (mixed
                                 // path), else from a pivoted elimination of x
  int* status = nullptr;         // status words
  int info_s = 0;                // the word of the overlap's factorisation
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// n x n matrix (ld n) into shared memory [column][row], zeros to np x np
__device__ void load_matrix(double* s, const double* g, int n, int np) {
  const int r = threadIdx.x & (kMax - 1);
  if (r >= np) return;
#pragma unroll 8
  for (int c = threadIdx.x / kMax; c < np; c += kThreads / kMax)
    s[c * P + r] = (r < n && c < n) ? __ldcg(g + (size_t)c * n + r) : 0.0;
}

// a working matrix (ld np, a multiple of 16) into shared memory: 16-byte copies
// all in flight at once; complete after copy_wait and a barrier
__device__ __forceinline__ void copy_matrix(double* s, const double* g, int np) {
  const int half = np / 2;                       // 16-byte pieces of a column
  const int per = kThreads / 64;                 // columns at a time, 64 threads each
  const int i = threadIdx.x & 63;
  if (i >= half) return;
  for (int c = threadIdx.x >> 6; c < np; c += per) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(s + c * P + 2 * i);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(g + (size_t)c * np + 2 * i)
                 : "memory");
  }
}
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// c(16 rows of this warp x 16 columns) += op(A)(rows, 0:kk) B(0:kk, panel), A
// [column][row] with op(A)(m, k) = TA ? A(k, m) : A(m, k), B a panel
// [column][row]; rows beyond np are not computed
template <bool TA>
__device__ __forceinline__ void warp_mm(const double* A, const double* B, int row0, int kk,
                                        double (&c)[2][2][2]) {
  const int lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
  for (int k = 0; k < kk; k += 4) {
    double a[2], b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int m = row0 + 8 * i + lr;
      a[i] = TA ? A[m * P + k + lk] : A[(k + lk) * P + m];
      b[i] = B[(8 * i + lr) * P + k + lk];
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) dmma(c[i][j], a[i], b[j]);
  }
}

// every entry (row, col) of the warp's 16 x 16 block
template <typename F> __device__ __forceinline__ void each(double (&c)[2][2][2], int row0, F f) {
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = 2 * (lane & 3);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) f(row0 + 8 * i + lr, 8 * j + lc + h, c[i][j][h]);
}

// f(row, panel column, value) of op(A) B for this CTA's column panel B [column][row]
template <bool TA, typename F>
__device__ __forceinline__ void panel_mm(const double* A, const double* B, int np, F f) {
  const int row0 = 16 * (threadIdx.x >> 5);
  if (row0 < np) {
    double c[2][2][2] = {};
    warp_mm<TA>(A, B, row0, np, c);
    each(c, row0, f);
  }
}

// f(0) ... f(E - 1) with compile-time indices (rows held in registers)
template <int I, int E, typename F> __device__ __forceinline__ void unroll(const F& f) {
  if constexpr (I < E) {
    f(std::integral_constant<int, I>{});
    unroll<I + 1, E>(f);
  }
}

// 1/sqrt(d) for a pivot: an FP32 estimate and two Newton steps y += y (1 - d y^2)/2,
// each doubling its 23 bits (the pivots form one serial chain, where the library
// function's handling of every exponent costs as much again); pivots beyond the
// FP32 range take the library function.
__device__ __forceinline__ double pivot_rsqrt(double d) {
  if (!(d > 1e-30 && d < 1e30)) return rsqrt(d);
  double y = (double)rsqrtf((float)d);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double e = fma(-d * y, y, 1.0);
    y = fma(0.5 * y, e, y);
  }
  return y;
}

// A (np x np in shared memory, lower triangle of an SPD matrix) <- inverse of
// its Cholesky factor, strictly upper triangle zero.  16-column panels: the
// diagonal block by one warp, the rest by MMAs.  Returns 0, or the order of the
// first pivot that is not positive (the factorisation then goes on with 1).
__device__ int cholesky_inverse(double* A, double* tmp, double* dia, int np, double* flag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) flag[0] = 0.0;
  __syncthreads();
  for (int p = 0; p < np; p += 16) {
    // diagonal block: L11 in place and its inverse in dia [row * 20 + col]
    if (warp == 0) {
      const int i = lane & 15;
      double row[16], inv = 0.0;   // row i of the block, 1 / L_ii
#pragma unroll
      for (int k = 0; k < 16; ++k) row[k] = A[(p + k) * P + p + i];
      unroll<0, 16>([&](auto j) {
        double d = __shfl_sync(0xffffffffu, row[j], j);
        if (!(d > 0.0)) {
          if (lane == 0 && flag[0] == 0.0) flag[0] = p + j + 1;
          d = 1.0;
        }
        const double si = pivot_rsqrt(d);
        if (i == j) inv = si;
        row[j] = i == j ? d * si : row[j] * si;
        unroll<decltype(j)::value + 1, 16>([&](auto k) {
          const double l = __shfl_sync(0xffffffffu, row[j], k);
          if (i >= k) row[k] -= row[j] * l;
        });
      });
      __syncwarp();
      if (lane < 16) {
#pragma unroll
        for (int k = 0; k < 16; ++k) A[(p + k) * P + p + i] = k <= i ? row[k] : 0.0;
      }
      __syncwarp();
      // column i of the inverse by forward substitution, each x_r taken out of
      // all later rows at once
      double x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r] = r == i ? 1.0 : 0.0;
      unroll<0, 16>([&](auto r) {
        x[r] *= __shfl_sync(0xffffffffu, inv, r);
        unroll<decltype(r)::value + 1, 16>([&](auto k) { x[k] -= A[(p + r) * P + p + k] * x[r]; });
      });
      __syncwarp();
      if (lane < 16) {
#pragma unroll
        for (int r = 0; r < 16; ++r) dia[r * 20 + i] = x[r];
      }
    }
    __syncthreads();
    // L21 = A21 L11^-T in place, 16 rows a warp; the inverse block waits in place
    // of L11
    const int below = np - p - 16;
    const int lr = lane >> 2, lk = lane & 3, lc = 2 * lk;
    if (16 * warp < below) {
      double c[2][2][2] = {};
      const int r0 = p + 16 + 16 * warp;
#pragma unroll
      for (int k = 0; k < 16; k += 4) {
        double a[2], b[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          a[h] = A[(p + k + lk) * P + r0 + 8 * h + lr];
          b[h] = dia[(8 * h + lr) * 20 + k + lk];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int g = 0; g < 2; ++g) dmma(c[h][g], a[h], b[g]);
      }
      __syncwarp();
      each(c, r0, [&](int r, int cc, double v) { A[(p + cc) * P + r] = v; });
    }
    {
      const int c = threadIdx.x >> 4, r = threadIdx.x & 15;
      A[(p + c) * P + p + r] = r >= c ? dia[r * 20 + c] : 0.0;
    }
    __syncthreads();
    // A22 -= L21 L21^T, lower 8 x 8 tiles
    const int nt = below / 8;
    for (int t = warp; t < nt * nt; t += 8) {
      const int ti = t / nt, tj = t - ti * nt;
      if (tj > ti) continue;
      const int r0 = p + 16 + 8 * ti, q0 = p + 16 + 8 * tj;
      double c[2] = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 16; k += 4)
        dmma(c, A[(p + k + lk) * P + r0 + lr], A[(p + k + lk) * P + q0 + lr]);
      A[(q0 + lc) * P + r0 + lr] -= c[0];
      A[(q0 + lc + 1) * P + r0 + lr] -= c[1];
    }
    __syncthreads();
  }
  // in-place inverse, last block column first: with Li = L^-1 of the trailing
  // blocks in place, the column below block p is -Li L21 L11^-1
  for (int p = np - 32; p >= 0; p -= 16) {
    const int below = np - p - 16;
    const int row0 = 16 * warp;
    double d[2][2][2] = {};
    if (row0 < below) {
      double c[2][2][2] = {};
      warp_mm<false>(A + (p + 16) * P + p + 16, A + p * P + p + 16, row0, row0 + 16, c);
      each(c, row0, [&](int r, int cc, double v) { tmp[cc * P + r] = -v; });
      __syncwarp();
      warp_mm<false>(tmp, A + p * P + p, row0, 16, d);
    }
    __syncthreads();                 // every warp has read the old column block
    if (row0 < below)
      each(d, row0, [&](int r, int cc, double v) { A[(p + cc) * P + p + 16 + r] = v; });
    __syncthreads();
  }
  const int zr = threadIdx.x & (kMax - 1);
  for (int c = threadIdx.x / kMax; c < np; c += kThreads / kMax)
    if (zr < c) A[c * P + zr] = 0.0;
  __syncthreads();
  return (int)flag[0];
}

// A (np x np in shared memory) <- its inverse by Gauss-Jordan elimination with
// row pivoting, in place; perm: np ints.  Returns 0 or the order of a zero
// pivot.
__device__ int gauss_inverse(double* A, double* colbuf, int* perm, double* flag, int np) {
  const int lane = threadIdx.x & 31;
  int bad = 0;
  for (int k = 0; k < np; ++k) {
    if (threadIdx.x < 32) {
      double best = -1.0;
      int at = k;
      for (int r = k + lane; r < np; r += 32) {
        const double v = fabs(A[k * P + r]);
        if (v > best) { best = v; at = r; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double b = __shfl_down_sync(0xffffffffu, best, o);
        const int i = __shfl_down_sync(0xffffffffu, at, o);
        if (b > best) { best = b; at = i; }
      }
      if (lane == 0) {
        perm[k] = at;
        flag[0] = best > 0.0 ? 0.0 : 1.0;
      }
    }
    __syncthreads();
    const int pr = perm[k];
    if (flag[0] != 0.0 && !bad) bad = k + 1;
    if (pr != k && threadIdx.x < np) {
      const double a = A[threadIdx.x * P + k];
      A[threadIdx.x * P + k] = A[threadIdx.x * P + pr];
      A[threadIdx.x * P + pr] = a;
    }
    __syncthreads();
    const double inv = 1.0 / (bad ? 1.0 : A[k * P + k]);
    if (threadIdx.x < np) colbuf[threadIdx.x] = A[k * P + threadIdx.x];
    __syncthreads();
    // row k scaled, the others eliminated; column k becomes the inverse's
    const int r = threadIdx.x & (kMax - 1);
    if (r < np && r != k) {
      const double m = -colbuf[r] * inv;
#pragma unroll 8
      for (int c = threadIdx.x / kMax; c < np; c += kThreads / kMax)
        A[c * P + r] = c == k ? m : A[c * P + r] + m * A[c * P + k];
    }
    __syncthreads();
    if (threadIdx.x < np)
      A[threadIdx.x * P + k] = ((int)threadIdx.x == k ? 1.0 : A[threadIdx.x * P + k]) * inv;
    __syncthreads();
  }
  // undo the row interchanges on the columns, last first
  for (int k = np - 1; k >= 0; --k) {
    const int pr = perm[k];
    if (pr != k && threadIdx.x < np) {
      const double a = A[k * P + threadIdx.x];
      A[k * P + threadIdx.x] = A[pr * P + threadIdx.x];
      A[pr * P + threadIdx.x] = a;
    }
    __syncthreads();
  }
  return bad;
}

__global__ void __launch_bounds__(kThreads, 1) k_ortho_small(SmallArgs a) {
  extern __shared__ __align__(16) double sm[];
  double* M = sm;                 // one matrix
  double* bp = M + kMat;          // a panel: this CTA's columns of x, then of y
  double* tmp = bp + kPanel;      // another: its columns of q
  double* dia = tmp + kPanel;
  double* flag = dia + 16 * 20;   // 64 doubles: a flag, block sums
  const int n = a.n, np = (n + 15) / 16 * 16;
  const int rank = blockIdx.x, size = gridDim.x, c0 = 16 * rank;
  const size_t nn = (size_t)np * np;
  // working matrices, ld np: the padding is zero in x and y
  double* x = a.work;             // the polar iterate and its successor
  double* y = a.work + nn;
  double* q = a.work + 2 * nn;
  double* z = a.work + 3 * nn;
  double* li = a.work + 4 * nn;
  double* sums = a.work + 5 * nn;
  const bool first = rank == 0 && threadIdx.x == 0;
  const int pr = threadIdx.x & (kMax - 1), pc = threadIdx.x / kMax;   // panel loops
  // this CTA's columns of B
  if (pr < np) {
#pragma unroll
    for (int c = pc; c < 16; c += kThreads / kMax)
      bp[c * P + pr] = (pr < n && c0 + c < n) ? a.B[(size_t)(c0 + c) * n + pr] : 0.0;
  }
  if (a.ortho) {
    load_matrix(M, a.S, n, np);
    __syncthreads();
    if (threadIdx.x >= n && threadIdx.x < np) M[threadIdx.x * P + threadIdx.x] = 1.0;
    __syncthreads();
    const int bad = cholesky_inverse(M, tmp, dia, np, flag);
    if (first) a.status[a.info_s] = bad;
    if (rank == 0 && pr < np)
      for (int c = pc; c < np; c += kThreads / kMax) li[(size_t)c * np + pr] = M[c * P + pr];
    // T = L^-1 B, the first iterate
    panel_mm<false>(M, bp, np, [&](int r, int c, double v) { tmp[c * P + r] = v; });
    __syncthreads();
    if (pr < np) {
#pragma unroll
      for (int c = pc; c < 16; c += kThreads / kMax) bp[c * P + pr] = tmp[c * P + pr];
    }
  }
  __syncthreads();
  if (pr < np) {
#pragma unroll
    for (int c = pc; c < 16; c += kThreads / kMax) x[(size_t)(c0 + c) * np + pr] = bp[c * P + pr];
  }
  cluster_sync();
  int iters = 0, info = 0;
  for (int it = 0; it < a.maxiter; ++it) {
    copy_matrix(M, x, np);
    copy_wait();
    __syncthreads();
    // the columns of q = I - x^T x, their squared norm, and z = x q
    double s = 0.0;
    panel_mm<true>(M, bp, np, [&](int r, int c, double v) {
      const double d = (r == c0 + c && r < n ? 1.0 : 0.0) - v;
      tmp[c * P + r] = d;
      s += d * d;
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) flag[8 + (threadIdx.x >> 5)] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double v = 0.0;
      for (int w = 0; w < kThreads / 32; ++w) v += flag[8 + w];
      sums[rank] = v;
    }
    panel_mm<false>(M, tmp, np, [&](int r, int c, double v) { z[(size_t)(c0 + c) * np + r] = v; });
    if (a.chol_higham && pr < np) {
#pragma unroll
      for (int c = pc; c < 16; c += kThreads / kMax) q[(size_t)(c0 + c) * np + pr] = tmp[c * P + pr];
    }
    cluster_sync();
    double norm2 = 0.0;
    for (int i = 0; i < size; ++i) norm2 += __ldcg(sums + i);
    const double qn = sqrt(norm2);
    iters = it + 1;
    if (qn < 1.0) {
      // y = x (I + q/2 + 3 q^2/8) = x + z/2 + 3/8 z q
      copy_matrix(M, z, np);
      copy_wait();
      __syncthreads();
      panel_mm<false>(M, tmp, np, [&](int r, int c, double v) {
        bp[c * P + r] += 0.5 * M[(c0 + c) * P + r] + 0.375 * v;
      });
    } else if (a.chol_higham) {
      // y = x (I + (x^T x)^-1) / 2 with x^T x = I - q
      copy_matrix(M, q, np);
      copy_wait();
      __syncthreads();
      if (pr < np)
        for (int c = pc; c < np; c += kThreads / kMax)
          M[c * P + pr] = (pr == c ? 1.0 : 0.0) - M[c * P + pr];
      __syncthreads();
      const int bad = cholesky_inverse(M, tmp, dia, np, flag);
      if (bad) info = bad;
      // W^T times this CTA's columns of W = M, then x times that
      panel_mm<true>(M, M + c0 * P, np, [&](int r, int c, double v) {
        tmp[c * P + r] = 0.5 * ((r == c0 + c ? 1.0 : 0.0) + v);
      });
      __syncthreads();
      copy_matrix(M, x, np);
      copy_wait();
      __syncthreads();
      panel_mm<false>(M, tmp, np, [&](int r, int c, double v) { bp[c * P + r] = v; });
    } else {
      // y = (x + x^-T) / 2
      copy_matrix(M, x, np);
      copy_wait();
      __syncthreads();
      if (threadIdx.x >= n && threadIdx.x < np) M[threadIdx.x * P + threadIdx.x] = 1.0;
      __syncthreads();
      const int bad = gauss_inverse(M, tmp, (int*)(tmp + 256), flag, np);
      if (bad) info = bad;
      if (pr < n) {
#pragma unroll
        for (int c = pc; c < 16; c += kThreads / kMax)
          if (c0 + c < n) bp[c * P + pr] = 0.5 * (bp[c * P + pr] + M[pr * P + c0 + c]);
      }
    }
    __syncthreads();
    if (pr < np) {
#pragma unroll
      for (int c = pc; c < 16; c += kThreads / kMax) y[(size_t)(c0 + c) * np + pr] = bp[c * P + pr];
    }
    cluster_sync();
    double* t = x;
    x = y;
    y = t;
    if (qn <= a.tol) break;
  }
  if (a.ortho) {
    copy_matrix(M, li, np);
    copy_wait();
    __syncthreads();
    panel_mm<true>(M, bp, np, [&](int r, int c, double v) {
      if (r >= n || c0 + c >= n) return;
      const size_t i = (size_t)(c0 + c) * n + r;
      a.X[i] = v;
      if (a.IX) a.IX[i] = (r == c0 + c ? 1.0 : 0.0) - v;
    });
  } else if (pr < n) {
#pragma unroll
    for (int c = pc; c < 16; c += kThreads / kMax)
      if (c0 + c < n) a.X[(size_t)(c0 + c) * n + pr] = bp[c * P + pr];
  }
  if (first) {
    a.status[ST_POLAR_ITERS] = iters;
    a.status[ST_INFO_POLAR] = info;
  }
}

void launch(Context& ctx, const SmallArgs& a) {
  allow_smem(k_ortho_small, kSmem);
  cudaLaunchConfig_t cfg = {};
  const int ctas = (a.n + 15) / 16;
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  QBX_CUDA(cudaLaunchKernelEx(&cfg, k_ortho_small, a));
  QBX_LAUNCHED(ctx);
}

}  // namespace

bool ortho_small_ok(const Context& ctx) { return ctx.nst <= kMax && ctx.d_small && ctx.ortho_small; }

size_t ortho_small_elems(int n) {
  const size_t np = (n + 15) / 16 * 16;
  return n <= kMax ? 5 * np * np + 16 : 0;
}

// X = L^-T polar(L^-1 B) with S = L L^T (lower triangle of S given, info code in
// status word `info`); with IX also I - X
void ortho_small(Context& ctx, const double* S, const double* B, double* X, double* IX, int info) {
  SmallArgs a;
  a.n = ctx.nst;
  a.S = S;
  a.B = B;
  a.X = X;
  a.IX = IX;
  a.work = ctx.d_small;
  a.tol = 1.e-6;
  a.maxiter = 20;
  a.ortho = true;
  a.chol_higham = ctx.precision == MIXED;
  a.status = ctx.d_status;
  a.info_s = info;
  launch(ctx, a);
}

// x <- its orthogonal polar factor
void polar_small(Context& ctx, double* x, double tol, int maxiter) {
  SmallArgs a;
  a.n = ctx.nst;
  a.B = x;
  a.X = x;
  a.work = ctx.d_small;
  a.tol = tol;
  a.maxiter = maxiter;
  a.chol_higham = ctx.precision == MIXED;
  a.status = ctx.d_status;
  launch(ctx, a);
}

}  // namespace qbx
