// quadrature.cu -- Gauss quadrature nodes and weights from the Lanczos tridiagonals.
//
// Replaces TridiagEigenVecSolve_NodesAndWeights (src/lsdft_tools.cc:912-1026): implicit QL
// with Wilkinson-type shifts (Numerical Recipes tqli), lambda_q = d[q], w_q = Z[0][q]^2,
// eigenvalues left unsorted, lambda_min / lambda_max by the reference's scan.  The rows of Z
// never mix in tqli, so only row 0 is carried: O(n) storage and O(n^2) work per node with
// results identical to the full-matrix form.
//
// One thread per node, FP64.  The three working arrays of a node (d, e and row 0 of Z, N_qp
// doubles each) live in shared memory, one column per thread (element i of thread t at
// i * blockDim + t): as local arrays the ~250 nodes per SM (1.5 KB each) overflow L1 and every
// rotation waits on L2.
//
// What bounds it is the FP64 pipe (2 lanes per SM and cycle) and, for a few nodes, the chain of
// dependent operations through the rotations.  Every result stays the correctly rounded one of the CPU
// reference (the order in which eigenvalues deflate turns on the last bits), so the products and sums
// are separate, rounded operations; but a rotation takes one reciprocal square root and corrects it
// by Markstein's residual steps to r = sqrt(x), f / r and g / r (IBM J. Res. Dev. 34, 1990) instead of
// a square root and two divisions; the next rotation's elements are loaded ahead; and the deflation
// test looks at the exponents first and does its FP64 comparison only where they leave it open.
#include <cuda_runtime.h>

#include "sq_kernels.hpp"

namespace sq {

namespace {

constexpr int kQuadBlock = 64;

// one thread's column of a shared array: element i at p[i * stride]
struct Col {
  double *p;
  int stride;
  __device__ __forceinline__ double &operator[](int i) const { return p[i * stride]; }
};

// r = sqrt(x), s = f / r, c = g / r, each correctly rounded: an estimate times the reciprocal root
// of x, and its residual against the exact product.  Outside [2^-900, 2^900], where a residual could
// leave the normal range, by the plain operations.
__device__ __forceinline__ double norm_and_quotients(double x, double f, double g, double &s, double &c) {
  const int ex = (__double2hiint(x) >> 20) & 2047;
  if (ex < 1023 - 900 || ex > 1023 + 900) {
    const double r = sqrt(x);
    s = f / r;
    c = g / r;
    return r;
  }
  const double y = rsqrt(x);
  const double r0 = __dmul_rn(x, y);
  const double r = fma(fma(-r0, r0, x), __dmul_rn(0.5, y), r0);
  const double inv = fma(fma(-r, y, 1.0), y, y);  // 1 / r
  const double s0 = __dmul_rn(f, inv), c0 = __dmul_rn(g, inv);
  s = fma(fma(-r, s0, f), inv, s0);
  c = fma(fma(-r, c0, g), inv, c0);
  return r;
}

__device__ __forceinline__ int exponent(double v) { return (__double2hiint(v) >> 20) & 2047; }

__global__ void __launch_bounds__(kQuadBlock)
    quadrature_kernel(const double *__restrict__ ab, long long n, int nqp,
                      double *__restrict__ lambda, double *__restrict__ wts,
                      double *__restrict__ lmin, double *__restrict__ lmax,
                      int *__restrict__ status) {
  extern __shared__ double qsm[];  // [3][nqp][blockDim]
  const Col d{qsm + threadIdx.x, (int)blockDim.x};
  const Col e{qsm + nqp * blockDim.x + threadIdx.x, (int)blockDim.x};
  const Col z{qsm + 2 * nqp * blockDim.x + threadIdx.x, (int)blockDim.x};
  for (long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x; node < n;
       node += (long long)gridDim.x * blockDim.x) {
    const double *a = ab + node * 2 * nqp;
    const double *b = a + nqp;
    for (int i = 0; i < nqp; i++) {
      d[i] = a[i];
      e[i] = b[i];
      z[i] = i == 0 ? 1.0 : 0.0;
    }
    e[nqp - 1] = 0.0;
    bool failed = false;
    for (int l = 0; l <= nqp - 1 && !failed; l++) {
      int iter = 0, m;
      do {
        for (m = l; m <= nqp - 2; m++) {
          const double em = e[m], dm = d[m], dn = d[m + 1];
          const int xe = exponent(em);
          if (xe > 0 && xe >= max(exponent(dm), exponent(dn)) - 51) continue;  // |e| > 2^-53 dd
          const double dd = fabs(dm) + fabs(dn);
          if (fabs(em) + dd == dd) break;
        }
        if (m != l) {
          if (iter++ == 50) {
            failed = true;
            break;
          }
          double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
          double r = sqrt(__dadd_rn(__dmul_rn(g, g), 1.0));
          g = __dadd_rn(d[m] - d[l], e[l] / (g + (g >= 0.0 ? fabs(r) : -fabs(r))));
          double s = 1.0, c = 1.0, p = 0.0;
          double dn = d[m], zn = z[m];                     // d[i + 1], z[i + 1]
          double ei = e[m - 1], di = d[m - 1], zi = z[m - 1];
          int i;
          bool zero = false;
          for (i = m - 1; i >= l; i--) {
            const double f = __dmul_rn(s, ei), bb = __dmul_rn(c, ei);
            const double x = __dadd_rn(__dmul_rn(g, g), __dmul_rn(f, f));
            const int q = i > l ? i - 1 : l;
            const double ep = e[q], dp = d[q], zp = z[q];  // the next rotation's
            if (x == 0.0) {
              e[i + 1] = 0.0;
              d[i + 1] = dn - p;
              e[m] = 0.0;
              z[i + 1] = zn;
              zero = true;
              break;
            }
            r = norm_and_quotients(x, f, g, s, c);
            e[i + 1] = r;
            g = dn - p;
            r = __dadd_rn(__dmul_rn(di - g, s), __dmul_rn(__dmul_rn(2.0, c), bb));
            p = __dmul_rn(s, r);
            d[i + 1] = __dadd_rn(g, p);
            g = __dadd_rn(__dmul_rn(c, r), -bb);
            z[i + 1] = __dadd_rn(__dmul_rn(s, zi), __dmul_rn(c, zn));
            zn = __dadd_rn(__dmul_rn(c, zi), -__dmul_rn(s, zn));
            dn = di;
            ei = ep;
            di = dp;
            zi = zp;
          }
          if (zero) continue;
          z[l] = zn;
          d[l] -= p;
          e[l] = g;
          e[m] = 0.0;
        }
      } while (m != l);
    }
    if (failed) atomicOr(status, kStatusNoConvergence);
    double emin = d[0], emax = d[0];
    double *lo = lambda + node * nqp, *wo = wts + node * nqp;
    for (int i = 0; i < nqp; i++) {
      lo[i] = d[i];
      wo[i] = z[i] * z[i];
      if (d[i] > emax) emax = d[i];
      else if (d[i] < emin) emin = d[i];
    }
    lmin[node] = emin;
    lmax[node] = emax;
  }
}

}  // namespace

cudaError_t launch_quadrature(const double *ab, long long n, int nqp, double *lambda, double *w,
                              double *lmin, double *lmax, int *status, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (nqp < 1 || nqp > 64) return cudaErrorInvalidValue;
  const int block = kQuadBlock;
  const size_t smem = sizeof(double) * 3 * (size_t)nqp * block;
  cudaError_t e = cudaFuncSetAttribute(quadrature_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const long long blocks = (n + block - 1) / block;
  const int grid = (int)(blocks < 152LL * 64 ? blocks : 152LL * 64);
  quadrature_kernel<<<grid, block, smem, s>>>(ab, n, nqp, lambda, w, lmin, lmax, status);
  return cudaGetLastError();
}

}  // namespace sq
