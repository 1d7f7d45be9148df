// quadrature.cu -- Gauss quadrature nodes and weights from the Lanczos tridiagonals.
//
// Replaces TridiagEigenVecSolve_NodesAndWeights (src/lsdft_tools.cc:912-1026): implicit QL
// with Wilkinson-type shifts (Numerical Recipes tqli), lambda_q = d[q], w_q = Z[0][q]^2,
// eigenvalues left unsorted, lambda_min / lambda_max by the reference's scan.  The rows of Z
// never mix in tqli, so only row 0 is carried: O(n) storage and O(n^2) work per node with
// results identical to the full-matrix form.
//
// One thread or a pair per node, FP64.  The three working arrays of a node (d, e and row 0 of Z, N_qp
// doubles each) live in shared memory, one column per node (element i of node t at
// i * nodes + t): as local arrays the ~250 nodes per SM (1.5 KB each) overflow L1 and every
// rotation waits on L2.
//
// What bounds it is the FP64 pipe: an instruction of a warp holds its SM sub-partition for 64 cycles,
// however many lanes are at work, so the time is their number (about 75 cycles each, 1870 rotations
// for 40 steps).  Every result stays the correctly rounded one of the CPU reference (the order in which
// eigenvalues deflate turns on the last bits), so the products and sums are separate, rounded
// operations.  But
//  * r = sqrt(x), f / r and g / r come from one FP32 reciprocal root, a Newton step and Markstein's
//    residual corrections (IBM J. Res. Dev. 34, 1990) instead of a square root and two divisions;
//  * factors of two go into the exponent, and the deflation test looks at the exponents first;
//  * where there are few nodes a pair of lanes works on each: one carries s, f, d, the other c, b,
//    g, so that most of a rotation's operations come in twos (20 instructions instead of 32).
// The next rotation's elements are loaded ahead.  For 40 steps: one node 3.69 -> 2.29 ms, 600 nodes
// 4.42 -> 3.17 ms, 39304 nodes 11.1 -> 8.0 ms (from a square root, two divisions and one lane per node).
#include <cuda_runtime.h>

#include "sq_kernels.hpp"

namespace sq {

namespace {

constexpr int kQuadBlock = 64;

// one node's column of a shared array: element i at p[i * stride]
struct Col {
  double *p;
  int stride;
  __device__ __forceinline__ double &operator[](int i) const { return p[i * stride]; }
};

__device__ __forceinline__ int exponent(double v) { return (__double2hiint(v) >> 20) & 2047; }
// v * 2^k through the exponent; v and the result normal numbers
__device__ __forceinline__ double scaled(double v, int k) {
  return __hiloint2double(__double2hiint(v) + (k << 20), __double2loint(v));
}
// 2 v; zero and the ends of the range by the addition
__device__ __forceinline__ double twice(double v) {
  const int e = exponent(v);
  return e == 0 || e >= 2046 ? v + v : scaled(v, 1);
}

// 1 / sqrt(x) to FP32 precision, as a double; x in [2^-120, 2^120].  By the bits: conversions run at
// the FP64 rate.
__device__ __forceinline__ bool root_range(double x) {
  const int e = exponent(x);
  return e >= 1023 - 120 && e <= 1023 + 120;
}
__device__ __forceinline__ double root_estimate(double x) {
  const unsigned hi = (unsigned)(__double2hiint(x) - (896 << 20));
  const int y = __float_as_int(rsqrtf(__int_as_float((int)((hi << 3) | ((unsigned)__double2loint(x) >> 29)))));
  return __hiloint2double((y >> 3) + (896 << 20), y << 29);
}

// r = sqrt(x), s = f / r, c = g / r: y = 1 / sqrt(x) by one Newton step from the estimate (to 5e-14), the
// products with it, and a residual correction of each, which leaves 3e-27: rounded correctly but where the
// exact value is that close to a midpoint (none in 3e9 random ones).
__device__ __forceinline__ double norm_and_quotients(double x, double f, double g, double &s, double &c) {
  if (!root_range(x)) {
    const double r = sqrt(x);
    s = f / r;
    c = g / r;
    return r;
  }
  const double y0 = root_estimate(x), t = __dmul_rn(x, y0), e = fma(-t, y0, 1.0);
  const double y = fma(scaled(y0, -1), e, y0), r0 = fma(scaled(t, -1), e, t);
  const double r = fma(fma(-r0, r0, x), scaled(y, -1), r0);
  const double s0 = __dmul_rn(f, y), c0 = __dmul_rn(g, y);
  s = fma(fma(-r, s0, f), y, s0);
  c = fma(fma(-r, c0, g), y, c0);
  return r;
}

// LANES threads of a warp per node (1 or 2).
template <int LANES>
__global__ void __launch_bounds__(kQuadBlock)
    quadrature_kernel(const double *__restrict__ ab, long long n, int nqp,
                      double *__restrict__ lambda, double *__restrict__ wts,
                      double *__restrict__ lmin, double *__restrict__ lmax,
                      int *__restrict__ status) {
  extern __shared__ double qsm[];  // [3][nqp][nodes of the block]
  const int nodes = blockDim.x / LANES, slot = threadIdx.x / LANES;
  const bool odd = LANES == 2 && (threadIdx.x & 1), writer = !odd;
  const unsigned pair = LANES == 2 ? 3u << (threadIdx.x & 30) : 0u;
  auto other = [&](double v) { return __shfl_xor_sync(pair, v, 1); };
  auto meet = [&]() {  // what one lane of the pair wrote is read by both
    if constexpr (LANES == 2) __syncwarp(pair);
  };
  const Col d{qsm + slot, nodes};
  const Col e{qsm + nqp * nodes + slot, nodes};
  const Col z{qsm + 2 * nqp * nodes + slot, nodes};
  for (long long node = blockIdx.x * (long long)nodes + slot; node < n;
       node += (long long)gridDim.x * nodes) {
    const double *a = ab + node * 2 * nqp;
    const double *b = a + nqp;
    for (int i = threadIdx.x % LANES; i < nqp; i += LANES) {
      d[i] = a[i];
      e[i] = i == nqp - 1 ? 0.0 : b[i];
      z[i] = i == 0 ? 1.0 : 0.0;
    }
    meet();
    bool failed = false;
    for (int l = 0; l <= nqp - 1 && !failed; l++) {
      int iter = 0, m;
      do {
        for (m = l; m <= nqp - 2; m++) {
          const double em = e[m], dm = d[m], dn = d[m + 1];
          const int xe = exponent(em), xd = max(exponent(dm), exponent(dn));
          if (xe > 0 && xe >= xd - 51 && xd < 2046) continue;  // |e| > 2^-53 dd, and dd does not overflow
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
          meet();  // both have read
          for (i = m - 1; i >= l; i--) {
            const int q = i > l ? i - 1 : l;
            const double ep = e[q], dp = d[q], zp = z[q];  // the next rotation's
            if constexpr (LANES == 1) {
              const double f = __dmul_rn(s, ei), bb = __dmul_rn(c, ei);
              const double x = __dadd_rn(__dmul_rn(g, g), __dmul_rn(f, f));
              if (x == 0.0) {
                zero = true;
                break;
              }
              e[i + 1] = norm_and_quotients(x, f, g, s, c);
              g = dn - p;
              r = __dadd_rn(__dmul_rn(di - g, s), __dmul_rn(c, twice(bb)));
              p = __dmul_rn(s, r);
              d[i + 1] = __dadd_rn(g, p);
              g = __dadd_rn(__dmul_rn(c, r), -bb);
              z[i + 1] = __dadd_rn(__dmul_rn(s, zi), __dmul_rn(c, zn));
              zn = __dadd_rn(__dmul_rn(c, zi), -__dmul_rn(s, zn));
            } else {
              // even lane: s, f, p, d[i+1], z[i+1]; odd lane: c (in s), bb, g, z[i]
              const double fb = __dmul_rn(s, ei), num = odd ? g : fb;
              const double sq = __dmul_rn(num, num), x = __dadd_rn(sq, other(sq));
              if (x == 0.0) {
                zero = true;
                break;
              }
              if (root_range(x)) {
                const double y0 = root_estimate(x), t = __dmul_rn(x, y0), err = fma(-t, y0, 1.0);
                const double v = fma(scaled(odd ? y0 : t, -1), err, odd ? y0 : t), o = other(v);
                const double y = odd ? v : o, r0 = odd ? o : v;
                r = fma(fma(-r0, r0, x), scaled(y, -1), r0);
                const double s0 = __dmul_rn(num, y);
                s = fma(fma(-r, s0, num), y, s0);
              } else {
                r = sqrt(x);
                s = num / r;
              }
              const double gd = dn - p, u = di - gd;
              const double m1 = __dmul_rn(odd ? twice(fb) : u, s);
              const double rr = __dadd_rn(m1, other(m1)), m2 = __dmul_rn(s, rr);
              const double nx = __dadd_rn(m2, odd ? -fb : gd);
              const double za = __dmul_rn(s, zi), zb = __dmul_rn(s, zn), zo = other(zb);
              const double zz = __dadd_rn(za, odd ? -zo : zo), zs = other(zz);
              if (writer) {
                e[i + 1] = r;
                d[i + 1] = nx;
                z[i + 1] = zz;
              }
              p = m2;                // even
              g = nx;                // odd
              zn = odd ? zz : zs;
            }
            dn = di;
            ei = ep;
            di = dp;
            zi = zp;
          }
          if constexpr (LANES == 2) {
            const double po = other(p), go = other(g);
            p = odd ? po : p;
            g = odd ? g : go;
          }
          if (writer) {
            if (zero) {
              e[i + 1] = 0.0;
              d[i + 1] = dn - p;
              z[i + 1] = zn;
            } else {
              z[l] = zn;
              d[l] -= p;
              e[l] = g;
            }
            e[m] = 0.0;
          }
          meet();
        }
      } while (m != l);
    }
    if (failed && writer) atomicOr(status, kStatusNoConvergence);
    double emin = d[0], emax = d[0];
    double *lo = lambda + node * nqp, *wo = wts + node * nqp;
    for (int i = 0; i < nqp; i++) {
      const double di = d[i];
      if (writer) {
        lo[i] = di;
        wo[i] = z[i] * z[i];
      }
      if (di > emax) emax = di;
      else if (di < emin) emin = di;
    }
    if (writer) {
      lmin[node] = emin;
      lmax[node] = emax;
    }
    meet();
  }
}

template <int LANES>
cudaError_t launch_lanes(const double *ab, long long n, int nqp, double *lambda, double *w, double *lmin,
                         double *lmax, int *status, cudaStream_t s) {
  const int nodes = kQuadBlock / LANES;
  const size_t smem = sizeof(double) * 3 * (size_t)nqp * nodes;
  cudaError_t e = cudaFuncSetAttribute(quadrature_kernel<LANES>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const long long blocks = (n + nodes - 1) / nodes;
  const int grid = (int)(blocks < 152LL * 64 ? blocks : 152LL * 64);
  quadrature_kernel<LANES><<<grid, kQuadBlock, smem, s>>>(ab, n, nqp, lambda, w, lmin, lmax, status);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_quadrature(const double *ab, long long n, int nqp, double *lambda, double *w,
                              double *lmin, double *lmax, int *status, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (nqp < 1 || nqp > 64) return cudaErrorInvalidValue;
  // a pair of lanes per node while that makes at most one warp per SM sub-partition (4 x 152): 600 nodes
  // of 40 steps take 3.17 ms in pairs and 3.28 ms alone, 9728 nodes 3.29 and 3.35; beyond, the pairs'
  // 2 x 20 instructions cost more than 32: 12000 nodes 3.71 and 3.48, 20000 nodes 5.77 and 4.71.
  return n <= 16LL * 4 * 152 ? launch_lanes<2>(ab, n, nqp, lambda, w, lmin, lmax, status, s)
                             : launch_lanes<1>(ab, n, nqp, lambda, w, lmin, lmax, status, s);
}

}  // namespace sq
