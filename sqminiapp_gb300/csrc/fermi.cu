// fermi.cu -- Fermi level, node densities and band energy from the quadrature (FP64).
//
// The reference declares this closure but never defines it (src/lsdft.h:98-102
// constraint_lssgq / FermiDirac / CalculateDensity_lssgq / findRootBrent, :209
// SystemEnergy_Calc_lssgq).  With the Gauss rule of node i (lambda_iq, w_iq):
//   N_e(lf) = 2 sum_i sum_q w_iq f(lambda_iq - lf),  f(x) = 1 / (1 + exp(beta x))
// lf is found by bisection on [min lambda - 1, max lambda + 1]; then
//   rho_i = (2/dV) sum_q w_iq f,  E_band = 2 sum w lambda f,
//   -TS = (2/beta) sum w [f ln f + (1-f) ln(1-f)].
//
// One cooperative persistent launch runs the whole search: each CTA reduces its slice into
// partials, a bounded grid barrier publishes them, and every CTA sums them in the same fixed
// order, so all CTAs take the same branch and the result does not depend on scheduling.  The
// barrier spins a bounded number of times and then reports kStatusTimeout instead of waiting
// forever.
//
// The bisection's midpoints are the same as ever, but few of them are evaluated: N_e grows with lf
// (weights are not negative; checked, else every midpoint is evaluated), so a midpoint outside a
// known interval [xl, xr] with N_e(xl) <= n_electrons < N_e(xr) needs no sum.  The interval comes from
// three levels per pass in FP32, taken as known only where the sum is off by more than its error,
// and from Newton steps in FP64.  FP64 exponentials are what a pass costs (2 lanes of FP64 per SM and
// cycle), so the FP64 passes run over the entries whose occupation can differ from 0 and 1 inside
// the interval, gathered in shared memory once; the others are a constant.
//   Before: about 45 passes of FP64 exponentials over all entries, 14.6 ms for 132651 x 40.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "sq_gb300.h"
#include "sq_kernels.hpp"

namespace sq {

namespace {

constexpr int kFermiBlock = 512;
constexpr long long kSpinLimit = 1LL << 22;

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ double block_sum_d(double v, double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum_d(v);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double t = 0.0;
  if (warp == 0) {
    t = lane < kFermiBlock / 32 ? red[lane] : 0.0;
    t = warp_sum_d(t);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// All CTAs meet here.  Returns false (in every thread of the CTA) if the wait gave up after
// spin_limit polls.
__device__ bool grid_barrier(unsigned *bar, int *status, int *flag_smem, long long spin_limit) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned *gen_p = bar + 1;
    const unsigned gen = *gen_p;
    __threadfence();
    const unsigned arrived = atomicAdd(bar, 1u);
    int ok = 1;
    if (arrived == gridDim.x - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      long long spins = 0;
      while (*gen_p == gen) {
        if (++spins > spin_limit) {
          atomicOr(status, kStatusTimeout);
          ok = 0;
          break;
        }
        __nanosleep(100);
      }
    }
    __threadfence();
    *flag_smem = ok;
  }
  __syncthreads();
  return *flag_smem != 0;
}

// Occupation 1 / (1 + exp(x)), x = beta (lam - lf), without the exponential where it rounds to 1 (x
// below -37.5: exp(x) < 2^-54) or underflows to 0 (x above 745.2).
__device__ __forceinline__ double fermi_dirac(double beta, double lam, double lf) {
  const double x = beta * (lam - lf);
  if (x < -37.5) return 1.0;
  if (x > 745.2) return 0.0;
  return 1.0 / (1.0 + exp(x));
}

// The float nearest towards zero, by the bits (conversions run at the FP64 rate); for |v| below 2^-126
// zero, above 2^127 infinity.
__device__ __forceinline__ float truncate_f32(double v) {
  const int hi = __double2hiint(v), mag = hi & 0x7fffffff;
  const int bits = (int)(((unsigned)(mag - (896 << 20)) << 3) | ((unsigned)__double2loint(v) >> 29));
  const int r = mag < (897 << 20) ? 0 : mag >= (1150 << 20) ? 0x7f800000 : bits;
  return __int_as_float(r | (hi & 0x80000000));
}

// In units of 1/beta: entries this far above a level count as empty in the gathered sums (their
// occupation is below 2e-20, 2e-13 of the electrons if all states of a cell that is filled to kFermiLeast
// lie there), and this far below as full (exactly 1 in FP64).
constexpr double kFermiAbove = 45.5, kFermiBelow = 37.5;
// With a smaller share of the states filled every midpoint is summed over all entries.
constexpr double kFermiLeast = 1e-7;
constexpr int kFermiLevels = 3;    // levels per FP32 pass
constexpr int kFermiRows = 2 * kFermiLevels + 2;  // scratch rows: partials of two passes, bracket
constexpr int kFermiEntries = 4096;  // entries of a CTA's slice gathered in shared memory
constexpr size_t kFermiSmem = sizeof(double) * 2 * kFermiEntries;

// Totals of up to N partials per CTA (rows scratch + j * G), the same order in every CTA.
template <int N>
__device__ void grid_totals(const double *rows, int G, double *bcast, double (&t)[N]) {
  if (threadIdx.x < 32) {
#pragma unroll
    for (int j = 0; j < N; j++) {
      double v = 0.0;
      for (int i = threadIdx.x; i < G; i += 32) v += __ldcg(rows + (long long)j * G + i);
      v = warp_sum_d(v);
      if (threadIdx.x == 0) bcast[j] = v;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < N; j++) t[j] = bcast[j];
  __syncthreads();
}

__global__ void __launch_bounds__(kFermiBlock)
    fermi_kernel(const double *__restrict__ lambda, const double *__restrict__ w,
                 long long n_nodes, int nqp, double beta, double n_electrons, double dV,
                 double tol, int maxit, double *__restrict__ rho, double *__restrict__ out,
                 double *__restrict__ scratch, unsigned *__restrict__ bar,
                 int *__restrict__ status, long long spin_limit, int skip_block) {
  extern __shared__ double gathered[];  // [2][kFermiEntries]: lambda, w of the open entries
  __shared__ double red[kFermiBlock / 32];
  // fault injection of the timeout self-test: one CTA leaves before its first arrival, so
  // every other CTA's first barrier wait runs out
  if ((int)blockIdx.x == skip_block) return;
  __shared__ double bcast[kFermiLevels];
  __shared__ int flag, n_open_s;
  const int G = gridDim.x;
  const long long n = n_nodes * nqp;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long stride = (long long)G * blockDim.x;
  double *bracket = scratch + (long long)(2 * kFermiLevels) * G;
  int parity = 0;  // which half of the partial rows the next pass writes

  // phase 0: bracket, the weights' sum, and whether N_e is known to grow with the level
  double lo = 1e300, hi = -1e300;
  float filled = 0.f;
  bool plain = false;
  for (long long e = tid; e < n; e += stride) {
    const double l = lambda[e];
    lo = fmin(lo, l);
    hi = fmax(hi, l);
    // a weight below zero or not finite, a value not finite (exponent all ones)
    const int wh = __double2hiint(w[e]), lh = __double2hiint(l);
    plain = plain || (wh < 0 && (wh & 0x7fffffff)) || ((wh >> 20) & 2047) == 2047 || ((lh >> 20) & 2047) == 2047;
    filled += truncate_f32(w[e]);
  }
  const double filled_all = block_sum_d(2.0 * (double)filled, red);  // in thread 0
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  plain = __syncthreads_or(plain);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = lo;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = red[0];
    for (int i = 1; i < kFermiBlock / 32; i++) m = fmin(m, red[i]);
    bracket[blockIdx.x] = m;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = hi;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = red[0];
    for (int i = 1; i < kFermiBlock / 32; i++) m = fmax(m, red[i]);
    bracket[G + blockIdx.x] = m;
    scratch[blockIdx.x] = plain ? 1.0 : 0.0;
    scratch[G + blockIdx.x] = filled_all;
  }
  if (!grid_barrier(bar, status, &flag, spin_limit)) return;
  {
    double a = 1e300, b = -1e300, q = 0.0, t = 0.0;
    if (threadIdx.x < 32) {
      for (int i = threadIdx.x; i < G; i += 32) {
        a = fmin(a, __ldcg(bracket + i));
        b = fmax(b, __ldcg(bracket + G + i));
        q += __ldcg(scratch + i);
        t += __ldcg(scratch + G + i);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a = fmin(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
        q += __shfl_xor_sync(0xffffffffu, q, o);
        t += __shfl_xor_sync(0xffffffffu, t, o);
      }
      if (threadIdx.x == 0) {
        bcast[0] = a - 1.0;
        bcast[1] = b + 1.0;
        // nearly empty: the electrons are no longer far more than what the gathered sums leave out
        // (kFermiAbove) and the FP32 passes cap (exponents above 80); or weights outside FP32's range
        bcast[2] = q != 0.0 || !(n_electrons >= kFermiLeast * t) || !(t > 1e-25);
      }
    }
    __syncthreads();
    lo = bcast[0];
    hi = bcast[1];
    plain = bcast[2] != 0.0;
    __syncthreads();
  }
  parity = 1;  // the first half still holds the flags

  // known interval: N_e(xl) <= n_electrons < N_e(xr)
  double xl = -1e300, xr = 1e300;
  const double inv_beta = 1.0 / beta;

  // phase 1a: kFermiLevels levels per pass in FP32.  Of a level's sum S the rounding of lambda (1e-7
  // of |lambda|, beta times that of the exponent), of the terms and of the float sums (2^-24 of S for
  // each term that a thread adds) stay below err S.
  if (!plain) {
    double cl = lo, cr = hi;
    const float bf = (float)beta;
    const double span = fmax(fabs(lo), fabs(hi));
    const double err = 1e-4 + 4e-7 * beta * span + 6e-8 * (double)((n + stride - 1) / stride);
    for (int pass = 0; pass < 24 && cr - cl > 0.25 * inv_beta && err < 0.25; pass++) {
      float lev[kFermiLevels], c[kFermiLevels];
#pragma unroll
      for (int j = 0; j < kFermiLevels; j++) {
        lev[j] = truncate_f32(cl + (cr - cl) * ((j + 1) / (double)(kFermiLevels + 1)));
        c[j] = 0.f;
      }
      for (long long e = tid; e < n; e += stride) {
        const float l = truncate_f32(lambda[e]), we = truncate_f32(w[e]);
#pragma unroll
        for (int j = 0; j < kFermiLevels; j++)
          c[j] += we * __fdividef(1.f, 1.f + __expf(fminf(bf * (l - lev[j]), 80.f)));
      }
      double *rows = scratch + (long long)parity * kFermiLevels * G, t[kFermiLevels];
      parity ^= 1;
#pragma unroll
      for (int j = 0; j < kFermiLevels; j++) {
        const double v = block_sum_d(2.0 * (double)c[j], red);
        if (threadIdx.x == 0) rows[(long long)j * G + blockIdx.x] = v;
      }
      if (!grid_barrier(bar, status, &flag, spin_limit)) return;
      grid_totals(rows, G, bcast, t);
      bool moved = false;
#pragma unroll
      for (int j = 0; j < kFermiLevels; j++) {
        const double m = (double)lev[j], slack = err * fmax(t[j], n_electrons);
        if (t[j] + slack < n_electrons && m > cl) {
          cl = m;
          moved = true;
        }
        if (t[j] - slack > n_electrons && m < cr) {
          cr = m;
          moved = true;
        }
      }
      if (!moved || !(cl < cr)) break;
    }
    if (cl < cr) {
      if (cl > lo) xl = cl;
      if (cr < hi) xr = cr;
    }
  }

  // phase 1b: the entries that are neither full nor empty for every level left; `full` their sum
  const double open_lo = fmax(xl, lo) - kFermiBelow * inv_beta, open_hi = fmin(xr, hi) + kFermiAbove * inv_beta;
  double full = 0.0;
  bool in_smem = !plain;
  if (threadIdx.x == 0) n_open_s = 0;
  __syncthreads();
  if (in_smem) {
    for (long long base = tid - threadIdx.x; base < n; base += stride) {
      const long long e = base + threadIdx.x;
      bool open = false;
      double l = 0.0;
      if (e < n) {
        l = lambda[e];
        open = l >= open_lo && l <= open_hi;
        if (l < open_lo) full += 2.0 * w[e];
      }
      // places by warp: one warp after another in a fixed order
      const unsigned m = __ballot_sync(0xffffffffu, open);
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      __shared__ int first[kFermiBlock / 32 + 1];
      if (lane == 0) first[warp] = __popc(m);
      __syncthreads();
      int at = n_open_s, all = 0;
      for (int i = 0; i < kFermiBlock / 32; i++) {
        at += i < warp ? first[i] : 0;
        all += first[i];
      }
      at += __popc(m & ((1u << lane) - 1u));
      if (open && at < kFermiEntries) {
        gathered[at] = l;
        gathered[kFermiEntries + at] = w[e];
      }
      __syncthreads();
      if (threadIdx.x == 0) n_open_s += all;
      __syncthreads();
      if (n_open_s > kFermiEntries) break;  // uniform: this CTA sums over its whole slice instead
    }
    in_smem = n_open_s <= kFermiEntries;
  }
  const int n_open = n_open_s;

  // N_e and its derivative at x, summed over all CTAs.  False if the barrier gave up.
  auto evaluate = [&](double x, double &ne, double &dne) {
    double c = 0.0, d = 0.0;
    if (in_smem) {
      c = full;
      for (int i = threadIdx.x; i < n_open; i += kFermiBlock) {
        const double f = fermi_dirac(beta, gathered[i], x), we = 2.0 * gathered[kFermiEntries + i];
        c += we * f;
        d += we * f * (1.0 - f);
      }
    } else {
      for (long long e = tid; e < n; e += stride) {
        const double f = fermi_dirac(beta, lambda[e], x), we = 2.0 * w[e];
        c += we * f;
        d += we * f * (1.0 - f);
      }
    }
    c = block_sum_d(c, red);
    d = block_sum_d(d, red);
    double *rows = scratch + (long long)parity * kFermiLevels * G, t[2];
    parity ^= 1;
    if (threadIdx.x == 0) {
      rows[blockIdx.x] = c;
      rows[G + blockIdx.x] = d;
    }
    if (!grid_barrier(bar, status, &flag, spin_limit)) return false;
    grid_totals(rows, G, bcast, t);
    ne = t[0];
    dne = beta * t[1];
    return true;
  };

  // phase 1c: Newton steps from inside the interval, every evaluation narrows it; once a step is
  // within tol, one more evaluation just across the root
  if (!plain && xl > -1e300 && xr < 1e300) {
    const double near = fmax(0.25 * tol, 4e-16 * fmax(fabs(xl), fabs(xr)));
    double x = 0.5 * (xl + xr);
    for (int k = 0; k < 12 && xr - xl > 2.0 * near; k++) {
      double ne, dne;
      if (!evaluate(x, ne, dne)) return;
      const bool above = ne > n_electrons;
      if (above) xr = x;
      else xl = x;
      double next = x - (ne - n_electrons) / dne;
      if (fabs(next - x) <= near) next = above ? next - near : next + near;  // the other side
      if (!(next > xl && next < xr)) next = 0.5 * (xl + xr);
      x = next;
    }
  }

  // phase 1: bisection on the electron count
  int it;
  for (it = 0; it < maxit; it++) {
    const double mid = 0.5 * (lo + hi);
    bool above = mid >= xr;
    if (!above && mid > xl) {
      double ne, dne;
      if (!evaluate(mid, ne, dne)) return;
      above = ne > n_electrons;
    }
    if (above) hi = mid;
    else lo = mid;
    if (hi - lo < tol) break;
  }
  const double lf = 0.5 * (lo + hi);

  // phase 2: densities, band energy, entropy term
  double eb = 0.0, ent = 0.0;
  for (long long node = tid; node < n_nodes; node += stride) {
    double r = 0.0;
    for (int q = 0; q < nqp; q++) {
      const long long e = node * nqp + q;
      const double l = lambda[e], x = beta * (l - lf);
      if (x > 745.2 && !plain) continue;  // empty (an infinite weight times 0 has to reach the sums)
      const double f = fermi_dirac(beta, l, lf);
      r += w[e] * f;
      eb += 2.0 * w[e] * l * f;
      double s = 0.0;
      if (f > 0.0 && f < 1.0) s = f * log(f) + (1.0 - f) * log(1.0 - f);
      ent += 2.0 * w[e] * s;
    }
    if (rho) rho[node] = 2.0 * r / dV;
  }
  eb = block_sum_d(eb, red);
  ent = block_sum_d(ent, red);
  double *rows = scratch + (long long)parity * kFermiLevels * G, t[2];
  if (threadIdx.x == 0) {
    rows[blockIdx.x] = eb;
    rows[G + blockIdx.x] = ent;
  }
  if (!grid_barrier(bar, status, &flag, spin_limit)) return;
  if (blockIdx.x == 0) {
    grid_totals(rows, G, bcast, t);
    if (threadIdx.x == 0) {
      out[0] = lf;
      out[1] = t[0];
      out[2] = t[1] / beta;
      out[3] = (double)it;
    }
  }
}

constexpr int kCountBlock = 256;

// Partial electron counts: one per CTA, in a fixed grid-stride order.
__global__ void __launch_bounds__(kCountBlock)
    count_partials_kernel(const double *__restrict__ lambda, const double *__restrict__ w,
                          long long n, double beta, double lf, double *__restrict__ partial) {
  __shared__ double red[kCountBlock / 32];
  double c = 0.0;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    c += 2.0 * w[e] * fermi_dirac(beta, lambda[e], lf);
  c = warp_sum_d(c);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < kCountBlock / 32; i++) t += red[i];
    partial[blockIdx.x] = t;
  }
}

__global__ void sum_partials_kernel(const double *__restrict__ partial, int n,
                                    double *__restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < n; i++) t += partial[i];
    *out = t;
  }
}

// Node densities, band energy and entropy term of a given Fermi level (the last phase of
// fermi_kernel on its own): part[2 * block] = (2 sum w lambda f, 2 sum w s(f)) per CTA.
__global__ void __launch_bounds__(kCountBlock)
    density_energy_kernel(const double *__restrict__ lambda, const double *__restrict__ w,
                          long long n_nodes, int nqp, double beta, double lf, double dV,
                          double *__restrict__ rho, double *__restrict__ part) {
  __shared__ double red[2][kCountBlock / 32];
  double eb = 0.0, ent = 0.0;
  for (long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x; node < n_nodes;
       node += (long long)gridDim.x * blockDim.x) {
    double r = 0.0;
    for (int q = 0; q < nqp; q++) {
      const long long e = node * nqp + q;
      const double f = fermi_dirac(beta, lambda[e], lf);
      r += w[e] * f;
      eb += 2.0 * w[e] * lambda[e] * f;
      double sv = 0.0;
      if (f > 0.0 && f < 1.0) sv = f * log(f) + (1.0 - f) * log(1.0 - f);
      ent += 2.0 * w[e] * sv;
    }
    if (rho) rho[node] = 2.0 * r / dV;
  }
  eb = warp_sum_d(eb);
  ent = warp_sum_d(ent);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = eb;
    red[1][threadIdx.x >> 5] = ent;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int i = 0; i < kCountBlock / 32; i++) {
      a += red[0][i];
      b += red[1][i];
    }
    part[2 * blockIdx.x] = a;
    part[2 * blockIdx.x + 1] = b;
  }
}

__global__ void sum_pairs_kernel(const double *__restrict__ part, int n, double *__restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int i = 0; i < n; i++) {
      a += part[2 * i];
      b += part[2 * i + 1];
    }
    out[0] = a;
    out[1] = b;
  }
}

}  // namespace

cudaError_t launch_density_energy(const double *lambda, const double *w, long long n_nodes, int nqp,
                                  double beta, double lf, double dV, double *rho, double *partial,
                                  int grid, double *out, cudaStream_t s) {
  density_energy_kernel<<<grid, kCountBlock, 0, s>>>(lambda, w, n_nodes, nqp, beta, lf, dV, rho,
                                                     partial);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  sum_pairs_kernel<<<1, 32, 0, s>>>(partial, grid, out);
  return cudaGetLastError();
}

cudaError_t launch_electron_count(const double *lambda, const double *w, long long n_nodes,
                                  int nqp, double beta, double lf, double *partial, int grid,
                                  double *out, cudaStream_t s) {
  const long long n = n_nodes * nqp;
  count_partials_kernel<<<grid, kCountBlock, 0, s>>>(lambda, w, n, beta, lf, partial);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  sum_partials_kernel<<<1, 32, 0, s>>>(partial, grid, out);
  return cudaGetLastError();
}

// The message of sq_fermi_density_energy_noalloc failures, reported by sq_last_error_string.
void set_noalloc_error(const std::string &msg);

size_t fermi_scratch_doubles(int grid, int maxit) {
  return (size_t)grid * std::max(maxit + 4, kFermiRows);
}

namespace {
cudaError_t launch_fermi_impl(const double *lambda, const double *w, long long n_nodes, int nqp,
                              double beta, double n_electrons, double dV, double tol, int maxit,
                              double *rho, double *out, double *scratch, unsigned *barrier,
                              int *status, int grid, cudaStream_t s, long long spin_limit,
                              int skip_block) {
  cudaError_t e = cudaMemsetAsync(barrier, 0, 2 * sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  void *args[] = {(void *)&lambda, (void *)&w,   (void *)&n_nodes, (void *)&nqp,
                  (void *)&beta,   (void *)&n_electrons, (void *)&dV, (void *)&tol,
                  (void *)&maxit,  (void *)&rho, (void *)&out,     (void *)&scratch,
                  (void *)&barrier, (void *)&status, (void *)&spin_limit, (void *)&skip_block};
  e = cudaFuncSetAttribute(fermi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFermiSmem);
  if (e != cudaSuccess) return e;
  return cudaLaunchCooperativeKernel((const void *)fermi_kernel, dim3(grid), dim3(kFermiBlock),
                                     args, kFermiSmem, s);
}
}  // namespace

cudaError_t launch_fermi(const double *lambda, const double *w, long long n_nodes, int nqp,
                         double beta, double n_electrons, double dV, double tol, int maxit,
                         double *rho, double *out, double *scratch, unsigned *barrier,
                         int *status, int grid, cudaStream_t s) {
  return launch_fermi_impl(lambda, w, n_nodes, nqp, beta, n_electrons, dV, tol, maxit, rho, out,
                           scratch, barrier, status, grid, s, kSpinLimit, -1);
}

// Fault-injection self-test of the grid barrier's bounded wait: the same cooperative launch
// with one CTA leaving before its first arrival and a short poll limit (about 4096 polls of
// 100 ns), so the other CTAs give up, record kStatusTimeout and return.  Nothing faults or
// hangs: the kernel ends and the context stays usable.
cudaError_t launch_fermi_timeout_selftest(const double *lambda, const double *w, long long n_nodes,
                                          int nqp, double *out, double *scratch,
                                          unsigned *barrier, int *status, int grid,
                                          cudaStream_t s) {
  return launch_fermi_impl(lambda, w, n_nodes, nqp, 30.0, 1.0, 1.0, 1e-12, 10, nullptr, out,
                           scratch, barrier, status, grid, s, 1LL << 12, 0);
}

// ---------------------------------------------------------------------------------------
// Allocation-free entry point.
//
// Some callers cannot call cudaMalloc: code running inside a host framework that owns the
// device allocator and forbids side allocations, plugin hosts that run with a fixed memory
// budget, and stream-ordered pipelines that must not hit the allocator's implicit device
// synchronisation between steps.  For them the Fermi-level kernel can run on a file-scope
// scratch array that is part of the loaded module instead of on handle-owned buffers.
//
// Scratch capacity: kNoallocMaxBlocks CTA partials for each of kNoallocMaxIters bisection
// steps plus four rows for the bracket and energy sums (about 410 KiB of doubles), the grid
// barrier, the four scalar results and a status word.  Every GPU that loads the library
// holds this array until the process exits.  All calls share it and it keeps the contents
// of the last call: the barrier and the status word are cleared at the start of each call,
// everything else is written before it is read.  Two calls whose work overlaps on the GPU
// (on different streams, or from different host threads) race on the array and give wrong
// results; calls must be ordered.
//
// The array's device address belongs to the CUDA context that is current when it is looked
// up, so every call looks it up again with cudaGetSymbolAddress (no allocation): a context
// that was destroyed and made again, or another context made current by the caller, never
// sees a stale address.
// ---------------------------------------------------------------------------------------
namespace {
constexpr int kNoallocMaxBlocks = 256;
constexpr int kNoallocMaxIters = 200;
constexpr size_t kNoallocPartials = (size_t)kNoallocMaxBlocks * (kNoallocMaxIters + 4);

struct NoallocScratch {
  double partials[kNoallocPartials];
  double out[4];
  unsigned barrier[2];
  int status;
  int pad;
};

static __device__ __align__(256) NoallocScratch g_noalloc_scratch;
}  // namespace

extern "C" sq_status sq_fermi_density_energy_noalloc(const double *d_lambda,
                                                     const double *d_weights, long n_nodes,
                                                     int n_qp, double beta, double n_electrons,
                                                     double dV, double tol, int maxit,
                                                     double *d_rho, double *out, void *stream) {
  if (!d_lambda || !d_weights || !out) {
    set_noalloc_error("null argument");
    return SQ_BAD_INPUT;
  }
  if (n_nodes <= 0 || n_qp <= 0 || !(beta > 0) || !(dV > 0) || !(tol > 0)) {
    set_noalloc_error("n_nodes, n_qp, beta, dV and tol must be positive");
    return SQ_BAD_INPUT;
  }
  if (maxit < 1 || maxit > kNoallocMaxIters) {
    set_noalloc_error("maxit must be 1.." + std::to_string(kNoallocMaxIters) +
                      " (capacity of the static scratch array)");
    return SQ_CAPACITY;
  }
  cudaStream_t s = (cudaStream_t)stream;
  // the call ends with a device-to-host copy and a stream synchronisation, neither of which a
  // stream capture allows: refuse before touching the stream
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(s, &cap);
  if (e != cudaSuccess) {
    set_noalloc_error(std::string("cudaStreamIsCapturing: ") + cudaGetErrorString(e));
    return SQ_CUDA_ERROR;
  }
  if (cap != cudaStreamCaptureStatusNone) {
    set_noalloc_error("the stream is being captured; this call synchronises it and cannot be "
                      "captured");
    return SQ_BAD_INPUT;
  }
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) {
    set_noalloc_error(std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    return SQ_CUDA_ERROR;
  }
  // the array's address in the current context (looked up on every call, see above)
  void *ptr = nullptr;
  if ((e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch)) != cudaSuccess) {
    set_noalloc_error(std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    return SQ_CUDA_ERROR;
  }
  NoallocScratch *scr = reinterpret_cast<NoallocScratch *>(ptr);
  int sms = 0, per_sm = 0;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(fermi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFermiSmem)) !=
          cudaSuccess ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fermi_kernel, kFermiBlock, kFermiSmem)) !=
          cudaSuccess) {
    set_noalloc_error(std::string("device query: ") + cudaGetErrorString(e));
    return SQ_CUDA_ERROR;
  }
  if (per_sm < 1) {
    set_noalloc_error("the Fermi kernel cannot be resident on this device");
    return SQ_CUDA_ERROR;
  }
  // one CTA per SM (co-resident for the cooperative launch), as the handle-based path uses
  const int grid = std::min(sms, kNoallocMaxBlocks);
  if ((e = cudaMemsetAsync(&scr->status, 0, sizeof(int), s)) != cudaSuccess ||
      (e = launch_fermi(d_lambda, d_weights, n_nodes, n_qp, beta, n_electrons, dV, tol, maxit,
                        d_rho, scr->out, scr->partials, scr->barrier, &scr->status, grid, s)) !=
          cudaSuccess) {
    set_noalloc_error(std::string("fermi kernel: ") + cudaGetErrorString(e));
    return SQ_CUDA_ERROR;
  }
  double res[4];
  int st = 0;
  if ((e = cudaMemcpyAsync(res, scr->out, sizeof(res), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (e = cudaMemcpyAsync(&st, &scr->status, sizeof(int), cudaMemcpyDeviceToHost, s)) !=
          cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess) {
    set_noalloc_error(std::string("result copy: ") + cudaGetErrorString(e));
    return SQ_CUDA_ERROR;
  }
  if (st & kStatusTimeout) {
    set_noalloc_error("a device-side wait gave up");
    return SQ_DEVICE_TIMEOUT;
  }
  out[0] = res[0];
  out[1] = res[1];
  out[2] = res[2];
  // res[3] = bisection steps taken; the kernel leaves the loop early once hi - lo < tol, so
  // reaching maxit means the bracket never got that narrow
  if (res[3] >= (double)maxit) {
    set_noalloc_error("Fermi bisection did not reach tol in maxit steps (outputs hold the last "
                      "midpoint)");
    return SQ_NO_CONVERGENCE;
  }
  return SQ_OK;
}

}  // namespace sq
