// BiCGStab on the device with the semantics of PETSc 3.10 KSPSolve_BCGS, the
// Krylov method of the reference's input/petsc_options_bcgs.dat:1 (read
// through SolverPetsc.cpp:101): left preconditioning, x0 = 0, the
// preconditioned residual norm in KSPConvergedDefault, breakdown when
// (v, rp) = 0 or rho = 0, and the t = 0 exit (x += alpha p) of the omega
// step.  Every scalar lives in a device control block updated by the last
// CTA of a deterministic reduction (grid and order fixed by n), so iterations
// can be enqueued in CUDA-graph chunks without host round trips; once the
// solve has ended every kernel of a later iteration returns at once.
//
// One iteration (vectors r, rp, p, v, s, t, x; M^-1 A applied by the caller
// between the kernels):
//   bcgs_p       p = r - omega_old beta v + beta p
//   (caller)     v = M^-1 A p
//   bcgs_alpha   alpha = rho / (v, rp)
//   bcgs_s       s = r - alpha v
//   (caller)     t = M^-1 A s
//   bcgs_omega   omega = (s, t) / (t, t)
//   bcgs_xr      x = alpha p + omega s + x, r = s - omega t, ||r||, rho = (r, rp)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "linalg_kernels.cuh"

namespace cfdgpu {

struct BcgsState {
  int its, reason, active, maxit;
  int tzero;                // (t, t) = 0 and (s, s) = 0: x += alpha p ends the solve
  int skip;                 // inner solve of a flexible GMRES step whose cycle has ended: nothing runs
  double rtol, atol, dtol, rnorm0, ttol;
  double rho, rhoold, alpha, omega, omegaold, beta, dp;
  unsigned int counter;
};

// KSPConvergedDefault on the BCGS control block
__device__ __forceinline__ int bcgs_converged(BcgsState *s, int n_its, double rnorm)
{
  if (n_its == 0) {
    s->rnorm0 = rnorm;
    s->ttol = fmax(s->rtol * rnorm, s->atol);
  }
  if (isnan(rnorm) || isinf(rnorm)) return -9;
  if (rnorm <= s->ttol) return (rnorm < s->atol) ? 3 : 2;
  if (rnorm >= s->dtol * s->rnorm0) return -4;
  return 0;
}

__global__ void bcgs_setup(BcgsState *st, int maxit, double rtol, double atol, double dtol,
                           const GmresState *__restrict__ outer = nullptr, int j = 0)
{
  if (threadIdx.x || blockIdx.x) return;
  st->skip = (outer && (!outer->active || outer->it != j)) ? 1 : 0;
  st->its = 0; st->reason = 0; st->active = 0; st->maxit = maxit; st->tzero = 0;
  st->rtol = rtol; st->atol = atol; st->dtol = dtol; st->rnorm0 = 0.0; st->ttol = 0.0;
  st->rho = 0.0; st->rhoold = 1.0; st->alpha = 1.0; st->omega = 1.0; st->omegaold = 1.0; st->beta = 0.0;
  st->dp = 0.0;
  st->counter = 0u;
}

// Reductions.  A kernel's CTAs leave one partial sum each; the last CTA to
// arrive adds them with all its threads (a fixed tree), and a small vector gets a
// small grid.  With 296 CTAs always and one thread adding 296 partials, alpha,
// omega and xr took 8.7, 24.3 and 12.6 us on 6,912 dofs and 14.5, 29.6 and 23.9 on
// 1.1 M; now 4.2, 5.0, 5.8 and 9.4, 11.4, 15.5 (1.1 M: bound by the vectors' 9 MB
// each from L2).  Inner products are carried as unevaluated pairs hi + lo
// (products split exactly by FMA, Knuth's two-sum; Ogita, Rump and Oishi, 2005):
// BiCGStab's (r, rp) and (v, rp) fall many orders below the sum of their terms'
// magnitudes, and a plain sum can then cancel to exactly 0.0, which the
// breakdown rule takes for an orthogonal vector.  The transformations are exact
// only as written, each operation rounded once: the _rn intrinsics are never
// contracted, where a compiler may turn x * y + a into one FMA.
struct Pair {
  double hi, lo;
};

__device__ __forceinline__ Pair pair_add(const Pair &a, const Pair &b)
{
  const double s = __dadd_rn(a.hi, b.hi), t = __dsub_rn(s, a.hi);
  return {s, (a.lo + b.lo) + (__dsub_rn(a.hi, __dsub_rn(s, t)) + __dsub_rn(b.hi, t))};
}

__device__ __forceinline__ void pair_fma(Pair &acc, double x, double y)
{
  const double p = __dmul_rn(x, y);
  acc = pair_add(acc, {p, fma(x, y, -p)});
}

// FP32 vectors (the inner solves of the mixed-precision path) have products that
// are exact in 64 bits and a tolerance of a digit or two: plain sums, and always in
// the same order (RED_BLOCKS CTAs, their partials one after another), because the
// outer solve carries the last bit of alpha and omega on into the pressure level
// that it ends at.  The partials are loaded by all threads and added from shared memory.
template <typename VT> struct SumOf { using type = Pair; };
template <> struct SumOf<float> { using type = double; };
template <typename VT> using Sum = typename SumOf<VT>::type;
template <typename VT> inline int bcgs_grid(int64_t n) { return sizeof(VT) == 4 ? RED_BLOCKS : red_grid(n); }
__device__ __forceinline__ void sum_fma(Pair &acc, double x, double y) { pair_fma(acc, x, y); }
__device__ __forceinline__ void sum_fma(double &acc, double x, double y) { acc = fma(x, y, acc); }
// a sum that has overflowed is what the plain sum would be: its error term is not a number
__device__ __forceinline__ double sum_value(const Pair &v) { return isfinite(v.hi) ? v.hi + v.lo : v.hi; }
__device__ __forceinline__ double sum_value(double v) { return v; }

// sum over the CTA, valid in every thread; sh: RED_THREADS / 32 entries
__device__ __forceinline__ Pair block_sum_pair(Pair v, Pair *sh)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = pair_add(v, {__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
  __syncthreads();
  if (threadIdx.x % 32 == 0) sh[threadIdx.x / 32] = v;
  __syncthreads();
  v = sh[0];
#pragma unroll
  for (int k = 1; k < RED_THREADS / 32; k++) v = pair_add(v, sh[k]);
  return v;
}

// The CTA's K sums to memory; true in the last CTA to arrive, whose threads
// then all hold the K totals in v.  partial: 2 * K * gridDim.x doubles.
template <int K>
__device__ __forceinline__ bool reduce_all(Pair (&v)[K], double *__restrict__ partial, unsigned int *counter)
{
  __shared__ Pair sh[RED_THREADS / 32];
  Pair *const mine = reinterpret_cast<Pair *>(partial);
#pragma unroll
  for (int q = 0; q < K; q++) {
    const Pair t = block_sum_pair(v[q], sh);
    if (threadIdx.x == 0) mine[q * gridDim.x + blockIdx.x] = t;
  }
  if (!last_block(counter, gridDim.x)) return false;
#pragma unroll
  for (int q = 0; q < K; q++) {
    Pair t{0.0, 0.0};
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += RED_THREADS) {
      const double2 p = __ldcg(reinterpret_cast<const double2 *>(partial) + q * gridDim.x + k);
      t = pair_add(t, {p.x, p.y});
    }
    v[q] = block_sum_pair(t, sh);
  }
  return true;
}

template <int K>
__device__ __forceinline__ bool reduce_all(double (&v)[K], double *__restrict__ partial, unsigned int *counter)
{
  __shared__ double sh[RED_THREADS / 32], all[K * RED_BLOCKS], total[K];
#pragma unroll
  for (int q = 0; q < K; q++) {
    const double t = block_sum<RED_THREADS>(v[q], sh);
    if (threadIdx.x == 0) partial[q * gridDim.x + blockIdx.x] = t;
  }
  if (!last_block(counter, gridDim.x)) return false;
  for (unsigned int k = threadIdx.x; k < K * gridDim.x; k += RED_THREADS) all[k] = __ldcg(partial + k);
  __syncthreads();
  if (threadIdx.x < K) total[threadIdx.x] = sum_in_order(all + threadIdx.x * gridDim.x, gridDim.x);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < K; q++) v[q] = total[q];
  return true;
}

// Start: r holds M^-1 b.  rp = r, p = v = 0, dp = ||r||, rho = (r, rp),
// convergence test at iteration 0.
template <typename VT>
__global__ void __launch_bounds__(RED_THREADS)
bcgs_init(int64_t n, const VT *__restrict__ r, VT *__restrict__ rp, VT *__restrict__ p, VT *__restrict__ v,
          BcgsState *st, double *__restrict__ partial)
{
  if (st->skip) return;
  Sum<VT> s[1] = {};
  for (int64_t i = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_THREADS) {
    const VT x = r[i];
    rp[i] = x;
    p[i] = VT(0);
    v[i] = VT(0);
    sum_fma(s[0], (double)x, (double)x);
  }
  if (reduce_all(s, partial, &st->counter) && threadIdx.x == 0) {
    const double t = sum_value(s[0]);
    const double dp = sqrt(t);
    st->dp = dp;
    st->its = 0;
    const int reason = bcgs_converged(st, 0, dp);
    st->reason = reason;
    st->active = (reason == 0 && st->maxit > 0) ? 1 : 0;
    // first iteration: rho = (r, rp), beta = (rho / 1) (1 / 1)
    st->rho = t;
    st->rhoold = 1.0; st->alpha = 1.0; st->omegaold = 1.0;
    st->beta = (st->rho / st->rhoold) * (st->alpha / st->omegaold);
  }
}

template <typename VT>
__global__ void bcgs_p(int64_t n, const VT *__restrict__ r, const VT *__restrict__ v, VT *__restrict__ p,
                       const BcgsState *__restrict__ st)
{
  if (!st->active) return;
  const double b = st->beta, c = -st->omegaold * st->beta;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = (VT)(1.0 * (double)r[i] + c * (double)v[i] + b * (double)p[i]);
}

// alpha = rho / (v, rp); (v, rp) = 0 is a breakdown
template <typename VT>
__global__ void __launch_bounds__(RED_THREADS)
bcgs_alpha(int64_t n, const VT *__restrict__ v, const VT *__restrict__ rp, BcgsState *st, double *__restrict__ partial)
{
  if (!st->active) return;
  Sum<VT> s[1] = {};
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_THREADS)
    sum_fma(s[0], (double)v[i], (double)rp[i]);
  if (reduce_all(s, partial, &st->counter) && threadIdx.x == 0) {
    const double d1 = sum_value(s[0]);
    if (isnan(d1) || isinf(d1)) {
      st->reason = -9; st->active = 0;      // KSP_DIVERGED_NANORINF
    } else if (d1 == 0.0) {
      st->reason = -5; st->active = 0;      // KSP_DIVERGED_BREAKDOWN
    } else {
      st->alpha = st->rho / d1;
    }
  }
}

template <typename VT>
__global__ void bcgs_s(int64_t n, const VT *__restrict__ r, const VT *__restrict__ v, VT *__restrict__ s,
                       const BcgsState *__restrict__ st)
{
  if (!st->active) return;
  const double a = -st->alpha;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s[i] = (VT)(a * (double)v[i] + (double)r[i]);
}

// omega = (s, t) / (t, t); (t, t) = 0 ends the solve (x += alpha p) when
// s = 0, else it is a breakdown
template <typename VT>
__global__ void __launch_bounds__(RED_THREADS)
bcgs_omega(int64_t n, const VT *__restrict__ s, const VT *__restrict__ t, BcgsState *st, double *__restrict__ partial)
{
  if (!st->active) return;
  Sum<VT> d[3] = {};
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_THREADS) {
    const double si = (double)s[i], ti = (double)t[i];
    sum_fma(d[0], si, ti);
    sum_fma(d[1], ti, ti);
    sum_fma(d[2], si, si);
  }
  if (reduce_all(d, partial, &st->counter) && threadIdx.x == 0) {
    const double d1 = sum_value(d[0]), d2 = sum_value(d[1]), d3 = sum_value(d[2]);
    if (d2 == 0.0) {
      if (d3 != 0.0) {
        st->reason = -5; st->active = 0;    // singular preconditioned operator
      } else {
        st->tzero = 1;
        st->omega = 0.0;
      }
    } else {
      st->omega = d1 / d2;
    }
  }
}

// x = alpha p + omega s + x, r = s - omega t; dp = ||r||, convergence test,
// then rho of the next iteration = (r, rp) and its beta
template <typename VT>
__global__ void __launch_bounds__(RED_THREADS)
bcgs_xr(int64_t n, double *__restrict__ x, const VT *__restrict__ p, const VT *__restrict__ s, const VT *__restrict__ t,
        VT *__restrict__ r, const VT *__restrict__ rp, BcgsState *st, double *__restrict__ partial)
{
  if (!st->active) return;
  const double alpha = st->alpha, omega = st->omega;
  const bool tz = st->tzero != 0;
  Sum<VT> d[2] = {};
#pragma unroll 2
  for (int64_t i = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_THREADS) {
    if (tz) {
      x[i] += alpha * (double)p[i];
    } else {
      x[i] = alpha * (double)p[i] + omega * (double)s[i] + 1.0 * x[i];
      const VT ri = (VT)(-omega * (double)t[i] + (double)s[i]);
      r[i] = ri;
      const double rd = (double)ri;
      sum_fma(d[0], rd, rd);
      sum_fma(d[1], rd, (double)rp[i]);
    }
  }
  if (reduce_all(d, partial, &st->counter) && threadIdx.x == 0) {
    st->its = st->its + 1;
    if (tz) {
      st->dp = 0.0;
      st->reason = 2;                       // KSP_CONVERGED_RTOL
      st->active = 0;
    } else {
      const double dp = sqrt(sum_value(d[0]));
      st->dp = dp;
      const double rho = st->rho;
      st->rhoold = rho;
      st->omegaold = omega;
      int reason = bcgs_converged(st, st->its, dp);
      if (reason == 0 && rho == 0.0) reason = -5;
      if (reason == 0 && st->its >= st->maxit) reason = -3;   // KSP_DIVERGED_ITS
      st->reason = reason;
      st->active = (reason == 0) ? 1 : 0;
      st->rho = sum_value(d[1]);
      st->beta = (st->rho / st->rhoold) * (st->alpha / st->omegaold);
    }
  }
}

}  // namespace cfdgpu
