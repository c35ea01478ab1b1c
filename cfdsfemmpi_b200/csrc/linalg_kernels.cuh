// Sparse and dense linear-algebra kernels for the nodal-block (BSR) system:
// SpMV with the preconditioner fused into its epilogue, deterministic
// reductions, and the device-side pieces of restarted GMRES (PETSc 3.10
// KSPGMRES semantics: classical Gram-Schmidt, left preconditioning,
// preconditioned-residual norm, KSPConvergedDefault; the reference calls it
// from src/base/SolverPetsc.cpp:253).
//
// Determinism: every reduction uses a fixed grid, a fixed per-thread stride,
// a fixed in-CTA tree, and a final pass (last CTA, or one warp per output)
// that adds the per-CTA partials in index order, so results do not depend on
// scheduling.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cfdgpu {

constexpr int RED_BLOCKS = 296;     // 2 x 148 SMs
constexpr int RED_THREADS = 256;

// ---------------------------------------------------------------------------
// GMRES control block (device memory).  One thread (the last CTA of a
// reduction kernel) updates it; every other kernel only reads it.
struct GmresState {
  int it;          // Arnoldi columns built in the current cycle
  int its;         // total iterations (KSP iteration count)
  int reason;      // KSPConvergedReason, 0 while iterating
  int active;      // current cycle continues
  int m;           // restart length
  int maxit;
  double rtol, atol, dtol;
  double rnorm0, ttol;
  double res;      // current residual-norm estimate
  double tt;       // norm of the newest Krylov vector
  double v0scale;  // 1/res for V_0 (kept for diagnostics; sigma[0] holds the scale)
  unsigned int counter;
};

struct GmresArrays {
  double *sigma;   // m+1: basis vector k is sigma[k] * V_k (the stored vectors are not normalised)
  double *H;       // (m+1) x m, column-major, see hidx()
  double *cs, *sn; // m
  double *grs;     // m+1
  double *y;       // m
  double *partial; // scratch for reductions: (m+1) * ntiles doubles
  double *coef;    // m+1: H(k, j) * sigma[k], the update coefficients of Arnoldi step j
  unsigned int *kcount;   // m/8+1 arrival counters of the multi-dot's k-groups (zero between launches)
};

__device__ __forceinline__ int ksp_converged(GmresState *s, int n_its, double rnorm)
{
  if (n_its == 0) {
    s->rnorm0 = rnorm;
    s->ttol = fmax(s->rtol * rnorm, s->atol);
  }
  if (isnan(rnorm) || isinf(rnorm)) return -9;            // KSP_DIVERGED_NANORINF
  if (rnorm <= s->ttol) return (rnorm < s->atol) ? 3 : 2; // KSP_CONVERGED_ATOL / RTOL
  if (rnorm >= s->dtol * s->rnorm0) return -4;            // KSP_DIVERGED_DTOL
  return 0;
}

// Block-level sum (fixed tree); result valid in thread 0.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sh)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x / 32, l = threadIdx.x % 32;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NT / 32; k++) r += sh[k];
  }
  __syncthreads();
  return r;
}

// Sum of an array in shared memory, one entry after another, by one thread.
__device__ __forceinline__ double sum_in_order(const double *v, unsigned int count)
{
  double t = 0.0;
#pragma unroll 8
  for (unsigned int k = 0; k < count; k++) t += v[k];
  return t;
}

// Returns true in exactly one CTA (the last to arrive), after all CTAs'
// partials are visible.
__device__ __forceinline__ bool last_block(unsigned int *counter, unsigned int nblocks)
{
  __shared__ bool amlast;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int t = atomicAdd(counter, 1u);
    amlast = (t == nblocks - 1);
  }
  __syncthreads();
  if (amlast) {
    __threadfence();
    if (threadIdx.x == 0) *counter = 0u;
  }
  return amlast;
}

// ---------------------------------------------------------------------------
// BSR SpMV, 4x4 blocks, FP64 vectors: one warp per block row; each lane loads
// two entries of a block (row q/2, columns 2(q%2), 2(q%2)+1 of block 'sub'),
// so a warp instruction reads four consecutive blocks (16-byte loads for FP64
// blocks).  MT = float gives the FP64 residual of the FP32 matrix used by the
// mixed-precision refinement.  MODE 0: y = M^-1 (A x), MODE 1: y = M^-1 (b - A x).
// PC: 0 none, 1 jacobi (dinv), 2 point-block (binv, 4x4 per node, row-major).
template <int MODE, int PC, typename MT>
__global__ void __launch_bounds__(256)
bsr4_spmv(int nrows, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
              const MT *__restrict__ val, const double *__restrict__ x, const double *__restrict__ b,
              const double *__restrict__ dinv, const double *__restrict__ binv, double *__restrict__ y,
              const GmresState *__restrict__ st, int j, const double *__restrict__ xscale,
              const int *__restrict__ active = nullptr)
{
  if (st && (!st->active || st->it != j)) return;
  if (active && !active[0]) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= nrows) return;
  const double xs = xscale ? xscale[0] : 1.0;
  const int sub = lane >> 3, q = lane & 7, row = q >> 1, cp = (q & 1) * 2;
  const int kb0 = rowptr[warp], kb1 = rowptr[warp + 1];
  double acc0 = 0.0, acc1 = 0.0;
  for (int kb = kb0 + sub; kb < kb1; kb += 4) {
    const int c = colidx[kb];
    double a0, a1;
    if constexpr (sizeof(MT) == 8) {
      const double2 a = *reinterpret_cast<const double2 *>(val + (int64_t)kb * 16 + row * 4 + cp);
      a0 = a.x; a1 = a.y;
    } else {
      const float2 a = *reinterpret_cast<const float2 *>(val + (int64_t)kb * 16 + row * 4 + cp);
      a0 = a.x; a1 = a.y;
    }
    const double2 xv = *reinterpret_cast<const double2 *>(x + (int64_t)c * 4 + cp);
    acc0 = fma(a0, xv.x, acc0);
    acc0 = fma(a1, xv.y, acc0);
  }
  double acc = acc0 + acc1;
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 8);
  acc += __shfl_xor_sync(0xffffffffu, acc, 16);
  acc *= xs;
  // lanes 0,2,4,6 hold rows 0..3
  const int64_t r = (int64_t)warp * 4 + row;
  double v = acc;
  if (MODE == 1) v = b[r] - acc;
  if (PC == 2) {
    const double v0 = __shfl_sync(0xffffffffu, v, 0), v1 = __shfl_sync(0xffffffffu, v, 2);
    const double v2 = __shfl_sync(0xffffffffu, v, 4), v3 = __shfl_sync(0xffffffffu, v, 6);
    if (lane < 8 && (lane & 1) == 0) {
      const double *Bi = binv + (int64_t)warp * 16 + row * 4;
      y[r] = Bi[0] * v0 + Bi[1] * v1 + Bi[2] * v2 + Bi[3] * v3;
    }
  } else if (lane < 8 && (lane & 1) == 0) {
    y[r] = (PC == 1) ? dinv[r] * v : v;
  }
}

// BSR SpMV, 4x4 FP32 blocks and FP32 vectors (inner solve of the mixed
// precision path): one warp per block row, lane = (block sub 0..7, row 0..3),
// each lane loads one 16-byte block row and the matching 16 bytes of x, so a
// warp instruction reads eight consecutive 64-byte blocks.
template <int PC>
__global__ void __launch_bounds__(256)
bsr4_spmv_f32(int nrows, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
              const float *__restrict__ val, const float *__restrict__ x, const float *__restrict__ dinv,
              const float *__restrict__ binv, float *__restrict__ y, const GmresState *__restrict__ st, int j,
              const double *__restrict__ xscale, const int *__restrict__ active = nullptr)
{
  if (st && (!st->active || st->it != j)) return;
  if (active && !active[0]) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= nrows) return;
  const float xs = xscale ? (float)xscale[0] : 1.f;
  const int sub = lane >> 2, row = lane & 3;
  const int kb0 = rowptr[warp], kb1 = rowptr[warp + 1];
  float acc = 0.f;
  for (int kb = kb0 + sub; kb < kb1; kb += 8) {
    const int c = colidx[kb];
    const float4 a = *reinterpret_cast<const float4 *>(val + (int64_t)kb * 16 + row * 4);
    const float4 xv = *reinterpret_cast<const float4 *>(x + (int64_t)c * 4);
    acc = fmaf(a.x, xv.x, acc);
    acc = fmaf(a.y, xv.y, acc);
    acc = fmaf(a.z, xv.z, acc);
    acc = fmaf(a.w, xv.w, acc);
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 4);
  acc += __shfl_xor_sync(0xffffffffu, acc, 8);
  acc += __shfl_xor_sync(0xffffffffu, acc, 16);
  acc *= xs;
  const int64_t r = (int64_t)warp * 4 + row;
  if (PC == 2) {
    const float v0 = __shfl_sync(0xffffffffu, acc, 0), v1 = __shfl_sync(0xffffffffu, acc, 1);
    const float v2 = __shfl_sync(0xffffffffu, acc, 2), v3 = __shfl_sync(0xffffffffu, acc, 3);
    if (lane < 4) {
      const float *Bi = binv + (int64_t)warp * 16 + row * 4;
      y[r] = Bi[0] * v0 + Bi[1] * v1 + Bi[2] * v2 + Bi[3] * v3;
    }
  } else if (lane < 4) {
    y[r] = (PC == 1) ? dinv[r] * acc : acc;
  }
}

// BSR SpMV, 3x3 blocks (2D): one warp per block row.  Lanes 3*sub + row load row
// 'row' of block 'sub' of ten and entry 'row' of its x, so the nine blocks of a
// quadrilateral mesh's row are one pass of contiguous loads; lanes 0, 1 and 2 then
// add a row each from shared memory, entry after entry.  Bound by the chain row
// pointer -> column -> x -> sum (27 FMAs); the preconditioner's entries are loaded
// ahead of it.  One thread per scalar row with the same sums, which waited for its
// blocks one after another and with point-block Jacobi went over the whole node
// three times, took 5.7 us (Jacobi, 363 unknowns) and 7.9 (point-block, 10,092);
// now 2.4 and 3.6.  ST: type of the vectors and of the sums; MT: of the blocks.
// With more rows than fill the chip it is bound by its instructions (three lanes of
// a warp add), and a thread per scalar row (bsr3_spmv_rows) is the better one from
// BSR3_WARPS rows on, those of the instances that share the chip taken together.
// Between events (about 5 us more), warps / threads, Jacobi and point-block:
// 10,201 nodes 11.0 / 11.9 and 11.6 / 13.0 us, 25,921 16.8 / 12.8 and 18.8 / 17.2,
// 160,801 72 / 36 and 81 / 67.  64 instances of 4,225 nodes: 127 / 118 ms a step.
constexpr int64_t BSR3_WARPS = 148 * 96;
template <int MODE, int PC, typename MT, typename ST>
__global__ void __launch_bounds__(256)
bsr3_spmv(int nrows, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
          const MT *__restrict__ val, const ST *__restrict__ x, const ST *__restrict__ b,
          const ST *__restrict__ dinv, const ST *__restrict__ binv, ST *__restrict__ y,
          const GmresState *__restrict__ st, int j, const double *__restrict__ xscale,
          const int *__restrict__ active = nullptr)
{
  if (st && (!st->active || st->it != j)) return;
  if (active && !active[0]) return;
  constexpr int PASS = 10;                       // blocks per pass; a row of 30 entries keeps 16-byte pairs
  __shared__ __align__(16) ST sa[8][3][3 * PASS], sx[8][3 * PASS];
  const int w = threadIdx.x >> 5, node = blockIdx.x * 8 + w;
  const int lane = threadIdx.x & 31;
  if (node >= nrows) return;
  const ST xs = xscale ? (ST)xscale[0] : (ST)1;
  const int sub = lane / 3, row = lane - 3 * sub;
  const int kb0 = rowptr[node], kb1 = rowptr[node + 1];
  const int64_t r = (int64_t)node * 3 + row;
  ST pc[3] = {}, br = 0;
  if (lane < 3) {
    if (MODE == 1) br = b[r];
    if (PC == 1) pc[0] = dinv[r];
    if (PC == 2) {
#pragma unroll
      for (int q = 0; q < 3; q++) pc[q] = binv[r * 3 + q];
    }
  }
  ST acc = 0;
  for (int k0 = kb0; k0 < kb1; k0 += PASS) {
    const int kb = k0 + sub;
    if (sub < PASS) {
      ST a[3] = {}, xv = 0;
      if (kb < kb1) {
        xv = x[(int64_t)colidx[kb] * 3 + row];
#pragma unroll
        for (int q = 0; q < 3; q++) a[q] = (ST)val[(int64_t)kb * 9 + row * 3 + q];
      }
#pragma unroll
      for (int q = 0; q < 3; q++) sa[w][row][3 * sub + q] = a[q];
      sx[w][3 * sub + row] = xv;
    }
    __syncwarp();
    if (lane < 3) {
#pragma unroll
      for (int k = 0; k < 3 * PASS; k++) acc = fma(sa[w][row][k], sx[w][k], acc);
    }
    __syncwarp();
  }
  ST v = (MODE == 1) ? br - xs * acc : xs * acc;
  if (PC == 1) v *= pc[0];
  if (PC == 2) {
    const ST v0 = __shfl_sync(0xffffffffu, v, 0), v1 = __shfl_sync(0xffffffffu, v, 1);
    const ST v2 = __shfl_sync(0xffffffffu, v, 2);
    v = fma(pc[2], v2, fma(pc[1], v1, pc[0] * v0));
  }
  if (lane < 3) y[r] = v;
}

// The same with one thread per scalar row, the same sums in the same order.  With
// point-block Jacobi a thread adds all three rows of its node.
template <int MODE, int PC, typename MT, typename ST>
__global__ void __launch_bounds__(256)
bsr3_spmv_rows(int nrows, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
               const MT *__restrict__ val, const ST *__restrict__ x, const ST *__restrict__ b,
               const ST *__restrict__ dinv, const ST *__restrict__ binv, ST *__restrict__ y,
               const GmresState *__restrict__ st, int j, const double *__restrict__ xscale,
               const int *__restrict__ active = nullptr)
{
  if (st && (!st->active || st->it != j)) return;
  if (active && !active[0]) return;
  const ST xs = xscale ? (ST)xscale[0] : (ST)1;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t node = t / 3;
  const int row = (int)(t % 3);
  if (node >= nrows) return;
  const int kb0 = rowptr[node], kb1 = rowptr[node + 1];
  auto sum = [&](int r) {
    ST acc = 0;
    for (int kb = kb0; kb < kb1; kb++) {
      const int64_t c = (int64_t)colidx[kb] * 3;
      const MT *a = val + (int64_t)kb * 9 + r * 3;
#pragma unroll
      for (int q = 0; q < 3; q++) acc = fma((ST)a[q], x[c + q], acc);
    }
    return (MODE == 1) ? b[node * 3 + r] - xs * acc : xs * acc;
  };
  ST v;
  if constexpr (PC == 2) {
    const ST v0 = sum(0), v1 = sum(1), v2 = sum(2);
    const ST *m = binv + node * 9 + row * 3;
    v = fma(m[2], v2, fma(m[1], v1, m[0] * v0));
  } else {
    v = sum(row);
    if (PC == 1) v *= dinv[t];
  }
  y[t] = v;
}

// The launch of either.
template <int MODE, int PC, typename MT, typename ST>
inline void launch_bsr3(cudaStream_t s, int sharers, int nrows, const int32_t *rowptr, const int32_t *colidx,
                        const MT *val, const ST *x, const ST *b, const ST *dinv, const ST *binv, ST *y,
                        const GmresState *st, int j, const double *xscale, const int *active = nullptr)
{
  if ((int64_t)nrows * sharers <= BSR3_WARPS)
    bsr3_spmv<MODE, PC, MT, ST><<<(int)((nrows * 32LL + 255) / 256), 256, 0, s>>>(nrows, rowptr, colidx, val, x, b, dinv, binv, y, st, j, xscale, active);
  else
    bsr3_spmv_rows<MODE, PC, MT, ST><<<(int)((nrows * 3LL + 255) / 256), 256, 0, s>>>(nrows, rowptr, colidx, val, x, b, dinv, binv, y, st, j, xscale, active);
}

// z = M^-1 r (stand-alone preconditioner application)
template <int NB, typename VT, typename PT>
__global__ void pc_apply(int64_t n, int pc, const PT *__restrict__ dinv, const PT *__restrict__ binv,
                         const VT *__restrict__ r, VT *__restrict__ z)
{
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  if (pc == 2) {
    const int64_t node = t / NB;
    const int row = (int)(t % NB);
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < NB; q++) s += (double)binv[node * NB * NB + row * NB + q] * (double)r[node * NB + q];
    z[t] = (VT)s;
  } else if (pc == 1) {
    z[t] = (VT)((double)dinv[t] * (double)r[t]);
  } else {
    z[t] = r[t];
  }
}

// Scalar-diagonal inverse and point-block inverses of the assembled matrix.
template <int NB, typename VT, typename PT>
__global__ void build_jacobi(int nnode, const int32_t *__restrict__ diag_slot, const VT *__restrict__ val,
                             PT *__restrict__ dinv, PT *__restrict__ binv, int pc)
{
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= nnode) return;
  const VT *B = val + (int64_t)diag_slot[node] * NB * NB;
  if (pc == 1) {
#pragma unroll
    for (int a = 0; a < NB; a++) {
      const double d = (double)B[a * NB + a];
      dinv[(int64_t)node * NB + a] = (PT)((d != 0.0) ? 1.0 / d : 1.0);
    }
    return;
  }
  // Gauss-Jordan with partial pivoting on the NB x NB diagonal block
  double A[NB][NB], I[NB][NB];
#pragma unroll
  for (int a = 0; a < NB; a++)
#pragma unroll
    for (int c = 0; c < NB; c++) { A[a][c] = (double)B[a * NB + c]; I[a][c] = (a == c) ? 1.0 : 0.0; }
#pragma unroll
  for (int c = 0; c < NB; c++) {
    int piv = c;
#pragma unroll
    for (int r = c + 1; r < NB; r++)
      if (fabs(A[r][c]) > fabs(A[piv][c])) piv = r;
#pragma unroll
    for (int k = 0; k < NB; k++) {
      if (piv != c) {
        double t = A[c][k]; A[c][k] = A[piv][k]; A[piv][k] = t;
        t = I[c][k]; I[c][k] = I[piv][k]; I[piv][k] = t;
      }
    }
    const double p = A[c][c];
    const double d = (p != 0.0) ? 1.0 / p : 1.0;
#pragma unroll
    for (int k = 0; k < NB; k++) { A[c][k] *= d; I[c][k] *= d; }
#pragma unroll
    for (int r = 0; r < NB; r++) {
      if (r == c) continue;
      const double f = A[r][c];
#pragma unroll
      for (int k = 0; k < NB; k++) { A[r][k] -= f * A[c][k]; I[r][k] -= f * I[c][k]; }
    }
  }
#pragma unroll
  for (int a = 0; a < NB; a++)
#pragma unroll
    for (int c = 0; c < NB; c++) binv[(int64_t)node * NB * NB + a * NB + c] = (PT)I[a][c];
}

// The last CTA's sum of a grid's partials, all threads loading (fixed tree);
// result valid in thread 0.
__device__ __forceinline__ double sum_partials(const double *partial, unsigned int count, double *sh)
{
  double t = 0.0;
  for (unsigned int k = threadIdx.x; k < count; k += RED_THREADS) t += __ldcg(partial + k);
  return block_sum<RED_THREADS>(t, sh);
}

// The same one after another, result valid in thread 0; count <= RED_BLOCKS.  One
// thread that also loaded the 296 partials was most of the 11 us that a norm took.
__device__ __forceinline__ double sum_partials_in_order(const double *partial, unsigned int count)
{
  __shared__ double all[RED_BLOCKS];
  for (unsigned int k = threadIdx.x; k < count; k += RED_THREADS) all[k] = __ldcg(partial + k);
  __syncthreads();
  return threadIdx.x == 0 ? sum_in_order(all, count) : 0.0;
}

// CTAs of a reduction over n entries: four entries per thread, at most RED_BLOCKS
inline int red_grid(int64_t n)
{
  const int64_t g = (n + 4 * RED_THREADS - 1) / (4 * RED_THREADS);
  return (int)(g < 1 ? 1 : g > RED_BLOCKS ? RED_BLOCKS : g);
}

// ---------------------------------------------------------------------------
// deterministic 2-norm: out[0] = ||x||; partials in scratch
__global__ void __launch_bounds__(RED_THREADS)
norm2_kernel(int64_t n, const double *__restrict__ x, double *__restrict__ partial, unsigned int *counter,
             double *__restrict__ out)
{
  __shared__ double sh[RED_THREADS / 32];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_THREADS)
    s = fma(x[i], x[i], s);
  s = block_sum<RED_THREADS>(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
  if (last_block(counter, gridDim.x)) {
    const double t = sum_partials_in_order(partial, gridDim.x);
    if (threadIdx.x == 0) out[0] = sqrt(t);
  }
}

// 16-byte chunks of a Krylov vector: 2 doubles or 4 floats.  Arithmetic on
// the values is FP64 in every kernel; FP32 vectors only change the storage.
template <typename VT> struct Chunk;
template <> struct Chunk<double> {
  static constexpr int E = 2;
  static __device__ __forceinline__ void load(const double *p, double (&v)[2])
  {
    const double2 t = *reinterpret_cast<const double2 *>(p);
    v[0] = t.x; v[1] = t.y;
  }
  static __device__ __forceinline__ void store(double *p, const double (&v)[2])
  {
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
  }
};
template <> struct Chunk<float> {
  static constexpr int E = 4;
  static __device__ __forceinline__ void load(const float *p, double (&v)[4])
  {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  }
  static __device__ __forceinline__ void store(float *p, const double (&v)[4])
  {
    *reinterpret_cast<float4 *>(p) = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
  }
};

// Gram data of two residual differences k_i = a - b_i (deterministic):
// out = [<a,k1>, <a,k2>, <k1,k1>, <k1,k2>, <k2,k2>]; partial holds 5*gridDim.x
__global__ void __launch_bounds__(RED_THREADS)
minres_dots2(int64_t n, const double *__restrict__ a, const double *__restrict__ b1, const double *__restrict__ b2,
             double *__restrict__ partial, unsigned int *counter, double *__restrict__ out)
{
  __shared__ double sh[RED_THREADS / 32];
  double s[5] = {0, 0, 0, 0, 0};
  for (int64_t i = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_THREADS) {
    const double k1 = a[i] - b1[i], k2 = a[i] - b2[i];
    s[0] = fma(a[i], k1, s[0]);
    s[1] = fma(a[i], k2, s[1]);
    s[2] = fma(k1, k1, s[2]);
    s[3] = fma(k1, k2, s[3]);
    s[4] = fma(k2, k2, s[4]);
  }
#pragma unroll
  for (int q = 0; q < 5; q++) {
    const double t = block_sum<RED_THREADS>(s[q], sh);
    if (threadIdx.x == 0) partial[5 * blockIdx.x + q] = t;
  }
  if (last_block(counter, gridDim.x)) {
    __shared__ double all[5][RED_BLOCKS];
    for (unsigned int k = threadIdx.x; k < 5 * gridDim.x; k += RED_THREADS) all[k % 5][k / 5] = __ldcg(partial + k);
    __syncthreads();
    if (threadIdx.x < 5) out[threadIdx.x] = sum_in_order(all[threadIdx.x], gridDim.x);
  }
}

// GMRES cycle start: res = ||V0||, convergence test at its, v0scale.
template <typename VT>
__global__ void __launch_bounds__(RED_THREADS)
gmres_start(int64_t n, const VT *__restrict__ v0, GmresState *st, GmresArrays ga)
{
  __shared__ double sh[RED_THREADS / 32];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_THREADS) {
    const double v = (double)v0[i];
    s = fma(v, v, s);
  }
  s = block_sum<RED_THREADS>(s, sh);
  if (threadIdx.x == 0) ga.partial[blockIdx.x] = s;
  if (last_block(&st->counter, gridDim.x)) {
    const double t = sum_partials_in_order(ga.partial, gridDim.x);
    if (threadIdx.x == 0) {
      const double res = sqrt(t);
      st->res = res;
      st->it = 0;
      ga.grs[0] = res;
      st->v0scale = (res != 0.0) ? 1.0 / res : 0.0;
      ga.sigma[0] = (res != 0.0) ? 1.0 / res : 1.0;
      if (res == 0.0) {
        if (st->its == 0) { st->rnorm0 = 0.0; st->ttol = st->atol; }
        st->reason = 3;   // KSP_CONVERGED_ATOL: zero residual on entry
        st->active = 0;
      } else {
        st->reason = ksp_converged(st, st->its, res);
        st->active = (st->reason == 0 && st->its < st->maxit && st->m > 0) ? 1 : 0;
      }
    }
  }
}

// Hessenberg storage: column-major, leading dimension m+1: H(r, c) = H[c*(m+1) + r].
__device__ __forceinline__ int64_t hidx(int r, int c, int m) { return (int64_t)c * (m + 1) + r; }

// Krylov vectors are stored with a leading dimension ldv that is a multiple
// of 512 entries; entries n..ldv-1 stay zero, so every kernel below processes
// 16-byte chunks (Chunk<VT>::E entries) over nchunk = ldv / E.
constexpr int ORTHO_THREADS = 256;
constexpr int MDOT_KC = 8;          // basis vectors per CTA in the multi-dot

// Classical Gram-Schmidt dot products <w, V_k> for a group of MDOT_KC
// vectors per grid row: grid (ntiles, ceil((j+1)/KC)).  Every CTA stores its
// tile partial sums; the last CTA to arrive in a grid row adds that row's
// partials (one warp per k, lanes strided over the tiles, then a fixed
// shuffle tree) and stores H(k, j) = sigma_k <w, V_k> and the update
// coefficient H(k, j) sigma_k.
template <typename VT>
__global__ void __launch_bounds__(ORTHO_THREADS)
gmres_mdot(int64_t nchunk, const VT *__restrict__ V, int64_t ldv, int j, const GmresState *__restrict__ st,
           GmresArrays ga)
{
  double *__restrict__ partial = ga.partial;
  if (!st->active || st->it != j) return;
  constexpr int E = Chunk<VT>::E;
  __shared__ double sh[MDOT_KC][ORTHO_THREADS / 32];
  const int k0 = blockIdx.y * MDOT_KC;
  const int nk = min(MDOT_KC, j + 1 - k0);
  const int64_t p = (int64_t)blockIdx.x * ORTHO_THREADS + threadIdx.x;
  const VT *w = V + (int64_t)(j + 1) * ldv;
  double acc[MDOT_KC];
#pragma unroll
  for (int q = 0; q < MDOT_KC; q++) acc[q] = 0.0;
  if (p < nchunk) {
    double wv[E];
    Chunk<VT>::load(w + E * p, wv);
#pragma unroll
    for (int q = 0; q < MDOT_KC; q++) {
      if (q < nk) {
        double v[E];
        Chunk<VT>::load(V + (int64_t)(k0 + q) * ldv + E * p, v);
        double a = wv[0] * v[0];
#pragma unroll
        for (int e = 1; e < E; e++) a = fma(wv[e], v[e], a);
        acc[q] = a;
      }
    }
  }
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < MDOT_KC; q++) {
    double v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sh[q][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < nk) {
    double t = 0.0;
#pragma unroll
    for (int w2 = 0; w2 < ORTHO_THREADS / 32; w2++) t += sh[threadIdx.x][w2];
    partial[(int64_t)(k0 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
  }
  if (last_block(&ga.kcount[blockIdx.y], gridDim.x)) {
    if (wid < nk) {
      const int k = k0 + wid;
      const double *pp = partial + (int64_t)k * gridDim.x;
      double t = 0.0;
      for (unsigned int b = lane; b < gridDim.x; b += 32) t += __ldcg(pp + b);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) {
        const double hkj = ga.sigma[k] * t;
        ga.H[hidx(k, j, st->m)] = hkj;
        ga.coef[k] = hkj * ga.sigma[k];
      }
    }
  }
}

// The same for few unknowns: one CTA per basis vector, which needs no second
// stage over partial sums (a fence, an atomic and a dependent read, a third of
// the multi-dot's 3.7 us at 363 unknowns; now 1.8).  256 threads up to MDOT_EACH
// chunks, 1024 up to MDOT_EACH_WIDE, where a CTA's two vectors take as long as the
// second stage; beyond, up to MDOT_EACH_FULL, only with a CTA for every SM (the
// tiles use the whole chip for a few vectors too).  Mean over a GMRES(400) solve,
// tiles -> this, us: 4,332 unknowns 5.1 -> 3.6, 10,092 6.1 -> 4.5, 15,987 7.4 -> 5.1,
// 30,603 11.5 -> 7.9, 51,483 20.2 -> 14.6.
constexpr int64_t MDOT_EACH = 8 * ORTHO_THREADS, MDOT_EACH_WIDE = 8 * 1024, MDOT_EACH_FULL = 32 * 1024;
inline bool mdot_each(int64_t nchunk, int vectors)
{
  return nchunk <= MDOT_EACH_WIDE || (nchunk <= MDOT_EACH_FULL && vectors >= 148);
}
template <typename VT, int NT>
__global__ void __launch_bounds__(NT)
gmres_mdot_each(int64_t nchunk, const VT *__restrict__ V, int64_t ldv, int j, const GmresState *__restrict__ st,
                GmresArrays ga)
{
  if (!st->active || st->it != j) return;
  constexpr int E = Chunk<VT>::E;
  __shared__ double sh[NT / 32];
  const int k = blockIdx.x;
  const VT *v = V + (int64_t)k * ldv, *w = V + (int64_t)(j + 1) * ldv;
  const double sigma = ga.sigma[k];
  double acc = 0.0;
  constexpr int UN = 4;
  for (int64_t p0 = threadIdx.x; p0 < nchunk; p0 += UN * NT) {
    double a[UN][E], b[UN][E];
#pragma unroll
    for (int t = 0; t < UN; t++) {
      if (p0 + t * NT < nchunk) {
        Chunk<VT>::load(v + E * (p0 + t * NT), a[t]);
        Chunk<VT>::load(w + E * (p0 + t * NT), b[t]);
      }
    }
#pragma unroll
    for (int t = 0; t < UN; t++) {
      if (p0 + t * NT < nchunk) {
#pragma unroll
        for (int e = 0; e < E; e++) acc = fma(a[t][e], b[t][e], acc);
      }
    }
  }
  acc = block_sum<NT>(acc, sh);
  if (threadIdx.x == 0) {
    const double hkj = sigma * acc;
    ga.H[hidx(k, j, st->m)] = hkj;
    ga.coef[k] = hkj * sigma;
  }
}

// The same sums, in the same order, for instances that share the chip (a batch):
// there no SM is idle and what counts is the work, so a CTA of 256 threads takes
// MDOT_SHARED vectors and reads w once for them.  Thread t does the part of threads
// t, t + 256, .. of a CTA of NT.  With a CTA per vector 64 instances of 12,675
// unknowns (up to 200 vectors) took 133 ms a step instead of 118.
constexpr int MDOT_SHARED = 4;
inline bool mdot_shared(int threads, int vectors, int sharers)
{
  return sharers > 1 && (int64_t)sharers * vectors * threads > 148 * 2048;
}
template <typename VT, int NT>
__global__ void __launch_bounds__(ORTHO_THREADS)
gmres_mdot_shared(int64_t nchunk, const VT *__restrict__ V, int64_t ldv, int j, const GmresState *__restrict__ st,
                  GmresArrays ga)
{
  if (!st->active || st->it != j) return;
  constexpr int E = Chunk<VT>::E, VEC = MDOT_SHARED, PARTS = NT / ORTHO_THREADS, W = ORTHO_THREADS / 32;
  constexpr int UN = PARTS > 1 ? 2 : 1;      // parts whose loads are in flight together
  static_assert(PARTS % UN == 0, "");
  __shared__ double sh[VEC][NT / 32];
  const int k0 = blockIdx.x * VEC;
  const VT *w = V + (int64_t)(j + 1) * ldv;
  const VT *v[VEC];
#pragma unroll
  for (int i = 0; i < VEC; i++) v[i] = V + (int64_t)min(k0 + i, j) * ldv;
  double acc[PARTS][VEC] = {};
  for (int64_t p0 = threadIdx.x; p0 < nchunk; p0 += NT) {
#pragma unroll
    for (int q0 = 0; q0 < PARTS; q0 += UN) {
      double a[UN][VEC][E], b[UN][E];
#pragma unroll
      for (int q = 0; q < UN; q++) {
        const int64_t p = p0 + (q0 + q) * ORTHO_THREADS;
        if (p < nchunk) {
          Chunk<VT>::load(w + E * p, b[q]);
#pragma unroll
          for (int i = 0; i < VEC; i++) Chunk<VT>::load(v[i] + E * p, a[q][i]);
        }
      }
#pragma unroll
      for (int q = 0; q < UN; q++) {
        if (p0 + (q0 + q) * ORTHO_THREADS < nchunk) {
#pragma unroll
          for (int i = 0; i < VEC; i++)
#pragma unroll
            for (int e = 0; e < E; e++) acc[q0 + q][i] = fma(a[q][i][e], b[q][e], acc[q0 + q][i]);
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < PARTS; q++)
#pragma unroll
    for (int i = 0; i < VEC; i++) {
      double t = acc[q][i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (threadIdx.x % 32 == 0) sh[i][q * W + threadIdx.x / 32] = t;
    }
  __syncthreads();
  const int k = k0 + threadIdx.x;
  if (threadIdx.x < VEC && k <= j) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < NT / 32; q++) t += sh[threadIdx.x][q];
    const double sigma = ga.sigma[k];
    const double hkj = sigma * t;
    ga.H[hidx(k, j, st->m)] = hkj;
    ga.coef[k] = hkj * sigma;
  }
}

// w -= sum_k h_k sigma_k V_k, then ||w||^2 partials.  A CTA covers CL * PER
// 16-byte chunks; its threads are 256 / CL sets of CL, and the k's fall into
// 256 / CL * RES groups, the residues of k modulo their number, RES of them to a
// set: a thread adds the terms of each of its groups for its PER chunks, UN * RES
// terms in flight, and the groups' sums are combined in a fixed order through
// shared memory.  One more CTA, the first, applies the stored Givens rotations to
// column j meanwhile (a serial chain of j steps, none of which needs the norm);
// the last CTA to arrive finishes the norm, forms the new rotation and runs the
// convergence test (KSPGMRESUpdateHessenberg, KSPConvergedDefault).  The last step
// of a chunk leaves a copy of the control block in pinned host memory (snap).
//
// Many unknowns (64 x 2 chunks): bound by reading V, 2 KB of a vector per CTA.  Few
// unknowns (16 x 1): V comes from L2 and the time is the latency of the terms that a
// thread adds one batch after another, so each CTA takes 16 chunks with 16
// groups, which fills the SMs and cuts the chain to j / 128 batches.
// With the wide form for every size and the rotations after the norm: 6.5 us at 363
// unknowns and 50 vectors, 15.5 at 10,092 and 300; now 5.0 and 7.5.
//
// The packed form (128 x 1, eight groups a thread) has an eighth of the narrow one's
// CTAs and the same 16 groups and partial sums, so the same bits.
constexpr int ROT_PER = 1024 / ORTHO_THREADS;      // columns per thread of the rotations (restart <= 1000)
constexpr int MAXPY_FEW_SPAN = 16, MAXPY_WIDE_SPAN = 128;
// The narrow form pays while its CTAs, three an SM, are resident at once (14,208 FP64
// unknowns): a step of the hex8 cavity with 19,652 and 37,044 unknowns took 9.6 and
// 13.6 ms with it and 8.8 and 11.0 with the wide one, quad4 with 30,603 25.8 and 23.2;
// with 12,675 5.9 and 6.9 the other way.  Instances that share the chip fill it
// together: 64 of 12,675 unknowns 148 ms a step with the narrow form, 118 with the
// packed one, 32 hex8 of 8,788 30.8 and 24.3.
constexpr int MAXPY_WAVE = 3 * 148;
constexpr int64_t MAXPY_FEW = (int64_t)MAXPY_FEW_SPAN * MAXPY_WAVE;
inline int maxpy_tiles(int64_t nchunk, bool few)
{
  const int span = few ? MAXPY_FEW_SPAN : MAXPY_WIDE_SPAN;
  return (int)((nchunk + span - 1) / span);
}
inline bool maxpy_narrow(int64_t nchunk, int sharers) { return (int64_t)maxpy_tiles(nchunk, true) * sharers <= MAXPY_WAVE; }
template <typename VT, int CL, int PER, int UN, int RES>
__global__ void __launch_bounds__(ORTHO_THREADS, PER > 1 ? 5 : RES > 1 ? 2 : 3)
gmres_maxpy_norm(int64_t nchunk, VT *__restrict__ V, int64_t ldv, int j, GmresState *st, GmresArrays ga,
                 GmresState *snap)
{
  if (!st->active || st->it != j) {
    if (snap && blockIdx.x == 0 && threadIdx.x == 0) *snap = *st;
    return;
  }
  constexpr int E = Chunk<VT>::E, SPAN = CL * PER, GROUPS = ORTHO_THREADS / CL * RES;
  constexpr int TILE = RES > 1 ? MAXPY_FEW_SPAN : SPAN;    // chunks of a partial sum
  static_assert(SPAN <= ORTHO_THREADS && (RES == 1 || (GROUPS == ORTHO_THREADS / MAXPY_FEW_SPAN && TILE == 16)), "");
  __shared__ double sh[ORTHO_THREADS / 32];
  __shared__ union {
    double qs[GROUPS][E][SPAN];
    struct {
      double2 step[1024 + 16];
      double a[1024 + 16];
    } rot;                         // the CTA of the rotations
  } u;
  const int m = st->m;
  if (blockIdx.x == 0) {
    // a_0 = h_0, a_{q+1} = c_q h_{q+1} - s_q a_q is the chain; the products
    // before it and the rotated entries c_q a_q + s_q h_{q+1} after it take all threads
    double2 *st2 = u.rot.step;
    double *a = u.rot.a;
    double *Hj = ga.H + hidx(0, j, m);
    double hq[ROT_PER], cq[ROT_PER], sq[ROT_PER];
#pragma unroll
    for (int i = 0; i < ROT_PER; i++) {
      const int q = i * ORTHO_THREADS + threadIdx.x;
      hq[i] = cq[i] = sq[i] = 0.0;
      if (q < j) { hq[i] = Hj[q + 1]; cq[i] = ga.cs[q]; sq[i] = ga.sn[q]; st2[q] = make_double2(sq[i], cq[i] * hq[i]); }
    }
    if (threadIdx.x == 0) a[0] = Hj[0];
    __syncthreads();
    if (threadIdx.x == 0) {
      // eight steps in registers, the next eight loaded ahead of them
      double v = a[0];
      double2 t[8], n[8];
#pragma unroll
      for (int i = 0; i < 8; i++) t[i] = st2[i];
      for (int q = 0; q < j; q += 8) {
#pragma unroll
        for (int i = 0; i < 8; i++) n[i] = st2[q + 8 + i];
        double o[8];
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = v = fma(-t[i].x, v, t[i].y);
#pragma unroll
        for (int i = 0; i < 8; i++) {
          a[q + 1 + i] = o[i];      // past j: not read
          t[i] = n[i];
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ROT_PER; i++) {
      const int q = i * ORTHO_THREADS + threadIdx.x;
      if (q < j) Hj[q] = cq[i] * a[q] + sq[i] * hq[i];
    }
    if (threadIdx.x == 0) Hj[j] = a[j];
  } else {
    // coefficients H(k, j) sigma_k (written by the multi-dot), read as
    // group-uniform broadcasts inside the loop
    const double *__restrict__ hk = ga.coef;
    VT *w = V + (int64_t)(j + 1) * ldv;
    const int lp = threadIdx.x % CL, g = threadIdx.x / CL;
    const int64_t c0 = (int64_t)(blockIdx.x - 1) * SPAN;
    // the chunk of w this thread finishes, loaded early; nchunk is a multiple
    // of 128 (ldv is one of 512 entries), the spans may reach past it
    const int64_t pfin = c0 + threadIdx.x;
    const bool fin = threadIdx.x < SPAN && pfin < nchunk;
    double wfin[E];
    if (fin) Chunk<VT>::load(w + E * pfin, wfin);
    double acc[RES][PER][E] = {};
    const VT *bp[PER];
    bool in[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const int64_t p = c0 + lp + i * CL;
      in[i] = p < nchunk;
      bp[i] = V + E * (in[i] ? p : c0);
    }
    if (in[0]) {
      for (int k = g * RES; k <= j; k += GROUPS * UN) {
        double v[UN][RES][PER][E], c[UN][RES];
#pragma unroll
        for (int t = 0; t < UN; t++)
#pragma unroll
          for (int r = 0; r < RES; r++) {
            const int kt = k + t * GROUPS + r;
            if (kt <= j) {
              c[t][r] = __ldg(hk + kt);
#pragma unroll
              for (int i = 0; i < PER; i++) Chunk<VT>::load(bp[i] + (int64_t)kt * ldv, v[t][r][i]);
            }
          }
#pragma unroll
        for (int t = 0; t < UN; t++)
#pragma unroll
          for (int r = 0; r < RES; r++) {
            if (k + t * GROUPS + r <= j) {
#pragma unroll
              for (int i = 0; i < PER; i++)
#pragma unroll
                for (int e = 0; e < E; e++) acc[r][i][e] = fma(c[t][r], v[t][r][i][e], acc[r][i][e]);
            }
          }
      }
    }
#pragma unroll
    for (int r = 0; r < RES; r++)
#pragma unroll
      for (int i = 0; i < PER; i++)
#pragma unroll
        for (int e = 0; e < E; e++) u.qs[g * RES + r][e][lp + i * CL] = acc[r][i][e];
    __syncthreads();
    double s = 0.0;
    if (fin) {
      double a[E];
#pragma unroll
      for (int e = 0; e < E; e++) {
        double q[GROUPS];
#pragma unroll
        for (int i = 0; i < GROUPS; i++) q[i] = u.qs[i][e][threadIdx.x];
#pragma unroll
        for (int d = 1; d < GROUPS; d *= 2)
#pragma unroll
          for (int i = 0; i < GROUPS; i += 2 * d) q[i] += q[i + d];
        a[e] = wfin[e] - q[0];
      }
      Chunk<VT>::store(w + E * pfin, a);
      // the norm is taken of the stored (possibly rounded) values
#pragma unroll
      for (int e = 0; e < E; e++) {
        const double v = (double)(VT)a[e];
        s = fma(v, v, s);
      }
    }
    if constexpr (RES > 1) {
      // half a warp each: the order of block_sum over 16 threads
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (fin && threadIdx.x % TILE == 0) ga.partial[pfin / TILE] = s;
    } else {
      s = block_sum<ORTHO_THREADS>(s, sh);
      if (threadIdx.x == 0) ga.partial[blockIdx.x - 1] = s;
    }
  }
  if (last_block(&st->counter, gridDim.x)) {
    double a = 0.0, g0 = 0.0;
    if (threadIdx.x == 0) { a = __ldcg(ga.H + hidx(j, j, m)); g0 = __ldcg(ga.grs + j); }
    const double t = sum_partials(ga.partial, (unsigned int)((nchunk + TILE - 1) / TILE), sh);
    if (threadIdx.x == 0) {
      const int it = j;
      const double tt = sqrt(t);
      st->tt = tt;
      ga.sigma[it + 1] = (tt != 0.0) ? 1.0 / tt : 1.0;   // VecNormalize, applied lazily
      double hapbnd = fabs(tt / g0);
      if (hapbnd > 1.0e-30) hapbnd = 1.0e-30;
      const bool hapend = tt < hapbnd;
      double res;
      int reason = 0;
      if (!hapend) {
        const double r = sqrt(a * a + tt * tt);
        if (r == 0.0) {
          reason = -2;   // KSP_DIVERGED_NULL
          res = st->res;
        } else {
          const double c = a / r, sn = tt / r;
          ga.cs[it] = c;
          ga.sn[it] = sn;
          res = -(sn * g0);
          ga.grs[it + 1] = res;
          ga.grs[it] = c * g0;
          ga.H[hidx(it, it, m)] = c * a + sn * tt;
          res = fabs(res);
        }
      } else {
        res = 0.0;
      }
      if (reason == 0) {
        st->it = it + 1;
        st->its = st->its + 1;
        st->res = res;
        reason = ksp_converged(st, st->its, res);
        if (hapend && reason == 0) reason = -5;   // KSP_DIVERGED_BREAKDOWN
      }
      st->reason = reason;
      st->active = (reason == 0 && st->it < m && st->its < st->maxit) ? 1 : 0;
      if (snap) *snap = *st;
    }
  }
}

// KSPGMRESBuildSoln back substitution, one CTA, 32 columns at a time from the
// last: one warp solves the diagonal block from registers (lane i holds row i,
// each y travels by shuffle), then the rows above take the block's columns, a
// thread each.  A quotient is r * (1/d) with one correction
// step, so the division is off the chain and the result as good as r / d.
// Bound by that chain, 60 cycles a column; a column at a time over the whole CTA,
// with a load, a division and two barriers in turn, took 280 us for 290 columns; now 45.
constexpr int BACKSUB_THREADS = 256;
__global__ void __launch_bounds__(BACKSUB_THREADS) gmres_backsub(GmresState *st, GmresArrays ga)
{
  __shared__ double r[1024];
  __shared__ double ys[32];
  const int it = st->it, m = st->m;
  if (it <= 0) return;
  for (int i = threadIdx.x; i < it; i += BACKSUB_THREADS) r[i] = ga.grs[i];
  const int lane = threadIdx.x & 31;
  for (int k1 = it; k1 > 0;) {
    const int k0 = (k1 - 1) & ~31, nc = k1 - k0;
    double col[32], inv = 0.0, d = 0.0;
    if (threadIdx.x < 32) {
#pragma unroll
      for (int c = 0; c < 32; c++) col[c] = (c < nc && lane < c) ? ga.H[hidx(k0 + lane, k0 + c, m)] : 0.0;
      if (lane < nc) d = ga.H[hidx(k0 + lane, k0 + lane, m)];
      inv = (d != 0.0) ? 1.0 / d : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      double v = (lane < nc) ? r[k0 + lane] : 0.0;
#pragma unroll
      for (int c = 31; c >= 0; c--) {
        double q = v * inv;
        q = isfinite(q) ? fma(fma(-q, d, v), inv, q) : v / d;
        const double y = __shfl_sync(0xffffffffu, q, c);
        if (lane < c) v = fma(-col[c], y, v);
        else if (lane == c) v = y;
      }
      if (lane < nc) ga.y[k0 + lane] = v;
      ys[lane] = (lane < nc) ? v : 0.0;
    }
    __syncthreads();
    // rows above the block, a thread each
    for (int i = threadIdx.x; i < k0; i += BACKSUB_THREADS) {
      double h[32], v = r[i];
#pragma unroll
      for (int c = 0; c < 32; c++) h[c] = (c < nc) ? ga.H[hidx(i, k0 + c, m)] : 0.0;
#pragma unroll
      for (int c = 31; c >= 0; c--) v = fma(-h[c], ys[c], v);
      r[i] = v;
    }
    k1 = k0;
  }
}

// x += scale * sum_{k < it} y_k sigma_k V_k  (x is FP64 whatever the basis
// type).  Up to 16 vectors a thread adds its entry's terms alone; from there on a
// CTA covers 32 entries, its eight warps taking the k's modulo 8 with eight loads
// in flight, so the latency of V is paid it / 64 times and not it / 4 times.
constexpr int UPDATE_SPAN = 32, UPDATE_ALONE = 16;
template <typename VT>
__global__ void __launch_bounds__(ORTHO_THREADS)
gmres_update_x(int64_t n, double *__restrict__ x, const VT *__restrict__ V, int64_t ldv,
               const GmresState *__restrict__ st, GmresArrays ga, double scale)
{
  constexpr int W = ORTHO_THREADS / 32;
  __shared__ double yk[1024];
  __shared__ double sh[W][UPDATE_SPAN];
  const int it = st->it;
  if (it <= 0) return;
  for (int k = threadIdx.x; k < it; k += blockDim.x) yk[k] = ga.y[k] * ga.sigma[k];
  __syncthreads();
  if (it <= UPDATE_ALONE) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
      double s = 0.0;
      for (int k = 0; k < it; k++) s = fma(yk[k], (double)V[(int64_t)k * ldv + i], s);
      x[i] += scale * s;
    }
    return;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t i0 = (int64_t)blockIdx.x * UPDATE_SPAN; i0 < n; i0 += (int64_t)gridDim.x * UPDATE_SPAN) {
    const int64_t i = i0 + lane;
    double s = 0.0;
    if (i < n) {
#pragma unroll 8
      for (int k = w; k < it; k += W) s = fma(yk[k], (double)V[(int64_t)k * ldv + i], s);
    }
    sh[w][lane] = s;
    __syncthreads();
    if (w == 0 && i < n) {
      double t = 0.0;
#pragma unroll
      for (int q = 0; q < W; q++) t += sh[q][lane];
      x[i] += scale * t;
    }
    __syncthreads();
  }
}

// FP32 copy of an FP64 array of any length
__global__ void k_round_to_f32(int64_t n, const double *__restrict__ a, float *__restrict__ b)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

// b32 = sigma * v (FP32): the normalised Arnoldi vector of a flexible GMRES
// step, the right-hand side of its inner solve; skipped once the cycle ended
__global__ void k_scale_v_to_f32(int64_t n, const double *__restrict__ v, const double *__restrict__ sigma,
                                 float *__restrict__ b32, const GmresState *__restrict__ st, int j)
{
  if (st && (!st->active || st->it != j)) return;
  const double s = sigma[0];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b32[i] = (float)(s * v[i]);
}

// mixed precision helpers: b32 = r64 * s (FP32), x64 += a * d64
__global__ void k_scale_to_f32(int64_t n, const double *__restrict__ r, const double *__restrict__ norm,
                               float *__restrict__ b32)
{
  const double s = (norm[0] != 0.0) ? 1.0 / norm[0] : 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b32[i] = (float)(r[i] * s);
}

__global__ void k_axpy_dev(int64_t n, const double *__restrict__ a, const double *__restrict__ d,
                           double *__restrict__ x)
{
  const double s = a[0];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] += s * d[i];
}

__global__ void gmres_init(GmresState *st, int m, int maxit, double rtol, double atol, double dtol)
{
  if (threadIdx.x || blockIdx.x) return;
  st->it = 0; st->its = 0; st->reason = 0; st->active = 0;
  st->m = m; st->maxit = maxit; st->rtol = rtol; st->atol = atol; st->dtol = dtol;
  st->rnorm0 = 0.0; st->ttol = 0.0; st->res = 0.0; st->tt = 0.0; st->v0scale = 0.0;
  st->counter = 0u;
}

}  // namespace cfdgpu
