// Block-Jacobi / block ILU(k) preconditioner on the nodal-block (BSR) matrix:
// numeric factorisation and the two triangular solves, for the reference's
// iterative option files (-pc_type bjacobi -sub_pc_type ilu
// -sub_pc_factor_levels k, input/petsc_options_gmres.dat:2-5 and
// input/petsc_options_bcgs.dat:2-5, read through SolverPetsc.cpp:101,111).
//
// Factor layout (pattern from build_ilu_pattern): per node row i the blocks
// fptr[i]..fptr[i+1]-1, columns fcol[] sorted, the diagonal at fdiag[i].
// Strictly lower blocks hold the multipliers L_ip (unit block-lower factor),
// the others U_ij; fdinv[i] holds the inverse of U_ii (pivoted Gauss-Jordan).
//
// Scheduling is sync-free.  Factorisation: one persistent grid whose warps draw
// rows from an atomic ticket in level-set order (computed on the host).  Rows of
// one level are independent, so a row only waits for rows handed out before it:
// a row whose inputs are not ready polls their flags (acquire loads with
// back-off), and a finished row publishes its flag after a fence.  Triangular solves: persistent CTAs draw groups of rows
// (trsv_plan.h), and the solved values are their own ready flags.  The earliest
// unfinished row always has its inputs, so progress is guaranteed; every wait
// is bounded and records a time-out in the control block instead of spinning
// forever.  Flags hold an epoch number: the last warp (CTA) of a launch resets
// the ticket and advances the epoch, so no per-launch reset kernel is needed
// and launches can be captured in CUDA graphs.  Every row's arithmetic runs in a
// fixed order, so results do not depend on scheduling.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "linalg_kernels.cuh"
#include "trsv_plan.h"
#include "warp_wait.h"

namespace cfdgpu {

__host__ __device__ constexpr size_t up_to_16(size_t x) { return (x + 15) / 16 * 16; }

struct TriCtl {
  unsigned int ticket;    // next chunk to hand out
  unsigned int exited;    // warps of the current launch that finished
  unsigned int epoch;     // launches completed; flags of this launch are set to epoch + 1
  unsigned int error;     // 0, or ILU_ERR_*
  int zero_pivot_row;     // factorisation: first row whose diagonal block is singular
};

constexpr unsigned int ILU_ERR_TIMEOUT = 1u;     // a dependency wait ran out (never expected)
constexpr unsigned int ILU_ERR_ZERO_PIVOT = 2u;  // singular diagonal block in the factorisation
constexpr int ILU_THREADS = 256;
constexpr int ILU_WARPS = ILU_THREADS / 32;
constexpr int ILU_SPIN_LIMIT = 1 << 21;          // ~1-2 s of polling per wait
#ifndef ILU_SPIN_HOT
#define ILU_SPIN_HOT 256
#endif
// polls without sleeping before the back-off starts: an input usually
// arrives within a few L2 round trips, and a sleeping warp wakes late
constexpr int ILU_SPIN_HOT_POLLS = ILU_SPIN_HOT;

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int *p)
{
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed_u32(unsigned int *p, unsigned int v)
{
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Wait (a whole warp on one flag, bounded) until *f == target: acquire loads,
// the first ILU_SPIN_HOT_POLLS back to back, then with exponential back-off.
// Returns false after a time-out, or when another warp has already timed out.
__device__ __forceinline__ bool wait_flag(const unsigned int *f, unsigned int target, TriCtl *ctl)
{
  unsigned int ns = 32;
  for (int it = 0; it < ILU_SPIN_LIMIT; it++) {
    if (ld_acquire_u32(f) == target) return true;
    if (it >= ILU_SPIN_HOT_POLLS) {
      __nanosleep(ns);
      if (ns < 1024) ns <<= 1;
      if (*(volatile unsigned int *)&ctl->error) return false;
    }
  }
  atomicCAS(&ctl->error, 0u, ILU_ERR_TIMEOUT);
  return false;
}

__device__ __forceinline__ int draw_ticket(TriCtl *ctl, int lane)
{
  unsigned int t = 0;
  if (lane == 0) t = atomicAdd(&ctl->ticket, 1u);
  return (int)__shfl_sync(0xffffffffu, t, 0);
}

// Exit accounting: the last warp of the launch resets the ticket and
// advances the epoch.
__device__ __forceinline__ void launch_done(TriCtl *ctl, int lane, unsigned int epoch)
{
  if (lane == 0) {
    __threadfence();
    const unsigned int nw = gridDim.x * (blockDim.x / 32);
    const unsigned int k = atomicAdd(&ctl->exited, 1u);
    if (k == nw - 1) {
      ctl->ticket = 0u;
      ctl->exited = 0u;
      __threadfence();
      *(volatile unsigned int *)&ctl->epoch = epoch + 1u;
      __threadfence();
    }
  }
}

// NB entries at p (a row of a block) past L1: other SMs write them
template <int NB, typename T>
__device__ __forceinline__ void ld_row(const T *p, double (&v)[NB])
{
  if constexpr (NB == 4 && sizeof(T) == 8) {
    const double2 a = __ldcg(reinterpret_cast<const double2 *>(p)), b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else if constexpr (NB == 4) {
    const float4 a = __ldcg(reinterpret_cast<const float4 *>(p));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  } else {
#pragma unroll
    for (int c = 0; c < NB; c++) v[c] = (double)__ldcg(p + c);
  }
}

// Inverse of the NB x NB block at A (row-major) by a warp: Gauss-Jordan with
// partial pivoting on [A | I], lane = (row, column) of its NB x 2 NB entries.
// Returns the lane's entry of the inverse (lanes with column >= NB); ok is
// false (in every lane) when a pivot column is zero.
template <int NB>
__device__ __forceinline__ double invert_block(const double *A, int lane, bool &ok)
{
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int C = 2 * NB;
  const int r = lane / C < NB ? lane / C : 0, c = lane % C;
  double v = c < NB ? A[r * NB + c] : (c - NB == r ? 1.0 : 0.0);
  ok = true;
#pragma unroll
  for (int k = 0; k < NB; k++) {
    double col[NB];
#pragma unroll
    for (int q = 0; q < NB; q++) col[q] = __shfl_sync(FULL, v, q * C + k);
    int piv = k;
    double best = col[k];
#pragma unroll
    for (int q = k + 1; q < NB; q++)
      if (fabs(col[q]) > fabs(best)) { piv = q; best = col[q]; }
    if (best == 0.0) ok = false;
    const double d = best != 0.0 ? 1.0 / best : 0.0;
    // rows k and piv change places
    const int from = r == k ? piv : r == piv ? k : r;
    double f = from == k ? col[k] : best;     // entry (r, k) after that
#pragma unroll
    for (int q = 0; q < NB; q++)
      if (q == r && q != k && q != piv) f = col[q];
    v = __shfl_sync(FULL, v, from * C + c);
    const double top = __shfl_sync(FULL, v, k * C + c) * d;
    v = r == k ? top : v - f * top;
  }
  return v;
}

// ---------------------------------------------------------------------------
// Numeric block ILU: one warp per node row, rows in level order.  For row i:
// W = the row of A on the factor pattern (fill blocks zero); for every pivot
// p < i of the row in increasing column order, L_ip = W_p U_pp^-1 and
// W_j -= L_ip U_pj for the blocks j > p of row p that lie in row i's pattern
// (list umap: the block's number in row p after the diagonal, and its place in
// row i: the halves of an ENT); then U_ii^-1.  AT is the type of the assembled
// matrix, FT of the factors; W is FP64 and lives in shared memory (with PLACES, rows
// of more than rowcap blocks in `scratch`).
//
// What bounds it: the dependency chain, per level the last pivot's hop.  With W
// in global memory, one fence per pivot and the inverse by one lane the kernel
// took 8.1 ms at 64^3 (hex8, ILU(0), 455 levels: 18 us each), 3.6 at 32^3, 0.58 at
// 11^3, 13.9 ms on the 256 x 128 O-grid with ILU(3) (1,404 levels) and 55.7 ms for
// the complete LU of the 64 x 64 cavity (4,224 levels).  Now a pivot's inverse and
// the blocks of its row are requested together once its flag is seen (pivots long
// done are found by one poll of all flags), and the row's blocks that others need
// are written and published before the rest: 2.9, 1.2, 0.25, 4.5 and 17.1 ms (FP32
// values are rounded where they were stored before, so the factors keep their bits).
// An instance whose rows all fit has no PLACES, and its accesses to W are known to be
// to shared memory: with a pointer to either it took 3.5, 1.5, 0.26, 4.5 and 18.8.
//
// UNR rounds of 32 / NB blocks are fetched at once.  Where a pivot's list takes more
// than two fetches of two rounds (rows of over factor_wide(NB) blocks: complete LU,
// high levels) the last pivot's fetches are on the chain one after another, and the
// WIDE form fetches seven rounds (four of 4x4 blocks) with one CTA per SM for the
// registers: complete LU of the 64 x 64 cavity 24.1 -> 18.9 ms (before the above).
// Seven rounds are 70 blocks of 3x3; a pivot's list has 84 on average there and the
// rest of it comes in a second fetch.  On shorter rows
// more rounds only cost registers (four on the O-grid: 4.5 -> 4.8 ms).
constexpr int factor_wide(int nb) { return 4 * (32 / nb) * 2; }
template <int NB, typename AT, typename FT, bool WIDE, bool PLACES, typename ENT>
__global__ void __launch_bounds__(ILU_THREADS, WIDE ? 1 : 2)
ilu_factor(int n, int rowcap, const int32_t *__restrict__ arow, const int32_t *__restrict__ aslot,
           const AT *__restrict__ aval, const int32_t *__restrict__ fptr, const int32_t *__restrict__ fcol,
           const int32_t *__restrict__ fdiag, const int64_t *__restrict__ uoff, const ENT *__restrict__ umap,
           const int32_t *__restrict__ order, const int32_t *__restrict__ perm, FT *fval, FT *fdinv,
           unsigned int *flags, TriCtl *ctl, double *scratch, const int32_t *__restrict__ place, int maxrow)
{
  constexpr int BB = NB * NB;
  constexpr int PER = 32 / NB;        // blocks updated at once: lane = (block, row)
  constexpr int UNR = WIDE ? (NB == 3 ? 7 : 4) : 2;
  constexpr int HALF = 4 * sizeof(ENT);      // bits of a block's place in the row
  constexpr ENT NONE = ~ENT(0), PLACE = NONE >> HALF;
  extern __shared__ __align__(16) double wsm[];
  __shared__ double Lsh[ILU_WARPS][BB];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned int epoch = *(volatile unsigned int *)&ctl->epoch;
  const unsigned int target = epoch + 1u;
  const int e = lane % BB, er = e / NB, ec = e % NB;
  const int ob = lane / NB, orow = lane % NB;
  while (true) {
    const int tk = draw_ticket(ctl, lane);
    if (tk >= n) break;
    const int i = order[tk];
    const int f0 = fptr[i], f1 = fptr[i + 1], fd = fdiag[i];
    double *W = wsm + (int64_t)w * rowcap * BB;
    if constexpr (PLACES) {
      if (f1 - f0 > rowcap) W = scratch + (int64_t)(place ? place[i] : blockIdx.x * (blockDim.x / 32) + w) * maxrow * BB;
    }
    for (int x = lane; x < (f1 - f0) * BB; x += 32) W[x] = 0.0;
    __syncwarp();
    {
      const int ai = perm ? perm[i] : i;   // node of factor row i
      const int a0 = arow[ai], a1 = arow[ai + 1];
      for (int x = lane; x < (a1 - a0) * BB; x += 32) {
        const int s = aslot[a0 + x / BB];
        if (s >= 0) W[(s - f0) * BB + x % BB] = (double)(FT)aval[(int64_t)a0 * BB + x];
      }
    }
    __syncwarp();
    unsigned done = 0;       // pivots of the current 32 whose flags have been seen
    int pl = 0;
    int64_t ul = 0, un = 0;  // this lane's pivot: column, its list
    for (int q = f0; q < fd; q++) {
      const int b = (q - f0) & 31;
      if (b == 0) {
        const bool in = q + lane < fd;
        pl = in ? fcol[q + lane] : 0;
        ul = in ? uoff[q + lane] : 0;
        un = in ? uoff[q + lane + 1] : 0;
        done = __ballot_sync(0xffffffffu, in && ld_acquire_u32(flags + pl) == target);
        __syncwarp();
      }
      const int p = __shfl_sync(0xffffffffu, pl, b);
      const int64_t o0 = __shfl_sync(0xffffffffu, ul, b), o1 = __shfl_sync(0xffffffffu, un, b);
      const int u0 = fdiag[p] + 1;
      // this lane's first blocks: entries of the list do not depend on the pivot's values
      ENT ent[UNR];
#pragma unroll
      for (int k = 0; k < UNR; k++) {
        const int64_t o = o0 + k * PER + ob;
        ent[k] = ob < PER && o < o1 ? umap[o] : NONE;
      }
      if (!((done >> b) & 1u)) {
        wait_flag(flags + p, target, ctl);
        __syncwarp();
        const int x = q - b + lane;
        done = __ballot_sync(0xffffffffu, x < fd && ld_acquire_u32(flags + pl) == target);
        __syncwarp();
      }
      double dcol[NB], ub[UNR][NB][NB];
#pragma unroll
      for (int k = 0; k < NB; k++) dcol[k] = (double)__ldcg(fdinv + (int64_t)p * BB + k * NB + ec);
      auto fetch = [&](int k) {
        if (ent[k] != NONE) {
#pragma unroll
          for (int c = 0; c < NB; c++) ld_row<NB>(fval + (int64_t)(u0 + (int)(ent[k] >> HALF)) * BB + c * NB, ub[k][c]);
        }
      };
#pragma unroll
      for (int k = 0; k < UNR; k++) fetch(k);
      {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NB; k++) s = fma(W[(q - f0) * BB + er * NB + k], dcol[k], s);
        if (lane < BB) Lsh[w][lane] = s;
      }
      __syncwarp();
      if (lane < BB) W[(q - f0) * BB + lane] = Lsh[w][lane];
      double lrow[NB];
#pragma unroll
      for (int k = 0; k < NB; k++) lrow[k] = Lsh[w][orow * NB + k];
      for (int64_t o = o0; o < o1; o += PER * UNR) {
#pragma unroll
        for (int k = 0; k < UNR; k++) {
          if (ent[k] != NONE) {
            double *const t = W + (int)(ent[k] & PLACE) * BB + orow * NB;
#pragma unroll
            for (int c = 0; c < NB; c++) {
              double s = 0.0;
#pragma unroll
              for (int z = 0; z < NB; z++) s = fma(lrow[z], ub[k][z][c], s);
              t[c] = (double)(FT)(t[c] - s);   // as stored
            }
          }
        }
        if (o + PER * UNR < o1) {
#pragma unroll
          for (int k = 0; k < UNR; k++) {
            const int64_t x = o + PER * (UNR + k) + ob;
            ent[k] = ob < PER && x < o1 ? umap[x] : NONE;
          }
#pragma unroll
          for (int k = 0; k < UNR; k++) fetch(k);
        }
      }
      __syncwarp();
    }
    {
      bool ok;
      const double v = invert_block<NB>(W + (fd - f0) * BB, lane, ok);
      if (!ok && lane == 0 && atomicCAS(&ctl->error, 0u, ILU_ERR_ZERO_PIVOT) == 0u) ctl->zero_pivot_row = i;
      const int r = lane / (2 * NB), c = lane % (2 * NB) - NB;
      if (r < NB && c >= 0) fdinv[(int64_t)i * BB + r * NB + c] = (FT)v;
    }
    // what later rows read, the flag, then the multipliers
    for (int x = (fd + 1 - f0) * BB + lane; x < (f1 - f0) * BB; x += 32) fval[(int64_t)f0 * BB + x] = (FT)W[x];
    __threadfence();
    __syncwarp();
    if (lane == 0) st_relaxed_u32(flags + i, target);
    for (int x = lane; x < (fd + 1 - f0) * BB; x += 32) fval[(int64_t)f0 * BB + x] = (FT)W[x];
    __syncwarp();
  }
  launch_done(ctl, lane, epoch);
}

// ---------------------------------------------------------------------------
// Triangular solves z = (L U)^-1 r.
//
// The values are their own ready flags: the intermediate vector y and the
// output z hold a signalling-NaN sentinel (a bit pattern no arithmetic
// produces) until their row is written, so whoever needs a value polls the value
// itself (relaxed loads) and needs no separate flag, fence or second round trip.  The lower solve writes y_i
// and resets z_i to the sentinel for the upper solve; the upper solve reads
// y_i, writes z_i and resets y_i to the sentinel for the next lower solve.
// y is the handle's own buffer (sentinel-filled at creation); r and z must
// not overlap.
//
// Lower:  y_i = r_i - sum_{p<i} L_ip y_p
// Upper:  z_i = U_ii^-1 (y_i - sum_{p>i} U_ip z_p)
// st/j: inside a GMRES chunk the launch is skipped once the cycle has ended;
// active: inside a BiCGStab chunk, once the solve has ended.
template <typename VT> struct Sentinel;
template <> struct Sentinel<double> {
  using U = unsigned long long;
  static constexpr U bits = 0x7FF4C0FFEE15BAD1ull;   // signalling NaN
  static __device__ __forceinline__ U load(const double *p)
  {
    U v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void load2(const double *p, U (&v)[2])
  {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "l"(p) : "memory");
  }
  static __device__ __forceinline__ void store(double *p, double x)
  {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(x) : "memory");
  }
  static __device__ __forceinline__ double value(U v) { return __longlong_as_double((long long)v); }
  static __device__ __forceinline__ double sentinel() { return __longlong_as_double((long long)bits); }
};
template <> struct Sentinel<float> {
  using U = unsigned int;
  static constexpr U bits = 0x7FA0C0DEu;               // signalling NaN
  static __device__ __forceinline__ U load(const float *p)
  {
    U v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void load2(const float *p, U (&v)[2])
  {
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(p) : "memory");
  }
  static __device__ __forceinline__ void store(float *p, float x)
  {
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(x) : "memory");
  }
  static __device__ __forceinline__ float value(U v) { return __uint_as_float(v); }
  static __device__ __forceinline__ float sentinel() { return __uint_as_float(bits); }
};

// value at p once it is no longer the sentinel (bounded wait; polls as in wait_flag)
template <typename VT>
__device__ __forceinline__ double wait_value(const VT *p, typename Sentinel<VT>::U v, TriCtl *ctl)
{
  using S = Sentinel<VT>;
  if (v != S::bits) return (double)S::value(v);
  unsigned int ns = 32;
  for (int it = 0; it < ILU_SPIN_LIMIT; it++) {
    if (it >= ILU_SPIN_HOT_POLLS) {
      __nanosleep(ns);
      if (ns < 256) ns <<= 1;
    }
    v = S::load(p);
    if (v != S::bits) return (double)S::value(v);
    if (*(volatile unsigned int *)&ctl->error) break;
  }
  atomicCAS(&ctl->error, 0u, ILU_ERR_TIMEOUT);
  return 0.0;
}

__global__ void fill_sentinel_f64(int64_t n, double *y)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = Sentinel<double>::sentinel();
}

__global__ void fill_sentinel_f32(int64_t n, float *y)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = Sentinel<float>::sentinel();
}

// Chains of rows on the device (IluPattern::lchain, lchain_order, or uchain, uchain_order).
struct ChainView {
  const int32_t *chains, *order;
  int nchains;
};

// Device form of a TrsvPlan (trsv_plan.h).
struct TrsvView {
  const TrsvGroup *groups;
  const int32_t *wptr;
  const TrsvPiece *pieces;
  const uint32_t *desc;
  const int32_t *ext;
  int ngroups, slots;
};

constexpr int TRSV_THREADS = 32 * (TRSV_WARPS + TRSV_LOADERS);
constexpr int TRSV_DEPTH = 4;   // pieces in flight per solving warp (a power of two)

// Shared-memory layout of ilu_trsv<NB, UPPER, T>: a ring of TRSV_DEPTH stages
// per solving warp, each holding one piece: its record (TrsvPlan::desc), its
// blocks, the row's right-hand side and the inverted diagonal block (upper
// solve), the last three copied from the 16-byte boundary below them.
template <int NB, bool UPPER, typename T>
struct TrsvStage {
  static constexpr int BB = NB * NB;
  static constexpr int CAP = trsv_cap(NB);
  static constexpr bool ALIGNED = (BB * sizeof(T)) % 16 == 0;
  // 16-byte lines that `count` units of `unit` bytes may touch
  static constexpr int lines(int unit, int count = 1)
  {
    return (unit * count + (unit % 16 ? 16 - (int)sizeof(T) : 0) + 15) / 16;
  }
  static constexpr bool BALIGNED = (NB * sizeof(T)) % 16 == 0;
  static constexpr int RECL = (16 + 4 * trsv_slots(NB)) / 16;
  static constexpr int DINVL = UPPER ? lines(BB * (int)sizeof(T)) : 0;
  static constexpr int BL = lines(NB * (int)sizeof(T));
  static constexpr int REC = 0;
  static constexpr int DINV = REC + 16 * RECL;
  static constexpr int B = DINV + 16 * DINVL;
  static constexpr int VAL = B + 16 * BL;
  static constexpr int VALL = lines(BB * (int)sizeof(T), CAP), VALI = (VALL + 31) / 32;
  static constexpr int BYTES = VAL + 16 * VALL;
};

template <int NB, bool UPPER, typename T>
constexpr size_t trsv_smem(int slots)
{
  return up_to_16((size_t)(slots + 1) * NB * 8) + (size_t)TRSV_WARPS * TRSV_DEPTH * TrsvStage<NB, UPPER, T>::BYTES;
}

constexpr size_t TRSV_SMEM = 226 * 1024;    // of the 227 KB that a CTA may have; some of it is static
static_assert(trsv_smem<4, true, double>(trsv_max_slots(4)) <= TRSV_SMEM &&
              trsv_smem<3, true, double>(trsv_max_slots(3)) <= TRSV_SMEM, "a group's slots and the rings must fit");

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// asynchronous copy of 16 bytes at src (16-byte aligned) to shared memory.
// (The form that fills with zeros past a given byte took 330 cycles for a row's
// four copies with 16 warps on an SM, this one 70.)
__device__ __forceinline__ void copy_line(uint32_t dst, uint64_t src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ bool bar_try_wait(uint32_t bar, uint32_t parity)
{
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

template <typename V>
__device__ __forceinline__ V ld_shared(uint32_t p)
{
  return *reinterpret_cast<const V *>(__cvta_shared_to_generic(p));
}

// slots of ilu_trsv: written by one warp, polled by others
__device__ __forceinline__ unsigned long long ld_slot(uint32_t p)
{
  unsigned long long v;
  asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint32_t ld_slot_hi(uint32_t p)
{
  uint32_t v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
  return v;
}

__device__ __forceinline__ void ld_slot2(uint32_t p, unsigned long long &u, unsigned long long &v)
{
  asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(u), "=l"(v) : "r"(p) : "memory");
}

__device__ __forceinline__ void st_slot(uint32_t p, double v)
{
  asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory");
}

// Bounded waits of ilu_trsv (warp_wait.h).  A wait gives up when its time is over
// or another wait of the CTA has given up: ctl->error is then set and the CTA goes
// on with what is there, so that its copies complete and it can leave.
struct TrsvEnv {
  volatile int *flag;
  TriCtl *ctl;
  __device__ __forceinline__ bool gave_up() const { return *flag != 0; }
  __device__ __forceinline__ void give_up() const
  {
    *flag = 1;
    atomicCAS(&ctl->error, 0u, ILU_ERR_TIMEOUT);
  }
  __device__ __forceinline__ unsigned long long now() const
  {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
  }
};
using TrsvWait = LaneWait<TrsvEnv>;

// Persistent CTAs take groups of rows (TrsvPlan) in topological order.  Every
// value a group needs has a slot in shared memory that holds the sentinel until
// the value is known: the loader warps poll the inputs that other groups write
// and copy them in, the solving warps poll the slots and write their own rows'
// results to them (and to global memory, for other groups).  So a value passes
// between rows of one group in about a shared-memory round trip, and only from
// group to group does it cross the L2.
//
// What bounds it: the dependency chain.  On a hex8 mesh with n elements per
// side the natural-order ILU(0) has 7n levels.  One warp per x-line with every
// value handed over through L2 (the kernel before this one) took, lower / upper:
//   ILU(0), hex8 11^3 / 32^3 / 64^3      0.113 / 0.165, 0.46 / 0.68, 1.06 / 1.53 ms
//   ILU(3), 256 x 128 O-grid of quad4    1.94 / 2.33 ms
//   complete LU of the 64 x 64 cavity    27.6 / 33.5 ms
// and this one 0.031 / 0.037, 0.14 / 0.15, 0.32 / 0.35, 0.49 / 0.54 and 1.4 / 1.5 ms.
// The factors' bytes at copy speed are 0.07 ms at 64^3.  What is left is the
// chain: a row's loads, products and shuffles after its last input (about 0.3
// us), and an L2 hop (about 2 us with the polls on both sides) per plane of x-lines
// and per TRSV_STRANDS lines in a plane.
//
// What does not depend on the solve is kept off the chain: a row's blocks,
// right-hand side and slots come through a ring of asynchronous copies
// TRSV_DEPTH - 1 pieces ahead, and a strand's rows go to four warps in turn, so
// that a row's blocks are in registers when its last input arrives.  Measured
// instead, lower / upper at 64^3: one warp per strand, 8 strands 0.40 / 0.39 ms;
// two, 8 strands 0.34 / 0.37; three, 6 strands 0.39 / 0.41 (before the loaders
// polled one unit per lane); bulk copies started by one lane per row 0.52 / 0.57
// (80 cycles to start each one); one warp that starts all of them 0.65 / 0.74.
//
// Lower:  y_i = r_P(i) - sum_{p<i} L_ip y_p
// Upper:  z_P(i) = U_ii^-1 (y_i - sum_{p>i} U_ip z_P(p))
// with P the factor's row order (perm; NULL: the identity): y is indexed by
// factor row, r and z by node.  Every sum has a fixed order, so the result does
// not depend on scheduling.
template <int NB, bool UPPER, typename T>
__global__ void __launch_bounds__(TRSV_THREADS, 1)
ilu_trsv(TrsvView P, const T *__restrict__ fval, const T *__restrict__ fdinv, const int32_t *__restrict__ perm,
         const T *__restrict__ r, T *y, T *z, TriCtl *ctl, const GmresState *__restrict__ st, int j,
         const int *__restrict__ active)
{
  if (st && (!st->active || st->it != j)) return;
  if (active && !active[0]) return;
  using S = Sentinel<T>;
  using D = Sentinel<double>;
  using G = TrsvStage<NB, UPPER, T>;
  using U64 = unsigned long long;
  constexpr int BB = NB * NB;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_ticket, s_gave_up;
  __shared__ U64 s_gate;
  const uint32_t gate = smem_u32(&s_gate);
  double *const xs = reinterpret_cast<double *>(smem);
  const uint32_t xs0 = smem_u32(xs);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t ring = xs0 + (uint32_t)up_to_16((size_t)(P.slots + 1) * NB * 8) + (uint32_t)(w * TRSV_DEPTH * G::BYTES);
  // a lane's share of what is not blocks in a piece: record, right-hand side, inverted diagonal block
  const int part = lane < G::RECL ? 0 : lane < G::RECL + G::BL ? 1 : lane < G::RECL + G::BL + G::DINVL ? 2 : 3;
  const uint32_t pline = (uint32_t)(part == 0 ? lane : part == 1 ? lane - G::RECL : lane - G::RECL - G::BL);
  const uint32_t pdst = (uint32_t)(part == 0 ? G::REC : part == 1 ? G::B : G::DINV) + 16u * pline;
  const uint64_t pbase = (part == 0 ? reinterpret_cast<uint64_t>(P.desc)
                          : part == 1 ? reinterpret_cast<uint64_t>(UPPER ? y : r) : reinterpret_cast<uint64_t>(fdinv)) +
                         (G::BALIGNED && G::ALIGNED ? 16u * pline : 0u);
  const uint32_t pstride = part == 0 ? 16u : (uint32_t)((part == 1 ? NB : BB) * sizeof(T));
  const unsigned int epoch = *(volatile unsigned int *)&ctl->epoch;
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(gate) : "memory");
    s_gave_up = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (tid < NB) xs[(size_t)P.slots * NB + tid] = 0.0;    // the slot of blocks past a piece's end
  uint32_t ngone = 0;    // groups this CTA has done

  while (true) {
    __syncthreads();
    if (tid == 0) s_ticket = (int)atomicAdd(&ctl->ticket, 1u);
    __syncthreads();
    const int tk = s_ticket;
    if (tk >= P.ngroups) break;
    const TrsvGroup gr = P.groups[tk];

    // pieces of this warp, copied TRSV_DEPTH - 1 ahead: one commit group each
    int np = 0;
    const int4 *pc = nullptr;
    int4 h = make_int4(0, 0, 0, 0), hn = h;      // headers of the next two pieces to copy
    auto copy = [&](int t) {
      if (t < np) {
        const uint32_t s0 = ring + (uint32_t)(t % TRSV_DEPTH) * (uint32_t)G::BYTES;
        uint64_t v = reinterpret_cast<uint64_t>(fval) + (uint64_t)(uint32_t)h.x * (uint32_t)(BB * sizeof(T)) + 16u * lane;
        int left = (h.y & 0xffff) * BB * (int)sizeof(T) - 16 * lane;
        if constexpr (!G::ALIGNED) {
          left += (int)(v & 15);
          v &= ~(uint64_t)15;
        }
        const uint32_t d0 = s0 + G::VAL + 16u * lane;
#pragma unroll
        for (int i = 0; i < G::VALI; i++)
          if (left > 512 * i) copy_line(d0 + 512u * i, v + 512 * i);
        if (part < 3) {
          uint64_t q = pbase + (uint64_t)(uint32_t)(part == 0 ? h.z : h.w) * pstride;
          if (!G::BALIGNED || !G::ALIGNED) q = (q & ~(uint64_t)15) + 16u * pline;
          copy_line(s0 + pdst, q);
        }
        h = hn;
        if (t + 2 < np) hn = __ldg(pc + t + 2);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (w < TRSV_WARPS) {
      const int p0 = P.wptr[tk * (TRSV_WARPS + 1) + w];
      np = P.wptr[tk * (TRSV_WARPS + 1) + w + 1] - p0;
      pc = reinterpret_cast<const int4 *>(P.pieces + p0);
      if (np > 0) h = __ldg(pc);
      if (np > 1) hn = __ldg(pc + 1);
      __syncwarp();     // the ring's last pieces have been read by every lane
      for (int t = 0; t < TRSV_DEPTH - 1; t++) copy(t);
    }
    for (int k = tid; k < (gr.rows + gr.next) * NB; k += TRSV_THREADS) xs[k] = D::sentinel();
    __syncthreads();

    if (w >= TRSV_WARPS) {
      // ---- inputs from other groups ----
      // A unit is a pair of a row's entries (4x4 blocks) or one entry; a lane polls
      // one unit until it is there, copies it to its slot and goes on to its next
      // (the place of the one after that is looked up meanwhile).  One unit per
      // lane: polls further ahead only load the L2 that the values have to cross.
      constexpr int UW = (NB == 4) ? 2 : 1, UPR = NB / UW, LT = 32 * TRSV_LOADERS;
      const T *const src = UPPER ? z : y;
      const int32_t *const ext = P.ext + gr.ext0;
      const int tot = gr.next * UPR;
      auto place = [&](int k) {
        if (k >= tot) return (int64_t)-1;
        const int row = ext[k / UPR];
        return (int64_t)((UPPER && perm) ? perm[row] : row) * NB + (k % UPR) * UW;
      };
      // Until the first thing that the group waits for is there, its solving warps
      // wait on a barrier, which costs nothing.
      const int lt = tid - 32 * TRSV_WARPS, gunit = gr.gate * UPR;
      bool opens = tot > 0 ? lt == gunit % LT : lt == 0;
      auto open_gate = [&] {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gate) : "memory");
        opens = false;
      };
      if (tot == 0 && opens) open_gate();
      int64_t at = place(lt), nat = place(lt + LT);
      TrsvWait wait{{&s_gave_up, ctl}};
      for (int k = lt; at >= 0;) {
        typename S::U v[UW];
        if constexpr (UW == 2) S::load2(src + at, v);
        else v[0] = S::load(src + at);
        bool there = true;
#pragma unroll
        for (int c = 0; c < UW; c++) there &= v[c] != S::bits;
        if (there) {
#pragma unroll
          for (int c = 0; c < UW; c++)
            st_slot(xs0 + 8u * (uint32_t)(gr.rows * NB + k * UW + c), (double)S::value(v[c]));
          if (opens && k == gunit) open_gate();
          k += LT;
          at = nat;
          nat = place(k + LT);
          wait.it = 0;
        } else if (!wait.go_on()) {
          break;
        }
      }
      if (opens) open_gate();    // the wait for it ran out
    } else {
      // ---- rows ----
      // 4x4 blocks: lane = (block of four, row, column pair); 3x3 blocks:
      // lane = (row, block of eight), lanes 24..31 idle.  4x4 blocks in FP32
      // (inside the mixed-precision solves): lane = (block of two, row, column),
      // every lane adding its products one after another from the farthest column
      // to the nearest.  What comes of an FP32 solve depends on the last bit of
      // these sums (a solve that stops at a relative residual of 1e-14 fixes the
      // pressure level of an enclosed cavity only to 1e-9), so their order is part
      // of the results; a chain of 8 products in place of 4 is what that costs.
      constexpr bool CHAIN = NB == 4 && sizeof(T) == 4;
      constexpr int PER = CHAIN ? 2 : (NB == 4) ? 4 : 8, W = CHAIN ? 1 : (NB == 4) ? 2 : 3;
      constexpr int PASS = (G::CAP + PER - 1) / PER;
      const int sub = CHAIN ? lane >> 4 : (NB == 4) ? lane >> 3 : lane & 7;
      const int row = CHAIN ? (lane & 15) >> 2 : (NB == 4) ? (lane & 7) >> 1 : (lane >> 3 < 3 ? lane >> 3 : 0);
      const int c0 = CHAIN ? lane & 3 : (NB == 4) ? (lane & 1) * 2 : 0;
      const bool writes = CHAIN ? (lane < 16 && c0 == 0) : (NB == 4) ? (lane < 8 && (lane & 1) == 0) : (lane < 24 && sub == 0);
      // first block of the lane in a piece of k: its PASS blocks are PER apart
      auto first = [&](int k) { return CHAIN && UPPER ? (k - 1 - sub) & 1 : sub; };
      // a piece in registers: its blocks' entries, where their inputs lie, and the row's own data
      struct Piece {
        T a[PASS][W];
        uint32_t x[PASS];
        T d[W], b;
        int4 m;     // factor row, node, blocks and flags, own slot and the input expected last
      };
      const uint32_t lane_a = ring + G::VAL + (uint32_t)((row * NB + c0) * sizeof(T));
      const uint32_t lane_d = ring + G::DINV + (uint32_t)((row * NB + c0) * sizeof(T));
      const uint32_t lane_b = ring + G::B + (uint32_t)(row * sizeof(T));
      const uint32_t lane_x = xs0 + 8u * c0, zero = xs0 + (uint32_t)P.slots * NB * 8u;
      // piece s from its stage; its copies must have landed
      auto take = [&](int s, Piece &q) {
        const uint32_t so = (uint32_t)(s % TRSV_DEPTH) * (uint32_t)G::BYTES;
        q.m = ld_shared<int4>(ring + G::REC + so);
        const int k = q.m.z & 0xffff, b0 = first(k);
        const uint4 ds = ld_shared<uint4>(ring + G::REC + 16 + 16 * b0 + so);
        uint32_t off[PASS];
        if constexpr (CHAIN) {
          // the record lists the blocks congruent to 0, 1, 2, 3 modulo 4 in turn
          const uint4 de = ld_shared<uint4>(ring + G::REC + 16 + 16 * (b0 + 2) + so);
          off[0] = ds.x; off[2] = ds.y; off[4] = ds.z; off[6] = ds.w;
          off[1] = de.x; off[3] = de.y; off[5] = de.z; off[7] = de.w;
        } else {
          const uint32_t o[4] = {ds.x, ds.y, ds.z, ds.w};
#pragma unroll
          for (int p = 0; p < PASS; p++) off[p] = o[p];
        }
        const uint32_t ov = G::ALIGNED ? 0u : (((uint32_t)q.m.z >> TRSV_Q0_SHIFT & 3u) * (uint32_t)(BB * sizeof(T))) & 15u;
#pragma unroll
        for (int p = 0; p < PASS; p++) {
          q.x[p] = lane_x + off[p];
          // past the piece's end the stage holds blocks of earlier pieces: the zero slot instead
          const bool in = PER * p + b0 < k;
          const uint32_t e = in ? lane_a + so + ov + (uint32_t)((PER * p + b0) * BB * (int)sizeof(T)) : zero;
          if constexpr (NB == 4 && !CHAIN) {
            using V2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
            const V2 t = ld_shared<V2>(e);
            q.a[p][0] = t.x; q.a[p][1] = t.y;
          } else {
#pragma unroll
            for (int c = 0; c < W; c++) q.a[p][c] = ld_shared<T>(e + (uint32_t)(c * sizeof(T)));
          }
        }
        const uint32_t at = (uint32_t)(UPPER ? q.m.x : q.m.y);
        const uint32_t ob = G::BALIGNED ? 0u : (at * (uint32_t)(NB * sizeof(T))) & 15u;
        q.b = ld_shared<T>(lane_b + so + ob);
        if constexpr (UPPER) {
          const uint32_t oi = G::ALIGNED ? 0u : ((uint32_t)q.m.x * (uint32_t)(BB * sizeof(T))) & 15u;
#pragma unroll
          for (int c = 0; c < W; c++) q.d[c] = ld_shared<T>(lane_d + so + oi + (uint32_t)(c * sizeof(T)));
        }
      };
      double acc[W];
#pragma unroll
      for (int c = 0; c < W; c++) acc[c] = 0.0;
      T *const zr = z + row, *const yr = y + row;
      for (int s = 0; s < np; s++) {
        // its copies have landed when at most TRSV_DEPTH - 2 younger groups are pending
        asm volatile("cp.async.wait_group %0;" ::"n"(TRSV_DEPTH - 2) : "memory");
        __syncwarp();
        Piece q;
        take(s, q);
        if (q.m.z & TRSV_FIRST) {
#pragma unroll
          for (int c = 0; c < W; c++) acc[c] = 0.0;
        }
        copy(s + TRSV_DEPTH - 1);     // into the stage of piece s - 1
        if (s == 0) {
          // the loader opens the gate even when its own wait runs out
          TrsvWait wait{{&s_gave_up, ctl}};
          wait_lanes([&] { return bar_try_wait(gate, ngone & 1u); }, wait, [] { __syncwarp(); });
        }
        // One load at a time for the input expected last; then the whole row,
        // done over in the rare case that another input was later still (the
        // check is off the path from the loads to the result).
        TrsvWait wait{{&s_gave_up, ctl}};
        const uint32_t last = xs0 + ((uint32_t)q.m.w >> 16) * 8u + 4u;
        wait_lanes([&] { return ld_slot_hi(last) != (uint32_t)(D::bits >> 32); }, wait, [] { __syncwarp(); });
        double t[W], x;
        auto row_sum = [&]() -> bool {
          U64 u[PASS][W];
          bool miss = false;
          if (q.m.z & TRSV_DIRECT) {
            const T *const src = (UPPER ? z : y) + c0;
#pragma unroll
            for (int p = 0; p < PASS; p++)
#pragma unroll
              for (int c = 0; c < W; c++) {
                u[p][c] = 0ull;
                if (PER * p + first(q.m.z & 0xffff) < (q.m.z & 0xffff)) {
                  const typename S::U v = S::load(src + (q.x[p] - lane_x) + c);
                  u[p][c] = v == S::bits ? D::bits : (U64)__double_as_longlong((double)S::value(v));
                }
              }
          } else {
#pragma unroll
            for (int p = 0; p < PASS; p++) {
              if constexpr (NB == 4 && !CHAIN) {
                ld_slot2(q.x[p], u[p][0], u[p][1]);
              } else {
#pragma unroll
                for (int c = 0; c < W; c++) u[p][c] = ld_slot(q.x[p] + 8u * c);
              }
            }
          }
#pragma unroll
          for (int c = 0; c < W; c++) t[c] = acc[c];
#pragma unroll
          for (int p = 0; p < PASS; p++) {
            const int f = CHAIN && UPPER ? PASS - 1 - p : p;
#pragma unroll
            for (int c = 0; c < W; c++) t[c] = fma((double)q.a[f][c], D::value(u[f][c]), t[c]);
          }
          // no number has the sentinel's upper half either
#pragma unroll
          for (int p = 0; p < PASS; p++)
#pragma unroll
            for (int c = 0; c < W; c++) miss |= (uint32_t)(u[p][c] >> 32) == (uint32_t)(D::bits >> 32);
          const bool again = __any_sync(FULL, miss);
          double sum = t[0];
          if constexpr (W > 1) sum += t[1];
          if constexpr (W == 3) sum += t[2];
          if constexpr (CHAIN) {
            sum += __shfl_xor_sync(FULL, sum, 1);
            sum += __shfl_xor_sync(FULL, sum, 2);
            sum += __shfl_xor_sync(FULL, sum, 16);
            x = (double)q.b - sum;
            if constexpr (UPPER) {
              x = (double)q.d[0] * __shfl_sync(FULL, x, 4 * c0);
              x += __shfl_xor_sync(FULL, x, 1);
              x += __shfl_xor_sync(FULL, x, 2);
            }
          } else if constexpr (NB == 4) {
            sum += __shfl_xor_sync(FULL, sum, 1);
            sum += __shfl_xor_sync(FULL, sum, 8);
            sum += __shfl_xor_sync(FULL, sum, 16);
            x = (double)q.b - sum;
            if constexpr (UPPER) {
              // lanes 2 row hold entry `row`; lane (row, c0) takes columns c0, c0 + 1 of U_ii^-1
              const double s0 = __shfl_sync(FULL, x, 2 * c0), s1 = __shfl_sync(FULL, x, 2 * c0 + 2);
              x = fma((double)q.d[0], s0, (double)q.d[1] * s1);
              x += __shfl_xor_sync(FULL, x, 1);
            }
          } else {
            sum += __shfl_xor_sync(FULL, sum, 4);
            sum += __shfl_xor_sync(FULL, sum, 2);
            sum += __shfl_xor_sync(FULL, sum, 1);
            x = (double)q.b - sum;
            if constexpr (UPPER) {
              const double s0 = __shfl_sync(FULL, x, 0), s1 = __shfl_sync(FULL, x, 8), s2 = __shfl_sync(FULL, x, 16);
              x = fma((double)q.d[0], s0, fma((double)q.d[1], s1, (double)q.d[2] * s2));
            }
          }
          return again;
        };
        retry_warp(row_sum, wait, [](bool v) { return (bool)__all_sync(FULL, v); });
#pragma unroll
        for (int c = 0; c < W; c++) acc[c] = t[c];
        if (q.m.z & TRSV_LAST) {
          if (writes) {
            const T v = (T)x;
            st_slot(xs0 + ((uint32_t)q.m.w & 0xffffu) * 8u + 8u * row, (double)v);
            // the sentinel goes to the place that the next solve fills
            if (UPPER) {
              S::store(zr + (int64_t)q.m.y * NB, v);
              yr[(int64_t)q.m.x * NB] = S::sentinel();
            } else {
              S::store(yr + (int64_t)q.m.x * NB, v);
              zr[(int64_t)q.m.y * NB] = S::sentinel();
            }
          }
        }
      }
    }
    ngone++;
  }
  if (tid == 0) {
    __threadfence();
    const unsigned int k = atomicAdd(&ctl->exited, 1u);
    if (k == gridDim.x - 1) {
      ctl->ticket = 0u;
      ctl->exited = 0u;
      __threadfence();
      *(volatile unsigned int *)&ctl->epoch = epoch + 1u;
      __threadfence();
    }
  }
}

// ---------------------------------------------------------------------------
constexpr int TRSV_BATCH = 4;        // input loads in flight per lane for blocks beyond the pipelined ones
constexpr int TRSV_ROW_BLOCKS = 14;  // blocks per row held in the pipeline registers (a 27-point row: 13)

// The same solves with one warp per chain of rows (see IluPattern::lchain /
// uchain), chains in level order of the chain DAG: for orders of the rows in which
// many rows can be solved at once but few of them follow one another (TrsvPlan::
// chains has the rule and both kernels' times).  There a row's inputs are long
// done, every warp reads its own from memory, and 2,368 rows are in flight.  The
// chain's rows are solved in order; inputs from the chain itself come from shared
// memory, inputs from other chains from global memory once they are no longer the
// sentinel.  Bound by the levels, 1 to 3 us each for the rows of ILU(0): 66,049 nodes
// in random order take 98 us a solve with ILU(0) (19 levels) and 161 with ILU(3) (90).
//
// The rows of a chain run through a three-stage software pipeline, so that
// the memory latencies of a row overlap the work of the row before it: while
// row s is finished, the warp already holds the matrix values and the other
// chains' input values of row s+1, the column indices of row s+2 are in
// flight, and so is the block range of row s+3.  A lane holds PF blocks of a
// row in registers (G blocks per warp pass, lanes g = lane / (NB*NB));
// further blocks (fill rows of ILU(k), k >= 1) are loaded when their row is
// finished.  Per lane the products are summed in block order, so the result
// does not depend on how far ahead the loads ran.
// Results as of ilu_trsv.
template <int NB, bool UPPER, typename T>
__global__ void __launch_bounds__(ILU_THREADS, 2)
ilu_trsv_chains(int nchains, const int32_t *__restrict__ order, const int32_t *__restrict__ chains,
                const int32_t *__restrict__ fptr, const int32_t *__restrict__ fcol, const int32_t *__restrict__ fdiag,
                const T *__restrict__ fval, const T *__restrict__ fdinv, const int32_t *__restrict__ perm, const T *r,
                T *y, T *z, TriCtl *ctl, const GmresState *__restrict__ st, int j, const int *__restrict__ active)
{
  if (st && (!st->active || st->it != j)) return;
  if (active && !active[0]) return;
  using S = Sentinel<T>;
  using U = typename S::U;
  constexpr int BB = NB * NB;
  constexpr int G = 32 / BB;
  constexpr int PF = (TRSV_ROW_BLOCKS + G - 1) / G;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ double red[ILU_WARPS][32];
  __shared__ double sv[ILU_WARPS][NB];
  __shared__ double cache[ILU_WARPS][ILU_CHAIN_MAX * NB];
  const unsigned int epoch = *(volatile unsigned int *)&ctl->epoch;
  const int g = lane / BB, e = lane % BB, ec = e % NB;
  const bool glane = g < G;
  // the vector the off-diagonal products read: y (lower) or z (upper)
  const T *src = UPPER ? z : y;
  // position of column p in src: z is indexed by node, y by factor row
  auto at = [&](int p) -> int64_t { return (int64_t)((UPPER && perm) ? perm[p] : p) * NB + ec; };
  while (true) {
    const int tk = draw_ticket(ctl, lane);
    if (tk >= nchains) break;
    const int c = order[tk];
    const int lo = chains[2 * c], hi = chains[2 * c + 1];
    const int len = hi - lo;
    auto row = [&](int s) { return UPPER ? hi - 1 - s : lo + s; };
    auto own = [&](int p) { return UPPER ? p < hi : p >= lo; };
    // strictly lower (upper) blocks [qa, qb) of the chain's s-th row; the
    // qq-th block of a row is the farthest column first, so the chain's own
    // previous row (the input finished last) is consumed last
    auto range = [&](int s, int &qa, int &qb) {
      qa = qb = 0;
      if (s < len) {
        const int i = row(s);
        qa = UPPER ? fdiag[i] + 1 : fptr[i];
        qb = UPPER ? fptr[i + 1] : fdiag[i];
      }
    };
    auto blk = [&](int qa, int qb, int qq) { return UPPER ? qb - 1 - qq : qa + qq; };
    auto cols = [&](int qa, int qb, int (&p)[PF]) {
#pragma unroll
      for (int k = 0; k < PF; k++) {
        const int qq = k * G + g;
        p[k] = (glane && qq < qb - qa) ? fcol[blk(qa, qb, qq)] : -1;
      }
    };
    // matrix values, other chains' inputs and the row's own data (r_P(i) or
    // y_i, and the row of U_ii^-1) of the s-th row
    auto vals = [&](int s, int qa, int qb, const int (&p)[PF], T (&a)[PF], U (&v)[PF], T &b, T (&d)[NB]) {
#pragma unroll
      for (int k = 0; k < PF; k++)
        a[k] = p[k] >= 0 ? fval[(int64_t)blk(qa, qb, k * G + g) * BB + e] : T(0);
#pragma unroll
      for (int k = 0; k < PF; k++) v[k] = (p[k] >= 0 && !own(p[k])) ? S::load(src + at(p[k])) : U(0);
      b = T(0);
#pragma unroll
      for (int cc = 0; cc < NB; cc++) d[cc] = T(0);
      if (s < len) {
        const int i = row(s);
        if constexpr (NB == 4) {
          // every lane: entry er of the row's vector, entry (er, ec) of U_ii^-1
          if (UPPER) {
            b = y[(int64_t)i * NB + e / NB];
            d[0] = fdinv[(int64_t)i * BB + e];
          } else {
            b = r[(int64_t)(perm ? perm[i] : i) * NB + e / NB];
          }
        } else if (lane < NB) {
          if (UPPER) {
            b = y[(int64_t)i * NB + lane];
#pragma unroll
            for (int cc = 0; cc < NB; cc++) d[cc] = fdinv[(int64_t)i * BB + lane * NB + cc];
          } else {
            b = r[(int64_t)(perm ? perm[i] : i) * NB + lane];
          }
        }
      }
    };

    int qa0, qb0, qa1, qb1, qa2, qb2;
    int p0[PF], p1[PF], p2[PF];
    T a0[PF], a1[PF], d0[NB], d1[NB];
    U v0[PF], v1[PF];
    T b0, b1;
    range(0, qa0, qb0);
    range(1, qa1, qb1);
    range(2, qa2, qb2);
    cols(qa0, qb0, p0);
    cols(qa1, qb1, p1);
    vals(0, qa0, qb0, p0, a0, v0, b0, d0);
    for (int s = 0; s < len; s++) {
      const int i = row(s);
      // loads for the rows ahead
      vals(s + 1, qa1, qb1, p1, a1, v1, b1, d1);
      cols(qa2, qb2, p2);
      int qa3, qb3;
      range(s + 3, qa3, qb3);

      // row s: products in block order, other chains' inputs once they are
      // no longer the sentinel, the chain's own from shared memory
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < PF; k++) {
        if (p0[k] < 0) continue;
        const double xv = own(p0[k]) ? cache[w][(UPPER ? hi - 1 - p0[k] : p0[k] - lo) * NB + ec]
                                     : wait_value<T>(src + at(p0[k]), v0[k], ctl);
        acc = fma((double)a0[k], xv, acc);
      }
      const int nq = qb0 - qa0;
      for (int qb = G * PF; qb < nq; qb += G * TRSV_BATCH) {
        U v[TRSV_BATCH];
        int p[TRSV_BATCH];
        double a[TRSV_BATCH];
#pragma unroll
        for (int k = 0; k < TRSV_BATCH; k++) {
          const int qq = qb + k * G + g;
          const bool ok = (glane && qq < nq);
          const int q = blk(qa0, qb0, qq);
          p[k] = ok ? fcol[q] : -1;
          a[k] = ok ? (double)fval[(int64_t)q * BB + e] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < TRSV_BATCH; k++) v[k] = (p[k] >= 0 && !own(p[k])) ? S::load(src + at(p[k])) : U(0);
#pragma unroll
        for (int k = 0; k < TRSV_BATCH; k++) {
          if (p[k] < 0) continue;
          const double xv = own(p[k]) ? cache[w][(UPPER ? hi - 1 - p[k] : p[k] - lo) * NB + ec]
                                      : wait_value<T>(src + at(p[k]), v[k], ctl);
          acc = fma(a[k], xv, acc);
        }
      }
      const int64_t node = perm ? perm[i] : i;
      if constexpr (NB == 4) {
        // 4x4 blocks, two per warp pass: lane = 16 g + 4 er + ec.  Sum the
        // products of block row er over ec (lane bits 0-1) and g (bit 4)
        // with shuffles; every lane then holds entry er of the row's vector.
        constexpr unsigned FULL = 0xffffffffu;
        double t = acc;
        t += __shfl_xor_sync(FULL, t, 1);
        t += __shfl_xor_sync(FULL, t, 2);
        t += __shfl_xor_sync(FULL, t, 16);
        const double sr = (double)b0 - t;
        const int er = e / NB;
        if (UPPER) {
          // z_i = U_ii^-1 s: lane (er, ec) forms (U_ii^-1)_{er,ec} s_ec, summed over ec
          double x = (double)d0[0] * __shfl_sync(FULL, sr, ec * NB);
          x += __shfl_xor_sync(FULL, x, 1);
          x += __shfl_xor_sync(FULL, x, 2);
          if (lane < BB && ec == 0) {
            const T vv = (T)x;
            cache[w][s * NB + er] = (double)vv;
            S::store(z + node * NB + er, vv);
            y[(int64_t)i * NB + er] = S::sentinel();
          }
        } else if (lane < BB && ec == 0) {
          const T vv = (T)sr;
          cache[w][s * NB + er] = (double)vv;
          z[node * NB + er] = S::sentinel();
          S::store(y + (int64_t)i * NB + er, vv);
        }
        __syncwarp();
      } else {
      red[w][lane] = acc;
      __syncwarp();
      if (lane < NB) {
        double sum = (double)b0;
#pragma unroll
        for (int gg = 0; gg < G; gg++)
#pragma unroll
          for (int cc = 0; cc < NB; cc++) sum -= red[w][gg * BB + lane * NB + cc];
        sv[w][lane] = sum;
      }
      __syncwarp();
      if (lane < NB) {
        if (UPPER) {
          double x = 0.0;
#pragma unroll
          for (int cc = 0; cc < NB; cc++) x = fma((double)d0[cc], sv[w][cc], x);
          const T vv = (T)x;
          cache[w][s * NB + lane] = (double)vv;
          S::store(z + node * NB + lane, vv);
          y[(int64_t)i * NB + lane] = S::sentinel();
        } else {
          const T vv = (T)sv[w][lane];
          cache[w][s * NB + lane] = (double)vv;
          z[node * NB + lane] = S::sentinel();
          S::store(y + (int64_t)i * NB + lane, vv);
        }
      }
      __syncwarp();
      }
      // advance the pipeline
      qa0 = qa1; qb0 = qb1; qa1 = qa2; qb1 = qb2; qa2 = qa3; qb2 = qb3;
      b0 = b1;
#pragma unroll
      for (int k = 0; k < PF; k++) {
        p0[k] = p1[k]; p1[k] = p2[k]; a0[k] = a1[k]; v0[k] = v1[k];
      }
#pragma unroll
      for (int cc = 0; cc < NB; cc++) d0[cc] = d1[cc];
    }
  }
  launch_done(ctl, lane, epoch);
}

}  // namespace cfdgpu
