// fix_kernel.cuh -- FP64 POTRF / POTRS / POSV of orders above 32 in fixed point
// (chol_fix.cuh): one system per CTA of NW warps.
#pragma once

#include "chol_fix.cuh"
#include "chol_kernels.cuh"
#include "posv_core.cuh"

namespace kgb {

// Systems [0, count) of a launch: system indices themselves (uniform), or the
// slots [off[hi] .. off[lo + 1] + cnt[lo + 1]) of the permutation that sorts a
// variable-size batch by descending order, which hold the orders lo < n <= hi.
struct FixArgs {
  long long batch;
  const int *off, *cnt, *perm, *narr;
  int lo, hi;
  int *queue;         // variable size: next slot (relative), zeroed before the launch
  int *info;
  // systems left to the FP64 path: listed (uniform), or marked (variable size)
  int *redo_count, *redo_list, *redo_mark;
  double *scratch;    // per-CTA factor, when it does not fit in shared memory
  long long slot;     // its doubles
};

template <int NW, bool FAC_SMEM>
__host__ __device__ __forceinline__ size_t fix_smem_bytes(int n) {
  const size_t b = (FAC_SMEM ? (size_t)make_fix_layout(n).total() * 8 : NW * sizeof(FixStage)) +
                   NW * sizeof(FixScratch) + (size_t)n * 24;
  return (b + 15) / 16 * 16;
}

// CTAs per SM that the registers are cut for: of one warp twelve (168 registers;
// with eight, 255 registers, POSV of order 64 took 16% longer), of two warps five
// (with four, 17% longer at order 80, 5% shorter at 100) or, with the factor in L2, the
// number that the scratch is for: 8 warps to an SM (12 would leave 168 registers, fewer
// than two rows a lane take).
template <int NW, bool FAC_SMEM>
__host__ __device__ constexpr int fix_min_ctas() {
  return FAC_SMEM ? (NW == 1 ? 12 : NW == 2 ? 5 : 1) : 8 / NW;
}

// The solves as a function of their own: inlined, they and the factorization take
// registers from each other (20,000 of order 64, factor only, with 56-bit entries: 1245
// us without spills, up to 1740 with). L and the reciprocals lie at these offsets of the dynamic shared memory.
template <int NW>
__device__ __noinline__ void fix_solve_smem(int n, int rinv_at, double *B, int ldb, int m)
{
  extern __shared__ __align__(16) unsigned char smem[];
  fx_solve_all<NW, false>(make_fix_layout(n), reinterpret_cast<const double *>(smem),
                          reinterpret_cast<const double *>(smem + rinv_at), B, ldb, m);
}

template <int NW>
__device__ __noinline__ void fix_solve_l2(int n, const double *Xs, int rinv_at, double *B, int ldb,
                                          int m)
{
  extern __shared__ __align__(16) unsigned char smem[];
  fx_solve_all<NW, true>(make_fix_layout(n), Xs, reinterpret_cast<const double *>(smem + rinv_at),
                         B, ldb, m);
}

// POTRS: A holds the factor; m = 0: factor only.
template <int NW, bool FAC_SMEM>
__global__ void __launch_bounds__(32 * NW, fix_min_ctas<NW, FAC_SMEM>())
fix_posv_kernel(SysArgs sys, FixArgs fa)
{
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_slot;
  int first = 0;
  long long count = fa.batch;
  const bool uniform = fa.perm == nullptr;
  if (!uniform) {
    first = fa.off[fa.hi];
    count = fa.off[fa.lo + 1] + fa.cnt[fa.lo + 1] - first;
  }
  long long q = blockIdx.x;
  for (;;) {
    if (!uniform) {
      if (threadIdx.x == 0) s_slot = atomicAdd(fa.queue, 1);
      fx_sync<NW>();
      q = s_slot;
    }
    if (q >= count) break;
    const long long sidx = uniform ? q : (long long)fa.perm[first + q];
    const int n = uniform ? sys.n : fa.narr[sidx];
    int m, lda, ldb;
    double *A, *B;
    sys.get(sidx, m, A, lda, B, ldb);
    const FixLayout F = make_fix_layout(n);
    double *Xs = FAC_SMEM ? reinterpret_cast<double *>(smem)
                          : fa.scratch + (size_t)blockIdx.x * fa.slot;
    FixStage *st = FAC_SMEM ? nullptr : reinterpret_cast<FixStage *>(smem) + (threadIdx.x >> 5);
    unsigned char *p = smem + (FAC_SMEM ? (size_t)F.total() * 8 : NW * sizeof(FixStage));
    FixScratch *fs = reinterpret_cast<FixScratch *>(p) + (threadIdx.x >> 5);
    p += NW * sizeof(FixScratch);
    double *rinv = reinterpret_cast<double *>(p);
    int *Es = reinterpret_cast<int *>(rinv + n), *zs = Es + n;
    float *qs = reinterpret_cast<float *>(zs + n);
    int *wk = reinterpret_cast<int *>(qs + n);
    bool ok = true;
    if (sys.op == 2) {
      fx_load<NW>(F, A, lda, Xs, rinv);
    } else {
      ok = fx_potrf<NW, !FAC_SMEM>(F, A, lda, Xs, Es, qs, wk, zs, rinv, fs, st);
      if (ok) fx_store<NW>(F, Xs, Es, zs, rinv, A, lda, m > 0);
      if (threadIdx.x == 0) {
        if (ok) {
          if (fa.info) fa.info[sidx] = 0;
        } else if (uniform) {
          fa.redo_list[atomicAdd(fa.redo_count, 1)] = (int)sidx;
        } else {
          fa.redo_mark[sidx] = 1;
        }
      }
    }
    if (ok && m > 0) {
      const int rinv_at = (int)(reinterpret_cast<unsigned char *>(rinv) - smem);
      if (FAC_SMEM) fix_solve_smem<NW>(n, rinv_at, B, ldb, m);
      else fix_solve_l2<NW>(n, Xs, rinv_at, B, ldb, m);
    }
    fx_sync<NW>();
    if (uniform) q += gridDim.x;
  }
}

// POTRF / POSV of orders up to 32, one warp per system and one row per lane,
// without workspace: a matrix that does not fit the fixed-point scheme is
// factored again in FP64 by the same warp or (leave) marked in info, with
// INFO_LEFT, for chol_team_kernel. 4 KB to 7 KB of shared memory; FIX_SMALL_CTAS
// CTAs per SM leave 128 registers to a thread.
constexpr int FIX_SMALL_CTAS = 16;
template <int MODE, class AccA, class AccB>
__global__ void __launch_bounds__(32, FIX_SMALL_CTAS)
fix_small_kernel(int n, int m, AccA Aa, int lda, AccB Ba, int ldb, int *info, int leave)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const FixLayout F = make_fix_layout(n);
  double *Xs = reinterpret_cast<double *>(smem);
  FixScratch *fs = reinterpret_cast<FixScratch *>(Xs + F.total());
  double *rinv = reinterpret_cast<double *>(fs + 1);
  int *Es = reinterpret_cast<int *>(rinv + n), *zs = Es + n;
  float *qs = reinterpret_cast<float *>(zs + n);
  int *wk = reinterpret_cast<int *>(qs + n);
  const long long b = blockIdx.x;
  double *A = Aa.get(b);
  int fail = 0;
  if (fx_potrf<1, false, 1>(F, A, lda, Xs, Es, qs, wk, zs, rinv, fs))
    fx_store<1>(F, Xs, Es, zs, rinv, A, lda, MODE == MODE_POSV);
  else if (leave)
    fail = INFO_LEFT;
  else
    fail = fx_potrf_fp64(F, A, lda, Xs, rinv);
  if (threadIdx.x == 0 && info) info[b] = fail;
  if (MODE == MODE_POSV && !fail) fix_solve_smem<1>(n, (int)(reinterpret_cast<unsigned char *>(rinv) - smem), Ba.get(b), ldb, m);
}

}  // namespace kgb
