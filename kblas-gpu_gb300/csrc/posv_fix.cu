// posv_fix.cu -- launches of the fixed-point FP64 Cholesky kernels
// (fix_kernel.cuh) by order: warps per system, factor in shared memory or not.
#include "fix_kernel.cuh"
#include "kblas_internal.h"
#include "launch_util.h"
#include "posv_fix.h"

namespace kgb {

// Orders lo < n <= hi and how a system of them runs. One warp holds 64 rows
// (lanes 0..7 the pivots', 24 + 32 below them), two hold 120, so up to there a
// block of columns passes over the rows once. Ten factors of order 64 fit into the
// shared memory of an SM (19 KB each), four of order 104; larger ones live in L2,
// eight systems of one warp to an SM (no barriers, and every warp busy to the last
// column) until the systems of an SM no longer fit into its share of L2 and a
// batch has fewer of them than warps: then four of two warps. us (POSV, one
// right-hand side) for 2 warps in shared memory / 1 / 2 warps in L2: 6,000 of order 80
// 1273 / 1483 / -; of 100 2366 / 2352 / -; 2,000 of 200 - / 3752 / 4708; 1,500 of 256
// - / 5757 / 6309; 500 of 400 (4 right-hand sides) - / 8349 / 7267.
struct FixClass {
  int lo, hi;
};
static const FixClass FIX_CLASSES[FIX_NCLS] = {{32, 64}, {64, 104}, {104, 320}, {320, PC_MAX_N}};
// A batch of at most two systems per SM waits for single systems: above order 104
// they get eight warps, the factor in shared memory up to 216 (197 KB). 50 of order
// 200 (two right-hand sides) with one warp each 1402 us, with eight 468; of 400 7450 and
// 2559.
static const FixClass FIX_FEW[FIX_NCLS] = {{32, 64}, {64, 104}, {104, 216}, {216, PC_MAX_N}};

template <int NW, bool FAC_SMEM>
static int launch_class(KBlasHandle *h, int hi, int class_hi, long long batch, const SysArgs &sys,
                        FixArgs fa) {
  auto kern = fix_posv_kernel<NW, FAC_SMEM>;
  const size_t smem = fix_smem_bytes<NW, FAC_SMEM>(hi);
  int st = set_smem(kern, fix_smem_bytes<NW, FAC_SMEM>(class_hi));  // the same from every thread
  if (st != KBLAS_Success) return st;
  long long grid = batch;
  if (!FAC_SMEM || fa.perm) {  // resident CTAs: their scratch, or their queue
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * NW, smem);
    if (e != cudaSuccess || per_sm < 1) per_sm = 1;
    if (!FAC_SMEM && per_sm > 8 / NW) per_sm = 8 / NW;  // as many as the scratch is for
    if (grid > (long long)h->sm_count * per_sm) grid = (long long)h->sm_count * per_sm;
  }
  kern<<<(unsigned)grid, 32 * NW, smem, h->stream>>>(sys, fa);
  KGB_LAUNCH_CHECK("fix_posv_kernel");
  return KBLAS_Success;
}

size_t fix_scratch_bytes(KBlasHandle *h, int max_n) {
  size_t most = 0;
  for (int c = 2; c < FIX_NCLS; c++) {
    const FixClass &k = FIX_CLASSES[c];
    if (max_n <= k.lo) continue;
    const size_t b = (size_t)(c == 2 ? 8 : 4) * make_fix_layout(max_n < k.hi ? max_n : k.hi).total() * 8;
    if (b > most) most = b;
  }
  return most * h->sm_count;
}

int fix_launch(KBlasHandle *h, int max_n, long long batch, const SysArgs &sys, FixArgs fa,
               int *queues) {
  const bool uniform = fa.perm == nullptr, few = batch <= 2 * h->sm_count;
  fa.batch = batch;
  for (int c = FIX_NCLS - 1; c >= 0; c--) {
    const FixClass &k = few ? FIX_FEW[c] : FIX_CLASSES[c];
    if (max_n <= k.lo || (uniform && max_n > k.hi)) continue;
    const int hi = max_n < k.hi ? max_n : k.hi;
    fa.lo = k.lo;
    fa.hi = hi;
    fa.queue = queues + c;
    fa.slot = make_fix_layout(hi).total();
    int st;
    switch (c) {
      case 0: st = launch_class<1, true>(h, hi, k.hi, batch, sys, fa); break;
      case 1: st = launch_class<2, true>(h, hi, k.hi, batch, sys, fa); break;
      case 2:
        st = few ? launch_class<8, true>(h, hi, k.hi, batch, sys, fa)
                 : launch_class<1, false>(h, hi, k.hi, batch, sys, fa);
        break;
      default:
        st = few ? launch_class<8, false>(h, hi, k.hi, batch, sys, fa)
                 : launch_class<2, false>(h, hi, k.hi, batch, sys, fa);
        break;
    }
    if (st != KBLAS_Success) return st;
  }
  return KBLAS_Success;
}

}  // namespace kgb
