// posv_fix.cu -- launches of the fixed-point FP64 Cholesky kernels
// (fix_kernel.cuh) by order: warps per system, factor in shared memory or not.
#include "fix_kernel.cuh"
#include "kblas_internal.h"
#include "launch_util.h"
#include "posv_fix.h"

namespace kgb {

// Orders lo < n <= hi and how a system of them runs. One warp holds 64 rows
// (lanes 0..7 the pivots', 24 + 32 below them), two hold 120, so up to there a
// block of columns passes over the rows once. The integer pipe wants 8 warps or
// more on an SM: ten factors of order 64 fit into shared memory (21 KB each), four
// of order 104; from there on the factors live in L2, which leaves four systems
// of two warps to an SM whatever their order. us for 1 / 2 warps, then 1 / 2 / 4 / 8
// with the factor in L2 (POSV, one right-hand side): 20,000 of order 64 1744 / 2326,
// 3274 / 4221 / 5965 / 10998; 6,000 of 100 - / 2007, 2273 / 2697 / 4283 / 7432; 3,000
// of 160 - / -, 3376 / 3087 / 4650 / 7372; 1,500 of 256 6203 / 5274 / 5967 / 8823.
struct FixClass {
  int lo, hi;
};
constexpr int FIX_L2_WARPS = 2, FIX_L2_CTAS = 4;  // per system; CTAs per SM that the scratch is for
static const FixClass FIX_CLASSES[FIX_NCLS] = {{32, 64}, {64, 104}, {104, PC_MAX_N}};

template <int NW, bool FAC_SMEM>
static int launch_class(KBlasHandle *h, int hi, long long batch, const SysArgs &sys, FixArgs fa) {
  auto kern = fix_posv_kernel<NW, FAC_SMEM>;
  const size_t smem = fix_smem_bytes<NW, FAC_SMEM>(hi);
  int st = set_smem(kern, smem);
  if (st != KBLAS_Success) return st;
  long long grid = batch;
  if (!FAC_SMEM || fa.perm) {  // resident CTAs: their scratch, or their queue
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * NW, smem);
    if (e != cudaSuccess || per_sm < 1) per_sm = 1;
    if (!FAC_SMEM && per_sm > FIX_L2_CTAS) per_sm = FIX_L2_CTAS;
    if (grid > (long long)h->sm_count * per_sm) grid = (long long)h->sm_count * per_sm;
  }
  kern<<<(unsigned)grid, 32 * NW, smem, h->stream>>>(sys, fa);
  KGB_LAUNCH_CHECK("fix_posv_kernel");
  return KBLAS_Success;
}

size_t fix_scratch_bytes(KBlasHandle *h, int max_n) {
  if (max_n <= FIX_CLASSES[FIX_NCLS - 1].lo) return 0;
  return (size_t)h->sm_count * FIX_L2_CTAS * make_fix_layout(max_n).total() * 8;
}

int fix_launch(KBlasHandle *h, int max_n, long long batch, const SysArgs &sys, FixArgs fa,
               int *queues) {
  const bool uniform = fa.perm == nullptr;
  fa.batch = batch;
  fa.slot = make_fix_layout(max_n).total();
  for (int c = FIX_NCLS - 1; c >= 0; c--) {
    const FixClass &k = FIX_CLASSES[c];
    if (max_n <= k.lo || (uniform && max_n > k.hi)) continue;
    const int hi = max_n < k.hi ? max_n : k.hi;
    fa.lo = k.lo;
    fa.hi = hi;
    fa.queue = queues + c;
    int st;
    switch (c) {
      case 0: st = launch_class<1, true>(h, hi, batch, sys, fa); break;
      case 1: st = launch_class<2, true>(h, hi, batch, sys, fa); break;
      default: st = launch_class<FIX_L2_WARPS, false>(h, hi, batch, sys, fa); break;
    }
    if (st != KBLAS_Success) return st;
  }
  return KBLAS_Success;
}

}  // namespace kgb
