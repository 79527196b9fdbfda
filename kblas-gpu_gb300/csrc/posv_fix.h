// posv_fix.h -- the fixed-point FP64 Cholesky launches (posv_fix.cu).
#pragma once

#include "fix_kernel.cuh"
#include "kblas_internal.h"

namespace kgb {

constexpr int FIX_NCLS = 4;

// Bytes of scratch for orders up to max_n (after ensure_device_props).
size_t fix_scratch_bytes(KBlasHandle *h, int max_n);

// One launch per class of orders, largest first (uniform: the one of max_n).
// queues: FIX_NCLS zeroed work counters.
int fix_launch(KBlasHandle *h, int max_n, long long batch, const SysArgs &sys, FixArgs fa,
               int *queues);

}  // namespace kgb
