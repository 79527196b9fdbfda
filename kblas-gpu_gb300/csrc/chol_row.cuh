// chol_row.cuh -- FP32 POTRF / POTRS / POSV of orders above 32 whose factor fits
// in shared memory: one system per CTA of NW warps, one matrix row per lane.
//
// Left-looking by blocks of 8 columns, as chol_fix.cuh: a lane keeps the 8 sums
// of each of its R rows, lanes 0..7 of every warp hold the 8 pivot rows, so each
// warp finds the pivots by itself and a block needs one barrier (none with one
// warp). Bound by shared-memory loads: per column k a warp loads the 8 pivot
// rows' entries as two 128-bit broadcasts (8 cycles of the load pipe) and its own
// R entries for 8 R FMAs, hence up to four rows a lane.
//
// Every warp reads the 8 pivot rows of the block from A, so with several warps no
// thread writes them to A before the block's barrier; every other row is read and
// written by one lane only.
#pragma once

#include "chol_fix.cuh"
#include "chol_kernels.cuh"

namespace kgb {

constexpr int CR_FOLD = 32;  // columns after which a sum is taken off its entry

// Leading dimensions 4 mod 8: columns start on 16 bytes, and the backward
// solve's accesses along a row spread over the banks.
__host__ __device__ __forceinline__ FixLayout make_row_layout(int n) {
  return FixLayout{n, ((n + 3) & ~7) + 4};
}
template <int NW>
__host__ __device__ __forceinline__ size_t row_smem_bytes(int n) {
  return ((size_t)make_row_layout(n).total() + (size_t)NW * FX_W * FX_W + n) * sizeof(float);
}
template <int NW, int R>
constexpr int row_max_n() { return FX_W + NW * (32 * R - FX_W); }

__device__ __forceinline__ void row_ld8(const float *p, float (&y)[FX_W]) {
  const float4 u = *reinterpret_cast<const float4 *>(p), v = *reinterpret_cast<const float4 *>(p + 4);
  y[0] = u.x; y[1] = u.y; y[2] = u.z; y[3] = u.w;
  y[4] = v.x; y[5] = v.y; y[6] = v.z; y[7] = v.w;
}

// The columns C..C+7 of R rows a lane; returns the failing column (1-based, the
// same in every warp) or 0. Finished columns go to Xs and to A, the pivot rows (with
// several warps) to Xs alone: row_store_pivots.
template <int NW, int R>
__device__ __forceinline__ int row_block(const FixLayout &F, float *A, int lda, float *Xs, int C,
                                         float *rinv, float *yd)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int row[R], ri[R];
  bool own[R];
  float a[R][FX_W], acc[R][FX_W];
#pragma unroll
  for (int r = 0; r < R; r++) {
    row[r] = r == 0 ? (lane < FX_W ? C + lane : C + w * (32 - FX_W) + lane)
                    : C + FX_W + NW * (32 - FX_W) + ((r - 1) * NW + w) * 32 + lane;
    ri[r] = min(row[r], F.n - 1);
    own[r] = row[r] < F.n && (r > 0 || lane >= FX_W || w == 0);
#pragma unroll
    for (int c = 0; c < FX_W; c++) {
      a[r][c] = (row[r] < F.n && C + c <= row[r]) ? A[(size_t)ri[r] + (size_t)(C + c) * lda] : 0.f;
      acc[r][c] = 0.f;
    }
  }
  const float *P = Xs;
  int ld = F.n2;
  for (int K = 0; K < C; K += FX_W) {
    const float *yp = P + (C - K), *xp = P - K;
#pragma unroll
    for (int k = 0; k < FX_W; k++, yp += ld, xp += ld) {
      float y[FX_W];
      row_ld8(yp, y);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const float x = xp[ri[r]];
#pragma unroll
        for (int c = 0; c < FX_W; c++) acc[r][c] = fmaf(x, y[c], acc[r][c]);
      }
    }
    P += FX_W * ld;
    ld -= FX_W;
    if (((K + FX_W) & (CR_FOLD - 1)) == 0 || K + FX_W >= C) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < FX_W; c++) {
          a[r][c] -= acc[r][c];
          acc[r][c] = 0.f;
        }
    }
  }
  float *col = Xs + F.col(C);
  ld = F.ld(C / FX_W);
#pragma unroll
  for (int c = 0; c < FX_W; c++) {
    if (C + c < F.n) {
      const float d = __shfl_sync(0xffffffffu, a[0][c], c);
      if (!is_pos_pivot(d)) return C + c + 1;
      float s, q;
      pivot_rs(d, s, q);
      if (threadIdx.x == c) rinv[C + c] = q;
      float x[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        x[r] = (r == 0 && lane == c) ? s : a[r][c] * q;
        if (own[r] && row[r] >= C + c) {
          col[row[r]] = x[r];
          if (NW == 1 || r > 0 || lane >= FX_W) A[(size_t)row[r] + (size_t)(C + c) * lda] = x[r];
        }
      }
      col += ld;
      if (c + 1 < FX_W) {
        if (lane < FX_W) yd[c * FX_W + lane] = x[0];
        __syncwarp();
        float y[FX_W];
        row_ld8(yd + c * FX_W, y);
#pragma unroll
        for (int c2 = c + 1; c2 < FX_W; c2++)
#pragma unroll
          for (int r = 0; r < R; r++) a[r][c2] = fmaf(-x[r], y[c2], a[r][c2]);
      }
    }
  }
  return 0;
}

// The pivot rows of the block of columns C..C+7 from Xs to A, the columns before the
// failing one (fail, 1-based, or 0): by the lanes that put them into Xs, after the
// barrier that ends every warp's reading of them.
__device__ __forceinline__ void row_store_pivots(const FixLayout &F, float *A, int lda, const float *Xs,
                                                 int C, int fail)
{
  const int i = C + (int)threadIdx.x, end = min(fail ? fail - 1 : F.n, C + FX_W);
  if (threadIdx.x < FX_W && i < F.n)
    for (int k = C; k < end && k <= i; k++) A[(size_t)i + (size_t)k * lda] = Xs[F.col(k) + i];
}

// MODE as in chol_kernels.cuh.
template <int NW, int R, int MODE, class AccA, class AccB>
__global__ void __launch_bounds__(32 * NW)
chol_row_kernel(int n, int m, AccA A, int lda, AccB B, int ldb, int *info)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const FixLayout F = make_row_layout(n);
  float *Xs = reinterpret_cast<float *>(smem);
  float *yd = Xs + F.total() + (threadIdx.x >> 5) * FX_W * FX_W;
  float *rinv = Xs + F.total() + NW * FX_W * FX_W;
  const long long b = blockIdx.x;
  float *Ag = A.get(b);
  if (MODE == MODE_POTRS) {
    fx_load<NW>(F, Ag, lda, Xs, rinv);
  } else {
    int fail = 0;
    for (int C = 0; C < n && !fail; C += FX_W) {
      // a warp without rows of its own sits the block out: the pivots' verdict
      // reaches it at the barrier
      const int w = threadIdx.x >> 5;
      if (w == 0 || C + w * (32 - FX_W) + FX_W < n) {
        if (R > 2 && n - C > row_max_n<NW, 2>())
          fail = row_block<NW, R>(F, Ag, lda, Xs, C, rinv, yd);
        else if (R > 1 && n - C > row_max_n<NW, 1>())
          fail = row_block<NW, 2>(F, Ag, lda, Xs, C, rinv, yd);
        else
          fail = row_block<NW, 1>(F, Ag, lda, Xs, C, rinv, yd);
      }
      if (NW == 1) __syncwarp();
      else if (__syncthreads_or(fail) && !fail) fail = n + 1;  // (its value is warp 0's to report)
      if (NW > 1) row_store_pivots(F, Ag, lda, Xs, C, fail);
    }
    if (threadIdx.x == 0 && info) info[b] = fail;
    if (fail) return;
  }
  if (MODE != MODE_POTRF) fx_solve_all<NW, false>(F, Xs, rinv, B.get(b), ldb, m);
}

}  // namespace kgb
