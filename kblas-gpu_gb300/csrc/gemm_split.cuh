// gemm_split.cuh -- double-precision C := alpha op(A) op(B) + beta C on the
// tensor cores by exact slicing (fp64_split.cuh): batched GEMM and SYRK,
// uniform and variable-size.
//
// A CTA takes 64-row tiles of C. Per 64-deep k chunk it cuts its 64 rows of
// op(A) once, then walks 32-column tiles: cut op(B), issue the MMAs (one
// thread), and combine the sums from TMEM. The two TMEM halves hold the sums
// of odd and even digits of the same rows, so the warps of a row exchange
// half of their integer partial sums through shared memory and each finishes
// 8 of 16 columns. 107 KB of shared memory and half the TMEM columns per CTA:
// two CTAs per SM, whose load, cut, MMA and combine phases overlap. Measured
// (GB300, 20,000 products of 64^3): 1049 us against 8771 us on the FP64 pipe,
// which that one kept 95% busy. Bound by instruction issue and latency (28,600
// warp instructions a product, issue slots 43% busy, tensor pipe 10%).
// A chunk beyond the first adds to C (one more rounding of C per 64 of k).
#pragma once

#include "fp64_split.cuh"
#include "gemm_tile.cuh"

namespace kgb {

// op(X) as element (row, k) of a strided array
struct SpOp {
  const double *p;
  long long si, sk;
  __device__ __forceinline__ double at(int i, int k) const { return p[i * si + k * sk]; }
};

struct SpTile {
  SpOp A, B;  // rows of op(A) and columns of op(B), both (row, k)
  double *C;
  int ldc;
  int m, n, k;
  int part;  // TILE_FULL / TILE_LOWER / TILE_UPPER
};

struct SpSmem {
  int eA[SP_TM], eB[SP_TN];  // scales (exponent fields) of the rows / columns
  uint32_t tmem;
  int bad;    // a bounded wait ran out
  int nlist;  // entries to compute again
  uint64_t bar;
  unsigned short list[SP_LIST];
};

// Elements k .. k + 7 of one row; zeros outside (ok: the row exists).
__device__ __forceinline__ void sp_load8(const SpOp &o, int row, bool ok, int k, int kend,
                                         double (&x)[8]) {
#pragma unroll
  for (int i = 0; i < 8; i++) x[i] = 0.0;
  if (!ok) return;
  const double *p = o.p + row * o.si + k * o.sk;
  if (k + 8 <= kend) {
    if (o.sk == 1 && ((uintptr_t)p & 15) == 0) {  // k contiguous: 128-bit loads
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const double2 d = *reinterpret_cast<const double2 *>(p + i);
        x[i] = d.x;
        x[i + 1] = d.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++, p += o.sk) x[i] = *p;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++, p += o.sk)
      if (k + i < kend) x[i] = *p;
  }
}

__device__ __forceinline__ bool sp_in_part(int part, int gi, int gj) {
  return !((part == TILE_LOWER && gi < gj) || (part == TILE_UPPER && gi > gj));
}

// Largest |x| bits over the 8 lanes that hold one row's k groups.
__device__ __forceinline__ uint32_t sp_rowmax(uint32_t mx) {
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}

// End of the k chunk that starts at k0. No chunk is shorter than SP_KMIN unless k
// itself is (a variable-size batch: those use FP64 FMAs): a remainder of 1..15 takes 16
// of the 64 before it, which costs the same MMAs.
__device__ __forceinline__ int sp_chunk_end(int k0, int k) {
  const int left = k - k0;
  return left <= SP_KC ? k : k0 + (left < SP_KC + SP_KMIN ? SP_KC - SP_KMIN : SP_KC);
}

// One 64-row tile at I0 against the column tiles cp, cp + ncp, ... (alpha != 0
// and k > 0). A warp cuts 4 rows at a time, lane = (row, k group): the lanes
// of a row find its scale by shuffles, and both operand orders load whole
// 32-byte sectors. The next tile's columns and this tile's C are loaded while
// the MMAs run. Returns false if a bounded wait ran out.
static __device__ bool sp_row_tile(const SpTile &j, int I0, int cp, int ncp, double alpha,
                                   double beta0, unsigned char *smem, SpSmem &s, uint32_t &phase)
{
  unsigned char *sA = smem, *sB = smem + SP_SMEM_A;
  long long *xch = reinterpret_cast<long long *>(sB);  // exchange; the digits of B are used up by then
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int rows = min(SP_TM, j.m - I0);
  const int q = w & 3, half = w >> 2;  // TMEM lane quadrant, 16-column half of the tile
  const bool lower = q >= 2;
  const int row = 32 * (q & 1) + lane;
  const int kg = lane & 7, rsub = 4 * w + (lane >> 3);  // cutting: k group, row / column
  int tn = (j.n + SP_TN - 1) / SP_TN;
  if (j.part == TILE_LOWER) tn = min(tn, (I0 + rows - 1) / SP_TN + 1);
  if (j.part == TILE_UPPER) {
    const int skip = I0 / SP_TN;  // column tiles wholly below the diagonal
    if (cp < skip) cp += (skip - cp + ncp - 1) / ncp * ncp;
  }
  if (cp >= tn) return true;
  for (int k0 = 0, kend; k0 < j.k; k0 = kend) {
    kend = sp_chunk_end(k0, j.k);
    const int ksteps = (kend - k0 + 15) >> 4;
    const double beta = k0 == 0 ? beta0 : 1.0;
    const bool kon = 8 * kg < 16 * ksteps;
    const int kk = k0 + 8 * kg;
    int special = kend - k0 < SP_KMIN;
    double xb[8];
    {
      double x0[8], x1[8];
      sp_load8(j.A, I0 + rsub, rsub < rows, kk, kend, x0);
      sp_load8(j.A, I0 + rsub + 32, rsub + 32 < rows, kk, kend, x1);
      sp_load8(j.B, cp * SP_TN + rsub, cp * SP_TN + rsub < j.n, kk, kend, xb);
      const uint32_t m0 = sp_rowmax(sp_maxbits(x0)), m1 = sp_rowmax(sp_maxbits(x1));
      special |= sp_special(m0) || sp_special(m1);
      const int e0 = sp_scale(m0), e1 = sp_scale(m1);
      if (kg == 0) {
        s.eA[rsub] = e0;
        s.eA[rsub + 32] = e1;
      }
      if (kon) {
        sp_cut8<2>(x0, e0, sA + kg * SP_LBO_A + rsub * 16, SP_TM * 16);
        sp_cut8<2>(x1, e1, sA + kg * SP_LBO_A + (rsub + 32) * 16, SP_TM * 16);
      }
    }
    for (int t = cp; t < tn; t += ncp) {
      const int J0 = t * SP_TN;
      {
        const uint32_t mb = sp_rowmax(sp_maxbits(xb));
        const int eb = sp_scale(mb);
        if (kg == 0) s.eB[rsub] = eb;
        if (tid == 0) s.nlist = 0;
        if (kon) sp_cut8<1>(xb, eb, sB + kg * SP_LBO_B + rsub * 16, SP_TN * 16);
        fence_async_smem();
        special = (special & 1) | (sp_special(mb) ? 2 : 0);
      }
      const bool native = __syncthreads_or(special) != 0;
      if (!native && tid == 0) {
        tc_fence_after_sync();
        sp_issue(s.tmem, smem_addr(sA), smem_addr(sB), ksteps);
        tc_commit(&s.bar);
      }
      const int gi = I0 + row, c0 = 16 * half + (lower ? 8 : 0);  // the 8 columns this thread finishes
      double *Cp = j.C + gi + (size_t)(J0 + c0) * j.ldc;
      // loads that need not wait for the MMAs
      if (t + ncp < tn) {
        const int r = (t + ncp) * SP_TN + rsub;
        sp_load8(j.B, r, r < j.n, kk, kend, xb);
      }
      unsigned mine = 0;  // columns of this thread inside C
      double cv[8];
      {
        const double *p = Cp;
#pragma unroll
        for (int c = 0; c < 8; c++, p += j.ldc) {
          const int gj = J0 + c0 + c;
          const bool in = gi < j.m && gj < j.n && sp_in_part(j.part, gi, gj);
          if (in) mine |= 1u << c;
          cv[c] = (in && beta != 0.0) ? *p : 0.0;
        }
      }
      bool whole = native;
      if (!native) {
        if (!mbar_wait_bounded(&s.bar, phase)) s.bad = 1;
        phase ^= 1u;
        tc_fence_after_sync();
        // ---- combine: send the partner's 8 columns, keep the own ones ----
        const uint32_t at = s.tmem + ((uint32_t)(32 * q) << 16) + 16 * half;
        // slot of the partner warp (quadrant q ^ 2, same half)
        long long *dst = xch + (size_t)((half << 2) + (q ^ 2)) * 256 + lane;
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
          long long snd[4];
          sp_partial4(at + (lower ? 0 : 8) + h, lower, snd);
#pragma unroll
          for (int c = 0; c < 4; c++) dst[(h + c) * 32] = snd[c];
        }
        long long own[8];
        unsigned redo = 0;
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
          long long o4[4];
          float est[4];
          tmem_ld4_issue(s.tmem + ((uint32_t)(32 * q) << 16) + 224 + c0 + h, est);
          sp_partial4(at + (lower ? 8 : 0) + h, lower, o4);
          tmem_pin4(est);
#pragma unroll
          for (int c = 0; c < 4; c++) {
            own[h + c] = o4[c];
            if (est[c] < 4096.0f) redo |= 1u << (h + c);
          }
        }
        redo &= mine;
        if (redo) {
          int at_ = atomicAdd(&s.nlist, __popc(redo));
          for (unsigned b = redo; b && at_ < SP_LIST; b &= b - 1)
            s.list[at_++] = (unsigned short)((row << 5) | (c0 + __ffs(b) - 1));
        }
        tc_fence_before_sync();
        __syncthreads();
        if (s.bad) return false;
        whole = s.nlist > SP_LIST;
        if (!whole) {
          mine &= ~redo;
          if (beta != 0.0 && beta != 1.0) {
#pragma unroll
            for (int c = 0; c < 8; c++) cv[c] *= beta;
          }
          const long long *src = xch + (size_t)w * 256 + lane;
          const int ei = s.eA[row] - 2044 - 56;
          double *p = Cp;
#pragma unroll
          for (int c = 0; c < 8; c++, p += j.ldc) {
            const double v = sp_to_double(own[c] + src[c * 32], ei + s.eB[c0 + c]);
            if ((mine >> c) & 1u) *p = fma(alpha, v, cv[c]);
          }
          for (int e = tid; e < s.nlist; e += SP_NT) {
            const int er = s.list[e] >> 5, ec = s.list[e] & 31;
            double acc = 0.0;
            for (int k = k0; k < kend; k++) acc += j.A.at(I0 + er, k) * j.B.at(J0 + ec, k);
            double *p = j.C + (I0 + er) + (size_t)(J0 + ec) * j.ldc;
            const double old = beta == 0.0 ? 0.0 : beta * *p;
            *p = fma(alpha, acc, old);
          }
        }
      }
      if (whole) {
        // FP64 FMAs: thread = row (tid & 63), 8 columns
        const int r = tid & 63, cb = 8 * (tid >> 6);
        if (r < rows) {
          double acc[8];
#pragma unroll
          for (int c = 0; c < 8; c++) acc[c] = 0.0;
          for (int k = k0; k < kend; k++) {
            const double a = j.A.at(I0 + r, k);
#pragma unroll
            for (int c = 0; c < 8; c++)
              if (J0 + cb + c < j.n) acc[c] += a * j.B.at(J0 + cb + c, k);
          }
#pragma unroll
          for (int c = 0; c < 8; c++) {
            const int gr = I0 + r, gc = J0 + cb + c;
            if (gc < j.n && sp_in_part(j.part, gr, gc)) {
              double *p = j.C + gr + (size_t)gc * j.ldc;
              const double old = beta == 0.0 ? 0.0 : beta * *p;
              *p = fma(alpha, acc[c], old);
            }
          }
        }
      }
      __syncthreads();  // list, scales and exchange are free again
    }
  }
  return true;
}

__device__ __forceinline__ void sp_setup(SpSmem &s) {
  if (threadIdx.x < 32) {
    tmem_alloc(&s.tmem, SP_TMEM);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    s.bad = 0;
    mbar_init(&s.bar, 1);
    mbar_init_fence();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
}
__device__ __forceinline__ void sp_finish(SpSmem &s, uint32_t phase, int *status) {
  if (s.bad) {
    // a wait ran out: once more, bounded, for the MMAs in flight
    mbar_wait_bounded(&s.bar, phase ^ 1u);
    if (threadIdx.x == 0 && status) atomicExch(status, 1);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (threadIdx.x < 32) tmem_dealloc(s.tmem, SP_TMEM);
}

// C := alpha op(A) op(B) + beta C; dims = (m, n, k, lda, ldb, ldc) for GEMM,
// (m, k, lda, ldc) for SYRK (B = A, part = one triangle). blockIdx.y runs over
// (row tile, column part); alpha != 0.
template <bool SYRK, class AccA, class AccB, class AccC, class Dims>
__global__ void __launch_bounds__(SP_NT, 2)
gemm_split_kernel(int ta, int tb, int part, double alpha, AccA A, AccB B, double beta, AccC Cm,
                  Dims dims, int ncp, int *status)
{
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ SpSmem s;
  const long long mat = blockIdx.x;
  SpTile j;
  int lda, ldb;
  if constexpr (SYRK) {
    int d[4];
    dims.get(mat, d);
    j.m = j.n = d[0];
    j.k = d[1];
    lda = ldb = d[2];
    j.ldc = d[3];
  } else {
    int d[6];
    dims.get(mat, d);
    j.m = d[0]; j.n = d[1]; j.k = d[2];
    lda = d[3]; ldb = d[4]; j.ldc = d[5];
  }
  if (j.m <= 0 || j.n <= 0) return;
  const int tm = (j.m + SP_TM - 1) / SP_TM;
  if ((int)blockIdx.y >= tm * ncp) return;
  j.part = part;
  j.C = Cm.get(mat);
  if (j.k <= 0) {  // C := beta C; A and B are not read
    for (int u = blockIdx.y; u < tm * ncp; u += gridDim.y) {
      const int I0 = (u % tm) * SP_TM, rows = min(SP_TM, j.m - I0);
      for (int c = u / tm; c < j.n; c += ncp)
        for (int r = threadIdx.x; r < rows; r += SP_NT)
          if (sp_in_part(part, I0 + r, c)) {
            double *p = j.C + I0 + r + (size_t)c * j.ldc;
            *p = beta == 0.0 ? 0.0 : beta * *p;
          }
    }
    return;
  }
  const double *Ap = A.get(mat), *Bp = B.get(mat);
  j.A = ta ? SpOp{Ap, lda, 1} : SpOp{Ap, 1, lda};
  j.B = tb ? SpOp{Bp, 1, ldb} : SpOp{Bp, ldb, 1};
  sp_setup(s);
  uint32_t phase = 0;
  for (int u = blockIdx.y; u < tm * ncp; u += gridDim.y)
    if (!sp_row_tile(j, (u % tm) * SP_TM, u / tm, ncp, alpha, beta, smem, s, phase)) break;
  sp_finish(s, phase, status);
}

constexpr int SP_SMEM = SP_SMEM_A + SP_SMEM_B;

// Which products the split kernel takes (largest sizes of the launch; a hint
// of 0 is unknown and stays on the FP64-FMA tiles). Measured on GB300, 20,000
// matrices, FP64-FMA tiles against split: 16^3 325 / 493 us, 24 x 24 x 16
// 622 / 541, 32 x 32 x 16 622 / 541, 24^3 1148 / 555, 64 x 64 x 16 2450 / 934,
// 64^3 8771 / 1049; 5,000 of 128 x 16 x 64 2299 / 341, of 128^3 17839 / 1784. A tile
// costs the split kernel about the same whatever its fill, hence the product; the FP64
// tiles do half their work for up to 16 rows and k in steps of 16, so there one step
// stays with them (16 x 48 x 16 637 / 823, 16 x 64 x 16 635 / 851, 8 x 128 x 16 1264 /
// 1478, but 16 x 48 x 24 1177 / 823). Below k = 16 the error of the split is no longer
// smaller than that of an FP64 chain.
static inline bool sp_worthwhile(int m, int n, int k) {
  return k >= 16 && (k > 16 || m > 16) && (long long)m * n * k >= 24 * 24 * 16;
}

// Grid of a split launch: row tiles of the largest matrix, each with as many
// column parts as it takes to give every SM two CTAs.
static inline void sp_grid(KBlasHandle *h, long long batch, int mmax, int nmax, dim3 &grid, int &ncp) {
  ensure_device_props(h);
  const long long tm = (mmax + SP_TM - 1) / SP_TM, tn = (nmax + SP_TN - 1) / SP_TN;
  const long long want = 2LL * (h->sm_count > 0 ? h->sm_count : 152);
  long long c = (want + batch * tm - 1) / (batch * tm);
  if (c > tn) c = tn;
  if (c < 1) c = 1;
  ncp = (int)c;
  long long y = tm * c;
  if (y > 65535) y = 65535;
  grid = dim3((unsigned)batch, (unsigned)y);
}

}  // namespace kgb
