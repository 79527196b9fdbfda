// chol_fix.cuh -- FP64 Cholesky in 64-bit fixed point on the integer pipe, and
// the FP64 triangular solves with its factor (panel path, n > 32).
//
// Why: the part retires 2 FP64 FMA lanes per clock and SM but about 30 lanes of
// a 32 x 32 -> 64-bit integer multiply-add, and three of those make a product
// of two 60-bit numbers. A Cholesky factor suits fixed point: row i of L is
// bounded by sqrt(a_ii), so its scale 2^E_i > sqrt(a_ii) is known beforehand.
//
//   L(i, k) = X 2^(E_i - 59),  X = hi 2^30 + lo, |X| < 2^59, lo in [-2^29, 2^29)
//   S(i, j) = a_ij - sum_k L(i, k) L(j, k) in units of 2^(E_i + E_j - 62)
//
// A product adds hi hi' to one 64-bit sum and hi lo' + lo hi' to another (lo lo'
// is below 2^-60 of the scales). The sums cannot overflow: sum |hi|^2 of a row
// is at most 2^58 (Cauchy-Schwarz), so |sum hi hi'| <= 2^58 and
// |sum hi lo' + lo hi'| <= 2 2^29 sqrt(K) 2^29: for K = FX_CARRY = 128 columns,
// after which the second sum's upper part is carried into the first, <= 2^62.6.
// The pivot's reciprocal square root (FP32 seed, one cubic step) and the scaling of
// a column are 64-bit integer work too. The backward error |dA_ij| is a few
// 2^-60 sqrt(K) sqrt(a_ii a_jj), where a chain of FP64 FMAs has, entry by entry,
// about 2^-53 (|L| |L^T|)_ij.
//
// So an entry far below sqrt(a_ii a_jj) would keep fewer bits than in FP64, and a
// component of a solution that hangs on such entries alone (the far end of a
// decaying covariance for a unit right-hand side, weakly coupled unknowns) would
// be wrong in as many. So these are counted (fx_share): a coupling of the unknowns
// i > j is an entry with a_ij or S(i, j) not zero, t the bits by which the larger of
// both lies below its scale 2^(E_i + E_j), and an unknown whose couplings have
// max(0, t - 8) at more than 1 in the mean leaves the matrix to the FP64 path.
// Single small entries among others of the same unknowns, as random matrices have
// them, do not matter: the others' rounding reaches every component that theirs
// reaches. That takes others that lead there: a matrix that has a coupling with t
// above 12 stays only if every unknown has couplings with t up to 12 to at least half
// of the unknowns, for then the two that it couples have at least two such neighbours
// in common. (Two strongly coupled halves of order 110 with one coupling of 1e-12
// between them, taken in fixed point: the components of A^-1 e_1 in the second half
// wrong by 2e-6.)
// Against quad precision, FP64 FMAs / fixed point, on the matrices that stay: root mean
// square of |A - L L^T|_ij / (|L| |L^T|)_ij in 2^-53, G G^T + n I of order 128 1.2 /
// 1.0, condition 1e6 of order 64 0.5 / 0.4, squared-exponential covariance of length
// 0.3 and order 160 0.35 / 0.41; the largest relative error of a component of A^-1 e_1
// 7e-14 / 4e-13, 4e-10 / 5e-11 and 1.8e-9 / 1.5e-9. The same covariance with length
// 0.05, taken in fixed point: 3e-11 / 3e-6. 56-bit entries with the cross products
// summed in FP32 are faster (10,000 POSV of order 64, four right-hand sides 968 us
// against 1139, 2,000 of order 150 1944 against 2405), but not as accurate as FP64 FMAs
// entry by entry: 1.2 / 4.8 on the shifted matrices.
//
// A matrix that does not fit the scheme -- a pivot below 2^-42 a_jj, an entry
// or a row of L above its bound (only when A is not positive definite), an
// infinity or NaN, a diagonal outside 2^+-800, weak couplings -- is left to the
// FP64 path, which starts again from A (nothing has been written), so info and
// the columns before a failing pivot are that path's.
//
// Work split: left-looking by blocks of 8 columns, one matrix row per lane (or
// two): a lane keeps the 8 pairs of sums of each of its rows, loads its own
// X(i, k) (8 bytes, lanes consecutive) and the 8 pivot rows' X(C + c, k) as four
// 128-bit broadcasts: 24 (48) multiply-adds for 5 (6) loads. Lanes 0..7 of every
// warp hold the block's 8 pivot rows, so each warp finds the pivots by itself:
// the chain of 8 pivots, which the other warps would have to wait for, costs
// every warp 8 lanes instead, and a block needs one barrier.
#pragma once

#include "device_util.cuh"
#include "fp64_split.cuh"

namespace kgb {

constexpr int FX_W = 8;         // columns per block
constexpr int FX_CARRY = 128;   // columns after which the sums of cross products are carried
constexpr int FX_DMIN_LOG = 20; // smallest pivot taken, in units of 2^(2 E - 62)

// The lower triangle in blocks of 8 columns: block b holds the rows 8 b .. of
// its columns, leading dimension 2 mod 4, so that columns start on 16 bytes and
// 64-bit accesses along a row of L (the backward solve) hit different banks.
struct FixLayout {
  int n, n2;  // n rounded up to 4, plus 2
  __host__ __device__ __forceinline__ int ld(int b) const { return n2 - b * FX_W; }
  __host__ __device__ __forceinline__ int base(int b) const {
    return FX_W * (b * n2 - (FX_W / 2) * b * (b - 1));
  }
  __host__ __device__ __forceinline__ int total() const { return base((n + FX_W - 1) / FX_W); }
  // column k, indexed by the row
  __host__ __device__ __forceinline__ int col(int k) const {
    const int b = k / FX_W;
    return base(b) + (k - b * FX_W) * ld(b) - b * FX_W;
  }
};
__host__ __device__ __forceinline__ FixLayout make_fix_layout(int n) {
  return FixLayout{n, ((n + 3) & ~3) + 2};
}

template <int NW>
__device__ __forceinline__ void fx_sync() {
  if (NW == 1) __syncwarp();
  else __syncthreads();
}

// E with a (1 + 2^-12) < 2^(2 E); bad unless a is positive and within 2^+-800.
__device__ __forceinline__ int fx_scale(double a, int &bad) {
  const int hi = __double2hiint(a);
  if (hi < (223 << 20) || hi >= (1823 << 20)) {
    bad = 1;
    return 0;
  }
  return ((((hi + 0x100) >> 20) - 1023) >> 1) + 1;
}

// a 2^(62 - es), cut towards zero (but 1 at least, unless a is zero); bad if
// |a| >= 2^es (infinities and NaNs too)
__device__ __forceinline__ long long fx_from(double a, int es, int &bad) {
  const uint32_t hi = (uint32_t)__double2hiint(a), lo = (uint32_t)__double2loint(a);
  const int r = es + 1022 - (int)((hi >> 20) & 0x7ffu);
  if (r < 0) bad = 1;
  long long m =
      (long long)(((((unsigned long long)((hi & 0xfffffu) | 0x100000u)) << 32) | lo) << 9 >> min(max(r, 0), 63));
  if (m == 0) m = (hi << 1 | lo) != 0;
  const long long s = (long long)((int)hi >> 31);
  return (m ^ s) - s;
}

// The two sums of products, in units of S.
__device__ __forceinline__ long long fx_sum(long long hh, long long mid) {
  return (long long)((unsigned long long)hh << 4) + ((mid + (1ll << 25)) >> 26);
}
// Moves what it can of the cross products to the sum of hi hi', without rounding.
__device__ __forceinline__ void fx_carry(long long &hh, long long &mid) {
  hh += mid >> 30;
  mid &= (1ll << 30) - 1;
}

// Reciprocal square root of a pivot: rho = rh 2^31 + rl = 2^92 / sqrt(d 4^z), z
// chosen so that dn = d 4^z is in [2^60, 2^62).
struct FixPivot {
  int rh, rl, z;
};
// Pivots and the pivot rows of the block at hand, one copy per warp.
struct FixScratch {
  double yd[FX_W][FX_W];  // limbs, [column][row]
  FixPivot pv[FX_W];
};

// FP32 seed y = Y 2^-24 of 1 / sqrt(m), m = dn 2^-60, and r = y (1 + e / 2 +
// 3 e^2 / 8), e = 1 - m y^2 (Halley's cubic iteration; |e| < 2^-20, so the next
// term is below 2^-61). |e| 2^78 < 2^63: the product m y^2 is formed modulo 2^64.
__device__ __forceinline__ FixPivot fx_rsqrt(long long d) {
  FixPivot p;
  p.z = (__clzll(d) - 2) >> 1;
  const unsigned long long dn = (unsigned long long)d << (2 * p.z);
  const unsigned dh = (unsigned)(dn >> 30), dl = (unsigned)dn & 0x3fffffffu;
  const float y = rsqrtf(__uint2float_rn(dh) * 9.31322574615478515625e-10f);  // 2^-30
  const unsigned Y = min(__float2uint_rn(y * 16777216.0f), 0xffffffu);
  const unsigned long long y2 = (unsigned long long)Y * Y;
  const unsigned yh = (unsigned)(y2 >> 24), yl = (unsigned)y2 & 0xffffffu;
  const long long e = -(long long)((((unsigned long long)dh * yh) << 24) +
                                   (unsigned long long)dh * yl +
                                   (((unsigned long long)dl * yh) >> 6) +
                                   (((unsigned long long)dl * yl) >> 30));  // 2^-78
  const int e1 = (int)(e >> 28);                                           // 2^-50
  const int e2 = (int)(((long long)e1 * e1) >> 42);                        // 2^-58
  const long long corr = (e >> 21) + ((3 * e2) >> 3);                      // 2^-58, < 2^38
  const long long r = ((long long)Y << 38) + ((corr * (long long)Y) >> 20);  // 2^62 / sqrt(m)
  p.rh = (int)(r >> 31);
  p.rl = (int)r & 0x7fffffff;
  if (p.rh < 0) p.rh = p.rl = 0x7fffffff;  // 2^62
  return p;
}

// s rho 2^(z - 64): the entry of L in units of 2^(E - 59). bad gets set bits if s
// or the entry is out of range (the row's squares then exceed a_ii).
__device__ __forceinline__ long long fx_scale_entry(long long s, const FixPivot &p, unsigned &bad) {
  const int sh = (int)(s >> 32);
  bad |= (unsigned)(sh ^ (sh >> 31)) >> (30 - p.z);
  const long long t = (long long)((unsigned long long)s << p.z);
  const int th = (int)(t >> 31), tl = (int)t & 0x7fffffff;
  long long m = (long long)th * p.rl;
  m += (long long)tl * p.rh;
  long long x = (m >> 31) + 2;
  x += (long long)th * p.rh;
  x >>= 2;
  const int xh = (int)(x >> 32);
  bad |= (unsigned)(xh ^ (xh >> 31)) >> 27;
  return x;
}

// Both limbs as the words of a double (never used as a floating-point value).
__device__ __forceinline__ double fx_pack(long long x) {
  const int lo = (int)((unsigned)x << 2) >> 2;
  return __hiloint2double((int)((x - lo) >> 30), lo);
}
__device__ __forceinline__ long long fx_unpack(double v) {
  return ((long long)__double2hiint(v) << 30) + __double2loint(v);
}

// The 8 products of x with y[c0..7], each kind of product in turn: the two that
// share a sum are then 8 instructions apart.
__device__ __forceinline__ void fx_mac(long long (&hh)[FX_W], long long (&mid)[FX_W], double x,
                                       const double (&y)[FX_W], int c0) {
  const int xh = __double2hiint(x), xl = __double2loint(x);
#pragma unroll
  for (int c = 0; c < FX_W; c++)
    if (c >= c0) hh[c] += (long long)xh * __double2hiint(y[c]);
#pragma unroll
  for (int c = 0; c < FX_W; c++)
    if (c >= c0) mid[c] += (long long)xh * __double2loint(y[c]);
#pragma unroll
  for (int c = 0; c < FX_W; c++)
    if (c >= c0) mid[c] += (long long)xl * __double2hiint(y[c]);
}
// 8 consecutive limbs, 16-byte aligned
__device__ __forceinline__ void fx_ld8(const double *p, double (&y)[FX_W]) {
#pragma unroll
  for (int c = 0; c < FX_W; c += 2) {
    const double2 v = *reinterpret_cast<const double2 *>(p + c);
    y[c] = v.x;
    y[c + 1] = v.y;
  }
}
// The bits by which a coupling lies below its scale, plus 2; 32: it has none of the upper
// 30 or is none at all.
__device__ __forceinline__ int fx_below(long long a, long long s) {
  const int ah = (int)(a >> 32), sh = (int)(s >> 32);
  return __clz((ah ^ (ah >> 31)) | (sh ^ (sh >> 31)));
}
// A coupling's share of its two unknowns' sums: an unknown whose sum of shares ends above
// zero has couplings that are too weak. Where the line lies: an entry's error is about
// 2^-59..2^-60 of its scale, which FP64 FMAs reach 6 bits below it, and with 8 bits free
// and 1 more in the mean all of G G^T + n I up to order 1024 (0.0..0.5 in the mean of the
// worst unknown) and random matrices of condition 1e2..1e8 (0.0..0.2) stay;
// squared-exponential covariances on the unit square stay from length 0.27 on (at 0.25
// 1.3..2.2, at 0.2 2.3..5.8).
__device__ __forceinline__ int fx_share(bool none, int below) {
  return none ? 0 : max(below - 10, 0) - 1;
}
// Couplings more than 12 bits below their scales (an entry that is the only way from one
// unknown to another is then good to 2^-47) and pairs without a coupling: rare in dense
// matrices, so these are not summed like the shares but added at once, to the upper half
// of both unknowns' sums. weak gets bit 0 if it is a coupling.
constexpr int FX_LOOSE = 14;  // of fx_below
constexpr int FX_COUNT = 1 << 16;
__device__ __forceinline__ void fx_count_loose(bool none, int *wi, int *wj, unsigned &weak) {
  if (!none) weak |= 1u;
  atomicAdd(wi, FX_COUNT);
  atomicAdd(wj, FX_COUNT);
}
// Whether an unknown's sum leaves the matrix to FP64; weak gets bit 1 if the unknown is
// strongly coupled to fewer than half of the unknowns.
__device__ __forceinline__ bool fx_too_weak(int sum, int n, unsigned &weak) {
  const int shares = (short)sum, loose = (sum - shares) / FX_COUNT;
  if (2 * (n - 1 - loose) < n) weak |= 2u;
  return shares > 0;
}

// R rows of a thread against the block of columns C..C+7: the sums over the
// columns before C.
template <int R>
__device__ __forceinline__ void fx_dot(const FixLayout &F, const double *Xs, int C,
                                       const int (&row)[R], long long (&hh)[R][FX_W],
                                       long long (&mid)[R][FX_W])
{
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int c = 0; c < FX_W; c++) hh[r][c] = mid[r][c] = 0;
  const double *P = Xs;
  int ld = F.n2;
  for (int K = 0; K < C; K += FX_W) {
    const double *yp = P + (C - K);
    const double *xp = P - K;
#pragma unroll 4
    for (int k = 0; k < FX_W; k++) {
      double y[FX_W], x[R];
      fx_ld8(yp, y);
#pragma unroll
      for (int r = 0; r < R; r++) x[r] = xp[row[r]];
      yp += ld;
      xp += ld;
#pragma unroll
      for (int r = 0; r < R; r++) fx_mac(hh[r], mid[r], x[r], y, 0);
    }
    P += FX_W * ld;
    ld -= FX_W;
    if (((K + FX_W) & (FX_CARRY - 1)) == 0) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < FX_W; c++) fx_carry(hh[r][c], mid[r][c]);
    }
  }
}

// The same with X in global memory: the next 8 columns of the warp's rows and of
// the pivot rows are copied to shared memory while the current 8 are multiplied,
// so the latency of L2 is paid once per block, not once per 4 columns (500 systems
// of order 512, with 56-bit entries: 13.6 -> 11.6 ms). A's 8 columns come last, the same way, and into av
// (zeros right of the diagonal and of the matrix): registers that hold them during the
// products spill.
struct FixStage {
  double x[2][FX_W][64];
  double y[2][FX_W][FX_W];
};
__device__ __forceinline__ void fx_copy8(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
template <int R>
__device__ __forceinline__ void fx_dot_staged(const FixLayout &F, const double *A, int lda,
                                              const double *Xs, int C, const int (&row)[R],
                                              const int (&ri)[R], long long (&hh)[R][FX_W],
                                              long long (&mid)[R][FX_W], double (&av)[R][FX_W],
                                              FixStage *st)
{
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int c = 0; c < FX_W; c++) hh[r][c] = mid[r][c] = 0;
  const double *P = Xs;  // the block to be copied next
  int ld = F.n2;
  auto copy = [&](int K) {
    const int buf = (K / FX_W) & 1;
    if (K < C) {
#pragma unroll
      for (int c = 0; c < FX_W; c++)
#pragma unroll
        for (int r = 0; r < R; r++) fx_copy8(&st->x[buf][c][r * 32 + lane], P + c * ld + (ri[r] - K));
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = e * 4 + (lane >> 3), j = lane & 7;
        fx_copy8(&st->y[buf][c][j], P + c * ld + (C - K) + j);
      }
      P += FX_W * ld;
      ld -= FX_W;
    } else {
#pragma unroll
      for (int c = 0; c < FX_W; c++)
#pragma unroll
        for (int r = 0; r < R; r++)
          if (row[r] < F.n && C + c <= row[r])
            fx_copy8(&st->x[buf][c][r * 32 + lane], A + (size_t)row[r] + (size_t)(C + c) * lda);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  copy(0);
  for (int K = 0; K < C; K += FX_W) {
    copy(K + FX_W);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const int buf = (K / FX_W) & 1;
#pragma unroll 2
    for (int k = 0; k < FX_W; k++) {
      double y[FX_W];
      fx_ld8(st->y[buf][k], y);
#pragma unroll
      for (int r = 0; r < R; r++) fx_mac(hh[r], mid[r], st->x[buf][k][r * 32 + lane], y, 0);
    }
    __syncwarp();  // before this buffer is copied to again
    if (((K + FX_W) & (FX_CARRY - 1)) == 0) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < FX_W; c++) fx_carry(hh[r][c], mid[r][c]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  const int buf = (C / FX_W) & 1;
#pragma unroll
  for (int c = 0; c < FX_W; c++)
#pragma unroll
    for (int r = 0; r < R; r++)  // (each lane reads what it copied itself)
      av[r][c] = (row[r] < F.n && C + c <= row[r]) ? st->x[buf][c][r * 32 + lane] : 0.0;
}

// The columns C..C+7 of R rows, after fx_dot. FIRST: row[0] of lanes 0..7 are the
// pivot rows; otherwise the pivots are the ones that FIRST left in fs (KEEP). own: rows
// that this thread stores. qs: the squares of each row's entries. wk: the sums of
// weak couplings, the rows' in wr. False if a pivot is too small: every warp sees the
// same pivots. bad gets set bits if a row is out of range.
template <int R, bool FIRST, bool KEEP>
__device__ __forceinline__ bool fx_columns(const FixLayout &F, double *Xs, int C,
                                           const int (&row)[R], const bool (&own)[R],
                                           int *zs, double *rho_s,
                                           long long (&hh)[R][FX_W], long long (&mid)[R][FX_W],
                                           long long (&a)[R][FX_W], FixScratch *fs,
                                           float (&qs)[R], int *wk, int (&wr)[R],
                                           unsigned &weak, unsigned &bad)
{
  const int lane = threadIdx.x & 31;
  const int ld = F.ld(C / FX_W);
  double *col = Xs + F.col(C);
  // the columns' sums of this lane, plus R, a byte each (0..44)
  unsigned wc[2] = {R * 0x01010101u, R * 0x01010101u};
#pragma unroll
  for (int c = 0; c < FX_W; c++) {
    if (C + c < F.n) {
      long long s[R];
      FixPivot pv;
#pragma unroll
      for (int r = 0; r < R; r++) s[r] = a[r][c] - fx_sum(hh[r][c], mid[r][c]);
      if (FIRST) {
        const long long d = __shfl_sync(0xffffffffu, s[0], c);
        if (d < (1ll << FX_DMIN_LOG) || d >= (1ll << 62)) return false;
        pv = fx_rsqrt(d);
        if (threadIdx.x == c) {
          rho_s[C + c] = __longlong_as_double(((long long)pv.rh << 31) + pv.rl);
          zs[C + c] = pv.z;
        }
      } else {
        pv = fs->pv[c];
      }
      double x[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        unsigned b = 0;
        x[r] = fx_pack(fx_scale_entry(s[r], pv, b));
        if (own[r] && row[r] >= C + c) {
          bad |= b;
          col[row[r]] = x[r];
          const float f = (float)__double2hiint(x[r]);
          qs[r] += f * f;
          if (row[r] > C + c) {
            const bool none = (a[r][c] | s[r]) == 0;
            const int below = fx_below(a[r][c], s[r]), w = fx_share(none, below);
            wr[r] += w;
            wc[c >> 2] += (unsigned)w << (8 * (c & 3));
            if (below > FX_LOOSE) fx_count_loose(none, wk + row[r], wk + C + c, weak);
          }
        }
      }
      col += ld;
      if (FIRST) {
        if (lane < FX_W) fs->yd[c][lane] = x[0];
        if (KEEP && lane == c) fs->pv[c] = pv;
        __syncwarp();
      }
      double y[FX_W];
      fx_ld8(fs->yd[c], y);
#pragma unroll
      for (int r = 0; r < R; r++) fx_mac(hh[r], mid[r], x[r], y, c + 1);
    }
  }
  // lane c adds up column c's: two columns to a word
  unsigned mine = 0;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const unsigned t = __reduce_add_sync(0xffffffffu, (wc[e >> 1] >> (8 * (e & 1))) & 0x00ff00ffu);
    // columns 4 (e / 2) + e % 2 and two further
    if ((lane & ~2) == (e >> 1) * 4 + (e & 1)) mine = (lane & 2) ? t >> 16 : t & 0xffffu;
  }
  if (lane < FX_W && C + lane < F.n) atomicAdd(wk + C + lane, (int)mine - 32 * R);
  return true;
}

// The block of columns C..C+7 for R rows of each thread.
template <int R, bool FIRST, bool BIG>
__device__ __forceinline__ bool fx_rows(const FixLayout &F, const double *A, int lda, double *Xs,
                                        int C, const int (&row)[R], const bool (&own)[R],
                                        const int *Es, float *q, int *wk, int *zs,
                                        double *rho_s, FixScratch *fs, FixStage *st,
                                        unsigned &weak, unsigned &bad)
{
  int ri[R];
  long long a[R][FX_W], hh[R][FX_W], mid[R][FX_W];
#pragma unroll
  for (int r = 0; r < R; r++) ri[r] = min(row[r], F.n - 1);
  auto fixed = [&](const double (&av)[R][FX_W]) {
    int b = 0;
#pragma unroll
    for (int c = 0; c < FX_W; c++) {
      const int Ec = Es[min(C + c, F.n - 1)];
#pragma unroll
      for (int r = 0; r < R; r++) a[r][c] = fx_from(av[r][c], Es[ri[r]] + Ec, b);
    }
    bad |= (unsigned)b;
  };
  double av[R][FX_W];
  if (BIG) {
    fx_dot_staged<R>(F, A, lda, Xs, C, row, ri, hh, mid, av, st);
    fixed(av);
  } else {
#pragma unroll
    for (int c = 0; c < FX_W; c++)
#pragma unroll
      for (int r = 0; r < R; r++)
        av[r][c] = (row[r] < F.n && C + c <= row[r]) ? A[(size_t)ri[r] + (size_t)(C + c) * lda] : 0.0;
    fixed(av);
    fx_dot<R>(F, Xs, C, ri, hh, mid);
  }
  float qs[R];
  int wr[R];
#pragma unroll
  for (int r = 0; r < R; r++) qs[r] = 0.f, wr[r] = 0;
  const bool ok =
      fx_columns<R, FIRST, BIG>(F, Xs, C, row, own, zs, rho_s, hh, mid, a, fs, qs, wk, wr, weak, bad);
  // a row whose squares add up to more than a_ii: A is not positive definite
#pragma unroll
  for (int r = 0; r < R; r++)
    if (own[r]) {
      const float v = q[row[r]] + qs[r];
      q[row[r]] = v;
      if (!(v < 288230376151711744.0f)) bad = 1;  // 2^58
      atomicAdd(wk + row[r], wr[r]);
    }
  return ok;
}

// One block of columns. Rows: lanes 0..7 of every warp hold C..C+7, the other
// lanes (and, R = 2, the second row of every lane) the rows below, warp by warp;
// what is left (BIG, whose X is in global memory) in turns of 64 rows a warp.
template <int NW, int R, bool BIG>
__device__ __forceinline__ bool fx_block(const FixLayout &F, const double *A, int lda, double *Xs,
                                         int C, const int *Es, float *q, int *wk, int *zs,
                                         double *rho_s, FixScratch *fs, FixStage *st,
                                         unsigned &weak, unsigned &bad)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int row[R];
  bool own[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    row[r] = r == 0 ? (lane < FX_W ? C + lane : C + w * (32 - FX_W) + lane)
                    : C + FX_W + NW * (32 - FX_W) + w * 32 + lane;
    own[r] = row[r] < F.n && (r > 0 || lane >= FX_W || w == 0);
  }
  // a warp without rows of its own sits the block out and hears the verdict on
  // the pivots at the barrier
  bool ok = true;
  if (w == 0 || C + w * (32 - FX_W) + FX_W < F.n)
    ok = fx_rows<R, true, BIG>(F, A, lda, Xs, C, row, own, Es, q, wk, zs, rho_s, fs, st, weak, bad);
  if (BIG && R == 2) {
    for (int g = C + FX_W + NW * (64 - FX_W); ok && g < F.n; g += NW * 64) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        row[r] = g + (w * R + r) * 32 + lane;
        own[r] = row[r] < F.n;
      }
      fx_rows<R, false, BIG>(F, A, lda, Xs, C, row, own, Es, q, wk, zs, rho_s, fs, st, weak, bad);
    }
  }
  if (NW == 1) __syncwarp();
  else ok = __syncthreads_and(ok);
  // the sums of this block's unknowns are complete and stay as they are
  const int i = C + (lane & (FX_W - 1));
  return ok && !__any_sync(0xffffffffu, i < F.n && fx_too_weak(wk[i], F.n, weak));
}

// Cholesky factor of the lower triangle of A into Xs (limbs), by a CTA of NW
// warps (n <= 8 + 56 NW, or BIG); rho_s, zs: the reciprocal roots of the pivots.
// Es, wk: n ints, q: n floats. False: the FP64 path has to take the matrix.
// RMAX = 1: n <= 8 + 24 NW.
template <int NW, bool BIG, int RMAX = 2>
__device__ __forceinline__ bool fx_potrf(const FixLayout &F, const double *A, int lda, double *Xs,
                                         int *Es, float *q, int *wk, int *zs, double *rho_s,
                                         FixScratch *fs, FixStage *st = nullptr)
{
  int b = 0;
  for (int i = threadIdx.x; i < F.n; i += 32 * NW) {
    Es[i] = fx_scale(A[(size_t)i + (size_t)i * lda], b);
    q[i] = 0.f;
    wk[i] = 0;
  }
  if (NW == 1) b = __any_sync(0xffffffffu, b);
  else b = __syncthreads_or(b);
  if (b) return false;
  if (NW == 1) __syncwarp();
  unsigned bad = 0, weak = 0;
  bool ok = true;
  int C = 0;
  if (RMAX > 1)
    for (; ok && F.n - C > FX_W + NW * (32 - FX_W); C += FX_W)
      ok = fx_block<NW, 2, BIG>(F, A, lda, Xs, C, Es, q, wk, zs, rho_s, fs, st, weak, bad);
  for (; ok && C < F.n; C += FX_W)
    ok = fx_block<NW, 1, BIG>(F, A, lda, Xs, C, Es, q, wk, zs, rho_s, fs, st, weak, bad);
  // (ok is the same in every warp; each finds every unknown's sum, hence bit 1 of weak)
  if (__any_sync(0xffffffffu, weak & 2u) && (weak & 1u)) bad = 1;
  if (NW == 1) return ok && !__any_sync(0xffffffffu, bad != 0);
  return !__syncthreads_or(!ok || bad != 0);
}

// The same by one warp in FP64, for n <= 32: the factor into Xs and A's lower
// triangle (up to the failing column), 1 / diagonal into rinv. Returns info.
__device__ __forceinline__ int fx_potrf_fp64(const FixLayout &F, double *A, int lda, double *Xs,
                                             double *rinv)
{
  const int i = threadIdx.x & 31;
  for (int c = 0; c < F.n; c++)
    if (i >= c && i < F.n) Xs[F.col(c) + i] = A[(size_t)i + (size_t)c * lda];
  __syncwarp();
  for (int c = 0; c < F.n; c++) {
    double *x = Xs + F.col(c);
    const double d = x[c];
    if (!is_pos_pivot(d)) return c + 1;
    double s, r;
    pivot_rs(d, s, r);
    __syncwarp();  // d is read
    const double l = i == c ? s : (i > c && i < F.n) ? x[i] * r : 0.0;
    if (i >= c && i < F.n) {
      x[i] = l;
      A[(size_t)i + (size_t)c * lda] = l;
    }
    if (i == c) rinv[c] = r;
    __syncwarp();
    for (int k = c + 1; k < F.n; k++)
      if (i >= k && i < F.n) Xs[F.col(k) + i] -= l * x[k];
    __syncwarp();
  }
  return 0;
}

// Limbs -> FP64, into A's lower triangle and (keep) in place; the reciprocals of
// the diagonal replace rho.
template <int NW>
__device__ __forceinline__ void fx_store(const FixLayout &F, double *Xs, const int *Es,
                                         const int *zs, double *rinv, double *A, int lda, bool keep)
{
  for (int i = threadIdx.x; i < F.n; i += 32 * NW)
    rinv[i] = sp_to_double(__double_as_longlong(rinv[i]), zs[i] - 61 - Es[i]);
  int ld = F.n2;
  double *P = Xs;
  for (int C = 0; C < F.n; C += FX_W, P += FX_W * ld, ld -= FX_W) {
    for (int i = C + threadIdx.x; i < F.n; i += 32 * NW) {
      const int e = Es[i] - 59;
      double *dst = A + (size_t)i + (size_t)C * lda, *src = P + (i - C);
      double v[FX_W];
      // (all loads before any store: the columns right of the diagonal, or of
      // the matrix, hold anything)
#pragma unroll
      for (int c = 0; c < FX_W; c++) v[c] = src[c * ld];
#pragma unroll
      for (int c = 0; c < FX_W; c++) v[c] = sp_to_double(fx_unpack(v[c]), e);
#pragma unroll
      for (int c = 0; c < FX_W; c++) {
        if (C + c <= i) {
          if (keep) src[c * ld] = v[c];
          dst[(size_t)c * lda] = v[c];
        }
      }
    }
  }
  fx_sync<NW>();
}

// A's lower triangle, a Cholesky factor, and the reciprocals of its diagonal.
template <int NW, typename T>
__device__ __forceinline__ void fx_load(const FixLayout &F, const T *A, int lda, T *Xs, T *rinv)
{
  int ld = F.n2;
  T *P = Xs;
  for (int C = 0; C < F.n; C += FX_W, P += FX_W * ld, ld -= FX_W) {
    for (int i = C + threadIdx.x; i < F.n; i += 32 * NW) {
      const T *src = A + (size_t)i + (size_t)C * lda;
#pragma unroll
      for (int c = 0; c < FX_W; c++)
        if (C + c <= i) {
          const T v = src[(size_t)c * lda];
          P[i - C + c * ld] = v;
          if (C + c == i) rinv[i] = T(1) / v;
        }
    }
  }
  fx_sync<NW>();
}

// ----------------------------------------------------------------------------
// X L L^T = B for up to G rows of B (right-hand sides) by one warp: lane = (row
// of a group of 32 / G, right-hand side); the vectors pass through registers in
// segments of FX_NR groups. One column of L at a time: the FP64 pipe issues one
// multiply and one FMA per remaining group of rows, so every lane of every FMA
// (but those of the diagonal group) is useful work. What a segment takes from
// the segments solved before it has no dependent chain.
constexpr int FX_NR = 8;

// PF: a column is loaded while the one before it is worked on (L in global memory;
// from shared memory the registers that takes cost more than the latency).
template <int G, bool PF, typename T>
__device__ __forceinline__ void fx_solve(const FixLayout &F, const T *Ps, const T *rinv, T *B,
                                         int ldb, int nrhs)
{
  constexpr int RR = 32 / G;         // rows per register
  constexpr int SEG = RR * FX_NR;    // rows of a segment
  const int lane = threadIdx.x & 31, sub = lane / G, rhs = lane % G;
  const int n = F.n;
  const bool on = rhs < nrhs;
  T *b = B + (on ? rhs : 0);
  T y[FX_NR];
  for (int s0 = 0; s0 < n; s0 += SEG) {
#pragma unroll
    for (int j = 0; j < FX_NR; j++) {
      const int i = s0 + j * RR + sub;
      y[j] = (on && i < n) ? b[(size_t)i * ldb] : T(0);
    }
    // (rows past n repeat the last one: what they add up to is not used)
    int ro[FX_NR];
#pragma unroll
    for (int j = 0; j < FX_NR; j++) ro[j] = min(s0 + j * RR + sub, n - 1);
#pragma unroll 4
    for (int k = 0; k < s0; k++) {
      const T *col = Ps + F.col(k);
      const T yc = b[(size_t)k * ldb];
      T l[FX_NR];
#pragma unroll
      for (int j = 0; j < FX_NR; j++) l[j] = col[ro[j]];
#pragma unroll
      for (int j = 0; j < FX_NR; j++)
        if (s0 + j * RR < n) y[j] -= l[j] * yc;
    }
#pragma unroll
    for (int jc = 0; jc < FX_NR; jc++) {
      const int c0 = s0 + jc * RR;
      const int cn = min(RR, n - c0);
      T l[FX_NR];  // column c0 + c below its group; (PF) loaded ahead
      auto load = [&](int k) {
        const T *col = Ps + F.col(k);
#pragma unroll
        for (int j = jc; j < FX_NR; j++) l[j] = col[ro[j]];
      };
      if (PF && cn > 0) load(c0);
      for (int c = 0; c < cn; c++) {
        const T yc = __shfl_sync(0xffffffffu, y[jc], c * G + rhs) * rinv[c0 + c];
        if constexpr (!PF) {
          const T *col = Ps + F.col(c0 + c) + (c0 + sub);
#pragma unroll
          for (int j = jc + 1; j < FX_NR; j++)
            if (s0 + j * RR < n)
              y[j] -= ((s0 + j * RR + sub < n) ? col[(j - jc) * RR] : T(0)) * yc;
          if (sub == c) y[jc] = yc;
          if (sub > c && c0 + sub < n) y[jc] -= col[0] * yc;
        } else {
          T lc[FX_NR];
#pragma unroll
          for (int j = jc; j < FX_NR; j++) lc[j] = l[j];
          if (c + 1 < cn) load(c0 + c + 1);
          if (sub == c) y[jc] = yc;
          if (sub > c) y[jc] -= lc[jc] * yc;
#pragma unroll
          for (int j = jc + 1; j < FX_NR; j++)
            if (s0 + j * RR < n) y[j] -= lc[j] * yc;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < FX_NR; j++) {
      const int i = s0 + j * RR + sub;
      if (on && i < n) b[(size_t)i * ldb] = y[j];
    }
    __syncwarp();
  }
  for (int s0 = (n - 1) / SEG * SEG; s0 >= 0; s0 -= SEG) {
    int off[FX_NR];  // column s0 + j RR + sub of L
#pragma unroll
    for (int j = 0; j < FX_NR; j++) {
      const int i = min(s0 + j * RR + sub, n - 1);
      off[j] = F.col(i);
      y[j] = (on && s0 + j * RR + sub < n) ? b[(size_t)i * ldb] : T(0);
    }
#pragma unroll 4
    for (int k = s0 + SEG; k < n; k++) {
      const T xc = b[(size_t)k * ldb];
      T l[FX_NR];
#pragma unroll
      for (int j = 0; j < FX_NR; j++) l[j] = Ps[off[j] + k];
#pragma unroll
      for (int j = 0; j < FX_NR; j++) y[j] -= l[j] * xc;
    }
#pragma unroll
    for (int jc = FX_NR - 1; jc >= 0; jc--) {
      const int c0 = s0 + jc * RR;
      // x_k, then row k of L times x_k off the rows before it
      T l[FX_NR];
      auto load = [&](int k) {
#pragma unroll
        for (int j = 0; j <= jc; j++) l[j] = Ps[off[j] + k];
      };
      const int cn = min(RR, n - c0);
      if (PF && cn > 0) load(c0 + cn - 1);
      for (int c = cn - 1; c >= 0; c--) {
        const T xc = __shfl_sync(0xffffffffu, y[jc], c * G + rhs) * rinv[c0 + c];
        if constexpr (!PF) {
#pragma unroll
          for (int j = 0; j < jc; j++) y[j] -= Ps[off[j] + c0 + c] * xc;
          if (sub == c) y[jc] = xc;
          if (sub < c) y[jc] -= Ps[off[jc] + c0 + c] * xc;
        } else {
          T lc[FX_NR];
#pragma unroll
          for (int j = 0; j <= jc; j++) lc[j] = l[j];
          if (c > 0) load(c0 + c - 1);
          if (sub == c) y[jc] = xc;
          if (sub < c) y[jc] -= lc[jc] * xc;
#pragma unroll
          for (int j = 0; j < jc; j++) y[j] -= lc[j] * xc;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < FX_NR; j++) {
      const int i = s0 + j * RR + sub;
      if (on && i < n) b[(size_t)i * ldb] = y[j];
    }
    __syncwarp();
  }
}

// X L L^T = B for the m rows of B: four right-hand sides to a warp, or one when
// that leaves warps idle (an FMA of four costs the FP64 pipe the same as four of
// one, but the chain of columns is walked once).
template <int NW, bool PF, typename T>
__device__ __forceinline__ void fx_solve_all(FixLayout F, const T *Ps, const T *rinv, T *B,
                                             int ldb, int m)
{
  const int w = threadIdx.x >> 5;
  if (m > 2 && m > NW) {
    for (int r = 4 * w; r < m; r += 4 * NW) fx_solve<4, PF>(F, Ps, rinv, B + r, ldb, m - r);
  } else {
    for (int r = w; r < m; r += NW) fx_solve<1, PF>(F, Ps, rinv, B + r, ldb, 1);
  }
}

}  // namespace kgb
