// fp64_split.cuh -- FP64 matrix products on the tensor cores by exact slicing
// (the Ozaki scheme: Ozaki, Ogita, Oishi, Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59, 2012; on half-precision tensor
// cores: Mukunoki, Ozaki, Ogita, Imamura, ISC 2020).
//
// Why: the part has 2 FP64 FMA lanes per clock and SM but 4096 FP16 tensor
// FMAs, so a product that is cut into 28 FP16 ones still costs a fraction of
// the FP64 pipe's time; the kernels here are bound by the integer work that
// cuts the operands and puts the results together.
//
// Each row of op(A) (and each column of op(B)) gets a power-of-two scale
// 2^E > |x| and every element becomes a 56-bit fixed-point number,
// x 2^(55 - E) cut towards zero = sum_i s_i 2^(8 (7 - i)), i = 1..7, with signed 8-bit
// digits s_i in [-128, 127] held exactly in FP16. The products s_i s_j' with
// i + j <= 8 are summed on the tensor cores; all with the same i + j share an
// FP32 accumulator, which stays exact: with at most 4 products per
// accumulator and a k chunk of 64 it is an integer of at most 2^22. The seven
// sums are put together in 64-bit integers and rounded once to FP64.
//
// Error: the cut loses up to 2^-55 2^E per element, always towards zero (2^-56 in
// the mean), and the dropped products (i + j = 9) are at most 6 2^-56 2^(Ei + Ej) per
// k (about 2^-56 in the mean), so against sum_k |a_ik| |b_kj| the result is as
// accurate as a chain of FP64 FMAs over 16 k or more whenever that sum is not far
// below 2^(Ei + Ej); shorter sums use FP64 FMAs. The former is checked for
// every entry: one more product, of |s_1| with |s_1'|, estimates the sum, and
// an entry whose estimate is below 2^-2 2^(Ei + Ej) is computed again with
// FP64 FMAs (graded or sparse data; at most a few entries of a dense tile).
// Tiles holding infinities, NaNs or exponents outside [-462, 458] use FP64
// FMAs altogether.
//
// Shared-memory operand layout (no swizzle, K-major; see tc_util.cuh for the
// descriptors): a "tall" matrix whose rows are (digit, row), 16 bytes (8 k)
// per row, 8-row groups contiguous (SBO = 128) and k in groups of 8 (LBO).
// M = 128 covers two digits of a 64-row tile, so one MMA computes s_i s_j and
// s_(i+1) s_j for all j at once; N runs over the digits of 32 columns.
#pragma once

#include <cuda_fp16.h>

#include "device_util.cuh"
#include "tc_util.cuh"

namespace kgb {

constexpr int SP_TM = 64;    // rows of a tile
constexpr int SP_TN = 32;    // columns of a tile
constexpr int SP_KC = 64;    // k chunk (one scale per row and chunk)
constexpr int SP_KMIN = 16;  // shortest k chunk that is cut (see the error above)
constexpr int SP_NT = 256;   // threads per CTA
constexpr int SP_APL = 9;    // A planes: digits 1..7, |digit 1| twice
constexpr int SP_BPL = 8;    // B planes: digits 1..7, |digit 1|
constexpr uint32_t SP_SBO = 128;
// The k groups are 16 bytes out of step with the banks, so that the 8 lanes
// which store the 8 k groups of one row hit different banks.
constexpr uint32_t SP_LBO_A = SP_APL * SP_TM * 16 + 16;
constexpr uint32_t SP_LBO_B = SP_BPL * SP_TN * 16 + 16;
constexpr int SP_SMEM_A = (SP_KC / 8) * SP_LBO_A;   // 73856
constexpr int SP_SMEM_B = (SP_KC / 8) * SP_LBO_B;   // 32896
constexpr int SP_TMEM = 256;  // TMEM columns: 7 sums and the estimate, 32 columns each
constexpr int SP_LIST = 512;  // entries of a tile redone one by one; above, the whole tile

// |x| bits of the largest element of a row -> exponent field er with
// |x| <= (1 - 2^-7) 2^(er - 1022): the first digit, carries of the lower ones
// included (2^47 (1 + 1/255) of 2^55), then never reaches 128.
__device__ __forceinline__ int sp_scale(uint32_t maxhi) {
  return maxhi ? (int)((maxhi + 0x4000u) >> 20) : 1022;
}
// rows whose products need FP64 FMAs: infinities, NaNs, exponents whose
// products could leave the normal range
__device__ __forceinline__ bool sp_special(uint32_t maxhi) {
  return maxhi != 0u && (maxhi >= (1480u << 20) || maxhi < (560u << 20));
}

// 8 k-neighbours of one row, zeros outside; returns the bits of the largest
// |x| (a denormal below 2^-1042 counts as the smallest non-zero value).
__device__ __forceinline__ uint32_t sp_maxbits(const double (&x)[8]) {
  uint32_t mx = 0, lo = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    mx = max(mx, (uint32_t)__double2hiint(x[i]) & 0x7fffffffu);
    lo |= (uint32_t)__double2loint(x[i]);
  }
  return mx ? mx : (lo ? 1u : 0u);
}

// Fixed-point form of x at scale er (cut towards zero), each byte biased by
// 128: bytes 6..0 are the digits 1..7 plus 128.
__device__ __forceinline__ void sp_fixed(double x, int er, uint32_t &ulo, uint32_t &uhi) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int sh = min(er - (int)((hi >> 20) & 0x7ffu), 63);
  const unsigned long long m =
      ((((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << 2) >> sh;
  const uint32_t s = (uint32_t)((int)hi >> 31);
  const unsigned long long v =
      ((unsigned long long)((uint32_t)(m >> 32) ^ s) << 32) | ((uint32_t)m ^ s);
  const unsigned long long u = v + (0x0080808000000000ull | (0x80808080u - s));
  ulo = (uint32_t)u;
  uhi = (uint32_t)(u >> 32);
}

// Bytes b, b + 1 (b = 0 or 2) of two neighbours along k as two FP16 pairs.
__device__ __forceinline__ uint32_t sp_half2(uint32_t inter, uint32_t sel) {
  const uint32_t t = __byte_perm(inter, 0x64646464u, sel);  // 1024 + byte, twice
  const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&t),
                            __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480)));
  return *reinterpret_cast<const uint32_t *>(&h);
}
// Digit planes of byte 0..3 of the words (w0, w1) of two neighbours along k.
__device__ __forceinline__ void sp_planes4(uint32_t w0, uint32_t w1, uint32_t (&o)[4]) {
  const uint32_t p0 = __byte_perm(w0, w1, 0x5140);  // w0.0 w1.0 w0.1 w1.1
  const uint32_t p1 = __byte_perm(w0, w1, 0x7362);  // w0.2 w1.2 w0.3 w1.3
  o[0] = sp_half2(p0, 0x4140);
  o[1] = sp_half2(p0, 0x4342);
  o[2] = sp_half2(p1, 0x4140);
  o[3] = sp_half2(p1, 0x4342);
}

// Cut 8 k-neighbours of one row and store digits 1..7 at dst + plane_bytes *
// (digit - 1); the planes of |digit 1| follow NABS times.
template <int NABS>
__device__ __forceinline__ void sp_cut8(const double (&x)[8], int er, unsigned char *dst,
                                        uint32_t plane_bytes) {
  uint32_t pl[7][4];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    uint32_t l0, h0, l1, h1, o[4];
    sp_fixed(x[i], er, l0, h0);
    sp_fixed(x[i + 1], er, l1, h1);
    sp_planes4(l0, l1, o);
#pragma unroll
    for (int b = 0; b < 4; b++) pl[6 - b][i >> 1] = o[b];
    sp_planes4(h0, h1, o);
#pragma unroll
    for (int b = 0; b < 3; b++) pl[2 - b][i >> 1] = o[b];
  }
#pragma unroll
  for (int d = 0; d < 7; d++)
    *reinterpret_cast<uint4 *>(dst + d * plane_bytes) = make_uint4(pl[d][0], pl[d][1], pl[d][2], pl[d][3]);
  if (NABS > 0) {
    const uint4 q = make_uint4(pl[0][0] & 0x7fff7fffu, pl[0][1] & 0x7fff7fffu,
                               pl[0][2] & 0x7fff7fffu, pl[0][3] & 0x7fff7fffu);
#pragma unroll
    for (int k = 0; k < NABS; k++) *reinterpret_cast<uint4 *>(dst + (7 + k) * plane_bytes) = q;
  }
}

// Instruction descriptor of kind::f16 with FP16 operands and FP32 sums.
__host__ __device__ __forceinline__ uint32_t idesc_f16_f32(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// All MMAs of one 64 x 32 tile and k extent of 16 ksteps; issued by one
// thread. TMEM columns 32 c .. 32 c + 31, c = 0..6: lanes 0..63 hold the sum
// of the products with i + j = c + 2, lanes 64..127 those with i + j = c + 3
// (c <= 5); c = 7: the estimate, in both halves.
__device__ __forceinline__ void sp_issue(uint32_t tmem, uint32_t sA, uint32_t sB, int ksteps) {
  for (int ks = 0; ks < ksteps; ks++) {
    const uint32_t a = sA + (uint32_t)ks * 2 * SP_LBO_A, b = sB + (uint32_t)ks * 2 * SP_LBO_B;
    const uint64_t bd = smem_desc(b, SP_LBO_B, SP_SBO);
#pragma unroll
    for (int p = 0; p < 4; p++) {  // digits (2p + 1, 2p + 2) of A, digits 1..7 - 2p of B
      const uint64_t ad = smem_desc(a + (uint32_t)p * 2 * SP_TM * 16, SP_LBO_A, SP_SBO);
      tc_mma_bf16(tmem + 64 * p, ad, bd, idesc_f16_f32(128, SP_TN * (7 - 2 * p)),
                  (ks | p) ? 1u : 0u);
    }
    tc_mma_bf16(tmem + 224, smem_desc(a + 7 * SP_TM * 16, SP_LBO_A, SP_SBO),
                smem_desc(b + 7 * SP_TN * 16, SP_LBO_B, SP_SBO), idesc_f16_f32(128, SP_TN),
                ks ? 1u : 0u);
  }
}

// 4 consecutive TMEM columns of this thread's lane, not waited for.
__device__ __forceinline__ void tmem_ld4_issue(uint32_t taddr, float (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Pins values loaded by tmem_ld4_issue after the wait.
__device__ __forceinline__ void tmem_pin4(float (&v)[4]) {
  asm volatile("" : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]));
}

// An integer-valued FP32 number of magnitude at most 2^22, plus SP_MAGIC.
constexpr int SP_MAGIC = 0x4b400000;  // bits of 1.5 2^23
__device__ __forceinline__ int sp_bits(float v) { return __float_as_int(v + 12582912.0f); }

// This lane's part of 4 columns (at = TMEM address of the first), as integers
// in units of 2^(Ei + Ej - 56).
__device__ __forceinline__ void sp_partial4(uint32_t at, bool lower, long long (&t)[4]) {
  // block of the sum i + j = d: d - 2 in the upper lanes, d - 3 in the lower
  float v[7][4];
  if (!lower) {
#pragma unroll
    for (int c = 0; c < 7; c++) tmem_ld4_issue(at + 32 * c, v[c]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++) v[0][q] = 0.0f;
#pragma unroll
    for (int c = 0; c < 6; c++) tmem_ld4_issue(at + 32 * c, v[c + 1]);
  }
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < 7; c++) tmem_pin4(v[c]);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    // pairs of neighbouring sums in 32 bits (wrap-around drops the magic)
    const unsigned k257 = 257u * (unsigned)SP_MAGIC;
    const int x1 = (int)((unsigned)sp_bits(v[0][q]) * 256u + ((unsigned)sp_bits(v[1][q]) - k257));
    const int x2 = (int)((unsigned)sp_bits(v[2][q]) * 256u + ((unsigned)sp_bits(v[3][q]) - k257));
    const int x3 = (int)((unsigned)sp_bits(v[4][q]) * 256u + ((unsigned)sp_bits(v[5][q]) - k257));
    const int y = (sp_bits(v[6][q]) - (SP_MAGIC - 32)) >> 6;
    const long long l = (long long)x2 * (1 << 18) + ((long long)x3 * 4 + y);
    t[q] = l + ((long long)((unsigned long long)((unsigned)x1 << 2) << 32));
  }
}

// The integer t 2^(e2) as FP64, rounded to nearest (ties away from zero); the
// result must be in the normal range (or t zero). Integer instructions only.
__device__ __forceinline__ double sp_to_double(long long t, int e2) {
  const uint32_t sgn = (uint32_t)(t >> 63);
  const unsigned long long a = (unsigned long long)(t < 0 ? -t : t);  // < 2^63
  const int lz = __clzll((long long)a) - 1;
  const unsigned long long m = ((a << (lz & 63)) + 0x200ull) >> 10;  // 2^52 <= m <= 2^53
  // value = m 2^(e2 + 10 - lz); adding m to the exponent field below it also
  // carries a rounding overflow into the exponent
  const uint32_t ef = (uint32_t)(e2 + 10 - lz + 52 + 1023 - 1);
  const uint32_t hi = (uint32_t)(m >> 32) + (ef << 20);
  const double r = __hiloint2double((int)(hi | (sgn & 0x80000000u)), (int)(uint32_t)m);
  return a ? r : 0.0;
}

}  // namespace kgb
