// Block fixed-point arithmetic for FP64 products on the tensor cores.
//
// GB300 issues about 2 FP64 FMAs per clock and SM; its half-precision
// `mma.sync` does 1,000 multiply-adds (measured), and adds integers exactly
// while the sums stay below 2^24 in its FP32 accumulators.  A product sum
// over columns is therefore formed from integer digits (the splitting of
// Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012): with E the
// largest biased exponent of a row's (or of a right-hand side's) entries, an
// entry v becomes
//   t = trunc(v 2^(1084 - E)),  |t| < 2^62,  t = sum_k d_k 256^(7 - k),
// eight digits |d_k| <= 128 (|d_0| <= 65) held as halves, and
//   t t' = sum_s 256^(14 - s) sum_{i + j = s} d_i d'_j,  s = 0 .. 7
// (36 of the 64 digit products).  The sum of each s is exact, and the eight
// are put together in an integer, which is rounded once: a right-hand side
// costs 36 of the 1,000 multiply-adds a real product, 0.15 clocks an SM for a
// complex one against 2.2 for its four FP64 FMAs.  (The factorization's
// products, whose operands are unitary or scaled by column, take seven digits:
// bfg_sketch.cu.)
//
// Error.  With m the product of the largest part of the row and the largest
// part of the right-hand side (the largest t is at least 2^61, so m at least
// 2^122): the digit products left out, s = 8 above all, are below 7 2^14
// 2^48 2^1.01 < 2^65 = 2^-57 m, and truncation is below 2^-61 of the largest
// part on either side: a real product is off by less than 2^-56.8 m, and
// typically (digits of either sign) by 2^-60 m.  That is an error against m,
// not against the product itself: an FP64 sum's error is about 2^-53 sum |a x|,
// which for operands graded in opposite directions may be far below m.  So the
// applies look at the gradings: see fixEven.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace bfg {

constexpr int kFixDigits = 8, kFixSums = 8;
// k-steps (8 complex columns) between flushes: a step adds eight digit
// products, two of them with a first digit, of 16 columns each to the sum
// s = 7, which stays below 2^24
constexpr int kFixMaxSteps = 8;
static_assert((6 * 128 * 128 + 2 * 65 * 128) * 16 * kFixMaxSteps < 1 << 24, "exact FP32 sums");
constexpr int kFixSpecial = 2047;   // exponent code: not for fixed point
// the scales of the sums' units, 2^56 2^(Ea - 1084) 2^(Ex - 1084) (exponent
// field Ea + Ex - 1089) and 2^60 2^(Ea - 1081) 2^(Ex - 1081) (Ea + Ex - 1079),
// and 2^32 times these are normal numbers in this range
constexpr int kFixMinSum = 1100, kFixMaxSum = 3090;
// smallest usable code: below it an entry that is zero (whose implicit bit
// fixInt sets all the same) would not be shifted out
constexpr int kFixMinCode = 64;

// Biased exponent of v; 1 for a subnormal (so that zero alone has code 0).
__device__ __forceinline__ int fixCode(double v) {
  uint32_t const h = (uint32_t)__double2hiint(v) & 0x7FFFFFFFu;
  int const e = (int)(h >> 20);
  return (e == 0 && (h | (uint32_t)__double2loint(v)) != 0u) ? 1 : e;
}
__device__ __forceinline__ int fixCode(double2 v) { return max(fixCode(v.x), fixCode(v.y)); }
// code of v >= least, for least from 1 to 2046 (a subnormal's is below all)
__device__ __forceinline__ bool fixLarge(double2 v, int least) {
  return max(__double2hiint(v.x) & 0x7FFFFFFF, __double2hiint(v.y) & 0x7FFFFFFF) >= least << 20;
}
// the scale used for a largest code: any for all-zero data, the special one
// for data whose range fixed point does not cover (subnormal, NaN, infinite)
__device__ __forceinline__ int fixScaleOf(int code) {
  return code == 0 ? 1023 : code < kFixMinCode ? kFixSpecial : code;
}
// the smallest and largest scale pass for a set of row scales and a
// right-hand side's scale
__device__ __forceinline__ bool fixCovers(int eaMin, int eaMax, int ex) {
  return eaMax < kFixSpecial && ex < kFixSpecial && eaMin + ex >= kFixMinSum &&
         eaMax + ex <= kFixMaxSum;
}
// the power of two with this exponent field
__device__ __forceinline__ double fixPow(int field) { return __hiloint2double(field << 20, 0); }

// Gradings.  A column counts as small in a row of n columns where its entry's
// code is more than fixRowGap(n) below the row's largest, and as small in a
// right-hand side where it is more than kFixInputGap below.  `graded`: the most
// small columns that a row of the block piece has.  If an eighth of the columns
// in hand are small in neither, every row's sum of |a||x| over these n of N
// columns is at least n / 8 2^-(fixRowGap(N) + 1) 2^-(kFixInputGap + 1) m
// >= (n / N) 2^-11 m, and the fixed-point sum is within N 2^-43 of it whatever
// the entries (typically, as in opposite geometric gradings of up to 2^10, at
// or below FP64's own 2^-53).  Otherwise the columns are summed in plain FP64.
// The gaps: wide enough for the factors' natural gradings (equivalent points
// near and far from a source: up to 2^9 within a row), so that of the products
// of circles, ellipses and stars none and of scattering operators 0.2 % take
// the plain form; an input gap of 3 would send 1 % there and a quarter instead
// of an eighth with it 3 %, at three to four times the cost.
constexpr int kFixInputGap = 4;
__device__ __forceinline__ int fixRowGap(int n) { return 33 - __clz(n - 1); }   // ceil(log2 n) + 1
__device__ __forceinline__ bool fixEven(int n, int big, int graded) {
  return 8 * (big - graded) >= n;
}

// t and a bias that makes its bytes the digits + 128.  Eight digits: t + 2^7
// (1 + 256 + ... + 256^7).  Seven (t = trunc(v 2^(1077 - E)), |t| <= 2^55):
// six such bytes, and the top 16 bits the first digit + 512.  v at scale E:
// kFixMinCode <= E < kFixSpecial, |v| < 2^(E - 1022).
template <int D>
__device__ __forceinline__ uint64_t fixInt(double v, int E) {
  static_assert(D == 7 || D == 8, "digits");
  constexpr int L = D == 8 ? 9 : 2;
  uint32_t const h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
  uint32_t const mh = (h & 0xFFFFFu) | 0x100000u;
  uint32_t const sh = (uint32_t)E - ((h >> 20) & 0x7FFu);
  int32_t const s = (int32_t)h >> 31;
  uint64_t y = ((uint64_t)__funnelshift_l(l, mh, L) << 32) | (l << L);
  asm("shr.u64 %0, %0, %1;" : "+l"(y) : "r"(sh));   // 0 from 64 on
  // the bias, and the 1 of a two's complement negation
  uint64_t const c = ((uint64_t)(D == 8 ? 0x80808080u : 0x02008080u) << 32) |
                     (uint32_t)(0x80808080 - s);
  return (y ^ (uint64_t)(int64_t)s) + c;
}
// the digits of a complex entry, most significant first, as half pairs (re, im)
template <int D>
__device__ __forceinline__ void fixSplit(double2 v, int E, uint32_t (&d)[D]) {
  uint64_t const r = fixInt<D>(v.x, E), i = fixInt<D>(v.y, E);
  uint32_t const rl = (uint32_t)r, rh = (uint32_t)(r >> 32);
  uint32_t const il = (uint32_t)i, ih = (uint32_t)(i >> 32);
  // bytes interleaved (re, im, re, im), then each pair under the exponent of
  // 1024 (halves 1024 + byte), less 1024 + 128 (512 for seven digits' first)
  uint32_t const p[4] = {__byte_perm(rl, il, 0x5140), __byte_perm(rl, il, 0x7362),
                         __byte_perm(rh, ih, 0x5140), __byte_perm(rh, ih, 0x7362)};
#pragma unroll
  for (int q = 0; q < D; ++q) {   // q: from the last digit on
    bool const wide = D == 7 && q == 6;
    uint32_t const b = wide ? __byte_perm(rh, ih, 0x7632) | 0x64006400u
                            : __byte_perm(p[q / 2], 0x64646464u, q % 2 ? 0x4342 : 0x4140);
    __half2 const off = __half2half2(__ushort_as_half(wide ? 0xE600 : 0xE480));   // -1536, -1152
    __half2 const x = __hadd2(*reinterpret_cast<__half2 const *>(&b), off);
    d[D - 1 - q] = *reinterpret_cast<uint32_t const *>(&x);
  }
}

// acc + the sum put together from the digit sums' element r, which are
// cleared; sumE: the scales' sum Ea + Ex
__device__ __forceinline__ double fixAdd(double acc, float (&sum)[kFixSums][4], int r, int sumE) {
  int v[kFixSums];
#pragma unroll
  for (int s = 0; s < kFixSums; ++s) {
    v[s] = __float2int_rn(sum[s][r]);
    sum[s][r] = 0.f;
  }
  int64_t const hi = ((int64_t)v[0] << 24) + ((int64_t)v[1] << 16) + ((int64_t)v[2] << 8) + v[3];
  int64_t const lo = ((int64_t)v[4] << 24) + ((int64_t)v[5] << 16) + ((int64_t)v[6] << 8) + v[7];
  // hi 2^32 + lo in 63 bits: one conversion and one FMA on the FP64 pipe, not
  // two (an apply of 16 right-hand sides at 65,536 points 5,141 -> 4,808 us,
  // with the FP64 sums still in registers)
  int const top = (int)(hi >> 12), sh = max(14 - __clz(top ^ (top >> 31)), 0);
  int64_t const t = (int64_t)((uint64_t)hi << (32 - sh)) + (lo >> sh);
  return fma((double)t, fixPow(sumE - 1089 + sh), acc);
}

// D += A B, 16 x 8 x 16, halves in, FP32 sums (of integers: exact)
__device__ __forceinline__ void fixMma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                       uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

}  // namespace bfg
