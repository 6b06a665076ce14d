// Block fixed-point arithmetic for FP64 products on the tensor cores.
//
// GB300 issues about 2 FP64 FMAs per clock and SM; its half-precision
// `mma.sync` does 1,000 multiply-adds (measured), and adds integers exactly
// while the sums stay below 2^24 in its FP32 accumulators.  A product sum
// over columns is therefore formed from integer digits (the splitting of
// Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012): with E the
// largest biased exponent of a row's (or of a right-hand side's) entries, an
// entry v becomes
//   t = trunc(v 2^(1077 - E)),  |t| <= 2^55,  t = sum_k d_k 256^(6 - k),
// seven digits |d_k| <= 129 held as halves, and
//   t t' = sum_s 256^(12 - s) sum_{i + j = s} d_i d'_j,  s = 0 .. 7
// (34 of the 49 digit products; the others are below 2^-66 of the largest
// t t').  The sum of each s is exact, and the eight are put together in
// 64-bit integers, in units of 2^56: a right-hand side costs 34 of the 1,000
// multiply-adds a real product, 0.14 clocks an SM for a complex one against
// 2.2 for its four FP64 FMAs.  An entry is off by less than 2^-55 of the
// largest one, a quarter of an FP64 rounding (2^-53), and the sum rounds once
// per flush instead of once per term, so the error against exact arithmetic
// is below that of the FP64 sum.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace bfg {

constexpr int kFixDigits = 7, kFixSums = 8;
// k-steps (8 complex columns) between flushes: a step adds seven digit
// products of 16 * 129^2 to the sum s = 6, which stays below 2^24
constexpr int kFixMaxSteps = 8;
static_assert(7 * kFixMaxSteps * 16 * 129 * 129 < 1 << 24, "exact FP32 sums");
constexpr int kFixSpecial = 2047;   // exponent code: not for fixed point
// V 2^56 2^(Ea - 1077) 2^(Ex - 1077) as a power of two: exponent field of the
// scale Ea + Ex - 1075, a normal number (and 2^-24 of it) in this range
constexpr int kFixMinSum = 1100, kFixMaxSum = 3121;
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
// 2^56 2^(Ea - 1077) 2^(Ex - 1077) for a covered pair of scales
__device__ __forceinline__ double fixScale(int sumE) {
  return __hiloint2double((sumE - 1075) << 20, 0);
}

// t + 0x0200808080808080: its bytes are the digits + 128, its top 16 bits the
// top digit + 512.  v at scale E: kFixMinCode <= E < kFixSpecial,
// |v| < 2^(E - 1022).
__device__ __forceinline__ uint64_t fixInt(double v, int E) {
  uint32_t const h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
  uint32_t const mh = (h & 0xFFFFFu) | 0x100000u;
  uint32_t const sh = (uint32_t)E - ((h >> 20) & 0x7FFu);
  int32_t const s = (int32_t)h >> 31;
  uint64_t y = ((uint64_t)__funnelshift_l(l, mh, 2) << 32) | (l << 2);
  asm("shr.u64 %0, %0, %1;" : "+l"(y) : "r"(sh));   // 0 from 64 on
  // the bias, and the 1 of a two's complement negation
  uint64_t const c = ((uint64_t)0x02008080u << 32) | (uint32_t)(0x80808080 - s);
  return (y ^ (uint64_t)(int64_t)s) + c;
}
// the digits of a complex entry, most significant first, as half pairs (re, im)
__device__ __forceinline__ void fixSplit(double2 v, int E, uint32_t (&d)[kFixDigits]) {
  uint64_t const r = fixInt(v.x, E), i = fixInt(v.y, E);
  uint32_t const rl = (uint32_t)r, rh = (uint32_t)(r >> 32);
  uint32_t const il = (uint32_t)i, ih = (uint32_t)(i >> 32);
  // bytes interleaved (re, im, re, im), then each pair under the exponent of
  // 1024 (halves 1024 + byte), less 1024 + 128 (512 for the top digit)
  uint32_t const p0 = __byte_perm(rl, il, 0x5140), p1 = __byte_perm(rl, il, 0x7362);
  uint32_t const p2 = __byte_perm(rh, ih, 0x5140);
  uint32_t const k = 0x64646464u;
  d[6] = __byte_perm(p0, k, 0x4140);
  d[5] = __byte_perm(p0, k, 0x4342);
  d[4] = __byte_perm(p1, k, 0x4140);
  d[3] = __byte_perm(p1, k, 0x4342);
  d[2] = __byte_perm(p2, k, 0x4140);
  d[1] = __byte_perm(p2, k, 0x4342);
  d[0] = __byte_perm(rh, ih, 0x7632) | 0x64006400u;
#pragma unroll
  for (int q = 0; q < kFixDigits; ++q) {
    __half2 const off = __half2half2(__ushort_as_half(q == 0 ? 0xE600 : 0xE480));   // -1536, -1152
    __half2 const x = __hadd2(*reinterpret_cast<__half2 const *>(&d[q]), off);
    d[q] = *reinterpret_cast<uint32_t const *>(&x);
  }
}

// the exact sum put together from the digit sums' element r, in units of 2^56
// (rounded), which are cleared
__device__ __forceinline__ int64_t fixTake(float (&sum)[kFixSums][4], int r) {
  int v[kFixSums];
#pragma unroll
  for (int s = 0; s < kFixSums; ++s) {
    v[s] = __float2int_rn(sum[s][r]);
    sum[s][r] = 0.f;
  }
  return ((int64_t)v[0] << 40) + ((int64_t)v[1] << 32) + ((int64_t)v[2] << 24) +
         ((int64_t)v[3] << 16) + ((int64_t)v[4] << 8) +
         (v[5] + ((v[6] + (v[7] >> 8) + 128) >> 8));
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
