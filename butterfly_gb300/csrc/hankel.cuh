// Hankel functions of the first kind of orders 0 and 1 for real x > 0:
//   H0(x) = J0(x) + i Y0(x),   H1(x) = J1(x) + i Y1(x).
//
// The reference evaluates these with glibc's j0/y0/j1/y1 (bessel.c:284-308).
// This evaluator is written from published methods only; no library's
// internal constants are used.  Three regimes:
//
//   x < kSeriesMax      ascending power series (Abramowitz & Stegun 9.1.10,
//                       9.1.11, 9.1.13), with psi(k+1) = -gamma + H_k.
//   x < kAsymptoticMin  Miller's backward recurrence J_{n-1} = (2n/x) J_n -
//                       J_{n+1} from a start index far above x, normalised by
//                       J0 + 2 sum J_2k = 1 (A&S 9.1.46); Y0 from the Neumann
//                       series Y0 = (2/pi)[(ln(x/2)+gamma) J0 - 2 sum (-1)^k
//                       J_2k / k] (A&S 9.1.88) and Y1 = -Y0' from the
//                       derivative of that series.
//   otherwise           Hankel's asymptotic expansion (A&S 9.2.5-9.2.10):
//                       H_nu(x) ~ sqrt(2/(pi x)) (P + i Q) exp(i chi),
//                       chi = x - (nu/2 + 1/4) pi, P and Q polynomials in
//                       1/x^2 with the coefficients
//                       a_k = a_{k-1} (4 nu^2 - (2k-1)^2) / (8 k), as many as
//                       lie above 1e-17 at x.  exp(i chi) is formed
//                       from sincos(x) and the exact rotation by pi/4 or
//                       3 pi/4, so no rounding of x - chi enters.
//
// GB300's FP64 pipe (2 lanes a clock and SM) bounds every kernel that
// evaluates these, so the coefficients of both the expansion and the
// recurrence are compile-time constants and nothing is divided: about 60
// FP64 instructions for the expansion at x >= 100 and 200 for the recurrence,
// against 350 and 1,300 when each term formed its own factor by division.
//
// The same source compiles for the host (tests) and the device (kernels).
#pragma once

#include <math.h>

#if defined(__CUDACC__)
#define BFG_HD __host__ __device__ __forceinline__
#else
#define BFG_HD inline
#endif

namespace bfg {

constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr double kTwoOverPi = 0.636619772367581343075535053490057448;
constexpr double kEulerGamma = 0.577215664901532860606512090082402431;
constexpr double kInvSqrtPi = 0.564189583547756286948079451560772586;
constexpr double kSeriesMax = 0.25;
constexpr double kAsymptoticMin = 20.0;

struct Bessel01 {
  double j0, y0, j1, y1;
};

BFG_HD void bfgSincos(double x, double *s, double *c) {
#if defined(__CUDA_ARCH__)
  sincos(x, s, c);
#else
  *s = sin(x);
  *c = cos(x);
#endif
}

// x < kSeriesMax: ascending series.  q = x^2/4 <= 1/64, so eight terms
// reach below 1e-20 relative.
BFG_HD Bessel01 besselSeries(double x) {
  double const h = 0.5 * x;
  double const q = h * h;
  double lnh = log(h);
  // J0 = sum (-q)^k/(k!)^2 ; J1 = h sum (-q)^k / (k!(k+1)!)
  // Y0 tail: sum_{k>=1} (-1)^{k+1} H_k q^k/(k!)^2
  // Y1 tail: sum_{k>=0} (psi(k+1)+psi(k+2)) (-q)^k / (k!(k+1)!)
  double t0 = 1.0;            // (-q)^k/(k!)^2
  double t1 = 1.0;            // (-q)^k/(k!(k+1)!)
  double j0 = 1.0, j1s = 1.0;
  double harm = 0.0;          // H_k
  double y0tail = 0.0;
  double psi1 = -kEulerGamma;            // psi(k+1)
  double psi2 = -kEulerGamma + 1.0;      // psi(k+2)
  double y1tail = psi1 + psi2;
  for (int k = 1; k <= 8; ++k) {
    double const dk = (double)k;
    t0 *= -q / (dk * dk);
    t1 *= -q / (dk * (dk + 1.0));
    harm += 1.0 / dk;
    psi1 += 1.0 / dk;
    psi2 += 1.0 / (dk + 1.0);
    j0 += t0;
    j1s += t1;
    y0tail -= harm * t0;   // (-1)^{k+1} H_k q^k/(k!)^2 = -H_k t0
    y1tail += (psi1 + psi2) * t1;
  }
  Bessel01 b;
  b.j0 = j0;
  b.j1 = h * j1s;
  b.y0 = kTwoOverPi * ((lnh + kEulerGamma) * j0 + y0tail);
  b.y1 = -kTwoOverPi / x + kTwoOverPi * lnh * b.j1 - h * y1tail / kPi;
  return b;
}

// kSeriesMax <= x < kAsymptoticMin: Miller's algorithm + Neumann series.
// Step N forms J_{N-1} from J_N (jn) and J_{N+1} (jn1), then its part of
//   norm = 2 sum_{even m>=2} J_m
//   s0   = sum_{even m>=2} (-1)^{m/2} (4/m) J_m
//   s1   = sum_{odd  m>=3} (-1)^{(m+1)/2} 4m/(m^2-1) J_m
struct MillerState {
  double jn1, jn, norm, s0, s1, j1;
};
template <int M>
BFG_HD void millerAdd(MillerState &s) {
  if constexpr (M >= 2 && M % 2 == 0) {
    constexpr double c = ((M / 2) % 2 ? -4.0 : 4.0) / M;
    s.norm += s.jn;
    s.s0 = fma(c, s.jn, s.s0);
  } else if constexpr (M >= 3) {
    constexpr double c = (((M + 1) / 2) % 2 ? -4.0 : 4.0) * M / ((double)M * M - 1.0);
    s.s1 = fma(c, s.jn, s.s1);
  }
}
template <int N>
BFG_HD void millerStep(MillerState &s, double twoOverX) {
  double const jm1 = fma((double)N * twoOverX, s.jn, -s.jn1);
  s.jn1 = s.jn;
  s.jn = jm1;
  millerAdd<N - 1>(s);
  if constexpr (N == 2) s.j1 = s.jn;
  if constexpr (N > 1) millerStep<N - 1>(s, twoOverX);
}

template <int kStart>   // even, above x + 34
BFG_HD Bessel01 besselMiller(double x) {
  double const twoOverX = 2.0 / x;
  MillerState s{0.0, 1e-30, 0.0, 0.0, 0.0, 0.0};   // J_kStart: an arbitrary small start
  millerAdd<kStart>(s);
  millerStep<kStart>(s, twoOverX);
  double const scale = 1.0 / fma(2.0, s.norm, s.jn);
  Bessel01 b;
  b.j0 = s.jn * scale;
  b.j1 = s.j1 * scale;
  double const l = log(0.5 * x) + kEulerGamma;
  b.y0 = kTwoOverPi * (l * b.j0 - s.s0 * scale);
  // Y1 = (2/pi) [ -J0/x + l J1 + (-J1 + s1) ]
  b.y1 = kTwoOverPi * (l * b.j1 - 0.5 * twoOverX * b.j0 - b.j1 + s.s1 * scale);
  return b;
}

// a_k of order nu
template <int kNu, int K>
struct HankelA {
  static constexpr double v =
      HankelA<kNu, K - 1>::v * (4.0 * kNu * kNu - (2.0 * K - 1.0) * (2.0 * K - 1.0)) / (8.0 * K);
};
template <int kNu>
struct HankelA<kNu, 0> {
  static constexpr double v = 1.0;
};
// sum of a_{First + 2j} w^j, j = J .. kTerms - 1, by Horner's rule
template <int kNu, int kFirst, int kTerms, int J = 0>
BFG_HD double hankelPoly(double w) {
  if constexpr (J + 1 == kTerms)
    return HankelA<kNu, kFirst + 2 * J>::v;
  else
    return fma(hankelPoly<kNu, kFirst, kTerms, J + 1>(w), w, HankelA<kNu, kFirst + 2 * J>::v);
}
// P = sum (-1)^j a_2j / x^2j, Q = sum (-1)^j a_{2j+1} / x^{2j+1}: kTerms each
template <bool kOrder1, int kTerms>
BFG_HD void hankelPQ(double z, double &p0, double &q0, double &p1, double &q1) {
  double const w = -z * z;
  p0 = hankelPoly<0, 0, kTerms>(w);
  q0 = z * hankelPoly<0, 1, kTerms>(w);
  if constexpr (kOrder1) {
    p1 = hankelPoly<1, 0, kTerms>(w);
    q1 = z * hankelPoly<1, 1, kTerms>(w);
  } else {
    p1 = q1 = 0.0;
  }
}

// x >= kAsymptoticMin: Hankel's expansion; order 1 only when kOrder1.
template <bool kOrder1 = true>
BFG_HD Bessel01 besselAsymptotic(double x) {
#if defined(__CUDA_ARCH__)
  double const rx = rsqrt(x);
#else
  double const rx = 1.0 / sqrt(x);
#endif
  double const z = rx * rx;
  double p0, q0, p1, q1;
  // terms from which a_k / x^k < 1e-17 (both orders): 8 at x = 200, 10 at
  // 100, 13 at 50, 17 at 30, 27 at 20
  if (x >= 200.0) hankelPQ<kOrder1, 4>(z, p0, q0, p1, q1);
  else if (x >= 100.0) hankelPQ<kOrder1, 5>(z, p0, q0, p1, q1);
  else if (x >= 50.0) hankelPQ<kOrder1, 7>(z, p0, q0, p1, q1);
  else if (x >= 30.0) hankelPQ<kOrder1, 9>(z, p0, q0, p1, q1);
  else hankelPQ<kOrder1, 14>(z, p0, q0, p1, q1);
  double s, c;
  bfgSincos(x, &s, &c);
  // sqrt(2 / (pi x)) and the 1 / sqrt(2) of the rotations by pi/4 (chi0 =
  // x - pi/4: cos chi0 = (c + s) / sqrt 2, sin chi0 = (s - c) / sqrt 2) and
  // 3 pi/4 (cos chi1 = sin chi0, sin chi1 = -cos chi0)
  double const amp = kInvSqrtPi * rx, cs = amp * (c + s), sc = amp * (s - c);
  Bessel01 b;
  b.j0 = p0 * cs - q0 * sc;
  b.y0 = p0 * sc + q0 * cs;
  if (kOrder1) {
    b.j1 = p1 * sc + q1 * cs;
    b.y1 = q1 * sc - p1 * cs;
  } else {
    b.j1 = b.y1 = 0.0;
  }
  return b;
}

// J0, Y0 (and J1, Y1 when kOrder1) at x > 0.
template <bool kOrder1 = true>
BFG_HD Bessel01 bessel01(double x) {
  if (x >= kAsymptoticMin) return besselAsymptotic<kOrder1>(x);
  // one start index for the whole range: a shorter one below x = 8 saves less
  // than the two paths cost in warps that meet both
  if (x >= kSeriesMax) return besselMiller<56>(x);
  return besselSeries(x);
}

}  // namespace bfg
