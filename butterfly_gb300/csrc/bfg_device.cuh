// Device helpers shared by the CUDA sources of the factorization: complex
// product, the kernel value of each layer potential, warp sums.
#pragma once

#include <cuda_runtime.h>

#include "bfg_kernels.cuh"
#include "hankel.cuh"

namespace bfg {

constexpr double kTwoPiDev = 6.283185307179586;   // const.h BF_TWO_PI

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// |(dx, dy)|; the plain form where no square over- or underflows takes half
// the FP64 instructions of hypot
__device__ __forceinline__ double planeDistance(double dx, double dy) {
  double const r2 = fma(dx, dx, dy * dy);
  if (r2 > 1e-280 && r2 < 1e280) return sqrt(r2);
  return hypot(dx, dy);
}

// Kernel value K(x_tgt, x_src) for the layer potential in kp (helm2.c:38-91;
// matrix fills return 0 at r == 0, helm2.c:114, 159-160, 207, 255).
__device__ __forceinline__ double2 kernelValue(KernelParams const &kp, double tx,
                                               double ty, double tnx, double tny,
                                               double sx, double sy, double snx,
                                               double sny) {
  double const r = planeDistance(sx - tx, sy - ty);
  if (r == 0.0) return make_double2(0.0, 0.0);
  double const kr = kp.k * r;
  if (kp.layerPot == kLpSingle) {
    Bessel01 b = bessel01<false>(kr);
    return make_double2(-0.25 * b.y0, 0.25 * b.j0);          // (i/4) H0
  }
  Bessel01 b = bessel01<true>(kr);
  // (i/4) k H1(kr) / r = (k/(4r)) (-Y1 + i J1)
  double const f = 0.25 * kp.k / r;
  double2 const scale = make_double2(-f * b.y1, f * b.j1);
  if (kp.layerPot == kLpPvDouble) {
    double const dot = snx * (tx - sx) + sny * (ty - sy);
    return make_double2(scale.x * dot, scale.y * dot);
  }
  if (kp.layerPot == kLpPvNormalDerivSingle) {
    double const dot = tnx * (tx - sx) + tny * (ty - sy);
    return make_double2(scale.x * dot, scale.y * dot);
  }
  // combined field alpha S + beta D
  double const dot = snx * (tx - sx) + sny * (ty - sy);
  double2 const S = make_double2(-0.25 * b.y0, 0.25 * b.j0);
  double2 const D = make_double2(scale.x * dot, scale.y * dot);
  double2 const a = cmul(make_double2(kp.alphaRe, kp.alphaIm), S);
  double2 const c = cmul(make_double2(kp.betaRe, kp.betaIm), D);
  return make_double2(a.x + c.x, a.y + c.y);
}

// (accr, acci) += a x as four fused multiply-adds: written out, the compiler
// forms a multiply, an FMA and an add per part (six instructions), and the
// FP64 forms are bound by GB300's FP64 pipe
__device__ __forceinline__ void cmacc(float &accr, float &acci, float2 a, float2 x) {
  accr = fmaf(a.x, x.x, accr);
  accr = fmaf(-a.y, x.y, accr);
  acci = fmaf(a.x, x.y, acci);
  acci = fmaf(a.y, x.x, acci);
}
__device__ __forceinline__ void cmacc(double &accr, double &acci, double2 a, double2 x) {
  accr = fma(a.x, x.x, accr);
  accr = fma(-a.y, x.y, accr);
  acci = fma(a.x, x.y, acci);
  acci = fma(a.y, x.x, acci);
}

__device__ __forceinline__ double warpSum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The warp's sums of four values: a's in lanes 0-7, b's in 8-15, c's in 16-23,
// d's in 24-31.  Six FP64 additions a lane against the twenty of four warpSums.
__device__ __forceinline__ double warpSum4(double a, double b, double c, double d) {
  int const lane = threadIdx.x & 31;
  bool const hi = lane & 16, odd = lane & 8;
  double p = hi ? c : a, q = hi ? d : b;
  p += __shfl_xor_sync(0xffffffffu, hi ? a : c, 16);
  q += __shfl_xor_sync(0xffffffffu, hi ? b : d, 16);
  double v = odd ? q : p;
  v += __shfl_xor_sync(0xffffffffu, odd ? p : q, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// two sums the same way: a's in lanes 0 .. 15, b's in lanes 16 .. 31
__device__ __forceinline__ double warpSum2(double a, double b) {
  bool const hi = threadIdx.x & 16;
  double v = hi ? b : a;
  v += __shfl_xor_sync(0xffffffffu, hi ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace bfg
