// Double-float ("df64") apply of up to three right-hand sides: the FP64
// factors and vectors carried as pairs of FP32 numbers (hi + lo, ~48
// significant bits) and multiplied with FP32 FMAs and their exact error terms.
// The same 16 bytes per stored entry as FP64, within ~1e-13 of it, and fewer
// instructions an entry than the FP64 apply's fixed-point products (32,768
// points: 269 us against 351).  More right-hand sides take the FP64 apply,
// which is both more exact and faster there.  Same apply program as the other
// precisions (mat_block_dense.c:512-572, mat_product.c:211-245, one item =
// rows of one block row summing its blocks in order), no atomics, reproducible.
//
// Arithmetic (error-free transformations, Dekker 1971 / Knuth TAOCP 4.2.2;
// the FMA form of the product and the double-word sums of Joldes, Muller and
// Popescu, "Tight and rigorous error bounds for basic building blocks of
// double-word arithmetic", 2017):
//   TwoSum(a, b)   = (s, e), s = fl(a + b), e = a + b - s exactly
//   TwoProd(a, b)  = (p, e), p = fl(a b),   e = fma(a, b, -p) exactly
//   (ah + al)(bh + bl) ~ ah bh + [fma(ah, bh, -ah bh) + ah bl + al bh]
// Each lane keeps its running sum unnormalised as (s, t): the high parts
// pass through TwoSum and every low-order term is added to t.
#include <cuda_runtime.h>

#include <cstdint>

#include "bfg_kernels.cuh"
#include "bfg_launch.cuh"

namespace bfg {
namespace {


// The _rn intrinsics are never contracted into FMAs, which would break the
// error-free transformations.
__device__ __forceinline__ void twoSum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  float const bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}
__device__ __forceinline__ void fastTwoSum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  e = __fsub_rn(b, __fsub_rn(s, a));
}
// (sh, sl) += (ah + al)(bh + bl), unnormalised
__device__ __forceinline__ void dfMac(float ah, float al, float bh, float bl, float &sh,
                                      float &sl) {
  float const ph = __fmul_rn(ah, bh);
  float pl = fmaf(ah, bh, -ph);
  pl = fmaf(ah, bl, pl);
  pl = fmaf(al, bh, pl);
  float s, e;
  twoSum(sh, ph, s, e);
  sh = s;
  sl += e + pl;
}
// (sh, sl) += (bh, bl)
__device__ __forceinline__ void dfAdd(float &sh, float &sl, float bh, float bl) {
  float s, e;
  twoSum(sh, bh, s, e);
  sh = s;
  sl += e + bl;
}
// a double as hi + lo
__device__ __forceinline__ float2 dfSplit(double d) {
  float const h = __double2float_rn(d);
  return make_float2(h, __double2float_rn(d - (double)h));
}
// complex entry: (re hi, re lo, im hi, im lo)
__device__ __forceinline__ float4 dfSplit(double2 v) {
  float2 const r = dfSplit(v.x), i = dfSplit(v.y);
  return make_float4(r.x, r.y, i.x, i.y);
}

__global__ void arenaToDfKernel(double2 const *__restrict__ a, float4 *__restrict__ b, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    b[i] = dfSplit(a[i]);
}

// out (nRows x R, leading dimension R) = X rows (perm[i] or i), split
__global__ void gatherToDfKernel(double2 const *X, int64_t ldx,
                                 int64_t const *__restrict__ perm, int64_t nRows, int R,
                                 float4 *__restrict__ out) {
  afterPrevious();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nRows;
       i += (int64_t)gridDim.x * blockDim.x) {
    double2 const *x = X + (perm ? perm[i] : i) * ldx;
    for (int r = 0; r < R; ++r) out[i * R + r] = dfSplit(x[r]);
  }
}

// One CTA per (item, right-hand side): lane = item row, the S warps take every
// S-th column with 4 entries in flight each, read past the caches where one
// right-hand side reads them (kOne; the input rows stay); the warps' sums are
// combined in a fixed order.  X and W hold double-float rows with leading
// dimension R.  Bound by the latency of the loads, and by HBM where the items
// are many and alike.  Fetching a batch ahead cost more registers than it hid.
// S = 8 halves an item's time, S = 4 keeps more items in flight: 8 where the
// longest item has 1 / 540 of the stage's columns and more (1 / 250 for three
// right-hand sides, which fill the chip better) and would end after the others.
// Stages of one right-hand side, 4 and 8 warps: of 65,536 points (0.05 % of the
// columns in the longest) 129 and 135 us, of 15,346 points on 64 circles
// (0.07 %) 171 and 186, of 32,768 points on a star (0.20 %) 144 and 102, of
// 4,096 points (0.59 %) 35 and 25.
template <int S, bool kOne>
__global__ void __launch_bounds__(32 * S)
applyGemvDfKernel(ApplyItem const *__restrict__ items, ApplyContrib const *__restrict__ contribs,
                  float4 const *__restrict__ arena, float4 const *X, float4 *W, int R) {
  __shared__ float4 part[S][32];
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int const rhs = kOne ? 0 : blockIdx.y;
  int64_t const ld = kOne ? 1 : R;
  ApplyItem const it = items[blockIdx.x];
  bool const active = lane < it.rows;
  afterPrevious();
  float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f;
  auto mac = [&](float4 a, float4 x) {
    // re += ar xr - ai xi, im += ar xi + ai xr
    dfMac(a.x, a.y, x.x, x.y, rh, rl);
    dfMac(-a.z, -a.w, x.z, x.w, rh, rl);
    dfMac(a.x, a.y, x.z, x.w, ih, il);
    dfMac(a.z, a.w, x.x, x.y, ih, il);
  };
  auto entry = [&](float4 const *a) { return kOne ? __ldcs(a) : __ldg(a); };
  for (int c = 0; c < it.nContrib; ++c) {
    ApplyContrib const cb = contribs[it.contrib0 + c];
    float4 const *a = arena + cb.aOff + lane;
    float4 const *x = (cb.inIsX ? X : W) + cb.inRow * ld + rhs;
    int const n = cb.n;
    int64_t const lda = cb.lda;
    int j = warp;
    for (; j + 3 * S < n; j += 4 * S) {
      float4 a0, a1, a2, a3;
      if (active) {
        a0 = entry(a + (int64_t)(j + 0 * S) * lda);
        a1 = entry(a + (int64_t)(j + 1 * S) * lda);
        a2 = entry(a + (int64_t)(j + 2 * S) * lda);
        a3 = entry(a + (int64_t)(j + 3 * S) * lda);
      } else {
        a0 = a1 = a2 = a3 = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      float4 const x0 = x[(j + 0 * S) * ld], x1 = x[(j + 1 * S) * ld];
      float4 const x2 = x[(j + 2 * S) * ld], x3 = x[(j + 3 * S) * ld];
      mac(a0, x0);
      mac(a1, x1);
      mac(a2, x2);
      mac(a3, x3);
    }
    for (; j < n; j += S) {
      float4 const a0 = active ? entry(a + (int64_t)j * lda) : make_float4(0.f, 0.f, 0.f, 0.f);
      mac(a0, x[j * ld]);
    }
  }
  part[warp][lane] = make_float4(rh, rl, ih, il);
  __syncthreads();
  if (warp == 0 && active) {
    float sh = 0.f, sl = 0.f, th = 0.f, tl = 0.f;
#pragma unroll
    for (int w = 0; w < S; ++w) {
      float4 const v = part[w][lane];
      dfAdd(sh, sl, v.x, v.y);
      dfAdd(th, tl, v.z, v.w);
    }
    float a, b, c, d;
    fastTwoSum(sh, sl, a, b);
    fastTwoSum(th, tl, c, d);
    W[(it.outRow + lane) * ld + rhs] = make_float4(a, b, c, d);
  }
}

int gridDf(int64_t n) {
  int64_t g = (n + 255) / 256;
  return (int)(g < 1 ? 1 : (g > 152 * 32 ? 152 * 32 : g));
}

}  // namespace

cudaError_t launchArenaToDf(double2 const *a64, float4 *adf, int64_t n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  arenaToDfKernel<<<gridDf(n), 256, 0, stream>>>(a64, adf, n);
  return cudaGetLastError();
}

cudaError_t launchGatherToDf(double2 const *X, int64_t ldx, int64_t const *perm, int64_t nRows,
                             int R, float4 *out, cudaStream_t stream) {
  if (nRows == 0) return cudaSuccess;
  return launchAfter(gatherToDfKernel, dim3(gridDf(nRows)), dim3(256), 0, stream, X, ldx, perm, nRows,
                     R, out);
}

cudaError_t launchApplyStageDf(ApplyItem const *items, int64_t nItems,
                               ApplyContrib const *contribs, float4 const *arena,
                               float4 const *X, float4 *W, int R, int64_t cols, int64_t longest,
                               cudaStream_t stream) {
  if (nItems == 0) return cudaSuccess;
  bool const wide = (R < 3 ? 540 : 250) * longest >= cols;
  auto kernel = R == 1 ? (wide ? applyGemvDfKernel<8, true> : applyGemvDfKernel<4, true>)
                       : (wide ? applyGemvDfKernel<8, false> : applyGemvDfKernel<4, false>);
  return launchAfter(kernel, dim3((unsigned)nItems, (unsigned)R), dim3(wide ? 256 : 128), 0, stream,
                     items, contribs, arena, X, W, R);
}

}  // namespace bfg
