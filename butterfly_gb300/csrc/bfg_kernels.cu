// CUDA kernels of the butterfly Helmholtz path (sm_103a).
//
//  * fillBlocksKernel      evaluation (LAST) and dense blocks: fused
//                          points -> distance -> H0/H1 -> complex entry,
//                          written column-major straight into the arena
//                          (helm2.c:93-319, fac_helm2.c:403-509, 741-775).
//  * reexpansionKernel     FIRST/MIDDLE blocks: both proxy kernel matrices
//                          (helm2.c:321-365) plus the pseudo-inverse
//                          least-squares solve (mat_dense_complex.c:1768-1849)
//                          by a one-sided Jacobi SVD (details at the kernel).
//  * applyGemvKernel /     one stage of the staged FP32 apply (single / many
//    applyRhsKernel        RHS), each item a row chunk of one block row summing
//                          its blocks in order; no atomics, so results are
//                          reproducible bit for bit.
//  * applyReduceKernel     sums the per-product outputs into Y in a fixed
//                          order (the reference's block-dense accumulation,
//                          mat_block_dense.c:512-572), optionally scattering
//                          to original point order.
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include <cstdint>

#include "bfg_device.cuh"
#include "bfg_kernels.cuh"
#include "bfg_launch.cuh"
#include "hankel.cuh"

namespace bfg {

namespace {

constexpr double kTwoPiD = 6.283185307179586;   // const.h BF_TWO_PI
constexpr double kEps = 2.220446049250313e-16;
constexpr int kMaxSweeps = 60;

// ---------------------------------------------------------------------------
// LAST and DENSE blocks
// ---------------------------------------------------------------------------
__global__ void fillBlocksKernel(FillDesc const *__restrict__ descs, PointsDev src,
                                 PointsDev tgt, KernelParams kp, double2 *arena,
                                 int32_t *status) {
  extern __shared__ double proxy[];   // 4 * n for LAST blocks
  FillDesc const d = descs[blockIdx.x];
  kp.k = d.k;
  int const m = d.m, n = d.n;
  double2 *out = arena + d.arenaOff;
  bool const useSrcN = kp.layerPot == kLpPvDouble || kp.layerPot == kLpCombinedField;
  bool const useTgtN = kp.layerPot == kLpPvNormalDerivSingle;
  if (d.kind == kLast) {
    double const scale = kTwoPiD / (double)d.nTot;
    for (int b = threadIdx.x; b < n; b += blockDim.x) {
      double s, c;
      sincos(scale * (d.j0 + b), &s, &c);
      proxy[b] = d.ceq[2] * c + d.ceq[0];
      proxy[n + b] = d.ceq[2] * s + d.ceq[1];
      proxy[2 * n + b] = c;
      proxy[3 * n + b] = s;
    }
    __syncthreads();
    int64_t const total = (int64_t)m * n;
    for (int64_t e = threadIdx.x; e < total; e += blockDim.x) {
      int const i = (int)(e % m), j = (int)(e / m);
      int64_t const ti = d.t0 + i;
      out[e] = kernelValue(kp, tgt.x[ti], tgt.y[ti], useTgtN ? tgt.nx[ti] : 0.0,
                           useTgtN ? tgt.ny[ti] : 0.0, proxy[j], proxy[n + j],
                           useSrcN ? proxy[2 * n + j] : 0.0,
                           useSrcN ? proxy[3 * n + j] : 0.0);
    }
  } else if (d.kind == kDense) {
    int64_t const total = (int64_t)m * n;
    for (int64_t e = threadIdx.x; e < total; e += blockDim.x) {
      int const i = (int)(e % m), j = (int)(e / m);
      int64_t const ti = d.t0 + i, sj = d.s0 + j;
      out[e] = kernelValue(kp, tgt.x[ti], tgt.y[ti], useTgtN ? tgt.nx[ti] : 0.0,
                           useTgtN ? tgt.ny[ti] : 0.0, src.x[sj], src.y[sj],
                           useSrcN ? src.nx[sj] : 0.0, useSrcN ? src.ny[sj] : 0.0);
    }
  } else if (threadIdx.x == 0) {
    atomicOr(status, kStatusBadDescriptor);
  }
}

// ---------------------------------------------------------------------------
// FIRST and MIDDLE blocks: proxy fills + Jacobi pseudo-inverse re-expansion
//
// Z_shift = pinv(Z_equiv) Z_orig with Z_equiv p x p.  One-sided Jacobi on
// the columns of M = [Z_equiv^H ; I]: rotations Q make the top part
// T = Z_equiv^H Q column-orthogonal (T = V S) while the bottom part
// accumulates Q (= U).  Then pinv_k(Z_equiv) = T diag(w) Q^H with
// w_a = 1/s_a^2 for kept singular values, 0 otherwise, and every column of
// the output is x_j = T (w .* (Q^H z_j)), z_j = Z_orig[:, j] evaluated on
// the fly.  Modes: 0 = M in shared memory (one CTA), 1 = M in global
// scratch (one CTA), 2 = M in global scratch shared by a thread-block
// cluster of kClusterCtas CTAs that split every Jacobi round and meet at
// hardware cluster barriers.
// The sweeps are bound by the FP64 pipe, where a warp instruction takes 16
// clocks of the SM whatever its lanes do.  A rotation's angle takes about a
// hundred of them, more than the products of a pair of 25-row columns, so a
// round goes in three steps: the warps' dot products, the angles of up to
// 16 kReexpPer pairs with one thread a pair, the rotations.  Measured:
// this path 40 -> 21 ms at 65,536 points, 48 -> 25 ms for twelve problems of up
// to 16,384 points, 10.4 -> 6.5 ms at 4,096 points.
// ---------------------------------------------------------------------------
constexpr int kClusterCtas = 8;
constexpr int kReexpPer = 8;   // pairs of a warp in one step

// ---- double-float arithmetic for the Jacobi sweeps (kDf): each complex
// entry of M held as FP32 pairs (re hi, re lo, im hi, im lo) in the same 16
// bytes, products by FMA error terms, sums by TwoSum (Dekker; Knuth TAOCP
// 4.2.2).  The _rn intrinsics are never contracted into FMAs, which would
// break the error-free steps.
__device__ __forceinline__ void jTwoSum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  float const bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}
// (sh, sl) += (ah + al)(bh + bl), unnormalised
__device__ __forceinline__ void jMac(float ah, float al, float bh, float bl, float &sh, float &sl) {
  float const ph = __fmul_rn(ah, bh);
  float pl = fmaf(ah, bh, -ph);
  pl = fmaf(ah, bl, pl);
  pl = fmaf(al, bh, pl);
  float s, e;
  jTwoSum(sh, ph, s, e);
  sh = s;
  sl += e + pl;
}
__device__ __forceinline__ float2 jNorm(float h, float l) {
  float const s = __fadd_rn(h, l);
  return make_float2(s, __fsub_rn(l, __fsub_rn(s, h)));
}
__device__ __forceinline__ float2 jSplit(double d) {
  float const h = __double2float_rn(d);
  return make_float2(h, __double2float_rn(d - (double)h));
}
// the sum over the warp as a double; TwoSum is commutative, so every lane of
// the butterfly gets the same bits
__device__ __forceinline__ double jWarpSum(float h, float l) {
  for (int o = 16; o > 0; o >>= 1) {
    float const oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
    float s, e;
    jTwoSum(h, oh, s, e);
    h = s;
    l = __fadd_rn(e, __fadd_rn(l, ol));
  }
  return (double)h + (double)l;
}

template <int kMode, bool kDf>
struct ReexpMem {
  static __device__ __forceinline__ double2 ld(double2 const *p) {
    if (kMode == 2) return __ldcg(p);   // other SMs of the cluster write M
    return *p;
  }
  static __device__ __forceinline__ void st(double2 *p, double2 v) {
    if (kMode == 2) __stcg(p, v);
    else *p = v;
  }
  static __device__ __forceinline__ float4 ld4(double2 const *p) {
    float4 const *q = reinterpret_cast<float4 const *>(p);
    if (kMode == 2) return __ldcg(q);
    return *q;
  }
  static __device__ __forceinline__ void st4(double2 *p, float4 v) {
    float4 *q = reinterpret_cast<float4 *>(p);
    if (kMode == 2) __stcg(q, v);
    else *q = v;
  }
  // an entry of M as a complex double, whichever way it is held
  static __device__ __forceinline__ double2 ldC(double2 const *p) {
    if (!kDf) return ld(p);
    float4 const v = ld4(p);
    return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
  }
  static __device__ __forceinline__ void stC(double2 *p, double2 v) {
    if (!kDf) {
      st(p, v);
      return;
    }
    float2 const r = jSplit(v.x), i = jSplit(v.y);
    st4(p, make_float4(r.x, r.y, i.x, i.y));
  }
  static __device__ __forceinline__ void sync() {
    if (kMode == 2) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  }
};

constexpr int kNoExp = -100000;   // no nonzero entry seen
constexpr int kColExpBias = 1100;  // makes ilogb of any positive double positive

// The double-float scale exponent s of a block: the largest e over its
// threads (|entry|^2 < 2^e) and the largest s with p^2 2^(e + 2s) <= 2^100,
// so that a column's squared norm stays below 2^100 / p (FP32 reaches 2^128)
// while its rounding-floor entries stay far above 2^-102, where the error
// terms of their products turn subnormal.  Mode 2 combines the cluster's
// CTAs through their flag slots (free until the first sweep ends); every
// thread of the block (or cluster) gets the same s.
template <int kMode>
__device__ int reexpScaleExp(int eTop, int p, int32_t *clusterFlags, int rank) {
  __shared__ int red[32];
  for (int o = 16; o > 0; o >>= 1) eTop = max(eTop, __shfl_xor_sync(0xffffffffu, eTop, o));
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
  if (lane == 0) red[warp] = eTop;
  __syncthreads();
  if (threadIdx.x == 0) {
    int m = kNoExp;
    for (int w = 0; w < nWarps; ++w) m = max(m, red[w]);
    red[0] = m;
    if (kMode == 2) __stcg(clusterFlags + rank, m);
  }
  if (kMode == 2) cooperative_groups::this_cluster().sync();
  else __syncthreads();
  int eMax = red[0];
  if (kMode == 2)
    for (int q = 0; q < kClusterCtas; ++q) eMax = max(eMax, __ldcg(clusterFlags + q));
  __syncthreads();   // red[] is read before any later use of the helper's storage
  if (eMax == kNoExp) return 0;
  int lp = 0;
  while ((1 << lp) < p) ++lp;
  int const t = 100 - 2 * lp - eMax;
  return t >= 0 ? t / 2 : -((1 - t) / 2);
}

// kDf: the Jacobi sweeps in double-float (~48 significant bits, FP32
// arithmetic, about 6x fewer FP64 instructions; the rotation angles, the
// singular values and the output stay FP64), else in FP64
// Blocks with the same Z_equiv (the same rank, equivalent and check circles
// and wavenumber) share one SVD: descriptor `blk` is a group's leader (its n
// the largest over the group), and with `members` non-null the group's
// blocks are members[groupStart[blk] .. groupStart[blk + 1]), each of which
// gets its own Z_shift from the one pseudo-inverse.
template <int kMode, bool kDf>
__global__ void __launch_bounds__(512, kMode == 0 ? 2 : 1) reexpansionKernel(
    FillDesc const *__restrict__ descs, PointsDev src, KernelParams kp, int32_t cutMode,
    double cutTol, double2 *arena, double2 *scratch, int64_t const *scratchOff,
    int32_t *flags, int32_t *status, FillDesc const *__restrict__ members,
    int32_t const *__restrict__ groupStart) {
  using Mem = ReexpMem<kMode, kDf>;
  extern __shared__ double2 smem2[];
  int const ctas = kMode == 2 ? kClusterCtas : 1;
  int const blk = kMode == 2 ? (int)(blockIdx.x / kClusterCtas) : (int)blockIdx.x;
  int const rank = kMode == 2 ? (int)(blockIdx.x % kClusterCtas) : 0;
  FillDesc const d = descs[blk];
  kp.k = d.k;
  int const p = d.m, n = d.n, LD = 2 * p;
  int const tid = threadIdx.x, nthr = blockDim.x;
  int const lane = tid & 31, warp = tid >> 5, nWarps = nthr >> 5;
  int const gWarp = rank * nWarps + warp, gWarps = ctas * nWarps;

  // working matrix M (LD x p), then per-warp vectors (2p each), then (in a
  // cluster) p shared squared singular values; see reexpansionScratchEntries
  double2 *M, *wscr;
  double *geo;
  if (kMode == 0) {
    M = smem2;
    wscr = smem2 + (int64_t)LD * p;
    geo = reinterpret_cast<double *>(wscr + (int64_t)2 * p * nWarps);
  } else {
    M = scratch + scratchOff[blk];
    wscr = M + (int64_t)LD * p;
    geo = reinterpret_cast<double *>(smem2);
  }
  double2 *myB = wscr + (int64_t)2 * p * (kMode == 0 ? warp : gWarp);
  double2 *myY = myB + p;
  double *chkX = geo, *chkY = geo + p;
  double *eqX = geo + 2 * p, *eqY = geo + 3 * p, *eqNx = geo + 4 * p, *eqNy = geo + 5 * p;
  double *orX = geo + 6 * p, *orY = orX + n, *orNx = orX + 2 * n, *orNy = orX + 3 * n;
  double *wgt = orX + 4 * n;
  __shared__ int sRotated;
  __shared__ unsigned long long sColMax;   // bits of a nonnegative double
  // pair k nWarps + w of a step: warp w's k-th; (|x|^2, |y|^2, <x, y>), then
  // the rotation (c, s, exp(-i phi)), c = 2 for none
  __shared__ double4 sPair[16 * kReexpPer];
  bool const useSrcN = kp.layerPot == kLpPvDouble || kp.layerPot == kLpCombinedField;

  // proxy geometry (every CTA of a cluster keeps its own copy); check points
  // on cchk and equivalent sources on ceq share theta_a = (2 pi / p) a
  {
    double const scale = kTwoPiD / (double)p;
    for (int a = tid; a < p; a += nthr) {
      double s, c;
      sincos(scale * a, &s, &c);
      chkX[a] = d.cchk[2] * c + d.cchk[0];
      chkY[a] = d.cchk[2] * s + d.cchk[1];
      eqX[a] = d.ceq[2] * c + d.ceq[0];
      eqY[a] = d.ceq[2] * s + d.ceq[1];
      eqNx[a] = c;
      eqNy[a] = s;
    }
  }
  __syncthreads();

  // M[a*LD + r] = conj(K(chk_a, eq_r)) for r < p, identity below.
  // Double-float holds the top part scaled by 2^sExp (exact), sExp chosen
  // from the largest entry so that the sweeps' products stay far above
  // FP32's subnormal range: there the products' error terms lose their bits,
  // and pairs of columns at the rounding floor (sigma^2 ~ 1e-31 of the
  // largest) rotate on noise until the sweep cap.  FP64 keeps sExp = 0.
  int sExp = 0;
  {
    int64_t const total = (int64_t)LD * p;
    int eTop = kNoExp;   // exponent bound of the largest |entry|^2 this thread wrote
    for (int64_t e = (int64_t)rank * nthr + tid; e < total; e += (int64_t)ctas * nthr) {
      int const a = (int)(e / LD), r = (int)(e % LD);
      double2 v;
      if (r < p) {
        double2 k = kernelValue(kp, chkX[a], chkY[a], 0.0, 0.0, eqX[r], eqY[r], eqNx[r], eqNy[r]);
        v = make_double2(k.x, -k.y);
        double const m2 = v.x * v.x + v.y * v.y;
        if (kDf && m2 > 0.0) eTop = max(eTop, ilogb(m2) + 1);
      } else {
        v = make_double2(r - p == a ? 1.0 : 0.0, 0.0);
      }
      if (kDf) Mem::st(M + e, v);   // FP64 until the scale is known
      else Mem::stC(M + e, v);
    }
    if (kDf) {
      sExp = reexpScaleExp<kMode>(eTop, p, flags ? flags + (int64_t)blk * kClusterCtas : nullptr,
                                  rank);
      // every thread converts the entries it wrote
      for (int64_t e = (int64_t)rank * nthr + tid; e < total; e += (int64_t)ctas * nthr) {
        double2 v = Mem::ld(M + e);
        if ((int)(e % LD) < p) v = make_double2(ldexp(v.x, sExp), ldexp(v.y, sExp));
        Mem::stC(M + e, v);
      }
    }
  }
  Mem::sync();

  // one-sided Jacobi, round-robin pair schedule
  int const P = p + (p & 1);
  int const nPairs = P / 2;
  // rotation threshold: FP64 eps, or (double-float) 2^-44, well above the
  // rounding noise of the pair sums (2^-46 left a large block cycling to the
  // sweep cap)
  double const tolRot = (kDf ? 5.684341886080802e-14 : kEps) * sqrt((double)p);
  // double-float: columns far under the pseudo-inverse cut carry the
  // rounding noise (2^-48 of the largest columns) that every rotation of a
  // large column injects, and rotations on that noise would go on to the
  // sweep cap.  Measured against the previous sweep's largest column norm^2
  // (a lower bound of sigma_max^2): a pair whose columns both lie below
  // 1e-4 cut^2 is not rotated (only rotations with larger columns, which
  // still run, could lift them toward the cut), and one whose columns both
  // lie below 1e-2 cut^2 is rotated without holding the sweeps open --
  // neither can change the kept part of the pseudo-inverse.
  // The second band keeps a column just above the first from cycling against
  // the unrotated noise columns until the cap.
  double const cutRel = cutMode == 0 ? (double)p * kEps : cutTol;
  double skipBelow = 0.0, quietBelow = 0.0;
  // the columns of pair pr of a round (false: the bye of an odd count)
  auto columns = [&](int round, int pr, double2 *&ci, double2 *&cj) {
    int i, j;
    if (pr == 0) {
      i = round;
      j = P - 1;
    } else {
      i = round + pr;
      if (i >= P - 1) i -= P - 1;
      j = round - pr;
      if (j < 0) j += P - 1;
    }
    ci = M + (int64_t)i * LD;
    cj = M + (int64_t)j * LD;
    return i < p && j < p;
  };
  bool converged = false;
  for (int sweep = 0; sweep < kMaxSweeps; ++sweep) {
    if (tid == 0) {
      sRotated = 0;
      sColMax = 0ull;
    }
    __syncthreads();
    double colMax = 0.0;   // the largest column norm^2 of this thread's pairs
    for (int round = 0; round < P - 1; ++round) {
      for (int pr0 = 0; pr0 < nPairs; pr0 += gWarps * kReexpPer) {
        // the pairs' dot products, a warp each
        for (int k = 0, pr = pr0 + gWarp; k < kReexpPer && pr < nPairs; ++k, pr += gWarps) {
          double2 *ci, *cj;
          bool const both = columns(round, pr, ci, cj);   // (else zeros: no rotation)
          double4 *const out = sPair + k * nWarps + warp;
          if (kDf) {
            float alh = 0, all = 0, beh = 0, bel = 0, grh = 0, grl = 0, gih = 0, gil = 0;
            if (both)
              for (int r = lane; r < p; r += 32) {
                float4 const x = Mem::ld4(ci + r), y = Mem::ld4(cj + r);
                jMac(x.x, x.y, x.x, x.y, alh, all);
                jMac(x.z, x.w, x.z, x.w, alh, all);
                jMac(y.x, y.y, y.x, y.y, beh, bel);
                jMac(y.z, y.w, y.z, y.w, beh, bel);
                jMac(x.x, x.y, y.x, y.y, grh, grl);      // conj(x) y
                jMac(x.z, x.w, y.z, y.w, grh, grl);
                jMac(x.x, x.y, y.z, y.w, gih, gil);
                jMac(-x.z, -x.w, y.x, y.y, gih, gil);
              }
            double const al = jWarpSum(alh, all), be = jWarpSum(beh, bel);
            double const gr = jWarpSum(grh, grl), gi = jWarpSum(gih, gil);
            if (lane == 0) *out = make_double4(al, be, gr, gi);
          } else {
            double al = 0, be = 0, gr = 0, gi = 0;
            if (both)
              for (int r = lane; r < p; r += 32) {
                double2 x = Mem::ld(ci + r), y = Mem::ld(cj + r);
                al = fma(x.x, x.x, fma(x.y, x.y, al));
                be = fma(y.x, y.x, fma(y.y, y.y, be));
                gr = fma(x.x, y.x, fma(x.y, y.y, gr));     // conj(x) y
                gi = fma(x.x, y.y, fma(-x.y, y.x, gi));
              }
            double const v = warpSum4(al, be, gr, gi);
            if ((lane & 7) == 0) reinterpret_cast<double *>(out)[lane >> 3] = v;
          }
        }
        __syncthreads();
        // their rotations, a thread each
        int const left = nPairs - pr0 - rank * nWarps;   // pairs from this CTA's first on
        for (int q = tid; q < kReexpPer * nWarps; q += nthr) {
          if ((q / nWarps) * gWarps + q % nWarps >= left) continue;
          double const al = sPair[q].x, be = sPair[q].y, gr = sPair[q].z, gi = sPair[q].w;
          double4 rot = make_double4(2.0, 0.0, 0.0, 0.0);
          double const ag = sqrt(gr * gr + gi * gi);
          // double-float: a column below 1e-14 of its partner in norm lies far
          // under the pseudo-inverse cut; rotating it only cycles on rounding
          if (kDf) colMax = fmax(colMax, fmax(al, be));
          bool const negligible =
              kDf && (fmin(al, be) <= 1e-28 * fmax(al, be) || fmax(al, be) < skipBelow);
          if (!negligible && ag > tolRot * sqrt(al * be) && ag > 0.0) {
            double const zeta = (be - al) / (2.0 * ag);
            double const t = (zeta >= 0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
            double const c = 1.0 / sqrt(1.0 + t * t);
            rot = make_double4(c, c * t, gr / ag, -gi / ag);   // exp(-i phi) = conj(gamma)/|gamma|
            if (!kDf || fmax(al, be) >= quietBelow) sRotated = 1;
          }
          sPair[q] = rot;
        }
        __syncthreads();
        for (int k = 0, pr = pr0 + gWarp; k < kReexpPer && pr < nPairs; ++k, pr += gWarps) {
          double4 const rot = sPair[k * nWarps + warp];
          if (rot.x > 1.5) continue;
          double const c = rot.x, s = rot.y, er = rot.z, ei = rot.w;
          double2 *ci, *cj;
          columns(round, pr, ci, cj);
          if (kDf) {
            float2 const cD = jSplit(c), sD = jSplit(s), erD = jSplit(er), eiD = jSplit(ei);
            for (int r = lane; r < LD; r += 32) {
              float4 const x = Mem::ld4(ci + r), y = Mem::ld4(cj + r);
              float h, l;
              // yt = y exp(-i phi)
              h = 0.f, l = 0.f;
              jMac(y.x, y.y, erD.x, erD.y, h, l);
              jMac(-y.z, -y.w, eiD.x, eiD.y, h, l);
              float2 const ytr = jNorm(h, l);
              h = 0.f, l = 0.f;
              jMac(y.x, y.y, eiD.x, eiD.y, h, l);
              jMac(y.z, y.w, erD.x, erD.y, h, l);
              float2 const yti = jNorm(h, l);
              // x' = c x - s yt, y' = s x + c yt
              h = 0.f, l = 0.f;
              jMac(cD.x, cD.y, x.x, x.y, h, l);
              jMac(-sD.x, -sD.y, ytr.x, ytr.y, h, l);
              float2 const xr = jNorm(h, l);
              h = 0.f, l = 0.f;
              jMac(cD.x, cD.y, x.z, x.w, h, l);
              jMac(-sD.x, -sD.y, yti.x, yti.y, h, l);
              float2 const xi = jNorm(h, l);
              h = 0.f, l = 0.f;
              jMac(sD.x, sD.y, x.x, x.y, h, l);
              jMac(cD.x, cD.y, ytr.x, ytr.y, h, l);
              float2 const yr = jNorm(h, l);
              h = 0.f, l = 0.f;
              jMac(sD.x, sD.y, x.z, x.w, h, l);
              jMac(cD.x, cD.y, yti.x, yti.y, h, l);
              float2 const yi = jNorm(h, l);
              Mem::st4(ci + r, make_float4(xr.x, xr.y, xi.x, xi.y));
              Mem::st4(cj + r, make_float4(yr.x, yr.y, yi.x, yi.y));
            }
          } else {
            for (int r = lane; r < LD; r += 32) {
              double2 x = Mem::ld(ci + r), y = Mem::ld(cj + r);
              double const ytr = y.x * er - y.y * ei, yti = y.x * ei + y.y * er;
              Mem::st(ci + r, make_double2(c * x.x - s * ytr, c * x.y - s * yti));
              Mem::st(cj + r, make_double2(s * x.x + c * ytr, s * x.y + c * yti));
            }
          }
        }
        if (pr0 + gWarps * kReexpPer < nPairs) __syncthreads();   // sPair is rewritten
      }
      Mem::sync();
    }
    if (kDf) {
      if (colMax > 0.0) atomicMax(&sColMax, (unsigned long long)__double_as_longlong(colMax));
      __syncthreads();
    }
    int rotated = sRotated;
    // the largest column norm^2 as a biased exponent (2^(colExp - bias) <= it)
    int colExp = 0;
    if (kDf) {
      double const cm = __longlong_as_double((long long)sColMax);
      colExp = cm > 0.0 ? ilogb(cm) + kColExpBias : 0;
    }
    if (kMode == 2) {
      // cluster-wide OR of the CTAs' flags (and maximum of their exponents),
      // read after a barrier so every CTA takes the same decisions
      if (tid == 0) __stcg(flags + (int64_t)blk * kClusterCtas + rank, rotated | (colExp << 1));
      Mem::sync();
      rotated = 0;
      colExp = 0;
      for (int q = 0; q < kClusterCtas; ++q) {
        int const v = __ldcg(flags + (int64_t)blk * kClusterCtas + q);
        rotated |= v & 1;
        colExp = max(colExp, v >> 1);
      }
    }
    __syncthreads();
    if (!rotated) {
      converged = true;
      break;
    }
    if (kDf && colExp > 0) {
      double const colMaxLow = ldexp(cutRel * cutRel, colExp - kColExpBias);
      skipBelow = 1e-4 * colMaxLow;
      quietBelow = 1e-2 * colMaxLow;
    }
  }
  if (!converged && tid == 0 && rank == 0) atomicOr(status, kStatusJacobiNotConverged);

  // singular values and the pseudo-inverse cut (mat_dense_complex.c:1797-1808)
  double2 *wg = kMode == 2 ? wscr + (int64_t)2 * p * gWarps : nullptr;   // shared sigma^2
  for (int a = gWarp; a < p; a += gWarps) {
    double2 const *ca = M + (int64_t)a * LD;
    double s2 = 0;
    for (int r = lane; r < p; r += 32) {
      double2 v = Mem::ldC(ca + r);
      s2 += v.x * v.x + v.y * v.y;
    }
    s2 = warpSum(s2);
    if (kDf) s2 = ldexp(s2, -2 * sExp);   // sigma^2 of the unscaled block
    if (lane == 0) {
      if (kMode == 2) Mem::st(wg + a, make_double2(s2, 0.0));
      else wgt[a] = s2;
    }
  }
  Mem::sync();
  if (kMode == 2)
    for (int a = tid; a < p; a += nthr) wgt[a] = Mem::ld(wg + a).x;
  __syncthreads();
  if (tid == 0) {
    double smax = 0;
    for (int a = 0; a < p; ++a) smax = fmax(smax, sqrt(wgt[a]));
    double const cut = cutMode == 0 ? (double)p * kEps * smax + kEps : cutTol * smax;
    for (int a = 0; a < p; ++a) {
      double const sa = sqrt(wgt[a]);
      // (double-float: T holds 2^sExp of its columns, so 2^-sExp goes here)
      wgt[a] = (sa < cut || sa == 0.0) ? 0.0 : ldexp(1.0 / wgt[a], -sExp);
    }
  }
  __syncthreads();

  // every block of the group: its source points (Z_orig's columns), then
  // x_j = T (w .* (Q^H z_j)), one warp per output column
  int const g0 = members ? groupStart[blk] : 0, g1 = members ? groupStart[blk + 1] : 1;
  for (int gm = g0; gm < g1; ++gm) {
  FillDesc const dm = members ? members[gm] : d;
  int const nm = dm.n;
  if (dm.kind == kFirst) {
    for (int b = tid; b < nm; b += nthr) {
      int64_t const sj = dm.s0 + b;
      orX[b] = src.x[sj];
      orY[b] = src.y[sj];
      orNx[b] = (useSrcN && src.nx) ? src.nx[sj] : 0.0;
      orNy[b] = (useSrcN && src.ny) ? src.ny[sj] : 0.0;
    }
  } else {
    double const scale2 = kTwoPiD / (double)nm;
    for (int b = tid; b < nm; b += nthr) {
      double s, c;
      sincos(scale2 * b, &s, &c);
      orX[b] = dm.corig[2] * c + dm.corig[0];
      orY[b] = dm.corig[2] * s + dm.corig[1];
      orNx[b] = c;
      orNy[b] = s;
    }
  }
  __syncthreads();
  double2 *out = arena + dm.arenaOff;
  for (int j = gWarp; j < nm; j += gWarps) {
    for (int r = lane; r < p; r += 32) {
      double2 z = kernelValue(kp, chkX[r], chkY[r], 0.0, 0.0, orX[j], orY[j], orNx[j], orNy[j]);
      myB[r] = z;
    }
    __syncwarp();
    for (int a = 0; a < p; ++a) {
      double const w = wgt[a];
      if (w == 0.0) {
        if (lane == 0) myY[a] = make_double2(0.0, 0.0);
        continue;
      }
      double2 const *qa = M + (int64_t)a * LD + p;
      double yr = 0, yi = 0;
      for (int r = lane; r < p; r += 32) {
        double2 q = Mem::ldC(qa + r), z = myB[r];
        yr = fma(q.x, z.x, fma(q.y, z.y, yr));        // conj(q) z
        yi = fma(q.x, z.y, fma(-q.y, z.x, yi));
      }
      yr = warpSum(yr);
      yi = warpSum(yi);
      if (lane == 0) myY[a] = make_double2(w * yr, w * yi);
    }
    __syncwarp();
    for (int i = lane; i < p; i += 32) {
      double sr = 0, si = 0;
      for (int a = 0; a < p; ++a) {
        double2 const y = myY[a];
        if (y.x == 0.0 && y.y == 0.0) continue;
        double2 const t = Mem::ldC(M + (int64_t)a * LD + i);
        cmacc(sr, si, t, y);
      }
      out[(int64_t)j * p + i] = make_double2(sr, si);
    }
    __syncwarp();
  }
  __syncthreads();   // the next member's points overwrite these
  }
}

// ---------------------------------------------------------------------------
// dense rows, kernel matrices, Bessel probes
// ---------------------------------------------------------------------------
__global__ void denseRowsKernel(PointsDev src, int64_t nSrc, PointsDev tgt,
                                int64_t const *rows, KernelParams kp,
                                double2 const *x, int64_t ldx, int64_t R,
                                double2 *out, int64_t ldo) {
  // one CTA per sampled row; threads stride over sources, R <= 8 per pass
  int64_t const s = blockIdx.x;
  int64_t const ti = rows[s];
  bool const useSrcN = kp.layerPot == kLpPvDouble || kp.layerPot == kLpCombinedField;
  bool const useTgtN = kp.layerPot == kLpPvNormalDerivSingle;
  __shared__ double red[2][32];
  for (int64_t r0 = 0; r0 < R; r0 += 8) {
    int const rc = (int)((R - r0) < 8 ? (R - r0) : 8);
    double accr[8] = {0, 0, 0, 0, 0, 0, 0, 0}, acci[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int64_t j = threadIdx.x; j < nSrc; j += blockDim.x) {
      double2 kv = kernelValue(kp, tgt.x[ti], tgt.y[ti], useTgtN ? tgt.nx[ti] : 0.0,
                               useTgtN ? tgt.ny[ti] : 0.0, src.x[j], src.y[j],
                               useSrcN ? src.nx[j] : 0.0, useSrcN ? src.ny[j] : 0.0);
      for (int c = 0; c < rc; ++c) {
        double2 xv = x[j * ldx + r0 + c];
        cmacc(accr[c], acci[c], kv, xv);
      }
    }
    for (int c = 0; c < rc; ++c) {
      double vr = warpSum(accr[c]), vi = warpSum(acci[c]);
      if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = vr;
        red[1][threadIdx.x >> 5] = vi;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        double sr = 0, si = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
          sr += red[0][w];
          si += red[1][w];
        }
        out[s * ldo + r0 + c] = make_double2(sr, si);
      }
      __syncthreads();
    }
  }
}

__global__ void kernelMatrixKernel(PointsDev src, int64_t n, PointsDev tgt, int64_t m,
                                   KernelParams kp, double2 *out) {
  bool const useSrcN = kp.layerPot == kLpPvDouble || kp.layerPot == kLpCombinedField;
  bool const useTgtN = kp.layerPot == kLpPvNormalDerivSingle;
  int64_t const total = m * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t const i = e / n, j = e % n;
    out[e] = kernelValue(kp, tgt.x[i], tgt.y[i], useTgtN ? tgt.nx[i] : 0.0,
                         useTgtN ? tgt.ny[i] : 0.0, src.x[j], src.y[j],
                         useSrcN ? src.nx[j] : 0.0, useSrcN ? src.ny[j] : 0.0);
  }
}

// FP64 fused multiply-add throughput: 8 independent chains per thread, the
// result written so that nothing is optimised away
__global__ void __launch_bounds__(256) fp64RateKernel(int32_t iters, double seed, double *out) {
  double a[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) a[c] = seed + 1e-3 * (threadIdx.x + 8 * c);
  double const b = 0.9999999, d = 1e-9;
  for (int i = 0; i < iters; ++i)
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = fma(a[c], b, d);
  double t = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) t += a[c];
  if (t == 12345.678) out[blockIdx.x] = t;   // never true for these inputs
}

__global__ void bessel01Kernel(double const *x, int64_t n, double *out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    Bessel01 b = bessel01<true>(x[i]);
    out[4 * i] = b.j0;
    out[4 * i + 1] = b.y0;
    out[4 * i + 2] = b.j1;
    out[4 * i + 3] = b.y1;
  }
}

__global__ void arenaToF32Kernel(double2 const *a, float2 *b, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double2 v = a[i];
    b[i] = make_float2((float)v.x, (float)v.y);
  }
}

__global__ void c128ToC64Kernel(double2 const *a, int64_t lda, int64_t rows, int64_t cols,
                                float2 *b, int64_t ldb, int64_t bTile, int64_t bTileStride) {
  int64_t const total = rows * cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t const i = e / cols, j = e % cols;
    double2 v = a[i * lda + j];
    int64_t const o = bTile ? (j / bTile) * bTileStride + i * bTile + j % bTile : i * ldb + j;
    b[o] = make_float2((float)v.x, (float)v.y);
  }
}

__global__ void c64ToC128Kernel(float2 const *a, int64_t lda, int64_t rows, int64_t cols,
                                double2 *b, int64_t ldb) {
  int64_t const total = rows * cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t const i = e / cols, j = e % cols;
    float2 v = a[i * lda + j];
    b[i * ldb + j] = make_double2((double)v.x, (double)v.y);
  }
}

// ---------------------------------------------------------------------------
// apply
// ---------------------------------------------------------------------------
template <typename T2> struct Real;
template <> struct Real<double2> { using T = double; };
template <> struct Real<float2> { using T = float; };

template <typename T2>
__device__ __forceinline__ T2 mk2(typename Real<T2>::T a, typename Real<T2>::T b) {
  T2 v;
  v.x = a;
  v.y = b;
  return v;
}

// R == 1: one CTA of 8 warps per item; lane = output row, warp w takes the
// columns j = w, w + 8, ... of every block in the row, four columns in
// flight at once; the 8 partial sums are reduced in shared memory in a
// fixed order.
constexpr int kGemvWarps = 8;

__global__ void __launch_bounds__(32 * kGemvWarps)
applyGemvKernel(ApplyItem const *__restrict__ items, ApplyContrib const *__restrict__ contribs,
                float2 const *__restrict__ arena, float2 const *__restrict__ X, int64_t ldx,
                float2 *__restrict__ W) {
  __shared__ float2 part[kGemvWarps][32];
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ApplyItem const it = items[blockIdx.x];
  bool const active = lane < it.rows;
  float accr = 0, acci = 0;
  for (int c = 0; c < it.nContrib; ++c) {
    ApplyContrib const cb = contribs[it.contrib0 + c];
    float2 const *a = arena + cb.aOff + lane;
    float2 const *x = cb.inIsX ? X + cb.inRow * ldx : W + cb.inRow;
    int64_t const xs = cb.inIsX ? ldx : 1;
    int const n = cb.n;
    int64_t const lda = cb.lda;
    int j = warp;
    constexpr int S = kGemvWarps;
    for (; j + 3 * S < n; j += 4 * S) {
      float2 a0, a1, a2, a3;
      if (active) {
        a0 = a[(int64_t)(j + 0 * S) * lda];
        a1 = a[(int64_t)(j + 1 * S) * lda];
        a2 = a[(int64_t)(j + 2 * S) * lda];
        a3 = a[(int64_t)(j + 3 * S) * lda];
      } else {
        a0 = a1 = a2 = a3 = make_float2(0, 0);
      }
      float2 const x0 = x[(j + 0 * S) * xs], x1 = x[(j + 1 * S) * xs];
      float2 const x2 = x[(j + 2 * S) * xs], x3 = x[(j + 3 * S) * xs];
      cmacc(accr, acci, a0, x0);
      cmacc(accr, acci, a1, x1);
      cmacc(accr, acci, a2, x2);
      cmacc(accr, acci, a3, x3);
    }
    for (; j < n; j += S) {
      float2 const a0 = active ? a[(int64_t)j * lda] : make_float2(0, 0);
      float2 const x0 = x[j * xs];
      cmacc(accr, acci, a0, x0);
    }
  }
  part[warp][lane] = make_float2(accr, acci);
  __syncthreads();
  if (warp == 0 && active) {
    float sr = 0, si = 0;
#pragma unroll
    for (int w = 0; w < kGemvWarps; ++w) {
      sr += part[w][lane].x;
      si += part[w][lane].y;
    }
    W[it.outRow + lane] = make_float2(sr, si);
  }
}

// R > 1 (FP32): one CTA of 4 warps per (item, tile of RT right-hand sides),
// lane = row; warp w multiplies columns w, w + 4, ... of every block.  The
// input rows are copied into shared memory a chunk ahead (cp.async) and read
// as broadcasts, two complex values a load; the factor entries go from global
// memory to registers, a batch of four columns a warp ahead over chunk and
// block ends.  A complex product is two packed FMAs (fma.rn.f32x2):
// (p, q) += a.re (x.re, x.im) and (u, v) += a.im (x.re, x.im), and y =
// (p - v, q + u) at the end, so nothing is swapped or negated on the way.
// Bound by issue and load latency together (at 8 right-hand sides HBM 32 %,
// FMA pipe 49 % busy; at 64 the FMA pipe 65 %).  Measured at 32,768 points
// (us; before: synchronous tiles up to 8 right-hand sides, a shared-memory
// pipeline with a 4 x 4 register tile above): R = 2 375 -> 161, R = 4 378 ->
// 177, R = 8 385 -> 220, R = 16 408 -> 317, R = 64 1,290 -> 1,020.  Two batches
// ahead (more registers) 237 and 367 us at R = 8 and 16; 64 registers for more
// warps 223 and, at 96, 430.
constexpr int kRhsWarps = 4, kRhsCols = 64, kRhsAhead = 4;

__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t x) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(x));
}
__device__ __forceinline__ uint64_t dup2(float a) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

template <int RT>
__global__ void __launch_bounds__(32 * kRhsWarps) applyRhsKernel(
    ApplyItem const *__restrict__ items, ApplyContrib const *__restrict__ contribs,
    float2 const *__restrict__ arena, float2 const *X, int64_t ldx, float2 *W, int64_t R,
    unsigned tiles) {
  constexpr int S = kRhsWarps, KC = kRhsCols, U = kRhsAhead, TH = 32 * S;
  constexpr int kPanel = 2 * KC * RT, kPart = S * 32 * (RT + 1);
  __shared__ __align__(16) float2 smem[kPanel > kPart ? kPanel : kPart];
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the tiles of an item run side by side and read its blocks from HBM once
  ApplyItem const it = items[blockIdx.x / tiles];
  int64_t const r0 = (int64_t)(blockIdx.x % tiles) * RT;
  int const nr = (R - r0) < RT ? (int)(R - r0) : RT;
  int const row = lane < it.rows ? lane : 0;   // inactive lanes re-read row 0

  // the chunk being fetched: columns [j0, j0 + n) of contribution c
  int c = 0, j0 = 0, n = 0, lda = 0;
  float2 const *a = nullptr, *x = nullptr;
  int64_t xld = 0;
  ApplyContrib cb{};
  auto begin = [&]() {   // the next chunk (c < nContrib)
    if (j0 == 0) {
      cb = contribs[it.contrib0 + c];
      lda = cb.lda;
      xld = cb.inIsX ? ldx : R;
      x = (cb.inIsX ? X + cb.inRow * ldx : W + cb.inRow * R) + r0;
      a = arena + cb.aOff + row;
    } else {
      x += KC * xld;
      a += (int64_t)KC * lda;
    }
    n = min(KC, cb.n - j0);
    j0 += KC;
    if (j0 >= cb.n) {
      j0 = 0;
      ++c;
    }
  };
  // the chunk's input rows; zeros for the columns that fill its last batch
  auto copyX = [&](float2 *panel) {
    int const full = (n + S * U - 1) / (S * U) * (S * U);
    for (int e = tid; e < full * RT; e += TH) {
      int const col = e / RT, q = e % RT;
      if (col < n && q < nr) {
        unsigned const d = (unsigned)__cvta_generic_to_shared(panel + e);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(x + col * xld + q)
                     : "memory");
      } else {
        panel[e] = make_float2(0.f, 0.f);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // this warp's entries of the batch at column b of the chunk (a column past
  // the end re-reads the last one, against zeros)
  float2 av[U];
  auto loadA = [&](int b) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      av[u] = a[(int64_t)min(b + warp + u * S, n - 1) * lda];
  };

  uint64_t p[RT], w[RT];
#pragma unroll
  for (int q = 0; q < RT; ++q) p[q] = w[q] = 0ull;
  int slot = 0;
  bool more = it.nContrib > 0;
  if (more) {
    begin();
    copyX(smem);
    loadA(0);
  }
  while (more) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();   // the chunk has landed, and every warp has left the other panel
    float2 const *panel = smem + slot * KC * RT + warp * RT;
    int const nNow = n;
    for (int b = 0; b < nNow; b += S * U) {
      float2 now[U];
#pragma unroll
      for (int u = 0; u < U; ++u) now[u] = av[u];
      if (b + S * U < nNow) {
        loadA(b + S * U);
      } else if ((more = c < it.nContrib)) {
        begin();
        copyX(smem + (slot ^ 1) * KC * RT);
        loadA(0);
      }
      float2 const *xs = panel + b * RT;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        uint64_t const re = dup2(now[u].x), im = dup2(now[u].y);
        ulonglong2 const *xv = reinterpret_cast<ulonglong2 const *>(xs + u * S * RT);
#pragma unroll
        for (int q = 0; q < RT; q += 2) {
          ulonglong2 const v = xv[q / 2];
          fma2(p[q], re, v.x);
          fma2(w[q], im, v.x);
          fma2(p[q + 1], re, v.y);
          fma2(w[q + 1], im, v.y);
        }
      }
    }
    slot ^= 1;
  }
  __syncthreads();
  float2 *const part = smem;   // [warp][row][RT + 1]
#pragma unroll
  for (int q = 0; q < RT; ++q) {
    float2 const s = unpack2(p[q]), t = unpack2(w[q]);
    part[(warp * 32 + lane) * (RT + 1) + q] = make_float2(s.x - t.y, s.y + t.x);
  }
  __syncthreads();
  for (int e = tid; e < it.rows * RT; e += TH) {
    int const i = e / RT, q = e % RT;
    if (q >= nr) continue;
    float sr = 0.f, si = 0.f;
#pragma unroll
    for (int v = 0; v < S; ++v) {
      float2 const t = part[(v * 32 + i) * (RT + 1) + q];
      sr += t.x;
      si += t.y;
    }
    W[(it.outRow + i) * R + r0 + q] = make_float2(sr, si);
  }
}

__device__ __forceinline__ void addTerm(double &sr, double &si, double2 v) {
  sr += v.x;
  si += v.y;
}
__device__ __forceinline__ void addTerm(float &sr, float &si, float2 v) {
  sr += v.x;
  si += v.y;
}
__device__ __forceinline__ void addTerm(double &sr, double &si, float4 v) {   // double-float
  sr += (double)v.x + (double)v.y;
  si += (double)v.z + (double)v.w;
}

// The last sum and the input copy run with threadIdx.x over right-hand sides
// (a power of two of them; blockIdx.y over the rest of them where the rows are
// few) and threadIdx.y over rows, so that nothing is divided per element.  A
// row's terms (of type TW) are read four at a time, and where the rows alone leave the chip idle (kSplit) eight warps share
// them: one after the other, each waits for its base's load and its own
// (2,073 rows, one right-hand side: 13.7 -> 6.6 us).  kSys adds a
// boundary-integral system's other terms to the sum of the one right-hand
// side, a row's corrections shared by the eight warps too (as a kernel of
// its own, 9.4 us more).
template <typename TW, typename T2, bool kSplit, bool kSys>
__global__ void __launch_bounds__(256)
    applyReduceKernel(int32_t const *__restrict__ rowSeg, int64_t const *__restrict__ segStart,
                      int64_t const *__restrict__ segContrib0,
                      int64_t const *__restrict__ segBase, TW const *W, int64_t R, T2 *Y,
                      int64_t ldy, int64_t nRows, int64_t const *__restrict__ outPerm,
                      int64_t wTile, int64_t wTileStride, SystemTerms sys) {
  using T = typename Real<T2>::T;
  constexpr int U = 4, kParts = kSplit ? 8 : 1;
  __shared__ T2 part[kParts][32];
  int const z = kSplit ? threadIdx.z : 0;
  int64_t const ld = wTile ? wTile : R;
  int64_t const step = (int64_t)gridDim.x * blockDim.y;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.y; i0 < nRows; i0 += step) {
    int64_t const i = i0 + threadIdx.y;
    bool const live = i < nRows;
    int64_t di = 0, c0 = 0, c1 = 0, o = i;
    if (live) {
      int const s = rowSeg[i];
      di = i - segStart[s];
      c0 = segContrib0[s];
      c1 = segContrib0[s + 1];
      if (outPerm) o = outPerm[i];
    }
    if (i0 == blockIdx.x * (int64_t)blockDim.y) afterPrevious();
    for (int64_t r0 = blockIdx.y * (int64_t)blockDim.x; r0 < R;
         r0 += (int64_t)gridDim.y * blockDim.x) {
      int64_t const r = r0 + threadIdx.x;
      bool const mine = live && r < R;
      T sr = 0, si = 0;
      if (mine) {
        // W row-major (ld R), or tile-major: panels of wTile (16 or 32) columns
        TW const *Wc = (wTile ? W + (r >> (wTile == 16 ? 4 : 5)) * wTileStride + (r & (wTile - 1))
                              : W + r) + di * ld;
        for (int64_t c = c0 + z; c < c1; c += U * kParts) {
          TW v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            int64_t const cu = c + u * kParts;
            v[u] = Wc[segBase[cu < c1 ? cu : c] * ld];
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (c + u * kParts < c1) addTerm(sr, si, v[u]);
        }
        if constexpr (kSys) {
          for (int q = z; q < sys.nc; q += kParts) {
            double2 const c = sys.val[o * sys.nc + q], v = sys.xw[sys.col[o * sys.nc + q]];
            sr += c.x * v.x - c.y * v.y;
            si += c.x * v.y + c.y * v.x;
          }
          if (z == 0) {
            double2 const v = sys.x[o];
            sr += sys.shift * v.x;
            si += sys.shift * v.y;
          }
        }
      }
      if (kSplit) {
        int const l = threadIdx.y * blockDim.x + threadIdx.x;
        part[z][l] = mk2<T2>(sr, si);
        __syncthreads();
        if (z == 0) {
#pragma unroll
          for (int q = 1; q < kParts; ++q) {
            sr += part[q][l].x;
            si += part[q][l].y;
          }
        }
        __syncthreads();
      }
      if (z == 0 && mine) Y[o * ldy + r] = mk2<T2>(sr, si);
    }
  }
}

__device__ __forceinline__ void storeAs(double2 v, double2 *out) { *out = v; }
__device__ __forceinline__ void storeAs(double2 v, float4 *out) {
  float const xh = (float)v.x, yh = (float)v.y;
  *out = make_float4(xh, (float)(v.x - (double)xh), yh, (float)(v.y - (double)yh));
}

// the input of a system's apply: xw = w x, and the same in tree order
template <typename TO>
__global__ void gatherScaledKernel(SystemTerms sys, int64_t const *__restrict__ perm, int64_t n,
                                   TO *__restrict__ out) {
  afterPrevious();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t const p = perm[i];
    double const w = sys.w[p];
    double2 const x = sys.x[p], v = make_double2(w * x.x, w * x.y);
    sys.xw[p] = v;
    storeAs(v, out + i);
  }
}

template <typename T2>
__global__ void gatherRowsKernel(T2 const *X, int64_t ldx,
                                 int64_t const *__restrict__ perm, int64_t nRows, int64_t R,
                                 T2 *__restrict__ out, int64_t outTile, int64_t outTileStride) {
  afterPrevious();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.y + threadIdx.y; i < nRows;
       i += (int64_t)gridDim.x * blockDim.y) {
    T2 const *x = X + (perm ? perm[i] : i) * ldx;
    for (int64_t r = blockIdx.y * (int64_t)blockDim.x + threadIdx.x; r < R;
         r += (int64_t)gridDim.y * blockDim.x) {
      int64_t const o = outTile ? (r >> (outTile == 16 ? 4 : 5)) * outTileStride + i * outTile +
                                      (r & (outTile - 1))
                                : i * R + r;
      out[o] = x[r];
    }
  }
}

template <int RT>
cudaError_t launchRhs(ApplyItem const *items, int64_t nItems, ApplyContrib const *contribs,
                      float2 const *arena, float2 const *X, int64_t ldx, float2 *W, int64_t R,
                      cudaStream_t stream) {
  int64_t const tiles = (R + RT - 1) / RT;
  if (tiles > 0x7fffffff / nItems) return cudaErrorInvalidConfiguration;
  applyRhsKernel<RT><<<(unsigned)(nItems * tiles), 32 * kRhsWarps, 0, stream>>>(
      items, contribs, arena, X, ldx, W, R, (unsigned)tiles);
  return cudaGetLastError();
}

// Eight warps share a row's terms where the rows have eight of them on
// average and are few: 15,346 points on 64 circles 19 us, 26 unshared; but
// 65,536 points with three terms a row 13 us, 5.5 unshared
constexpr int64_t kReduceSplitOut = 1 << 17, kReduceSplitTerms = 8;

// 128 threads over (right-hand sides, rows): all right-hand sides up to 64
dim3 rowBlock(int64_t R) {
  unsigned x = 1;
  while (x < 64 && x < R) x *= 2;
  return dim3(x, 128 / x);
}

// the grid for that: thread blocks over rows, and over right-hand sides as far
// as the rows alone leave the chip idle (40 points, 65,536 right-hand sides in
// points' order and FP32: 1,350 us with 20 thread blocks a kernel, 246 so)
dim3 rowGrid(int64_t rowBlocks, int64_t R, dim3 block) {
  int64_t const cols = (R + block.x - 1) / block.x, want = (152 * 16 + rowBlocks - 1) / rowBlocks;
  return dim3((unsigned)rowBlocks, (unsigned)(cols < want ? cols : want));
}

int gridFor(int64_t total, int threads) {
  int64_t g = (total + threads - 1) / threads;
  if (g > 152 * 64) g = 152 * 64;
  return (int)(g < 1 ? 1 : g);
}

}  // namespace

int64_t reexpansionSmemBytes(int32_t m, int32_t n, int32_t warps) {
  return (int64_t)16 * (2 * (int64_t)m * m + 2 * (int64_t)m * warps) +
         reexpansionGeoBytes(m, n);
}

int64_t reexpansionGeoBytes(int32_t m, int32_t n) {
  return (int64_t)8 * (7 * (int64_t)m + 4 * (int64_t)n);
}

int64_t reexpansionScratchEntries(int32_t m, int32_t warps) {
  // M (2m x m), 2m per warp, m shared squared singular values
  int64_t e = 2 * (int64_t)m * m + 2 * (int64_t)m * warps + m;
  return (e + 15) & ~int64_t(15);
}

int32_t reexpansionClusterCtas() { return kClusterCtas; }

cudaError_t launchFillBlocks(FillDesc const *descs, int32_t nDesc, PointsDev src,
                             PointsDev tgt, KernelParams kp, double2 *arena,
                             int32_t maxProxyN, int32_t *status, cudaStream_t stream) {
  if (nDesc == 0) return cudaSuccess;
  size_t const smem = 4 * (size_t)(maxProxyN > 0 ? maxProxyN : 1) * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(fillBlocksKernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  fillBlocksKernel<<<nDesc, 256, smem, stream>>>(descs, src, tgt, kp, arena, status);
  return cudaGetLastError();
}

template <bool kDf>
cudaError_t launchReexpansionT(FillDesc const *descs, int32_t nDesc, PointsDev src,
                               KernelParams kp, int32_t cutMode, double cutTol,
                               double2 *arena, double2 *scratch, int64_t const *scratchOff,
                               int32_t *flags, int32_t *status, int32_t mode,
                               int32_t smemBytes, int32_t threads, cudaStream_t stream,
                               FillDesc const *members, int32_t const *groupStart) {
  if (nDesc == 0) return cudaSuccess;
  cudaError_t e;
  if (mode == 0) {
    e = cudaFuncSetAttribute(reexpansionKernel<0, kDf>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smemBytes);
    if (e != cudaSuccess) return e;
    reexpansionKernel<0, kDf><<<nDesc, threads, smemBytes, stream>>>(
        descs, src, kp, cutMode, cutTol, arena, scratch, scratchOff, flags, status, members,
        groupStart);
  } else if (mode == 1) {
    e = cudaFuncSetAttribute(reexpansionKernel<1, kDf>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smemBytes);
    if (e != cudaSuccess) return e;
    reexpansionKernel<1, kDf><<<nDesc, threads, smemBytes, stream>>>(
        descs, src, kp, cutMode, cutTol, arena, scratch, scratchOff, flags, status, members,
        groupStart);
  } else {
    e = cudaFuncSetAttribute(reexpansionKernel<2, kDf>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smemBytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nDesc * kClusterCtas, 1, 1);
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = (size_t)smemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, reexpansionKernel<2, kDf>, descs, src, kp, cutMode, cutTol,
                           arena, scratch, scratchOff, flags, status, members, groupStart);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

cudaError_t launchReexpansion(FillDesc const *descs, int32_t nDesc, PointsDev src,
                              KernelParams kp, int32_t cutMode, double cutTol,
                              double2 *arena, double2 *scratch, int64_t const *scratchOff,
                              int32_t *flags, int32_t *status, int32_t mode,
                              int32_t smemBytes, int32_t threads, int32_t doubleFloat,
                              cudaStream_t stream, FillDesc const *members,
                              int32_t const *groupStart) {
  if (doubleFloat)
    return launchReexpansionT<true>(descs, nDesc, src, kp, cutMode, cutTol, arena, scratch,
                                    scratchOff, flags, status, mode, smemBytes, threads, stream,
                                    members, groupStart);
  return launchReexpansionT<false>(descs, nDesc, src, kp, cutMode, cutTol, arena, scratch,
                                   scratchOff, flags, status, mode, smemBytes, threads, stream,
                                   members, groupStart);
}

cudaError_t launchDenseRows(PointsDev src, int64_t nSrc, PointsDev tgt,
                            int64_t const *rows, int64_t nRows, KernelParams kp,
                            double2 const *x, int64_t ldx, int64_t R, double2 *out,
                            int64_t ldo, cudaStream_t stream) {
  if (nRows == 0) return cudaSuccess;
  denseRowsKernel<<<(unsigned)nRows, 256, 0, stream>>>(src, nSrc, tgt, rows, kp, x, ldx, R,
                                                       out, ldo);
  return cudaGetLastError();
}

cudaError_t launchKernelMatrix(PointsDev src, int64_t n, PointsDev tgt, int64_t m,
                               KernelParams kp, double2 *out, cudaStream_t stream) {
  if (m * n == 0) return cudaSuccess;
  kernelMatrixKernel<<<gridFor(m * n, 256), 256, 0, stream>>>(src, n, tgt, m, kp, out);
  return cudaGetLastError();
}

cudaError_t launchFp64Rate(int32_t blocks, int32_t iters, double *out, cudaStream_t stream) {
  fp64RateKernel<<<(unsigned)blocks, 256, 0, stream>>>(iters, 0.5, out);
  return cudaGetLastError();
}

cudaError_t launchBessel01(double const *x, int64_t n, double *out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  bessel01Kernel<<<gridFor(n, 256), 256, 0, stream>>>(x, n, out);
  return cudaGetLastError();
}

cudaError_t launchArenaToF32(double2 const *a64, float2 *a32, int64_t n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  arenaToF32Kernel<<<gridFor(n, 256), 256, 0, stream>>>(a64, a32, n);
  return cudaGetLastError();
}

cudaError_t launchC128ToC64(double2 const *a, int64_t lda, int64_t rows, int64_t cols,
                            float2 *b, int64_t ldb, cudaStream_t stream, int64_t bTile,
                            int64_t bTileStride) {
  if (rows * cols == 0) return cudaSuccess;
  c128ToC64Kernel<<<gridFor(rows * cols, 256), 256, 0, stream>>>(a, lda, rows, cols, b, ldb,
                                                                 bTile, bTileStride);
  return cudaGetLastError();
}

cudaError_t launchC64ToC128(float2 const *a, int64_t lda, int64_t rows, int64_t cols,
                            double2 *b, int64_t ldb, cudaStream_t stream) {
  if (rows * cols == 0) return cudaSuccess;
  c64ToC128Kernel<<<gridFor(rows * cols, 256), 256, 0, stream>>>(a, lda, rows, cols, b, ldb);
  return cudaGetLastError();
}

cudaError_t launchApplyStage(ApplyItem const *items, int64_t nItems,
                             ApplyContrib const *contribs, float2 const *arena,
                             float2 const *X, int64_t ldx, float2 *W, int64_t R,
                             cudaStream_t stream) {
  if (nItems == 0) return cudaSuccess;
  if (R == 1) {
    applyGemvKernel<<<(unsigned)nItems, 32 * kGemvWarps, 0, stream>>>(items, contribs, arena, X,
                                                                      ldx, W);
    return cudaGetLastError();
  }
  // the narrowest tile that holds the right-hand sides
  if (R <= 2) return launchRhs<2>(items, nItems, contribs, arena, X, ldx, W, R, stream);
  if (R <= 4) return launchRhs<4>(items, nItems, contribs, arena, X, ldx, W, R, stream);
  if (R <= 8) return launchRhs<8>(items, nItems, contribs, arena, X, ldx, W, R, stream);
  return launchRhs<16>(items, nItems, contribs, arena, X, ldx, W, R, stream);
}

template <typename TW, typename T2>
cudaError_t launchApplyReduce(int32_t const *rowSeg, int64_t const *segStart,
                              int64_t const *segContrib0, int64_t const *segBase,
                              int64_t nTerms, TW const *W, int64_t R, T2 *Y, int64_t ldy,
                              int64_t nRows, int64_t const *outPerm,
                              cudaStream_t stream, int64_t wTile, int64_t wTileStride,
                              SystemTerms const *sys) {
  if (wTile != 0 && wTile != 16 && wTile != 32) return cudaErrorInvalidValue;
  if (sys && R != 1) return cudaErrorInvalidValue;
  bool const split = nRows * R < kReduceSplitOut && nTerms >= kReduceSplitTerms * nRows;
  dim3 block = rowBlock(R);
  if (split) {
    unsigned const x = block.x < 32 ? block.x : 32;
    block = dim3(x, 32 / x, 8);
  }
  auto run = [&](auto kernel) {
    return launchAfter(kernel, rowGrid(gridFor(nRows, block.y), R, block), block, 0, stream, rowSeg,
                       segStart,
                       segContrib0, segBase, W, R, Y, ldy, nRows, outPerm, wTile, wTileStride,
                       sys ? *sys : SystemTerms{});
  };
  if constexpr (std::is_same_v<T2, double2>) {
    if (sys) {
      return split ? run(applyReduceKernel<TW, T2, true, true>)
                   : run(applyReduceKernel<TW, T2, false, true>);
    }
  }
  return split ? run(applyReduceKernel<TW, T2, true, false>)
               : run(applyReduceKernel<TW, T2, false, false>);
}

template <typename TO>
cudaError_t launchGatherScaled(SystemTerms const &sys, int64_t const *perm, int64_t n, TO *out,
                               cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  return launchAfter(gatherScaledKernel<TO>, dim3(gridFor(n, 64)), dim3(64), 0, stream, sys, perm, n,
                     out);
}
template cudaError_t launchGatherScaled<double2>(SystemTerms const &, int64_t const *, int64_t,
                                                 double2 *, cudaStream_t);
template cudaError_t launchGatherScaled<float4>(SystemTerms const &, int64_t const *, int64_t,
                                                float4 *, cudaStream_t);

template <typename T2>
cudaError_t launchGatherRows(T2 const *X, int64_t ldx, int64_t const *perm,
                             int64_t nRows, int64_t R, T2 *out, cudaStream_t stream,
                             int64_t outTile, int64_t outTileStride) {
  if (outTile != 0 && outTile != 16 && outTile != 32) return cudaErrorInvalidValue;
  dim3 const block = rowBlock(R);
  return launchAfter(gatherRowsKernel<T2>, rowGrid(gridFor(nRows, block.y), R, block), block, 0,
                     stream, X, ldx, perm, nRows, R, out, outTile, outTileStride);
}

template cudaError_t launchApplyReduce<double2, double2>(
    int32_t const *, int64_t const *, int64_t const *, int64_t const *, int64_t, double2 const *, int64_t,
    double2 *, int64_t, int64_t, int64_t const *, cudaStream_t, int64_t, int64_t, SystemTerms const *);
template cudaError_t launchApplyReduce<float2, float2>(
    int32_t const *, int64_t const *, int64_t const *, int64_t const *, int64_t, float2 const *, int64_t,
    float2 *, int64_t, int64_t, int64_t const *, cudaStream_t, int64_t, int64_t, SystemTerms const *);
template cudaError_t launchApplyReduce<float4, double2>(
    int32_t const *, int64_t const *, int64_t const *, int64_t const *, int64_t, float4 const *, int64_t,
    double2 *, int64_t, int64_t, int64_t const *, cudaStream_t, int64_t, int64_t, SystemTerms const *);
template cudaError_t launchGatherRows<double2>(double2 const *, int64_t, int64_t const *, int64_t,
                                               int64_t, double2 *, cudaStream_t, int64_t, int64_t);
template cudaError_t launchGatherRows<float2>(float2 const *, int64_t, int64_t const *, int64_t,
                                              int64_t, float2 *, cudaStream_t, int64_t, int64_t);

}  // namespace bfg
