// Randomized re-expansion of FIRST/MIDDLE blocks (sm_103a, FP64).
//
// The reference computes every re-expansion block as
//   Z_shift = pinv(Z_equiv) Z_orig          (helm2.c:321-365,
//                                            mat_dense_complex.c:1768-1849)
// with Z_equiv p x p and p the a-priori rank estimate of helm2.c:14-36,
// p = k r1 r2 / (R - r1 - r2) - log10(eps).  That estimate divides by the
// gap between the two proxy circles, so for nearly touching circles p is many
// times the numerical rank of Z_equiv, which follows k r1 r2 / R: at 262,144
// points and k = 2048 a block with p = 9,982 has 482 singular values above
// 1e-13 sigma0, and one with p = 3,710 has 173 above 1e-12 sigma0.  The
// reference's SVD spends O(p^3) on directions that the pseudo-inverse cut
// then drops.  This path spends its work on the numerical rank instead
// (a randomized range finder; Halko, Martinsson and Tropp, SIAM Review 53,
// 2011, algorithms 4.1 and 5.1), its results in FP64 precision (only the
// Jacobi's first sweeps run in FP32; the products are exact digit sums,
// bfg_fixed.cuh):
//
//   Y  = Z_equiv Omega        Omega p x l with iid complex Gaussian entries
//   Q  = qr(Y)                Householder (explicit Q, p x l)
//   G  = Z_equiv^H Q          so Z_equiv ~ Q G^H
//   G  = Q2 R2                Householder
//   [R2^H ; I] W  ->  [T ; W] one-sided Jacobi, first in FP32, then in FP64:
//                             T = R2^H W has orthogonal columns,
//                             sigma_a = |t_a|, W unitary
//   Z_equiv ~ (Q T diag(1/sigma)) diag(sigma) (Q2 W)^H, hence
//   Z_shift = Q2 (W (diag(w) (T^H (Q^H Z_orig))))
//             with w_a = 1/sigma_a^2 for sigma_a >= cut, else 0 -- the
//             reference's cut rule applied to the same singular values.
//
// The sketch is accepted when its smallest sigma_a lies below
// capture * sigma_max: Y then reached Z_equiv's rounding floor (about 1e-14
// sigma0 for these kernels), so Q holds every direction above the cut to
// within that floor.  Otherwise the block is sketched again with l doubled.
// No atomics: results are reproducible bit for bit.
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include <algorithm>
#include <array>
#include <map>
#include <climits>
#include <cmath>
#include <cstdint>
#include <vector>

#include "bfg_device.cuh"
#include "bfg_fixed.cuh"
#include "bfg_kernels.cuh"

namespace bfg {

namespace {

constexpr double kEpsS = 2.220446049250313e-16;
constexpr int kSketchMaxSweeps = 60;
constexpr int kSketchCluster = 8;      // CTAs per block in cluster mode
constexpr int kGM = 64, kGN = 32;      // GEMM tile
constexpr int kFillTile = 16384;       // entries per fill CTA

// one block of the randomized path, as the kernels read it (offsets in
// complex entries from the scratch base)
struct SketchDev {
  int32_t kind, p, n, l;
  int64_t arenaOff, s0;
  double corig[3], ceq[3], cchk[3];
  double k;
  uint64_t seed;
  int64_t oZ, oB0, oB1, oB2, oM, oZo, oC, oD, oTau, oSW, oFlags;
  int64_t oStep;
  int64_t oT, oTo;   // unit circles: p points, and (MIDDLE) the n source points
};

struct FillTileDesc {
  int32_t blk, what;        // what: 0 Z_equiv, 1 Omega, 2 Z_orig
  int32_t cnt, pad;
  int64_t e0;
};

struct GemmDesc {
  double2 const *A, *B;
  double2 *C;
  double const *rowScale;   // optional: row i of C scaled by rowScale[i]
  int64_t lda, ldb, ldc;
  int32_t M, N, K, opA;     // opA 0: A is M x K; 1: C = A^H B with A stored K x M
  double const *colScale;   // optional: column j of C scaled by colScale[j]
  int32_t newton = 0;       // 1: C = 3/2 I - 1/2 op(A) B instead
  int16_t *rowCode = nullptr, *colCode = nullptr;   // scale codes of op(A)'s rows and B's
                                                    // columns (set at launch)
};

struct HqrDesc {
  double2 *A;     // rows x cols, ld rows: overwritten by the reflectors and R
  double2 *Q;     // rows x cols, ld rows: receives the explicit Q
  double2 *tau;   // cols
  double2 *step;  // 4 entries: the reflector in hand (cluster mode)
  double2 *Rt;    // optional: R^H (cols x cols, lower triangular) and the
                  // identity below it, ld = 2 cols
  int32_t rows, cols;
};

struct JacobiDesc {
  double2 *M;     // ld x cols; dot products over the first rowsDot rows,
                  // rotations over all ld rows
  double *s2;     // cols: squared column norms over the first rowsDot rows
  int32_t *flags; // kSketchCluster ints (cluster mode)
  int32_t cols, rowsDot, ld, pad;
};

struct WeightDesc {
  double const *s2;
  double *w;
  int32_t cols, p;          // p: order of Z_equiv (the reference cut's max(m, n))
};

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// a complex Gaussian with iid N(0,1) parts from a counter (Box-Muller)
__device__ __forceinline__ double2 gaussianAt(uint64_t seed, int64_t e) {
  uint64_t const h1 = splitmix64(seed ^ ((uint64_t)e * 0xD1B54A32D192ED03ull));
  uint64_t const h2 = splitmix64(h1);
  double const u1 = ((double)(h1 >> 11) + 0.5) * 0x1.0p-53;
  double const u2 = (double)(h2 >> 11) * 0x1.0p-53;
  double const r = sqrt(-2.0 * log(u1));
  double s, c;
  sincospi(2.0 * u2, &s, &c);
  return make_double2(r * c, r * s);
}

template <int kMode>
struct SMem {
  static __device__ __forceinline__ double2 ld(double2 const *p) {
    if (kMode == 2) return __ldcg(p);   // other CTAs of the cluster write it
    return *p;
  }
  static __device__ __forceinline__ void st(double2 *p, double2 v) {
    if (kMode == 2) __stcg(p, v);
    else *p = v;
  }
  static __device__ __forceinline__ void sync() {
    if (kMode == 2) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  }
};

__device__ __forceinline__ double2 conjD(double2 a) { return make_double2(a.x, -a.y); }

// ---------------------------------------------------------------------------
// Z_equiv, Omega and Z_orig of every block, column-major (entry e: row
// e % p, column e / p).  Proxy points are those of the full path: theta_a =
// (2 pi / p) a on the check and equivalent circles, (2 pi / n) b on the
// source-child circle of a MIDDLE block.
// ---------------------------------------------------------------------------
// (cos, sin) of theta_a = (2 pi / p) a of every group (blocks 0 .. nGroups-1)
// and of (2 pi / n) b of every MIDDLE member: one sincos a point, not one for
// both points of every entry
__global__ void __launch_bounds__(256) sketchCircleKernel(SketchDev const *__restrict__ blks,
                                                          int nGroups, double2 *scratch) {
  SketchDev const b = blks[blockIdx.x];
  bool const group = (int)blockIdx.x < nGroups;
  if (!group && b.kind == kFirst) return;
  int const n = group ? b.p : b.n;
  double2 *out = scratch + (group ? b.oT : b.oTo);
  double const scale = kTwoPiDev / (double)n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double s, c;
    sincos(scale * i, &s, &c);
    out[i] = make_double2(c, s);
  }
}

__global__ void __launch_bounds__(256) sketchFillKernel(SketchDev const *__restrict__ blks,
                                                        FillTileDesc const *__restrict__ tiles,
                                                        PointsDev src, KernelParams kp,
                                                        double2 *scratch) {
  FillTileDesc const t = tiles[blockIdx.x];
  SketchDev const b = blks[t.blk];
  kp.k = b.k;
  int const p = b.p;
  bool const useSrcN = kp.layerPot == kLpPvDouble || kp.layerPot == kLpCombinedField;
  double2 *out = scratch + (t.what == 0 ? b.oZ : t.what == 1 ? b.oB0 : b.oZo);
  double2 const *circ = scratch + b.oT, *circo = scratch + b.oTo;
  for (int q = threadIdx.x; q < t.cnt; q += blockDim.x) {
    int64_t const e = t.e0 + q;
    if (t.what == 1) {
      out[e] = gaussianAt(b.seed, e);
      continue;
    }
    int const i = (int)(e % p);
    int64_t const j = e / p;
    double2 const u = circ[i];
    double const tx = b.cchk[2] * u.x + b.cchk[0], ty = b.cchk[2] * u.y + b.cchk[1];
    double sx, sy, snx, sny;
    if (t.what == 0 || b.kind != kFirst) {
      double2 const v = t.what == 0 ? circ[j] : circo[j];
      double const *cc = t.what == 0 ? b.ceq : b.corig;
      sx = cc[2] * v.x + cc[0];
      sy = cc[2] * v.y + cc[1];
      snx = v.x;
      sny = v.y;
    } else {
      int64_t const sj = b.s0 + j;
      sx = src.x[sj];
      sy = src.y[sj];
      snx = (useSrcN && src.nx) ? src.nx[sj] : 0.0;
      sny = (useSrcN && src.ny) ? src.ny[sj] : 0.0;
    }
    out[e] = kernelValue(kp, tx, ty, 0.0, 0.0, sx, sy, snx, sny);
  }
}

// ---------------------------------------------------------------------------
// Batched complex FP64 GEMM, C = diag(rowScale) op(A) B diag(colScale), one
// 64 x 32 tile per CTA (tiles of all problems in one launch), the products
// formed from integer digits on the tensor cores (bfg_fixed.cuh).  A row of
// op(A) and a column of B have one scale each (gemmCodeKernel, one pass over
// the operands); a tile that meets a row or column without one (NaN,
// infinities, subnormals) is summed in plain FP64.
//
// 8 warps: four 16-row tiles times two groups of 16 columns.  Per k-step of 8:
// each thread splits two entries of A and one of B into shared memory in the
// fragments' order -- while the MMAs of the step before run from the other
// buffer -- and fetches the ones after.  34 MMAs of 16 x 8 x 16 per four
// columns; the exact sums go to FP64 every kFixMaxSteps k-steps.
// Bound by the tensor pipe and by splitting the entries.  Measured, against the
// FP64-FMA form (64 x 64 tiles, FP64 pipe 99.9 % busy): all products of the
// 65,536-point factorization 296 -> 52 ms (the output products 225 -> 41), of
// twelve problems of up to 16,384 points 257 -> 45 ms.
// ---------------------------------------------------------------------------
// Seven digits: t = trunc(v 2^(1077 - E)), |t| <= 2^55, |d_k| <= 129, and the
// products of digits i + j <= 7 (34 of 49): an entry is off by less than 2^-54
// of the largest of its row or column, and so is a product.
constexpr int kGemmDigits = 7;
constexpr int kGemmStageWords = kGemmDigits * (4 * 32 * 4 + 8 * 32 * 2);
static_assert(7 * kFixMaxSteps * 16 * 129 * 129 < 1 << 24, "exact FP32 sums");

// the exact sum put together from the digit sums' element r, in units of 2^56
// (rounded), which are cleared
__device__ __forceinline__ int64_t gemmTake(float (&sum)[kFixSums][4], int r) {
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

__device__ __forceinline__ double2 gemmA(GemmDesc const &g, int i, int k) {
  if (i >= g.M || k >= g.K) return make_double2(0.0, 0.0);
  return g.opA == 0 ? g.A[i + (int64_t)k * g.lda] : conjD(g.A[k + (int64_t)i * g.lda]);
}
__device__ __forceinline__ double2 gemmB(GemmDesc const &g, int k, int j) {
  return (j < g.N && k < g.K) ? g.B[k + (int64_t)j * g.ldb] : make_double2(0.0, 0.0);
}

// scale codes of 64 rows of op(A) (what 0) or of 64 columns of B (what 1):
// tile (desc, what, first row or column)
__global__ void __launch_bounds__(256) gemmCodeKernel(GemmDesc const *__restrict__ descs,
                                                      int4 const *__restrict__ tiles) {
  int4 const t = tiles[blockIdx.x];
  GemmDesc const g = descs[t.x];
  int const tid = threadIdx.x;
  if (t.y == 0 && g.opA == 0) {   // along the stored rows: 64 rows, 4 column slices
    __shared__ int red[4][64];
    int const i = t.z + (tid & 63);
    int code = 0;
    for (int k = tid >> 6; k < g.K; k += 4) code = max(code, fixCode(gemmA(g, i, k)));
    red[tid >> 6][tid & 63] = code;
    __syncthreads();
    if (tid < 64 && i < g.M)
      g.rowCode[i] = (int16_t)fixScaleOf(
          max(max(red[0][tid], red[1][tid]), max(red[2][tid], red[3][tid])));
    return;
  }
  int const lane = tid & 31, n = t.y == 0 ? g.M : g.N;
  double2 const *p = t.y == 0 ? g.A : g.B;
  int64_t const ld = t.y == 0 ? g.lda : g.ldb;
  for (int q = tid >> 5; q < 64 && t.z + q < n; q += 8) {   // a stored column per warp
    int code = 0;
    for (int k = lane; k < g.K; k += 32) code = max(code, fixCode(p[k + (t.z + q) * ld]));
    code = __reduce_max_sync(0xffffffffu, code);
    if (lane == 0) (t.y == 0 ? g.rowCode : g.colCode)[t.z + q] = (int16_t)fixScaleOf(code);
  }
}

__global__ void __launch_bounds__(256, 1) zgemmKernel(GemmDesc const *__restrict__ descs,
                                                      int4 const *__restrict__ tiles) {
  constexpr int D = kGemmDigits;
  extern __shared__ __align__(16) uint32_t gemmSmem[];   // two stages
  __shared__ int16_t sRow[kGM], sCol[kGN];
  int4 const tile = tiles[blockIdx.x];
  GemmDesc const g = descs[tile.x];
  int const i0 = tile.y * kGM, j0 = tile.z * kGN;
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t = lane & 3, gr = lane >> 2;
  int const mt = warp & 3, nh = warp >> 2;
  if (tid < kGM) sRow[tid] = i0 + tid < g.M ? g.rowCode[i0 + tid] : 1023;
  if (tid >= 64 && tid < 64 + kGN) sCol[tid - 64] = j0 + tid - 64 < g.N ? g.colCode[j0 + tid - 64] : 1023;
  __syncthreads();
  bool covered = true;
  for (int e = tid; e < kGM * kGN; e += 256)
    covered = covered && fixCovers(sRow[e % kGM], sRow[e % kGM], sCol[e / kGM]);
  bool const plain = __syncthreads_or(!covered);

  // this lane's results: rows 16 mt + gr, + 8; columns 16 nh + 4 u + t
  double acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[u][r] = 0.0;

  if (!plain) {
    float sum[4][kFixSums][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int s = 0; s < kFixSums; ++s)
#pragma unroll
        for (int r = 0; r < 4; ++r) sum[u][s][r] = 0.f;
    // the entries this thread splits: of A, row 16 (warp / 2) + gr + 8 h with
    // h = warp % 2 at columns t and t + 4; of B, columns 8 (warp / 2) + gr at
    // row t + 4 h
    int const h = warp & 1, ra = 16 * (warp >> 1) + gr + 8 * h, cb = 8 * (warp >> 1) + gr;
    int const ea = sRow[ra], eb = sCol[cb];
    double2 a0, a1, b0;
    auto fetch = [&](int k0) {
      a0 = gemmA(g, i0 + ra, k0 + t);
      a1 = gemmA(g, i0 + ra, k0 + t + 4);
      b0 = gemmB(g, k0 + t + 4 * h, j0 + cb);
    };
    // A: word ((digit 4 + row tile) 32 + lane) 4 + register (register h of
    // column t, 2 + h of t + 4); B: word ((digit 8 + n tile) 32 + lane) 2 +
    // register
    auto put = [&](uint32_t *sA) {
      uint32_t *sB = sA + D * 4 * 32 * 4;
      uint32_t d[D];
      fixSplit(a0, ea, d);
      uint32_t *p = sA + ((warp >> 1) * 32 + lane) * 4 + h;
#pragma unroll
      for (int q = 0; q < D; ++q) p[q * 512] = d[q];
      fixSplit(a1, ea, d);
#pragma unroll
      for (int q = 0; q < D; ++q) p[q * 512 + 2] = d[q];
      fixSplit(b0, eb, d);
      p = sB + ((cb >> 2) * 32 + 8 * (cb & 3) + t) * 2 + h;
#pragma unroll
      for (int q = 0; q < D; ++q) {
        p[q * 512] = d[q] ^ 0x80000000u;              // (Re b, -Im b)
        p[q * 512 + 8] = __byte_perm(d[q], 0, 0x1032);   // (Im b, Re b)
      }
    };
    int const ea0 = sRow[16 * mt + gr], ea1 = sRow[16 * mt + gr + 8];
    auto flush = [&]() {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        int const ec = sCol[16 * nh + 4 * u + t];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          acc[u][r] = fma((double)gemmTake(sum[u], r),
                          fixPow((r < 2 ? ea0 : ea1) + ec - 1075), acc[u][r]);
      }
    };
    fetch(0);
    put(gemmSmem);
    fetch(8);
    int buf = 0, steps = 0;
    for (int k0 = 0; k0 < g.K; k0 += 8, buf ^= 1) {
      __syncthreads();
      if (k0 + 8 < g.K) {
        put(gemmSmem + (buf ^ 1) * kGemmStageWords);
        if (k0 + 16 < g.K) fetch(k0 + 16);
      }
      uint4 const *sA = reinterpret_cast<uint4 const *>(gemmSmem + buf * kGemmStageWords) +
                        mt * 32 + lane;
      uint2 const *sB = reinterpret_cast<uint2 const *>(gemmSmem + buf * kGemmStageWords +
                                                        D * 4 * 32 * 4) + nh * 4 * 32 + lane;
#pragma unroll
      for (int i = 0; i < D; ++i) {
        uint4 const a = sA[i * 128];
#pragma unroll
        for (int j = 0; j < D && i + j < kFixSums; ++j)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint2 const b = sB[(j * 8 + u) * 32];
            fixMma(sum[u][i + j], a.x, a.y, a.z, a.w, b.x, b.y);
          }
      }
      if (++steps == kFixMaxSteps) {
        flush();
        steps = 0;
      }
    }
    if (steps > 0) flush();
  } else {
    for (int k = 0; k < g.K; ++k) {
      double2 const x0 = gemmA(g, i0 + 16 * mt + gr, k), x1 = gemmA(g, i0 + 16 * mt + gr + 8, k);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        double2 const y = gemmB(g, k, j0 + 16 * nh + 4 * u + t);
        cmacc(acc[u][0], acc[u][1], x0, y);
        cmacc(acc[u][2], acc[u][3], x1, y);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    int const j = j0 + 16 * nh + 4 * u + t;
    if (j >= g.N) continue;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      int const i = i0 + 16 * mt + gr + 8 * r;
      if (i >= g.M) continue;
      double const sc = g.rowScale ? g.rowScale[i] : 1.0;
      double const scc = g.newton ? -0.5 : g.colScale ? sc * g.colScale[j] : sc;
      double2 v = make_double2(scc * acc[u][2 * r], scc * acc[u][2 * r + 1]);
      if (g.newton && i == j) v.x += 1.5;
      g.C[i + (int64_t)j * g.ldc] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// Householder QR (LAPACK zgeqr2 / zlarfg conventions: H = I - tau v v^H,
// v_0 = 1, H^H [alpha; x] = [beta; 0] with beta real) and the explicit Q
// (zung2r), one block per CTA (mode 1) or per cluster of kSketchCluster
// CTAs (mode 2).  Half a warp updates a trailing column; the one that updates
// column k + 1 goes on to that column's reflector (its norm, square root and
// divisions) while the others update the rest, so a step ends at one barrier.
// CTA 0 stores the scaled reflector of column k while the others work on
// step k + 1, which no longer reads it.
//
// Bound by the FP64 pipe, where a warp instruction takes 16 clocks of the SM
// whatever its lanes do: a column's sums and coefficients take as many as its
// products at 60 rows, hence two columns a warp, and a reflector's scalars
// about eighty, hence one warp instead of all 16.  Measured, both QRs of
// a factorization: 126 -> 87 ms at 65,536 points (k = 512), 171 -> 73 ms for
// twelve problems of up to 16,384 points, 7.0 -> 3.8 ms at 4,096.
// ---------------------------------------------------------------------------
// the sums of a and b over each half warp, in every lane of the half
__device__ __forceinline__ void halfSum2(double &a, double &b) {
  int const lane = threadIdx.x & 31;
  bool const hi = lane & 8;
  double v = hi ? b : a;
  v += __shfl_xor_sync(0xffffffffu, hi ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  a = __shfl_sync(0xffffffffu, v, lane & 16);
  b = __shfl_sync(0xffffffffu, v, (lane & 16) | 8);
}

// the reflector of [alpha; x], s = |x|^2: v = [1; sc x]
struct Reflector {
  double2 tau, sc;
  double beta;
  __device__ __forceinline__ void form(double2 alpha, double s) {
    if (s == 0.0 && alpha.y == 0.0) {
      tau = sc = make_double2(0.0, 0.0);
      beta = alpha.x;
    } else {
      beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + s), alpha.x);
      tau = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
      double2 const den = make_double2(alpha.x - beta, alpha.y);   // sc = 1 / (alpha - beta)
      double const dd = den.x * den.x + den.y * den.y;
      sc = make_double2(den.x / dd, -den.y / dd);
    }
  }
};

template <int kMode>
__global__ void __launch_bounds__(512) hqrKernel(HqrDesc const *__restrict__ descs) {
  using Mem = SMem<kMode>;
  int const ctas = kMode == 2 ? kSketchCluster : 1;
  int const blk = kMode == 2 ? (int)(blockIdx.x / kSketchCluster) : (int)blockIdx.x;
  int const rank = kMode == 2 ? (int)(blockIdx.x % kSketchCluster) : 0;
  HqrDesc const d = descs[blk];
  int const m = d.rows, nc = d.cols;
  int const tid = threadIdx.x, nthr = blockDim.x;
  int const lane = tid & 31, warp = tid >> 5, nWarps = nthr >> 5;
  int const hl = lane & 15, half = lane >> 4;
  int const gWarp = rank * nWarps + warp, gWarps = ctas * nWarps;
  __shared__ Reflector sRef[2];   // by the step's parity
  double2 *A = d.A;

  if (warp == 0 && nc > 0) {   // (every CTA of a cluster: the same bits)
    double s = 0.0;
    for (int i = 1 + lane; i < m; i += 32) {
      double2 const v = Mem::ld(A + i);
      s = fma(v.x, v.x, fma(v.y, v.y, s));
    }
    s = warpSum(s);
    Reflector r;
    r.form(Mem::ld(A), s);
    if (lane == 0) sRef[0] = r;
    if (rank == 0 && lane == 0) Mem::st(d.tau, r.tau);
  }
  __syncthreads();
  Reflector prev{};
  for (int k = 0; k < nc; ++k) {
    double2 const *col = A + (int64_t)k * m;
    Reflector ref;
    if (kMode == 2 && k > 0) {   // formed by the cluster's first CTA
      double2 const *p = d.step + 2 * (k & 1);
      ref.sc = Mem::ld(p);
      ref.beta = Mem::ld(p + 1).x;
      ref.tau = Mem::ld(d.tau + k);
    } else {
      ref = sRef[k & 1];
    }
    if (rank == 0 && k > 0) {
      double2 *pc = A + (int64_t)(k - 1) * m;
      for (int i = k + tid; i < m; i += nthr) Mem::st(pc + i, cmul(prev.sc, Mem::ld(pc + i)));
      if (tid == 0) Mem::st(pc + (k - 1), make_double2(prev.beta, 0.0));
    }
    // a_j -= conj(tau) v (v^H a_j) for j > k, v = [1; sc x]
    for (int jb = k + 1 + 2 * gWarp; jb < nc; jb += 2 * gWarps) {
      bool const next = jb == k + 1;            // this warp's first half has column k + 1
      bool const on = jb + half < nc;
      double2 *cj = A + (int64_t)(on ? jb + half : jb) * m;
      double sr = 0.0, si = 0.0;
      for (int i = k + 1 + hl; i < m; i += 16) {
        double2 const x = Mem::ld(col + i), a = Mem::ld(cj + i);
        sr = fma(x.x, a.x, fma(x.y, a.y, sr));
        si = fma(x.x, a.y, fma(-x.y, a.x, si));
      }
      halfSum2(sr, si);
      double2 const akj = Mem::ld(cj + k);
      double2 const cs = cmul(conjD(ref.sc), make_double2(sr, si));
      double2 const w = make_double2(akj.x + cs.x, akj.y + cs.y);
      double2 const tw = cmul(conjD(ref.tau), w);
      double2 const f = cmul(ref.sc, tw);
      __syncwarp();
      if (on && hl == 0) Mem::st(cj + k, make_double2(akj.x - tw.x, akj.y - tw.y));
      double n2 = 0.0;
      double2 alpha = make_double2(0.0, 0.0);
      for (int i = k + 1 + hl; i < m; i += 16) {
        double2 const x = Mem::ld(col + i);
        double2 a = Mem::ld(cj + i);
        a.x = fma(-f.x, x.x, fma(f.y, x.y, a.x));
        a.y = fma(-f.x, x.y, fma(-f.y, x.x, a.y));
        if (on) Mem::st(cj + i, a);
        if (next) {
          if (i == k + 1) alpha = a;
          else n2 = fma(a.x, a.x, fma(a.y, a.y, n2));
        }
      }
      if (next) {
        double unused = 0.0;
        halfSum2(n2, unused);
        alpha.x = __shfl_sync(0xffffffffu, alpha.x, 0);
        alpha.y = __shfl_sync(0xffffffffu, alpha.y, 0);
        Reflector r;
        r.form(alpha, n2);
        if (lane == 0) {
          sRef[(k + 1) & 1] = r;
          Mem::st(d.tau + k + 1, r.tau);
          if (kMode == 2) {
            Mem::st(d.step + 2 * ((k + 1) & 1), r.sc);
            Mem::st(d.step + 2 * ((k + 1) & 1) + 1, make_double2(r.beta, 0.0));
          }
        }
      }
    }
    Mem::sync();
    prev = ref;
  }
  if (rank == 0 && nc > 0) {
    double2 *pc = A + (int64_t)(nc - 1) * m;
    for (int i = nc + tid; i < m; i += nthr) Mem::st(pc + i, cmul(prev.sc, Mem::ld(pc + i)));
    if (tid == 0) Mem::st(pc + (nc - 1), make_double2(prev.beta, 0.0));
  }
  Mem::sync();

  // R^H (lower triangular) and the identity below it
  if (d.Rt) {
    int64_t const ldR = 2 * (int64_t)nc, total = ldR * nc;
    for (int64_t e = (int64_t)rank * nthr + tid; e < total; e += (int64_t)ctas * nthr) {
      int const a = (int)(e % ldR), b = (int)(e / ldR);
      double2 v = make_double2(0.0, 0.0);
      if (a < nc) {
        if (a >= b) v = conjD(Mem::ld(A + b + (int64_t)a * m));
      } else if (a - nc == b) {
        v = make_double2(1.0, 0.0);
      }
      Mem::st(d.Rt + e, v);
    }
  }
  // Q = H_0 ... H_{nc-1} [I ; 0]
  double2 *Q = d.Q;
  {
    int64_t const total = (int64_t)m * nc;
    for (int64_t e = (int64_t)rank * nthr + tid; e < total; e += (int64_t)ctas * nthr)
      Mem::st(Q + e, make_double2((e % m) == (e / m) ? 1.0 : 0.0, 0.0));
  }
  Mem::sync();
  for (int i = nc - 1; i >= 0; --i) {
    double2 const t = Mem::ld(d.tau + i);
    double2 const *v = A + (int64_t)i * m;
    for (int jb = i + 2 * gWarp; jb < nc; jb += 2 * gWarps) {
      bool const on = jb + half < nc;
      double2 *qj = Q + (int64_t)(on ? jb + half : jb) * m;
      double sr = 0.0, si = 0.0;
      for (int r = i + 1 + hl; r < m; r += 16) {
        double2 const x = Mem::ld(v + r), a = Mem::ld(qj + r);
        sr = fma(x.x, a.x, fma(x.y, a.y, sr));
        si = fma(x.x, a.y, fma(-x.y, a.x, si));
      }
      halfSum2(sr, si);
      double2 const qij = Mem::ld(qj + i);
      double2 const w = make_double2(qij.x + sr, qij.y + si);
      double2 const tw = cmul(t, w);
      __syncwarp();
      if (on && hl == 0) Mem::st(qj + i, make_double2(qij.x - tw.x, qij.y - tw.y));
      if (on)
        for (int r = i + 1 + hl; r < m; r += 16) {
          double2 const x = Mem::ld(v + r);
          double2 q = Mem::ld(qj + r);
          q.x = fma(-tw.x, x.x, fma(tw.y, x.y, q.x));
          q.y = fma(-tw.x, x.y, fma(-tw.y, x.x, q.y));
          Mem::st(qj + r, q);
        }
    }
    Mem::sync();
  }
}

// ---------------------------------------------------------------------------
// One-sided Jacobi (Hestenes) on the columns of M, FP64: a round-robin pair
// schedule, one warp per column pair, rotation when |<x, y>| > eps sqrt(n)
// |x| |y|; sweeps until none rotates (cap kSketchMaxSweeps).  Then the
// squared column norms over the first rowsDot rows.
//
// Bound by the FP64 pipe, where a warp instruction takes 16 clocks of the SM
// whatever its lanes do.  A rotation's angle takes about a hundred of them
// (square roots, divisions), more than the products of a pair of 50-row
// columns: so a round goes in three steps -- every warp's dot products, the
// angles of up to kJacSlots pairs with one thread a pair, the rotations --
// and the angles cost one pair's instructions for 32 pairs.  The squared norms
// are formed once a sweep and follow the rotations (|x|^2 - t |<x, y>|,
// |y|^2 + t |<x, y>|): they only choose angles and say which pairs are done,
// the rotation is orthogonal whatever they are (make: 331 -> 319 ms at 65,536
// points, 387 -> 363 for the twelve problems).  Measured: the
// sweeps of the re-expansions 436 -> 234 ms at 65,536 points (k = 512), 762 ->
// 416 ms for twelve problems of up to 16,384 points, 21 -> 11 ms at 4,096 (and
// less again after the FP32 sweeps below).
// ---------------------------------------------------------------------------
constexpr int kJacPer = 8, kJacSlots = 16 * kJacPer;   // pairs a warp / a CTA of 16 warps a step

template <int kMode>
__global__ void __launch_bounds__(512) sketchJacobiKernel(JacobiDesc const *__restrict__ descs,
                                                          int32_t *status) {
  using Mem = SMem<kMode>;
  int const ctas = kMode == 2 ? kSketchCluster : 1;
  int const blk = kMode == 2 ? (int)(blockIdx.x / kSketchCluster) : (int)blockIdx.x;
  int const rank = kMode == 2 ? (int)(blockIdx.x % kSketchCluster) : 0;
  JacobiDesc const d = descs[blk];
  int const nc = d.cols, rd = d.rowsDot, LD = d.ld;
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nWarps = blockDim.x >> 5;
  int const gWarp = rank * nWarps + warp, gWarps = ctas * nWarps;
  double2 *M = d.M;
  __shared__ int sRotated;
  // pair k nWarps + w of a step: warp w's k-th; (-, -, <x, y>), then
  // the rotation (c, s, exp(-i phi)), c = 2 for none
  __shared__ double4 sPair[kJacSlots];
  static_assert(kJacSlots <= 512, "one thread a pair");

  int const P = nc + (nc & 1), nPairs = P / 2;
  double const tolRot = kEpsS * sqrt((double)rd);
  // the columns of pair pr of a round (false: the bye of an odd count)
  auto columns = [&](int round, int pr, int &i, int &j) {
    if (pr == 0) {
      i = round;
      j = P - 1;
    } else {
      i = round + pr;
      if (i >= P - 1) i -= P - 1;
      j = round - pr;
      if (j < 0) j += P - 1;
    }
    return i < nc && j < nc;
  };
  // |column|^2 over the first rowsDot rows of every column into d.s2
  auto norms = [&]() {
    for (int a = gWarp; a < nc; a += gWarps) {
      double2 const *ca = M + (int64_t)a * LD;
      double s2 = 0;
      for (int r = lane; r < rd; r += 32) {
        double2 const v = Mem::ld(ca + r);
        s2 += v.x * v.x + v.y * v.y;
      }
      s2 = warpSum(s2);
      if (lane == 0) __stcg(d.s2 + a, s2);
    }
  };
  bool converged = nc < 2;
  for (int sweep = 0; sweep < kSketchMaxSweeps && !converged; ++sweep) {
    if (tid == 0) sRotated = 0;
    norms();
    Mem::sync();
    for (int round = 0; round < P - 1; ++round) {
      for (int pr0 = 0; pr0 < nPairs; pr0 += gWarps * kJacPer) {
        // the pair whose angle this thread finds, its norms fetched ahead
        int const mine = pr0 + rank * nWarps + (tid / nWarps) * gWarps + tid % nWarps;
        bool const angle = tid < kJacPer * nWarps && mine < nPairs;
        int mi = 0, mj = 0;
        if (angle && !columns(round, mine, mi, mj)) mi = mj = 0;
        double const al = __ldcg(d.s2 + mi), be = __ldcg(d.s2 + mj);
        for (int k = 0, pr = pr0 + gWarp; k < kJacPer && pr < nPairs; ++k, pr += gWarps) {
          int i, j;
          double gr = 0, gi = 0;
          if (columns(round, pr, i, j)) {
            double2 const *ci = M + (int64_t)i * LD, *cj = M + (int64_t)j * LD;
            for (int r = lane; r < rd; r += 32) {
              double2 const x = Mem::ld(ci + r), y = Mem::ld(cj + r);
              gr = fma(x.x, y.x, fma(x.y, y.y, gr));
              gi = fma(x.x, y.y, fma(-x.y, y.x, gi));
            }
          }
          // (a bye's zeros do not rotate)
          double const v = warpSum2(gr, gi);
          if ((lane & 15) == 0)
            reinterpret_cast<double *>(sPair + k * nWarps + warp)[2 + (lane >> 4)] = v;
        }
        __syncthreads();
        if (angle) {
          double const gr = sPair[tid].z, gi = sPair[tid].w;
          double4 rot = make_double4(2.0, 0.0, 0.0, 0.0);
          double const ag = sqrt(gr * gr + gi * gi);
          if (ag > tolRot * sqrt(al * be) && ag > 0.0) {
            double const zeta = (be - al) / (2.0 * ag);
            double const t = (zeta >= 0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
            double const c = 1.0 / sqrt(1.0 + t * t);
            rot = make_double4(c, c * t, gr / ag, -gi / ag);
            __stcg(d.s2 + mi, fmax(al - t * ag, 0.0));
            __stcg(d.s2 + mj, fmax(be + t * ag, 0.0));
            sRotated = 1;
          }
          sPair[tid] = rot;
        }
        __syncthreads();
        for (int k = 0, pr = pr0 + gWarp; k < kJacPer && pr < nPairs; ++k, pr += gWarps) {
          double4 const rot = sPair[k * nWarps + warp];
          if (rot.x > 1.5) continue;
          double const c = rot.x, s = rot.y, er = rot.z, ei = rot.w;
          int i, j;
          columns(round, pr, i, j);
          double2 *ci = M + (int64_t)i * LD, *cj = M + (int64_t)j * LD;
          // x <- c x - w y, y <- c y + conj(w) x (a column's phase is free)
          double const wr = s * er, wi = s * ei;
          if (c == 1.0) {
            // most of the rotations after the first-order step: a third fewer FMAs
            for (int r = lane; r < LD; r += 32) {
              double2 const x = Mem::ld(ci + r), y = Mem::ld(cj + r);
              Mem::st(ci + r, make_double2(fma(-wr, y.x, fma(wi, y.y, x.x)),
                                           fma(-wr, y.y, fma(-wi, y.x, x.y))));
              Mem::st(cj + r, make_double2(fma(wr, x.x, fma(wi, x.y, y.x)),
                                           fma(wr, x.y, fma(-wi, x.x, y.y))));
            }
            continue;
          }
          for (int r = lane; r < LD; r += 32) {
            double2 const x = Mem::ld(ci + r), y = Mem::ld(cj + r);
            Mem::st(ci + r, make_double2(fma(-wr, y.x, fma(wi, y.y, c * x.x)),
                                         fma(-wr, y.y, fma(-wi, y.x, c * x.y))));
            Mem::st(cj + r, make_double2(fma(wr, x.x, fma(wi, x.y, c * y.x)),
                                         fma(wr, x.y, fma(-wi, x.x, c * y.y))));
          }
        }
        if (pr0 + gWarps * kJacPer < nPairs) __syncthreads();   // sPair is rewritten
      }
      Mem::sync();
    }
    int rotated = sRotated;
    if (kMode == 2) {
      if (tid == 0) __stcg(d.flags + rank, rotated);
      Mem::sync();
      rotated = 0;
      for (int q = 0; q < kSketchCluster; ++q) rotated |= __ldcg(d.flags + q);
      Mem::sync();   // the flags are rewritten by the next sweep
    }
    __syncthreads();
    if (!rotated) converged = true;
  }
  if (!converged && tid == 0 && rank == 0) atomicOr(status, kStatusJacobiNotConverged);
  norms();
}

// ---------------------------------------------------------------------------
// The first sweeps of the Jacobi in FP32: one-sided Jacobi on [X ; I], X the
// top half of M scaled to FP32's range, one CTA per block; M's bottom half
// receives the rotations' product V (unitary to ~1e-5).  On the tensor cores
// follow a Newton-Schulz step V <- V (3/2 I - 1/2 V^H V), a first-order step
// V <- V (I + S) from the Gram matrix of X V (jacRefineKernel), and
// Newton-Schulz again, which leaves V unitary to FP64.  The FP64 sweeps then
// run on [X V ; V]: two, the second of which rotates next to nothing, instead
// of seven or eight, at FP32's 64 times higher rate for the rest
// (mixed-precision Jacobi: Zhang, Gao and Bai, SIAM J. Matrix Anal. Appl.
// 2022).  The first rotates nearly every pair whatever was done before: X V
// has an error of 2^-53 |X|, which shows in every column shorter than that.
// The FP64 sweeps' stopping rule is unchanged, and so is the accuracy of what
// they leave.
// [X ; I] lives in shared memory where it fits (l <= 118), else in `scr`.
// Measured, FP32 sweeps: all sweeps 234 -> 117 ms at 65,536 points (k = 512),
// 416 -> 195 ms for twelve problems of up to 16,384 points, 11.9 -> 6.8 ms at
// 4,096; the first-order step: FP64 sweeps of the twelve 146 -> 91 ms for 15 ms
// of products (make 363 -> 347, 319 -> 310 and 15.2 -> 14.5 ms).
// ---------------------------------------------------------------------------
struct Jac32Desc {
  double2 *M;    // 2 l x l, ld 2 l
  float2 *scr;   // 2 l x l
  int32_t l, pad;
};
constexpr int kJac32Sweeps = 12, kJac32MaxSmem = 220 * 1024;
constexpr float kEps32 = 1.1920929e-7f;

__device__ __forceinline__ float4 warpSum4f(float a, float b, float c, float d) {
  int const lane = threadIdx.x & 31;
  bool const hi = lane & 16, odd = lane & 8;
  float p = hi ? c : a, q = hi ? d : b;
  p += __shfl_xor_sync(0xffffffffu, hi ? a : c, 16);
  q += __shfl_xor_sync(0xffffffffu, hi ? b : d, 16);
  float v = odd ? q : p;
  v += __shfl_xor_sync(0xffffffffu, odd ? p : q, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return make_float4(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 8),
                     __shfl_sync(0xffffffffu, v, 16), __shfl_sync(0xffffffffu, v, 24));
}

__global__ void __launch_bounds__(512) jac32Kernel(Jac32Desc const *__restrict__ descs,
                                                   int32_t inShared) {
  extern __shared__ __align__(16) float2 jac32Smem[];
  __shared__ int sRotated, sExp;
  Jac32Desc const d = descs[blockIdx.x];
  int const l = d.l, LD = 2 * l;
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nWarps = blockDim.x >> 5;
  float2 *A = inShared ? jac32Smem : d.scr;
  if (tid == 0) sExp = -100000;
  __syncthreads();
  int top = -100000;   // exponent of the largest part (integer work, no FP64)
  for (int e = tid; e < l * l; e += blockDim.x) {
    double2 const v = d.M[(int64_t)(e / l) * LD + e % l];
    int const c = max(((__double2hiint(v.x) >> 20) & 0x7FF), ((__double2hiint(v.y) >> 20) & 0x7FF));
    if (c) top = max(top, c - 1023);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) atomicMax(&sExp, top);
  __syncthreads();
  double const scale = sExp > -100000 ? scalbn(1.0, 25 - sExp) : 1.0;
  for (int e = tid; e < l * LD; e += blockDim.x) {
    int const j = e / LD, r = e % LD;
    float2 v = make_float2(r - l == j ? 1.f : 0.f, 0.f);
    if (r < l) {
      double2 const x = d.M[(int64_t)j * LD + r];
      v = make_float2((float)(x.x * scale), (float)(x.y * scale));
    }
    A[e] = v;
  }
  __syncthreads();
  int const P = l + (l & 1), nPairs = P / 2;
  float const tolRot = kEps32 * sqrtf((float)l);
  for (int sweep = 0; sweep < kJac32Sweeps; ++sweep) {
    if (tid == 0) sRotated = 0;
    __syncthreads();
    for (int round = 0; round < P - 1; ++round) {
      for (int pr = warp; pr < nPairs; pr += nWarps) {
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
        if (i >= l || j >= l) continue;
        float2 *ci = A + i * LD, *cj = A + j * LD;
        float al = 0.f, be = 0.f, gr = 0.f, gi = 0.f;
        for (int r = lane; r < l; r += 32) {
          float2 const x = ci[r], y = cj[r];
          al = fmaf(x.x, x.x, fmaf(x.y, x.y, al));
          be = fmaf(y.x, y.x, fmaf(y.y, y.y, be));
          gr = fmaf(x.x, y.x, fmaf(x.y, y.y, gr));     // conj(x) y
          gi = fmaf(x.x, y.y, fmaf(-x.y, y.x, gi));
        }
        float4 const w = warpSum4f(al, be, gr, gi);
        float const ag = sqrtf(w.z * w.z + w.w * w.w);
        if (!(ag > tolRot * (sqrtf(w.x) * sqrtf(w.y))) || !(ag > 0.f)) continue;
        float const zeta = (w.y - w.x) / (2.f * ag), az = fabsf(zeta);
        float t = az > 1e8f ? 0.5f / az : 1.f / (az + sqrtf(1.f + az * az));
        if (zeta < 0.f) t = -t;
        float const c = rsqrtf(1.f + t * t), s = c * t;
        float const er = w.z / ag, ei = -w.w / ag;   // exp(-i phi)
        for (int r = lane; r < LD; r += 32) {
          float2 const x = ci[r], y = cj[r];
          float const ytr = y.x * er - y.y * ei, yti = y.x * ei + y.y * er;
          ci[r] = make_float2(c * x.x - s * ytr, c * x.y - s * yti);
          cj[r] = make_float2(s * x.x + c * ytr, s * x.y + c * yti);
        }
        if (lane == 0) sRotated = 1;
      }
      __syncthreads();
    }
    bool const rotated = sRotated;
    __syncthreads();   // the flag is cleared by the next sweep
    if (!rotated) break;
  }
  for (int e = tid; e < l * l; e += blockDim.x) {
    int64_t const o = (int64_t)(e / l) * LD + l + e % l;
    float2 const v = A[o];
    d.M[o] = make_double2((double)v.x, (double)v.y);
  }
}

// I + S into M's bottom half from Y^H Y in `scr` (l x l FP64, ld l): the
// first-order step S_ij = G_ij / (G_jj - G_ii) that orthogonalises Y's columns,
// S anti-Hermitian.  An entry above 1e-5 (two singular values close together,
// or columns of rounding errors) is left to the sweeps.  The quotient needs no
// more than FP32: its error is of the second order.
// (I + S)^H (I + S) - I = -S^2, and the Newton-Schulz step squares that.  The
// entries' limit alone bounds |S| by l 1e-5 only, but most entries lie far
// below it: emulated on circles' Z_equiv at widths l = 64 to 640, |S| is 6e-6
// to 9e-5 and V before it unitary to 2e-11 .. 2e-8, both growing about as l,
// and V after it to 1e-15 .. 2e-15: the rounding of the products.  The FP64
// sweeps that follow keep V as unitary as they find it.
__global__ void __launch_bounds__(256) jacRefineKernel(Jac32Desc const *__restrict__ descs) {
  constexpr float kMost = 1e-5f;
  Jac32Desc const d = descs[blockIdx.x];
  int const l = d.l;
  double2 const *G = reinterpret_cast<double2 const *>(d.scr);
  double2 *T = d.M + l;
  for (int e = threadIdx.x; e < l * l; e += blockDim.x) {
    int const i = e % l, j = e / l;
    double2 t = make_double2(i == j ? 1.0 : 0.0, 0.0);
    if (i != j) {
      double2 const v = G[e];
      float const inv = 1.f / (float)(G[(int64_t)j * l + j].x - G[(int64_t)i * l + i].x);
      float const sx = (float)v.x * inv, sy = (float)v.y * inv;
      if (sx * sx + sy * sy <= kMost * kMost) t = make_double2(sx, sy);
    }
    T[(int64_t)j * 2 * l + i] = t;
  }
}

// M's top half = T (l x l, ld l)
__global__ void __launch_bounds__(256) jacTopKernel(Jac32Desc const *__restrict__ descs,
                                                    double2 const *const *__restrict__ T) {
  Jac32Desc const d = descs[blockIdx.x];
  double2 const *t = T[blockIdx.x];
  for (int e = threadIdx.x; e < d.l * d.l; e += blockDim.x)
    d.M[(int64_t)(e / d.l) * 2 * d.l + e % d.l] = t[e];
}

// pseudo-inverse weights with the reference's cut rule
// (mat_dense_complex.c:1797-1808: sigma < max(m,n) eps sigma0 + eps) or the
// relative cut sigma < tol sigma0 (linalg.c:26-36), and the capture test
__global__ void __launch_bounds__(256) sketchWeightsKernel(WeightDesc const *__restrict__ descs,
                                                           int32_t cutMode, double cutTol,
                                                           double capture, int32_t *fail) {
  WeightDesc const d = descs[blockIdx.x];
  __shared__ double rmax[32], rmin[32];
  double mx = 0.0, mn = INFINITY;
  for (int a = threadIdx.x; a < d.cols; a += blockDim.x) {
    mx = fmax(mx, d.s2[a]);
    mn = fmin(mn, d.s2[a]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) {
    rmax[warp] = mx;
    rmin[warp] = mn;
  }
  __syncthreads();
  mx = 0.0;
  mn = INFINITY;
  for (int w = 0; w < nw; ++w) {
    mx = fmax(mx, rmax[w]);
    mn = fmin(mn, rmin[w]);
  }
  double const smax = sqrt(mx);
  double const cut = cutMode == 0 ? (double)d.p * kEpsS * smax + kEpsS : cutTol * smax;
  for (int a = threadIdx.x; a < d.cols; a += blockDim.x) {
    double const sa = sqrt(d.s2[a]);
    d.w[a] = (sa < cut || sa == 0.0) ? 0.0 : 1.0 / d.s2[a];
  }
  if (threadIdx.x == 0) fail[blockIdx.x] = sqrt(mn) > capture * smax ? 1 : 0;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct Buf {
  void *p = nullptr;
  size_t bytes = 0;
  ~Buf() {
    if (p) cudaFree(p);
  }
  cudaError_t ensure(size_t n) {
    if (n <= bytes) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    cudaError_t e = cudaMalloc(&p, n);
    if (e == cudaSuccess) bytes = n;
    return e;
  }
};

// Side by side launches of one stream: the blocks of a phase go in several
// launches (by shared memory, with and without clusters), and one after the
// other each left most of the chip idle while its largest blocks ended (twelve
// problems of up to 16,384 points: make 347 -> 330 ms; 310 -> 295 at 65,536
// points, 14.5 -> 13.9 at 4,096).
// next() gives the stream itself, then side streams that start where fork()
// was called; after join() the stream waits for them.
struct Fork {
  cudaStream_t s, side[3] = {};
  cudaEvent_t start = nullptr, end[3] = {};
  int used = 0;
  explicit Fork(cudaStream_t stream) : s(stream) {}
  Fork(Fork const &) = delete;
  Fork &operator=(Fork const &) = delete;
  ~Fork() {
    for (int i = 0; i < 3; ++i) {
      if (side[i]) {
        cudaStreamSynchronize(side[i]);   // (idle unless an error came between)
        cudaStreamDestroy(side[i]);
      }
      if (end[i]) cudaEventDestroy(end[i]);
    }
    if (start) cudaEventDestroy(start);
  }
  cudaError_t fork() {
    used = 0;
    cudaError_t e = cudaSuccess;
    if (!start && (e = cudaEventCreateWithFlags(&start, cudaEventDisableTiming)) != cudaSuccess)
      return e;
    return cudaEventRecord(start, s);
  }
  cudaError_t next(cudaStream_t *out) {
    if (used == 0 || used > 3) {
      used = std::max(used, 1);
      *out = s;
      return cudaSuccess;
    }
    int const i = used++ - 1;
    cudaError_t e = cudaSuccess;
    if (!side[i]) {
      int priority = 0;
      if ((e = cudaStreamGetPriority(s, &priority)) != cudaSuccess) return e;
      e = cudaStreamCreateWithPriority(&side[i], cudaStreamNonBlocking, priority);
      if (e != cudaSuccess) return e;
    }
    if (!end[i] && (e = cudaEventCreateWithFlags(&end[i], cudaEventDisableTiming)) != cudaSuccess)
      return e;
    *out = side[i];
    return cudaStreamWaitEvent(side[i], start, 0);
  }
  cudaError_t join() {
    for (int i = 0; i + 1 < used; ++i) {
      cudaError_t e = cudaEventRecord(end[i], side[i]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(s, end[i], 0);
      if (e != cudaSuccess) return e;
    }
    used = 0;
    return cudaSuccess;
  }
};

template <typename T>
cudaError_t put(Buf &b, std::vector<T> const &v, cudaStream_t s) {
  cudaError_t e = b.ensure(std::max<size_t>(1, v.size()) * sizeof(T));
  if (e != cudaSuccess || v.empty()) return e;
  return cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s);
}

uint64_t splitmixHost(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}


// modes of the HQR / Jacobi launches: a whole cluster for large blocks
// (factorization of twelve problems of up to 16,384 points / of 65,536 points:
// QR clusters from p l = 2^17 386 and 331 ms, from 2^16 402 and 332, from 2^15
// 413 and 331; Jacobi clusters from l = 128 386 and 338 ms, from 96 462 and 359)
bool hqrCluster(int64_t p, int64_t l) { return p * l >= (int64_t)1 << 17; }
bool jacobiCluster(int64_t l) { return l >= 160; }

// device buffers of the GEMM launches, reused from one to the next
struct GemmBufs {
  Buf desc, tiles, code;
};

cudaError_t launchGemms(std::vector<GemmDesc> &g, GemmBufs &b, cudaStream_t s) {
  if (g.empty()) return cudaSuccess;
  int64_t codes = 0;
  for (GemmDesc const &d : g) codes += d.M + d.N;
  cudaError_t e = b.code.ensure((size_t)std::max<int64_t>(1, codes) * sizeof(int16_t));
  if (e != cudaSuccess) return e;
  int16_t *code = static_cast<int16_t *>(b.code.p);
  for (GemmDesc &d : g) {
    d.rowCode = code;
    d.colCode = code + d.M;
    code += d.M + d.N;
  }
  // the scale codes' tiles, then the products': longest K first, so that the
  // longest tiles start in the first wave
  std::vector<int4> tiles;
  std::vector<int> order(g.size());
  for (size_t i = 0; i < g.size(); ++i) order[i] = (int)i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return g[a].K > g[c].K; });
  for (int i : order) {
    for (int a = 0; a < g[i].M; a += 64) tiles.push_back(make_int4(i, 0, a, 0));
    for (int a = 0; a < g[i].N; a += 64) tiles.push_back(make_int4(i, 1, a, 0));
  }
  size_t const nCode = tiles.size();
  for (int i : order) {
    int const tm = (g[i].M + kGM - 1) / kGM, tn = (g[i].N + kGN - 1) / kGN;
    for (int a = 0; a < tm; ++a)
      for (int c = 0; c < tn; ++c) tiles.push_back(make_int4(i, a, c, 0));
  }
  if (tiles.size() == nCode) return cudaSuccess;
  if ((e = put(b.desc, g, s)) != cudaSuccess) return e;
  if ((e = put(b.tiles, tiles, s)) != cudaSuccess) return e;
  GemmDesc const *desc = static_cast<GemmDesc const *>(b.desc.p);
  int4 const *dt = static_cast<int4 const *>(b.tiles.p);
  constexpr int smem = 2 * kGemmStageWords * (int)sizeof(uint32_t);
  e = cudaFuncSetAttribute(zgemmKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  // grids are limited to 2^31 - 1 CTAs in x; one launch per 2^30 tiles
  size_t const step = (size_t)1 << 30;
  for (size_t t0 = 0; t0 < nCode; t0 += step) {
    gemmCodeKernel<<<(unsigned)std::min(step, nCode - t0), 256, 0, s>>>(desc, dt + t0);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  for (size_t t0 = nCode; t0 < tiles.size(); t0 += step) {
    zgemmKernel<<<(unsigned)std::min(step, tiles.size() - t0), 256, smem, s>>>(desc, dt + t0);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int kMode>
cudaError_t launchHqr(std::vector<HqrDesc> const &v, Buf &d, cudaStream_t s) {
  if (v.empty()) return cudaSuccess;
  cudaError_t e = put(d, v, s);
  if (e != cudaSuccess) return e;
  if (kMode == 1) {
    hqrKernel<1><<<(unsigned)v.size(), 512, 0, s>>>(static_cast<HqrDesc const *>(d.p));
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(v.size() * kSketchCluster));
  cfg.blockDim = dim3(512);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kSketchCluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, hqrKernel<2>, static_cast<HqrDesc const *>(d.p));
}

template <int kMode>
cudaError_t launchJacobi(std::vector<JacobiDesc> const &v, Buf &d, int32_t *status,
                         cudaStream_t s) {
  if (v.empty()) return cudaSuccess;
  cudaError_t e = put(d, v, s);
  if (e != cudaSuccess) return e;
  if (kMode == 1) {
    sketchJacobiKernel<1><<<(unsigned)v.size(), 512, 0, s>>>(
        static_cast<JacobiDesc const *>(d.p), status);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(v.size() * kSketchCluster));
  cfg.blockDim = dim3(512);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kSketchCluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, sketchJacobiKernel<2>, static_cast<JacobiDesc const *>(d.p),
                            status);
}

}  // namespace

int32_t sketchWidth(FillDesc const &d, double widthScale, int32_t widthPad) {
  double const R = std::hypot(d.ceq[0] - d.cchk[0], d.ceq[1] - d.cchk[1]);
  double const est = R > 0.0 ? d.k * d.ceq[2] * d.cchk[2] / R : (double)d.m;
  double l = std::ceil((widthScale * est + widthPad) / 32.0) * 32.0;
  if (!(l < (double)d.m)) return d.m;
  return std::max<int32_t>(32, (int32_t)l);
}

cudaError_t runSketchReexpansion(std::vector<SketchInput> const &in, PointsDev src,
                                 KernelParams kp, int32_t cutMode, double cutTol, double capture,
                                 double2 *arena, int64_t budgetEntries, cudaStream_t s,
                                 std::vector<FillDesc> *fallback, SketchReport *rep) {
  *rep = SketchReport{};
  if (in.empty()) return cudaSuccess;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t err = cudaEventCreate(&e0);
  if (err != cudaSuccess) return err;
  err = cudaEventCreate(&e1);
  if (err != cudaSuccess) {
    cudaEventDestroy(e0);
    return err;
  }
  struct Ev {
    cudaEvent_t a, b;
    ~Ev() {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  } evs{e0, e1};
  cudaEventRecord(e0, s);

  // phase boundaries of each batch (timed after the batch's final sync)
  struct PhaseEvents {
    cudaEvent_t e[9] = {};
    ~PhaseEvents() {
      for (cudaEvent_t x : e)
        if (x) cudaEventDestroy(x);
    }
  } pev;
  for (cudaEvent_t &x : pev.e)
    if ((err = cudaEventCreate(&x)) != cudaSuccess) return err;
  auto mark = [&](int i) { cudaEventRecord(pev.e[i], s); };

  Fork beside(s);
  // the cluster launch of a phase and the other one, side by side
  auto bothModes = [&](auto launch2, auto const &v2, Buf &d2, auto launch1, auto const &v1, Buf &d1) {
    if (v1.empty()) return launch2(v2, d2, s);
    if (v2.empty()) return launch1(v1, d1, s);
    cudaStream_t q;
    cudaError_t e = beside.fork();
    if (e == cudaSuccess) e = beside.next(&q);
    if (e == cudaSuccess) e = launch2(v2, d2, q);
    if (e == cudaSuccess) e = beside.next(&q);
    if (e == cudaSuccess) e = launch1(v1, d1, q);
    return e == cudaSuccess ? beside.join() : e;
  };

  // blocks with the same Z_equiv (rank, equivalent and check circles,
  // wavenumber) form one group: one sketch, QR and SVD; every member its own
  // Z_orig and Z_shift
  struct Group {
    std::vector<FillDesc> mem;
    int32_t l, fullOk;
  };
  std::vector<Group> queue;
  {
    std::map<std::array<double, 8>, size_t> key;
    for (SketchInput const &x : in) {
      std::array<double, 8> const k8 = {(double)x.d.m, x.d.ceq[0], x.d.ceq[1], x.d.ceq[2],
                                        x.d.cchk[0], x.d.cchk[1], x.d.cchk[2], x.d.k};
      auto it = key.find(k8);
      if (it == key.end()) {
        key.emplace(k8, queue.size());
        queue.push_back(Group{{x.d}, x.l, x.fullOk});
      } else {
        Group &g = queue[it->second];
        g.mem.push_back(x.d);
        g.l = std::max(g.l, x.l);
        g.fullOk = g.fullOk && x.fullOk;
      }
    }
  }
  // largest first, so that the longest groups start in the first wave
  auto cost = [](Group const &g) {
    double n = 0;
    for (auto const &d : g.mem) n += d.n;
    return (double)g.mem[0].m * g.l * (g.l + g.mem[0].m) + (double)g.l * g.mem[0].m * n;
  };
  std::stable_sort(queue.begin(), queue.end(),
                   [&](Group const &a, Group const &b) { return cost(a) > cost(b); });
  GemmBufs gemmBufs;
  Buf scratch, dBlk, dTiles, dJ32, dTops, dHqr1, dHqr2, dJac1, dJac2, dW, dFail, dStatus;
  err = dStatus.ensure(sizeof(int32_t));
  if (err != cudaSuccess) return err;
  err = cudaMemsetAsync(dStatus.p, 0, sizeof(int32_t), s);
  if (err != cudaSuccess) return err;
  int32_t *status = static_cast<int32_t *>(dStatus.p);
  uint64_t seedCounter = 0x5EED5EEDull;

  size_t q0 = 0;
  while (q0 < queue.size()) {
    // a batch of groups within the scratch budget (at least one): descs
    // holds the groups' leaders (the sketch, QRs and SVD), then their
    // members (Z_orig and the output products), memberOf[i] the leader of
    // member nb + i
    std::vector<SketchDev> blks, mems;
    std::vector<size_t> memberOf;
    int64_t total = 0;
    size_t q1 = q0;
    while (q1 < queue.size()) {
      Group const &gr = queue[q1];
      int64_t const p = gr.mem[0].m, l = gr.l;
      int64_t e = p * p + 3 * p * l + 2 * l * l + l + l + 8 + p;
      for (auto const &d : gr.mem) e += p * d.n + 2 * l * d.n + d.n;
      if (q1 > q0 && total + e > budgetEntries) break;
      FillDesc const &d0 = gr.mem[0];
      SketchDev b{};
      b.kind = d0.kind;
      b.p = d0.m;
      b.n = d0.n;
      b.l = gr.l;
      b.arenaOff = d0.arenaOff;
      b.s0 = d0.s0;
      for (int c = 0; c < 3; ++c) {
        b.corig[c] = d0.corig[c];
        b.ceq[c] = d0.ceq[c];
        b.cchk[c] = d0.cchk[c];
      }
      b.k = d0.k;
      b.seed = splitmixHost(seedCounter++);
      int64_t o = total;
      b.oZ = o; o += p * p;
      b.oB0 = o; o += p * l;
      b.oB1 = o; o += p * l;
      b.oB2 = o; o += p * l;
      b.oM = o; o += 2 * l * l;
      b.oTau = o; o += l;
      b.oSW = o; o += l;
      b.oFlags = o; o += 4;
      b.oStep = o; o += 4;
      b.oT = o; o += p;
      for (auto const &d : gr.mem) {
        SketchDev m = b;
        m.kind = d.kind;
        m.n = d.n;
        m.arenaOff = d.arenaOff;
        m.s0 = d.s0;
        for (int c = 0; c < 3; ++c) m.corig[c] = d.corig[c];
        m.oZo = o; o += p * d.n;
        m.oC = o; o += l * d.n;
        m.oD = o; o += l * d.n;
        m.oTo = o; o += d.n;
        mems.push_back(m);
        memberOf.push_back(blks.size());
      }
      total = o;
      blks.push_back(b);
      ++q1;
    }
    err = scratch.ensure((size_t)total * sizeof(double2));
    if (err != cudaSuccess) return err;
    double2 *S = static_cast<double2 *>(scratch.p);
    size_t const nb = blks.size();
    std::vector<SketchDev> descs = blks;
    descs.insert(descs.end(), mems.begin(), mems.end());

    // fill: Z_equiv and Omega per group, Z_orig per member
    mark(0);
    std::vector<FillTileDesc> tiles;
    auto addTiles = [&](size_t di, int w, int64_t cnt) {
      for (int64_t e0 = 0; e0 < cnt; e0 += kFillTile) {
        FillTileDesc t{};
        t.blk = (int32_t)di;
        t.what = w;
        t.e0 = e0;
        t.cnt = (int32_t)std::min<int64_t>(kFillTile, cnt - e0);
        tiles.push_back(t);
      }
    };
    for (size_t i = 0; i < nb; ++i) {
      addTiles(i, 0, (int64_t)blks[i].p * blks[i].p);
      addTiles(i, 1, (int64_t)blks[i].p * blks[i].l);
    }
    for (size_t i = 0; i < mems.size(); ++i)
      addTiles(nb + i, 2, (int64_t)mems[i].p * mems[i].n);
    if ((err = put(dBlk, descs, s)) != cudaSuccess) return err;
    if ((err = put(dTiles, tiles, s)) != cudaSuccess) return err;
    sketchCircleKernel<<<(unsigned)descs.size(), 256, 0, s>>>(static_cast<SketchDev const *>(dBlk.p),
                                                              (int)nb, S);
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
    for (size_t t0 = 0; t0 < tiles.size(); t0 += ((size_t)1 << 30)) {
      size_t const cnt = std::min<size_t>((size_t)1 << 30, tiles.size() - t0);
      sketchFillKernel<<<(unsigned)cnt, 256, 0, s>>>(
          static_cast<SketchDev const *>(dBlk.p), static_cast<FillTileDesc const *>(dTiles.p) + t0,
          src, kp, S);
      if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }

    // Y = Z Omega
    mark(1);
    std::vector<GemmDesc> g;
    for (auto const &b : blks)
      g.push_back(GemmDesc{S + b.oZ, S + b.oB0, S + b.oB1, nullptr, b.p, b.p, b.p, b.p, b.l, b.p, 0});
    if ((err = launchGemms(g, gemmBufs, s)) != cudaSuccess) return err;
    // Q = qr(Y) into B0
    mark(2);
    std::vector<HqrDesc> h1, h2;
    for (auto const &b : blks) {
      HqrDesc h{S + b.oB1, S + b.oB0, S + b.oTau, S + b.oStep, nullptr, b.p, b.l};
      (hqrCluster(b.p, b.l) ? h2 : h1).push_back(h);
    }
    if ((err = bothModes(launchHqr<2>, h2, dHqr2, launchHqr<1>, h1, dHqr1)) != cudaSuccess)
      return err;
    // G = Z^H Q into B1
    mark(3);
    g.clear();
    for (auto const &b : blks)
      g.push_back(GemmDesc{S + b.oZ, S + b.oB0, S + b.oB1, nullptr, b.p, b.p, b.p, b.p, b.l, b.p, 1});
    if ((err = launchGemms(g, gemmBufs, s)) != cudaSuccess) return err;
    // G = Q2 R2: Q2 into B2, [R2^H ; I] into M
    mark(4);
    h1.clear();
    h2.clear();
    for (auto const &b : blks) {
      HqrDesc h{S + b.oB1, S + b.oB2, S + b.oTau, S + b.oStep, S + b.oM, b.p, b.l};
      (hqrCluster(b.p, b.l) ? h2 : h1).push_back(h);
    }
    if ((err = bothModes(launchHqr<2>, h2, dHqr2, launchHqr<1>, h1, dHqr1)) != cudaSuccess)
      return err;
    // Jacobi on [R2^H ; I]: FP32 sweeps give V (M's bottom half), products by
    // way of Z's and G's buffers refine it, then FP64 sweeps on [R2^H V ; V]
    mark(5);
    {
      // by shared memory: four, two and one CTA an SM, and in global memory
      constexpr int64_t most[4] = {55 * 1024, 110 * 1024, kJac32MaxSmem, INT64_MAX};
      std::vector<Jac32Desc> js;
      std::vector<double2 const *> tops;
      size_t at[5] = {0, 0, 0, 0, 0};
      int64_t smem[4] = {0, 0, 0, 0};
      for (int c = 0; c < 4; ++c) {
        for (auto const &b : blks) {
          int64_t const bytes = 16 * (int64_t)b.l * b.l;
          if (bytes > most[c] || (c > 0 && bytes <= most[c - 1])) continue;
          js.push_back(Jac32Desc{S + b.oM, reinterpret_cast<float2 *>(S + b.oB1), b.l, 0});
          tops.push_back(S + b.oZ);
          if (c < 3) smem[c] = std::max(smem[c], bytes);
        }
        at[c + 1] = js.size();
      }
      if ((err = put(dJ32, js, s)) != cudaSuccess) return err;
      if ((err = put(dTops, tops, s)) != cudaSuccess) return err;
      Jac32Desc const *jd = static_cast<Jac32Desc const *>(dJ32.p);
      err = cudaFuncSetAttribute(jac32Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kJac32MaxSmem);
      if (err != cudaSuccess) return err;
      if ((err = beside.fork()) != cudaSuccess) return err;
      for (int c = 3; c >= 0; --c) {   // the largest first
        if (at[c + 1] == at[c]) continue;
        cudaStream_t q;
        if ((err = beside.next(&q)) != cudaSuccess) return err;
        jac32Kernel<<<(unsigned)(at[c + 1] - at[c]), 512, (size_t)smem[c], q>>>(jd + at[c], c < 3);
        if ((err = cudaGetLastError()) != cudaSuccess) return err;
      }
      if ((err = beside.join()) != cudaSuccess) return err;
      // C = op(A) B (kGram: A^H B, kNewton: 3/2 I - 1/2 A^H B) over every
      // block's l x l matrices: M's halves, Z's and G's buffers
      enum Where { kTop, kLow, kInZ, kInG };
      enum What { kPlain, kGram, kNewton };
      auto product = [&](What what, Where wa, Where wb, Where wc) {
        g.clear();
        for (auto const &b : blks) {
          auto at = [&](Where w) {
            return w == kTop ? S + b.oM : w == kLow ? S + b.oM + b.l : w == kInZ ? S + b.oZ : S + b.oB1;
          };
          auto ld = [&](Where w) { return (w == kTop || w == kLow ? 2 : 1) * (int64_t)b.l; };
          GemmDesc d{};
          d.M = d.N = d.K = b.l;
          d.A = at(wa); d.lda = ld(wa);
          d.B = at(wb); d.ldb = ld(wb);
          d.C = at(wc); d.ldc = ld(wc);
          d.opA = what != kPlain;
          d.newton = what == kNewton;
          g.push_back(d);
        }
        return launchGemms(g, gemmBufs, s);
      };
      // V to FP64 unitarity, its refinement, and the same again
      if ((err = product(kNewton, kLow, kLow, kInG)) != cudaSuccess) return err;
      if ((err = product(kPlain, kLow, kInG, kInZ)) != cudaSuccess) return err;
      if ((err = product(kPlain, kTop, kInZ, kLow)) != cudaSuccess) return err;   // Y = X V
      if ((err = product(kGram, kLow, kLow, kInG)) != cudaSuccess) return err;    // Y^H Y
      jacRefineKernel<<<(unsigned)js.size(), 256, 0, s>>>(jd);                    // I + S
      if ((err = cudaGetLastError()) != cudaSuccess) return err;
      if ((err = product(kPlain, kInZ, kLow, kInG)) != cudaSuccess) return err;   // V (I + S)
      if ((err = product(kNewton, kInG, kInG, kInZ)) != cudaSuccess) return err;
      if ((err = product(kPlain, kInG, kInZ, kLow)) != cudaSuccess) return err;
      if ((err = product(kPlain, kTop, kLow, kInZ)) != cudaSuccess) return err;
      jacTopKernel<<<(unsigned)js.size(), 256, 0, s>>>(jd, static_cast<double2 const *const *>(dTops.p));
      if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }
    std::vector<JacobiDesc> j1, j2;
    for (auto const &b : blks) {
      JacobiDesc j{};
      j.M = S + b.oM;
      j.s2 = reinterpret_cast<double *>(S + b.oSW);
      j.flags = reinterpret_cast<int32_t *>(S + b.oFlags);
      j.cols = b.l;
      j.rowsDot = b.l;
      j.ld = 2 * b.l;
      (jacobiCluster(b.l) ? j2 : j1).push_back(j);
    }
    auto jac1 = [&](auto const &v, Buf &d, cudaStream_t q) { return launchJacobi<1>(v, d, status, q); };
    auto jac2 = [&](auto const &v, Buf &d, cudaStream_t q) { return launchJacobi<2>(v, d, status, q); };
    if ((err = bothModes(jac2, j2, dJac2, jac1, j1, dJac1)) != cudaSuccess) return err;
    // weights and capture
    mark(6);
    std::vector<WeightDesc> wd;
    for (auto const &b : blks) {
      double *sw = reinterpret_cast<double *>(S + b.oSW);
      wd.push_back(WeightDesc{sw, sw + b.l, b.l, b.p});
    }
    if ((err = put(dW, wd, s)) != cudaSuccess) return err;
    if ((err = dFail.ensure(nb * sizeof(int32_t))) != cudaSuccess) return err;
    sketchWeightsKernel<<<(unsigned)nb, 256, 0, s>>>(static_cast<WeightDesc const *>(dW.p),
                                                     cutMode, cutTol, capture,
                                                     static_cast<int32_t *>(dFail.p));
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
    std::vector<int32_t> failed(nb, 0);
    if ((err = cudaMemcpyAsync(failed.data(), dFail.p, nb * sizeof(int32_t), cudaMemcpyDeviceToHost,
                               s)) != cudaSuccess)
      return err;
    if ((err = cudaStreamSynchronize(s)) != cudaSuccess) return err;

    // accepted groups: X = Q2 (W (diag(w) (T^H (Q^H Z_orig)))) per member.
    // A group whose members have more columns in all than Z_equiv has rows
    // forms E = Q2 W and F^H = Q T diag(w) once (in the free Z and G
    // buffers), and each member then takes X = E (F Z_orig): two products
    // per member instead of four
    std::vector<GemmDesc> gc, gd, ge, gx, gE, gF;
    std::vector<char> fused(nb, 0);
    std::vector<Group> requeue;
    for (size_t i = 0; i < nb; ++i) {
      SketchDev const &b = blks[i];
      Group const &gr = queue[q0 + i];
      bool const full = b.l >= b.p;
      if (failed[i] && !full) {
        Group r = gr;
        r.l = std::min<int32_t>(b.p, 2 * b.l);
        rep->retries += (int64_t)gr.mem.size();
        if (r.fullOk && r.l > (int32_t)(0.8 * b.p)) {
          fallback->insert(fallback->end(), r.mem.begin(), r.mem.end());
          rep->fallbacks += (int64_t)gr.mem.size();
        } else {
          requeue.push_back(r);
        }
        continue;
      }
      (b.p < kSketchCounted ? rep->smallGroups : rep->groups) += 1;
      int64_t sumN = 0;
      for (auto const &d : gr.mem) sumN += d.n;
      if (sumN > b.p) {
        fused[i] = 1;
        double const *w = reinterpret_cast<double const *>(S + b.oSW) + b.l;
        gE.push_back(GemmDesc{S + b.oB2, S + b.oM + b.l, S + b.oZ, nullptr, b.p, 2 * b.l, b.p, b.p,
                              b.l, b.l, 0, nullptr});
        gF.push_back(GemmDesc{S + b.oB0, S + b.oM, S + b.oB1, nullptr, b.p, 2 * b.l, b.p, b.p, b.l,
                              b.l, 0, w});
      }
    }
    for (size_t mi = 0; mi < mems.size(); ++mi) {
      size_t const i = memberOf[mi];
      SketchDev const &b = blks[i];
      if (failed[i] && b.l < b.p) continue;
      SketchDev const &m = mems[mi];
      double const *w = reinterpret_cast<double const *>(S + b.oSW) + b.l;
      if (fused[i]) {
        // Y1 = F Z_orig = (F^H)^H Z_orig into C, X = E Y1
        gc.push_back(GemmDesc{S + b.oB1, S + m.oZo, S + m.oC, nullptr, b.p, b.p, b.l, b.l, m.n,
                              b.p, 1, nullptr});
        gx.push_back(GemmDesc{S + b.oZ, S + m.oC, arena + m.arenaOff, nullptr, b.p, b.l, b.p, b.p,
                              m.n, b.l, 0, nullptr});
      } else {
        gc.push_back(GemmDesc{S + b.oB0, S + m.oZo, S + m.oC, nullptr, b.p, b.p, b.l, b.l, m.n,
                              b.p, 1, nullptr});
        gd.push_back(GemmDesc{S + b.oM, S + m.oC, S + m.oD, w, 2 * b.l, b.l, b.l, b.l, m.n, b.l, 1,
                              nullptr});
        ge.push_back(GemmDesc{S + b.oM + b.l, S + m.oD, S + m.oC, nullptr, 2 * b.l, b.l, b.l, b.l,
                              m.n, b.l, 0, nullptr});
        gx.push_back(GemmDesc{S + b.oB2, S + m.oC, arena + m.arenaOff, nullptr, b.p, b.l, b.p, b.p,
                              m.n, b.l, 0, nullptr});
      }
      if (b.p < kSketchCounted) continue;
      ++rep->blocks;
      rep->maxWidth = std::max<int64_t>(rep->maxWidth, b.l);
      rep->sumWidth += b.l;
    }
    mark(7);
    if ((err = launchGemms(gE, gemmBufs, s)) != cudaSuccess) return err;
    if ((err = launchGemms(gF, gemmBufs, s)) != cudaSuccess) return err;
    if ((err = launchGemms(gc, gemmBufs, s)) != cudaSuccess) return err;
    if ((err = launchGemms(gd, gemmBufs, s)) != cudaSuccess) return err;
    if ((err = launchGemms(ge, gemmBufs, s)) != cudaSuccess) return err;
    if ((err = launchGemms(gx, gemmBufs, s)) != cudaSuccess) return err;
    mark(8);
    // descriptors and scratch are reused by the next batch
    if ((err = cudaStreamSynchronize(s)) != cudaSuccess) return err;
    for (int i = 0; i < 8; ++i) {
      float pm = 0.f;
      cudaEventElapsedTime(&pm, pev.e[i], pev.e[i + 1]);
      rep->phaseMs[i] += pm;
    }
    queue.insert(queue.end(), requeue.begin(), requeue.end());
    q0 = q1;
  }
  int32_t hst = 0;
  if ((err = cudaMemcpy(&hst, dStatus.p, sizeof hst, cudaMemcpyDeviceToHost)) != cudaSuccess)
    return err;
  rep->notConverged = (hst & kStatusJacobiNotConverged) ? 1 : 0;
  cudaEventRecord(e1, s);
  if ((err = cudaEventSynchronize(e1)) != cudaSuccess) return err;
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  rep->ms = ms;
  return cudaSuccess;
}

}  // namespace bfg
