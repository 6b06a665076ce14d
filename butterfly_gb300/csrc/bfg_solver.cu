// Boundary-integral systems on a butterfly factorization, their block-Jacobi
// preconditioner, and flexible GMRES -- the solver side of the reference's
// multiple-scattering example:
//
//   A = 1/2 I + (K + C) diag(w)         assembleButterfliedK
//                                       (multiple_scattering_context.c:457-507)
//   K   the butterfly-compressed kernel (any layer potential; CFIE in the
//       example), applied through bfgFacApply in original point order
//   C   Kapur-Rokhlin correction of order 2, 6 or 10 inside every closed curve
//       (quadrature.c:124-269), built from the reference's kernel callback
//       K_helm2 (multiple_scattering_context.c:27-42)
//   w   quadrature weights
//   M   block-Jacobi: the inverse of every curve's diagonal block of A
//       (assemblePreconditioner, multiple_scattering_context.c:545-634),
//       formed and inverted on the GPU
//
// GMRES is the right-preconditioned flexible variant (Saad's FGMRES) with
// classical Gram-Schmidt applied twice; Arnoldi, Givens rotations and the
// Hessenberg solve are FP64.  The reference's bfSolveGMRES (linalg.c:47-317)
// is left-preconditioned; with right preconditioning the Arnoldi residual is
// the true residual of A x = b, which is what the convergence test checks.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bfg.h"
#include "bfg_kernels.cuh"
#include "bfg_launch.cuh"
#include "bfg_mlp.cuh"
#include "bfg_system.hpp"
#include "hankel.cuh"

namespace {

using cd = std::complex<double>;

// Kapur-Rokhlin end-correction weights (Kapur & Rokhlin, SIAM J. Numer.
// Anal. 34 (1997)), the values the reference tabulates (quadrature.c:12-40)
__constant__ double cKr2[2] = {1.825748064736159, -1.325748064736159};
__constant__ double cKr6[6] = {4.967362978287758, -16.20501504859126, 25.85153761832639,
                               -22.22599466791883, 9.930104998037539, -1.817995878141594};
__constant__ double cKr10[10] = {7.832432020568779, -4.565161670374749, 1.452168846354677,
                                 -2.901348302886379, 3.870862162579900, -3.523821383570681,
                                 2.172421547519342, -8.707796087382991, 2.053584266072635,
                                 -2.166984103403823};

__device__ double krWeight(int order, int p) {
  return order == 2 ? cKr2[p] : order == 6 ? cKr6[p] : cKr10[p];
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// bfHelm2GetKernelValue(helm, xsrc, xtgt, nsrc, NULL) (helm2.c:61-91); the
// point value returns NaN at r == 0 like get_S_value, never reached here.
__device__ double2 pointKernel(bfg::KernelParams const &kp, double sx, double sy, double snx,
                               double sny, double tx, double ty) {
  double const r = hypot(tx - sx, ty - sy);
  double const kr = kp.k * r;
  bfg::Bessel01 b = bfg::bessel01<true>(kr);
  double2 const S = make_double2(-0.25 * b.y0, 0.25 * b.j0);
  double const f = 0.25 * kp.k / r;
  double2 const sc = make_double2(-f * b.y1, f * b.j1);
  double const dot = snx * (tx - sx) + sny * (ty - sy);
  double2 const D = make_double2(sc.x * dot, sc.y * dot);
  if (kp.layerPot == bfg::kLpSingle) return S;
  if (kp.layerPot == bfg::kLpPvDouble) return D;
  double2 const a = cmul(make_double2(kp.alphaRe, kp.alphaIm), S);
  double2 const c = cmul(make_double2(kp.betaRe, kp.betaIm), D);
  return make_double2(a.x + c.x, a.y + c.y);
}

// Matrix-fill kernel value, target i / source j with source normal
// (helm2.c:93-280): 0 at r == 0.
__device__ double2 matrixKernel(bfg::KernelParams const &kp, double tx, double ty, double sx,
                                double sy, double snx, double sny) {
  double const r = hypot(sx - tx, sy - ty);
  if (r == 0.0) return make_double2(0.0, 0.0);
  double const kr = kp.k * r;
  bfg::Bessel01 b = bfg::bessel01<true>(kr);
  double2 const S = make_double2(-0.25 * b.y0, 0.25 * b.j0);
  if (kp.layerPot == bfg::kLpSingle) return S;
  double const f = 0.25 * kp.k / r;
  double2 const sc = make_double2(-f * b.y1, f * b.j1);
  double const dot = snx * (tx - sx) + sny * (ty - sy);
  double2 const D = make_double2(sc.x * dot, sc.y * dot);
  if (kp.layerPot == bfg::kLpPvDouble) return D;
  double2 const a = cmul(make_double2(kp.alphaRe, kp.alphaIm), S);
  double2 const c = cmul(make_double2(kp.betaRe, kp.betaIm), D);
  return make_double2(a.x + c.x, a.y + c.y);
}

// KR correction entries: row i gets 2*order entries w_KR[p] K(i, j) with
// j = i +- (p+1) cyclically inside i's curve (bf_get_KR_corr_block_spmat,
// quadrature.c:124-164), where K(i, j) is the reference's callback with
// source x_i, normal n_i and target x_j (multiple_scattering_context.c:27-42).
__global__ void krEntriesKernel(int64_t n, int64_t const *curveOf, int64_t const *offsets,
                                double const *x, double const *y, double const *nx,
                                double const *ny, bfg::KernelParams kp, int order,
                                double2 *val, int64_t *col) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t const b = curveOf[i];
    int64_t const i0 = offsets[b], m = offsets[b + 1] - i0;
    for (int p = 0; p < order; ++p) {
      double const w = krWeight(order, p);
      int64_t const jf = ((i + p + 1 - i0) % m) + i0;
      int64_t const jb = (((i + m) - p - 1 - i0) % m) + i0;
      double2 kf = pointKernel(kp, x[i], y[i], nx[i], ny[i], x[jf], y[jf]);
      double2 kb = pointKernel(kp, x[i], y[i], nx[i], ny[i], x[jb], y[jb]);
      int64_t const e = i * 2 * order + 2 * p;
      val[e] = make_double2(w * kf.x, w * kf.y);
      col[e] = jf;
      val[e + 1] = make_double2(w * kb.x, w * kb.y);
      col[e + 1] = jb;
    }
  }
}

// dense diagonal block of A for every curve, row-major n_b x n_b at blkOff[b]
__global__ void diagBlocksKernel(int64_t const *offsets, int64_t const *blkOff, double const *x,
                                 double const *y, double const *nx, double const *ny,
                                 double const *w, bfg::KernelParams kp, double shift,
                                 double2 *blocks) {
  int64_t const b = blockIdx.x;
  int64_t const i0 = offsets[b], m = offsets[b + 1] - i0;
  double2 *A = blocks + blkOff[b];
  for (int64_t e = threadIdx.x; e < m * m; e += blockDim.x) {
    int64_t const i = e / m, j = e % m;
    double2 k = matrixKernel(kp, x[i0 + i], y[i0 + i], x[i0 + j], y[i0 + j],
                             nx ? nx[i0 + j] : 0.0, ny ? ny[i0 + j] : 0.0);
    A[e] = k;
  }
}

// add the KR entries of each curve's rows, scale columns by w, add shift I
__global__ void diagBlocksFinishKernel(int64_t const *offsets, int64_t const *blkOff,
                                       double2 const *val, int64_t const *col, int nc,
                                       double const *w, double shift, double2 *blocks) {
  int64_t const b = blockIdx.x;
  int64_t const i0 = offsets[b], m = offsets[b + 1] - i0;
  double2 *A = blocks + blkOff[b];
  // KR entries: one thread per row, so the += of a row never races
  for (int64_t i = threadIdx.x; i < m; i += blockDim.x)
    for (int q = 0; q < nc; ++q) {
      int64_t const j = col[(i0 + i) * nc + q] - i0;
      double2 const c = val[(i0 + i) * nc + q];
      A[i * m + j].x += c.x;
      A[i * m + j].y += c.y;
    }
  __syncthreads();
  for (int64_t e = threadIdx.x; e < m * m; e += blockDim.x) {
    int64_t const i = e / m, j = e % m;
    double const wj = w[i0 + j];
    double2 v = A[e];
    v = make_double2(v.x * wj, v.y * wj);
    if (i == j) v.x += shift;
    A[e] = v;
  }
}

// In-place inversion of every block by Gauss-Jordan elimination with
// partial pivoting; inv receives the inverse (row-major).  One CTA per block.
__global__ void gaussJordanKernel(int64_t const *offsets, int64_t const *blkOff, double2 *A,
                                  double2 *inv, double2 *colBuf, int32_t *singular) {
  int64_t const b = blockIdx.x;
  int64_t const m = offsets[b + 1] - offsets[b];
  double2 *a = A + blkOff[b];
  double2 *v = inv + blkOff[b];
  double2 *colk = colBuf + offsets[b];
  __shared__ double red[32];
  __shared__ int64_t redIdx[32];
  __shared__ int64_t sPiv;
  for (int64_t e = threadIdx.x; e < m * m; e += blockDim.x)
    v[e] = make_double2((e / m) == (e % m) ? 1.0 : 0.0, 0.0);
  __syncthreads();
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int64_t k = 0; k < m; ++k) {
    // pivot: argmax_{r >= k} |a[r,k]|
    double best = -1;
    int64_t bi = k;
    for (int64_t r = k + threadIdx.x; r < m; r += blockDim.x) {
      double2 z = a[r * m + k];
      double mag = z.x * z.x + z.y * z.y;
      if (mag > best) { best = mag; bi = r; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      double ob = __shfl_xor_sync(0xffffffffu, best, o);
      int64_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { red[warp] = best; redIdx[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      double bb = -1;
      int64_t ii = k;
      for (int q = 0; q < nw; ++q)
        if (red[q] > bb || (red[q] == bb && redIdx[q] < ii)) { bb = red[q]; ii = redIdx[q]; }
      sPiv = ii;
      if (!(bb > 0)) atomicOr(singular, 1);
    }
    __syncthreads();
    int64_t const piv = sPiv;
    if (piv != k)
      for (int64_t c = threadIdx.x; c < m; c += blockDim.x) {
        double2 t = a[k * m + c]; a[k * m + c] = a[piv * m + c]; a[piv * m + c] = t;
        t = v[k * m + c]; v[k * m + c] = v[piv * m + c]; v[piv * m + c] = t;
      }
    __syncthreads();
    double2 const d = a[k * m + k];
    double const dd = d.x * d.x + d.y * d.y;
    double2 const dinv = dd > 0 ? make_double2(d.x / dd, -d.y / dd) : make_double2(0.0, 0.0);
    __syncthreads();
    for (int64_t c = threadIdx.x; c < m; c += blockDim.x) {
      a[k * m + c] = cmul(a[k * m + c], dinv);
      v[k * m + c] = cmul(v[k * m + c], dinv);
    }
    __syncthreads();
    for (int64_t r = threadIdx.x; r < m; r += blockDim.x) colk[r] = a[r * m + k];
    __syncthreads();
    for (int64_t e = threadIdx.x; e < m * m; e += blockDim.x) {
      int64_t const r = e / m, c = e % m;
      if (r == k) continue;
      double2 const f = colk[r];
      double2 const ak = a[k * m + c], vk = v[k * m + c];
      double2 t = cmul(f, ak);
      a[e] = make_double2(a[e].x - t.x, a[e].y - t.y);
      t = cmul(f, vk);
      v[e] = make_double2(v[e].x - t.x, v[e].y - t.y);
    }
    __syncthreads();
  }
}

// z = blockdiag(inv) r: one warp per row
__global__ void blockDiagApplyKernel(int64_t n, int64_t const *curveOf, int64_t const *offsets,
                                     int64_t const *blkOff, double2 const *inv, double2 const *r,
                                     double2 *z) {
  int64_t const row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  int const lane = threadIdx.x & 31;
  int64_t const b = curveOf[row];
  int64_t const i0 = offsets[b], m = offsets[b + 1] - i0;
  double2 const *a = inv + blkOff[b] + (row - i0) * m;
  double sr = 0, si = 0;
  for (int64_t j = lane; j < m; j += 32) {
    double2 const c = a[j], v = r[i0 + j];
    sr += c.x * v.x - c.y * v.y;
    si += c.x * v.y + c.y * v.x;
  }
  for (int o = 16; o > 0; o >>= 1) {
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    si += __shfl_xor_sync(0xffffffffu, si, o);
  }
  if (lane == 0) z[row] = make_double2(sr, si);
}

// The same product from an FP32 copy of the inverses, FP32 arithmetic: the
// preconditioner inside flexible GMRES (its accuracy does not change the
// solution the solver converges to, only possibly the iteration count).
// z = blockdiag(inv) (r - sub) + add; sub and add may be null.  A warp takes
// four rows, so that a residual entry is read and converted once for four
// products and four times the loads are in flight (15,346 points on 64
// curves: 22 us, 45 with a row a warp; 2,073 on 16: 5.4 and 5.5).
constexpr int kBjRows = 4, kBjWarps = 4;
__global__ void __launch_bounds__(32 * kBjWarps)
    blockDiagApply32Kernel(bfg::CurveTile const *tiles, int64_t const *offsets,
                           int64_t const *blkOff, float2 const *inv, double2 const *r,
                           double2 const *sub, double2 const *add, double2 *z) {
  constexpr int Q = kBjRows, U = 4;
  bfg::CurveTile const tile = tiles[blockIdx.x];
  int const lane = threadIdx.x & 31;
  int64_t const i0 = offsets[tile.curve], m = offsets[tile.curve + 1] - i0;
  int64_t const blk = blkOff[tile.curve], row = tile.first + (threadIdx.x >> 5) * Q;
  bfg::afterPrevious();
  if (row < m) {
    float2 const *a[Q];   // a row past the end repeats the last one
#pragma unroll
    for (int q = 0; q < Q; ++q) a[q] = inv + blk + min(row + q, m - 1) * m;
    float sr[Q], si[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) sr[q] = si[q] = 0.f;
    for (int64_t j0 = lane; j0 < m; j0 += 32 * U) {
      float2 c[U][Q];
      float vx[U], vy[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        int64_t const j = j0 + 32 * u < m ? j0 + 32 * u : j0;
#pragma unroll
        for (int q = 0; q < Q; ++q) c[u][q] = a[q][j];
        double2 rv = r[i0 + j];
        if (sub) {
          double2 const t = sub[i0 + j];
          rv = make_double2(rv.x - t.x, rv.y - t.y);
        }
        vx[u] = (float)rv.x;
        vy[u] = (float)rv.y;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (j0 + 32 * u < m)
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            sr[q] += c[u][q].x * vx[u] - c[u][q].y * vy[u];
            si[q] += c[u][q].x * vy[u] + c[u][q].y * vx[u];
          }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        sr[q] += __shfl_xor_sync(0xffffffffu, sr[q], o);
        si[q] += __shfl_xor_sync(0xffffffffu, si[q], o);
      }
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (lane == q && row + q < m) {
        double2 const t = add ? add[i0 + row + q] : make_double2(0.0, 0.0);
        z[i0 + row + q] = make_double2(t.x + sr[q], t.y + si[q]);
      }
  }
}

// Learned preconditioner, one CTA per chunk c (start, len <= chunk points).
// The chunk is brought to a canonical scale and phase: s = ||r_c|| and
// p = rho / |rho| with rho = sum_t |r_t| r_t, so that the preconditioner
// commutes with every complex scaling of r (a Krylov method's vectors carry
// arbitrary phases).  scale[3c .. 3c+2] = (s, Re p, Im p); features_c =
// conj(p) (r_c, zbj_c) / s as (re, im) pairs, zero-padded to `chunk` points.
__global__ void learnedFeaturesKernel(int chunk, int64_t const *start, int32_t const *len,
                                      double2 const *r, double2 const *zbj, float *feat,
                                      float *scale) {
  __shared__ double red[3][32];
  __shared__ double2 rot;   // conj(p) / s
  int64_t const c = blockIdx.x, a = start[c];
  int const L = len[c];
  double q = 0, ux = 0, uy = 0;
  for (int t = threadIdx.x; t < L; t += blockDim.x) {
    double2 const v = r[a + t];
    double const m2 = v.x * v.x + v.y * v.y, m = sqrt(m2);
    q += m2;
    ux += m * v.x;
    uy += m * v.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    q += __shfl_xor_sync(0xffffffffu, q, o);
    ux += __shfl_xor_sync(0xffffffffu, ux, o);
    uy += __shfl_xor_sync(0xffffffffu, uy, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = q;
    red[1][threadIdx.x >> 5] = ux;
    red[2][threadIdx.x >> 5] = uy;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0, x = 0, y = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      t += red[0][w];
      x += red[1][w];
      y += red[2][w];
    }
    double const sN = sqrt(t), rm = sqrt(x * x + y * y);
    double px = 1, py = 0;
    if (rm > 0) {
      px = x / rm;
      py = y / rm;
    }
    scale[3 * c] = (float)sN;
    scale[3 * c + 1] = (float)px;
    scale[3 * c + 2] = (float)py;
    double const inv = sN > 0 ? 1.0 / sN : 0.0;
    rot = make_double2(px * inv, -py * inv);
  }
  __syncthreads();
  double2 const w = rot;
  float *f = feat + c * 4 * (int64_t)chunk;
  for (int t = threadIdx.x; t < chunk; t += blockDim.x) {
    double2 const rv = t < L ? r[a + t] : make_double2(0, 0);
    double2 const zv = t < L ? zbj[a + t] : make_double2(0, 0);
    f[2 * t] = (float)(rv.x * w.x - rv.y * w.y);
    f[2 * t + 1] = (float)(rv.x * w.y + rv.y * w.x);
    f[2 * chunk + 2 * t] = (float)(zv.x * w.x - zv.y * w.y);
    f[2 * chunk + 2 * t + 1] = (float)(zv.x * w.y + zv.y * w.x);
  }
}
// targets_c = conj(p) (e_c - zbj_c) / s
__global__ void learnedTargetsKernel(int chunk, int64_t const *start, int32_t const *len,
                                     double2 const *e, double2 const *zbj, float const *scale,
                                     float *tgt) {
  int64_t const c = blockIdx.x, a = start[c];
  int const L = len[c];
  double const sN = scale[3 * c];
  double const inv = sN > 0 ? 1.0 / sN : 0.0;
  double const wx = scale[3 * c + 1] * inv, wy = -scale[3 * c + 2] * inv;
  float *t0 = tgt + c * 2 * (int64_t)chunk;
  for (int t = threadIdx.x; t < chunk; t += blockDim.x) {
    double2 const d = t < L ? make_double2(e[a + t].x - zbj[a + t].x, e[a + t].y - zbj[a + t].y)
                            : make_double2(0, 0);
    t0[2 * t] = (float)(d.x * wx - d.y * wy);
    t0[2 * t + 1] = (float)(d.x * wy + d.y * wx);
  }
}
// z_c += s p out_c
__global__ void learnedApplyKernel(int chunk, int64_t const *start, int32_t const *len,
                                   float const *out, float const *scale, double2 *z) {
  int64_t const c = blockIdx.x, a = start[c];
  int const L = len[c];
  double const sN = scale[3 * c], px = scale[3 * c + 1] * sN, py = scale[3 * c + 2] * sN;
  float const *o = out + c * 2 * (int64_t)chunk;
  for (int t = threadIdx.x; t < L; t += blockDim.x) {
    double const ox = o[2 * t], oy = o[2 * t + 1];
    z[a + t] = make_double2(z[a + t].x + px * ox - py * oy, z[a + t].y + px * oy + py * ox);
  }
}

// The same inversion in FP32 and in place (the preconditioner of the
// iterations needs no more): Gauss-Jordan with partial pivoting, a_kk <-
// 1 / pivot, column k <- -a_ik / pivot, the row exchanges undone on the
// columns at the end (perm: one int per row of the block).
__global__ void __launch_bounds__(1024) gaussJordan32Kernel(int64_t const *offsets,
                                                            int64_t const *blkOff, float2 *A,
                                                            int32_t *permBuf, float2 *colBuf,
                                                            int32_t *singular) {
  int64_t const b = blockIdx.x;
  int64_t const m = offsets[b + 1] - offsets[b];
  float2 *a = A + blkOff[b];
  int32_t *perm = permBuf + offsets[b];
  float2 *colk = colBuf + offsets[b];
  __shared__ float red[32];
  __shared__ int64_t redIdx[32];
  __shared__ int64_t sPiv;
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int64_t k = 0; k < m; ++k) {
    float best = -1.f;
    int64_t bi = k;
    for (int64_t r = k + threadIdx.x; r < m; r += blockDim.x) {
      float2 const z = a[r * m + k];
      float const mag = z.x * z.x + z.y * z.y;
      if (mag > best) { best = mag; bi = r; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      float const ob = __shfl_xor_sync(0xffffffffu, best, o);
      int64_t const oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { red[warp] = best; redIdx[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      float bb = -1.f;
      int64_t ii = k;
      for (int q = 0; q < nw; ++q)
        if (red[q] > bb || (red[q] == bb && redIdx[q] < ii)) { bb = red[q]; ii = redIdx[q]; }
      sPiv = ii;
      perm[k] = (int32_t)ii;
      if (!(bb > 0.f)) atomicOr(singular, 1);
    }
    __syncthreads();
    int64_t const piv = sPiv;
    if (piv != k)
      for (int64_t c = threadIdx.x; c < m; c += blockDim.x) {
        float2 const t = a[k * m + c]; a[k * m + c] = a[piv * m + c]; a[piv * m + c] = t;
      }
    __syncthreads();
    float2 const d = a[k * m + k];
    float const dd = d.x * d.x + d.y * d.y;
    float2 const dinv = dd > 0.f ? make_float2(d.x / dd, -d.y / dd) : make_float2(0.f, 0.f);
    __syncthreads();
    for (int64_t c = threadIdx.x; c < m; c += blockDim.x) {
      float2 const v = a[k * m + c];
      a[k * m + c] = c == k ? dinv : make_float2(v.x * dinv.x - v.y * dinv.y,
                                                 v.x * dinv.y + v.y * dinv.x);
    }
    for (int64_t r = threadIdx.x; r < m; r += blockDim.x) colk[r] = a[r * m + k];
    __syncthreads();
    for (int64_t e = threadIdx.x; e < m * m; e += blockDim.x) {
      int64_t const r = e / m, c = e % m;
      if (r == k || c == k) continue;
      float2 const f = colk[r], ak = a[k * m + c];
      float2 v = a[e];
      v.x -= f.x * ak.x - f.y * ak.y;
      v.y -= f.x * ak.y + f.y * ak.x;
      a[e] = v;
    }
    __syncthreads();
    for (int64_t r = threadIdx.x; r < m; r += blockDim.x)
      if (r != k) {
        float2 const f = colk[r];
        a[r * m + k] = make_float2(-(f.x * dinv.x - f.y * dinv.y), -(f.x * dinv.y + f.y * dinv.x));
      }
    __syncthreads();
  }
  for (int64_t k = m - 1; k >= 0; --k) {
    int64_t const p = perm[k];
    if (p != k)
      for (int64_t r = threadIdx.x; r < m; r += blockDim.x) {
        float2 const t = a[r * m + k]; a[r * m + k] = a[r * m + p]; a[r * m + p] = t;
      }
    __syncthreads();
  }
}

__global__ void c128ToC64FlatKernel(int64_t n, double2 const *a, float2 *b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    b[i] = make_float2((float)a[i].x, (float)a[i].y);
}

// Classical Gram-Schmidt of w against k basis vectors, by kernels that end in
// their own last CTA (the one that draws a counter's last ticket adds the
// partial sums in order, so results are reproducible, and resets it):
//   arnoldiDots  h = V^H w, and ||w||^2
//   arnoldiAxpy  w -= V h, ||w||^2 again and whether a second pass is due
// Twice, then the scaling: 5 launches an iteration.  A finishing kernel for
// every reduction and one for the criterion took 13, each a few microseconds
// of latency at 2,073 unknowns (1.8 ms of a
// solve's 49 iterations more than these).

// draws a ticket; true in every thread of the CTA that drew the last of `total`
__device__ __forceinline__ bool lastOf(uint32_t *counter, uint32_t total) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(counter, 1u) == total - 1;
    if (last) *counter = 0;
  }
  __syncthreads();
  __threadfence();
  return last;
}
// the sum of a double2 over the CTA, in every thread of warp 0
template <int kWarps>
__device__ __forceinline__ double2 ctaSum(double2 v) {
  __shared__ double2 red[kWarps];
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = make_double2(0.0, 0.0);
  for (int w = 0; w < kWarps; ++w) {
    v.x += red[w].x;
    v.y += red[w].y;
  }
  return v;
}

// h[i] = sum_r conj(V_i[r]) w[r], i < k (CTA (c, i): row chunk c of vector i),
// and for i = k, if the grid has it, *self = ||w||^2.  gate: nothing to do if
// it is closed.
constexpr int kDotThreads = 128, kDotRows = 8 * kDotThreads;
__global__ void __launch_bounds__(kDotThreads)
arnoldiDotsKernel(int64_t n, double2 const *V, int64_t ldv, int k, double2 const *w,
                  double2 *part, uint32_t *counters, double2 *h, double2 *self,
                  int32_t const *gate) {
  bfg::afterPrevious();
  if (gate && !*gate) return;
  constexpr int U = kDotRows / kDotThreads, kWarps = kDotThreads / 32;
  int const i = blockIdx.y;
  double2 const *v = i < k ? V + (int64_t)i * ldv : w;
  int64_t const r0 = blockIdx.x * (int64_t)kDotRows + threadIdx.x;
  double2 a[U], b[U];
#pragma unroll
  for (int q = 0; q < U; ++q) {
    bool const in = r0 + q * kDotThreads < n;
    a[q] = in ? v[r0 + q * kDotThreads] : make_double2(0.0, 0.0);
    b[q] = in ? w[r0 + q * kDotThreads] : make_double2(0.0, 0.0);
  }
  double sr = 0, si = 0;
#pragma unroll
  for (int q = 0; q < U; ++q) {
    sr = fma(a[q].y, b[q].y, fma(a[q].x, b[q].x, sr));
    si = fma(-a[q].y, b[q].x, fma(a[q].x, b[q].y, si));
  }
  double2 t = ctaSum<kWarps>(make_double2(sr, si));
  if (gridDim.x > 1) {
    double2 *p = part + (int64_t)i * gridDim.x;
    if (threadIdx.x == 0) p[blockIdx.x] = t;
    if (!lastOf(counters + i, gridDim.x)) return;
    t = make_double2(0.0, 0.0);
    for (unsigned c = threadIdx.x; c < gridDim.x; c += kDotThreads) {
      double2 const u = __ldcg(p + c);
      t.x += u.x;
      t.y += u.y;
    }
    t = ctaSum<kWarps>(t);
  }
  if (threadIdx.x == 0) *(i < k ? h + i : self) = t;
}
int dotChunks(int64_t n) { return (int)((n + kDotRows - 1) / kDotRows); }

// w += sign * sum_{i<k} V_i h_i.  A CTA takes 16 rows; its 16 half warps split
// the k basis vectors (slice s takes i = s, s + 16, ...), and the 16 partial
// sums are added in a fixed order.
// With `norm`: ||w||^2 to *norm (the partial sums in `part`), and, on the
// first pass of two (before = ||w||^2 ahead of it), the DGKS criterion: the
// second pass is due when the first removed more than half of the squared
// norm (||w_after|| < ||w_before|| / sqrt 2); if not, its coefficients h2 = 0.
constexpr int kAxpyRows = 16, kAxpySlices = 16;
__global__ void __launch_bounds__(kAxpyRows * kAxpySlices)
arnoldiAxpyKernel(int64_t n, double2 const *V, int64_t ldv, int k, double2 const *h, double sign,
                  double2 *w, int32_t const *gate, double2 *norm, double2 *part,
                  uint32_t *counter, double2 const *before, int32_t *gateOut, double2 *h2) {
  bfg::afterPrevious();
  if (gate && !*gate) return;
  constexpr int kThreads = kAxpyRows * kAxpySlices, U = 4;
  __shared__ double2 sum[kAxpySlices][kAxpyRows];
  int const lr = threadIdx.x % kAxpyRows, sl = threadIdx.x / kAxpyRows;
  int64_t const r = blockIdx.x * (int64_t)kAxpyRows + lr;
  double2 const old = sl == 0 && r < n ? w[r] : make_double2(0.0, 0.0);
  double sr = 0, si = 0;
  if (r < n)
    for (int i0 = sl; i0 < k; i0 += U * kAxpySlices) {
      double2 a[U], c[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        int const i = min(i0 + u * kAxpySlices, k - 1);
        a[u] = V[(int64_t)i * ldv + r];
        c[u] = h[i];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * kAxpySlices < k) {
          sr = fma(-a[u].y, c[u].y, fma(a[u].x, c[u].x, sr));
          si = fma(a[u].y, c[u].x, fma(a[u].x, c[u].y, si));
        }
    }
  sum[sl][lr] = make_double2(sr, si);
  __syncthreads();
  double2 q = make_double2(0.0, 0.0);   // |w[r]|^2 after
  if (sl == 0 && r < n) {
    double tr = 0, ti = 0;
#pragma unroll
    for (int s = 0; s < kAxpySlices; ++s) {
      tr += sum[s][lr].x;
      ti += sum[s][lr].y;
    }
    double2 const v = make_double2(old.x + sign * tr, old.y + sign * ti);
    w[r] = v;
    q.x = v.x * v.x + v.y * v.y;
  }
  if (!norm) return;
  if (threadIdx.x < 32) {
    for (int o = kAxpyRows / 2; o > 0; o >>= 1) q.x += __shfl_xor_sync(0xffffffffu, q.x, o);
    if (threadIdx.x == 0) part[blockIdx.x] = q;
  }
  if (!lastOf(counter, gridDim.x)) return;
  double2 t = make_double2(0.0, 0.0);
  for (unsigned c = threadIdx.x; c < gridDim.x; c += kThreads) t.x += __ldcg(&part[c].x);
  t = ctaSum<kThreads / 32>(t);
  if (threadIdx.x == 0) *norm = t;
  if (before) {
    bool const again = t.x < 0.5 * before->x;
    if (threadIdx.x == 0) *gateOut = again ? 1 : 0;
    if (!again)
      for (int i = threadIdx.x; i < k; i += kThreads) h2[i] = make_double2(0.0, 0.0);
  }
}
int axpyGrid(int64_t n) { return (int)((n + kAxpyRows - 1) / kAxpyRows); }

// y = x / sqrt(nrm2->x) (0 if the norm is 0), the norm read on the device
__global__ void scaleByNormKernel(int64_t n, double2 const *nrm2, double2 const *x, double2 *y) {
  bfg::afterPrevious();
  double const q = nrm2->x;
  double const s = q > 0 ? 1.0 / sqrt(q) : 0.0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x)
    y[r] = make_double2(s * x[r].x, s * x[r].y);
}

__global__ void scaleCopyKernel(int64_t n, double s, double2 const *x, double2 *y) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x)
    y[r] = make_double2(s * x[r].x, s * x[r].y);
}

// y = x - y
__global__ void subFromKernel(int64_t n, double2 const *x, double2 *y) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x)
    y[r] = make_double2(x[r].x - y[r].x, x[r].y - y[r].y);
}

int gridFor(int64_t n, int t) {
  int64_t g = (n + t - 1) / t;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, 152 * 32));
}

using bfg::Dev;

}  // namespace


namespace {

bfgStatus sysFail(bfgSystem s, bfgStatus st, std::string const &msg) {
  if (s) s->err = msg;
  return st;
}

#define SYS_CK(expr)                                                         \
  do {                                                                       \
    cudaError_t e_ = (expr);                                                 \
    if (e_ != cudaSuccess) return sysFail(sys, BFG_ERROR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
  } while (0)

}  // namespace

cudaStream_t bfgSystem_s::stream() const {
  void *s = nullptr;
  bfgContextGetStream(ctx, &s);
  return static_cast<cudaStream_t>(s);
}

extern "C" {

bfgStatus bfgSystemCreate(bfgContext ctx, bfgFac fac, bfgHelm2 const *helm, double const *xy,
                          double const *normals, double const *weights,
                          int64_t const *curveOffsets, int64_t numCurves, int32_t krOrder,
                          double diagShift, bfgSystem *out) {
  if (!ctx || !fac || !helm || !xy || !weights || !curveOffsets || !out || numCurves < 1)
    return BFG_ERROR_INVALID_ARGUMENTS;
  *out = nullptr;
  int64_t rows = 0, cols = 0;
  if (bfgFacGetShape(fac, &rows, &cols) != BFG_OK || rows != cols) return BFG_ERROR_INCOMPATIBLE_SHAPES;
  int64_t const n = rows;
  if (curveOffsets[0] != 0 || curveOffsets[numCurves] != n) return BFG_ERROR_INVALID_ARGUMENTS;
  if (krOrder != 0 && krOrder != 2 && krOrder != 6 && krOrder != 10) return BFG_ERROR_INVALID_ARGUMENTS;
  for (int64_t b = 0; b < numCurves; ++b)
    if (curveOffsets[b + 1] - curveOffsets[b] < (krOrder ? 2 * krOrder + 1 : 1))
      return BFG_ERROR_INVALID_ARGUMENTS;   // quadrature.c:58-59, 114-115
  bool const needN = helm->layerPot == bfg::kLpPvDouble || helm->layerPot == bfg::kLpCombinedField;
  if (needN && !normals) return BFG_ERROR_INVALID_ARGUMENTS;
  if (helm->layerPot == bfg::kLpPvNormalDerivSingle) return BFG_ERROR_NOT_IMPLEMENTED;
  auto *sys = new bfgSystem_s;
  sys->ctx = ctx;
  sys->fac = fac;
  sys->n = n;
  sys->numCurves = numCurves;
  sys->order = krOrder;
  sys->shift = diagShift;
  sys->kp.k = helm->k;
  sys->kp.layerPot = helm->layerPot;
  sys->kp.alphaRe = helm->alphaRe;
  sys->kp.alphaIm = helm->alphaIm;
  sys->kp.betaRe = helm->betaRe;
  sys->kp.betaIm = helm->betaIm;
  sys->offsets.assign(curveOffsets, curveOffsets + numCurves + 1);
  sys->weights.assign(weights, weights + sys->offsets.back());
  cudaStream_t s = sys->stream();
  std::vector<int64_t> curveOf(n);
  for (int64_t b = 0; b < numCurves; ++b)
    for (int64_t i = curveOffsets[b]; i < curveOffsets[b + 1]; ++i) curveOf[i] = b;
  std::vector<double> planes(4 * n, 0.0);
  for (int64_t i = 0; i < n; ++i) {
    planes[i] = xy[2 * i];
    planes[n + i] = xy[2 * i + 1];
    if (normals) {
      planes[2 * n + i] = normals[2 * i];
      planes[3 * n + i] = normals[2 * i + 1];
    }
  }
  bfgStatus st = [&]() -> bfgStatus {
    SYS_CK(sys->dOffsets.alloc((numCurves + 1) * 8));
    SYS_CK(sys->dCurveOf.alloc(n * 8));
    SYS_CK(sys->dX.alloc(4 * n * 8));
    SYS_CK(sys->dW.alloc(n * 8));
    SYS_CK(sys->tmpXw.alloc(n * 16));
    SYS_CK(cudaMemcpyAsync(sys->dOffsets.p, curveOffsets, (numCurves + 1) * 8, cudaMemcpyHostToDevice, s));
    SYS_CK(cudaMemcpyAsync(sys->dCurveOf.p, curveOf.data(), n * 8, cudaMemcpyHostToDevice, s));
    SYS_CK(cudaMemcpyAsync(sys->dX.p, planes.data(), 4 * n * 8, cudaMemcpyHostToDevice, s));
    SYS_CK(cudaMemcpyAsync(sys->dW.p, weights, n * 8, cudaMemcpyHostToDevice, s));
    int const nc = 2 * krOrder;
    SYS_CK(sys->dKrVal.alloc(std::max<int64_t>(1, n * nc) * 16));
    SYS_CK(sys->dKrCol.alloc(std::max<int64_t>(1, n * nc) * 8));
    if (krOrder) {
      double const *X = sys->dX.as<double>();
      krEntriesKernel<<<gridFor(n, 128), 128, 0, s>>>(
          n, sys->dCurveOf.as<int64_t>(), sys->dOffsets.as<int64_t>(), X, X + n, X + 2 * n,
          X + 3 * n, sys->kp, krOrder, sys->dKrVal.as<double2>(), sys->dKrCol.as<int64_t>());
      SYS_CK(cudaGetLastError());
    }
    SYS_CK(cudaStreamSynchronize(s));
    return BFG_OK;
  }();
  if (st != BFG_OK) {
    delete sys;
    return st;
  }
  *out = sys;
  return BFG_OK;
}

bfgStatus bfgSystemDestroy(bfgSystem sys) {
  if (!sys) return BFG_ERROR_INVALID_ARGUMENTS;
  cudaStreamSynchronize(sys->stream());
  delete sys;
  return BFG_OK;
}

char const *bfgSystemGetErrorString(bfgSystem sys) { return sys ? sys->err.c_str() : "no system"; }

namespace {
bfgStatus systemApply(bfgSystem sys, bfgPrecision prec, void const *X, void *Y);
}

bfgStatus bfgSystemApply(bfgSystem sys, void const *X, void *Y) {
  if (!sys || !X || !Y) return BFG_ERROR_INVALID_ARGUMENTS;
  return systemApply(sys, sys->applyPrec, X, Y);
}

bfgStatus bfgSystemSetApplyPrecision(bfgSystem sys, bfgPrecision prec) {
  if (!sys) return BFG_ERROR_INVALID_ARGUMENTS;
  if (prec != BFG_PRECISION_FP64 && prec != BFG_PRECISION_DF64)
    return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "system: FP64 or DF64 applies only");
  bfgStatus st = bfgFacPrepare(sys->fac, prec);
  if (st != BFG_OK) return sysFail(sys, st, "system: preparing the factors failed");
  sys->applyPrec = prec;
  return BFG_OK;
}

namespace {
bfgStatus systemApply(bfgSystem sys, bfgPrecision prec, void const *X, void *Y) {
  bfg::SystemTerms t;
  t.w = sys->dW.as<double>();
  t.x = static_cast<double2 const *>(X);
  t.xw = sys->tmpXw.as<double2>();
  t.shift = sys->shift;
  t.val = sys->dKrVal.as<double2>();
  t.col = sys->dKrCol.as<int64_t>();
  t.nc = 2 * sys->order;
  bfgStatus st = bfg::facApplySystem(sys->fac, prec, t, static_cast<double2 *>(Y));
  if (st != BFG_OK) return sysFail(sys, st, "system apply: butterfly apply failed");
  return BFG_OK;
}
}  // namespace

bfgStatus bfgSystemBuildBlockJacobi(bfgSystem sys) {
  if (!sys) return BFG_ERROR_INVALID_ARGUMENTS;
  cudaStream_t s = sys->stream();
  int64_t const nb = sys->numCurves;
  sys->blkOff.assign(nb + 1, 0);
  for (int64_t b = 0; b < nb; ++b) {
    int64_t m = sys->offsets[b + 1] - sys->offsets[b];
    sys->blkOff[b + 1] = sys->blkOff[b] + m * m;
  }
  int64_t const tot = sys->blkOff[nb];
  SYS_CK(sys->dBlkOff.alloc((nb + 1) * 8));
  SYS_CK(sys->dWork.alloc(tot * 16));
  SYS_CK(sys->dInv32.alloc(tot * 8));
  SYS_CK(sys->dColBuf.alloc(sys->n * 16));
  SYS_CK(sys->dPerm.alloc(sys->n * 4));
  SYS_CK(sys->dFlag.alloc(4));
  SYS_CK(cudaMemcpyAsync(sys->dBlkOff.p, sys->blkOff.data(), (nb + 1) * 8, cudaMemcpyHostToDevice, s));
  std::vector<bfg::CurveTile> const tiles = bfg::curveTiles(sys->offsets, kBjRows * kBjWarps);
  sys->bjTiles = (int64_t)tiles.size();
  SYS_CK(sys->dBjTiles.alloc(tiles.size() * sizeof(bfg::CurveTile)));
  SYS_CK(cudaMemcpyAsync(sys->dBjTiles.p, tiles.data(), tiles.size() * sizeof(bfg::CurveTile),
                         cudaMemcpyHostToDevice, s));
  SYS_CK(cudaMemsetAsync(sys->dFlag.p, 0, 4, s));
  double const *X = sys->dX.as<double>();
  int64_t const n = sys->n;
  bool const useN = sys->kp.layerPot != bfg::kLpSingle;
  diagBlocksKernel<<<(unsigned)nb, 256, 0, s>>>(sys->dOffsets.as<int64_t>(),
                                                 sys->dBlkOff.as<int64_t>(), X, X + n,
                                                 useN ? X + 2 * n : nullptr,
                                                 useN ? X + 3 * n : nullptr, sys->dW.as<double>(),
                                                 sys->kp, sys->shift, sys->dWork.as<double2>());
  SYS_CK(cudaGetLastError());
  diagBlocksFinishKernel<<<(unsigned)nb, 256, 0, s>>>(
      sys->dOffsets.as<int64_t>(), sys->dBlkOff.as<int64_t>(), sys->dKrVal.as<double2>(),
      sys->dKrCol.as<int64_t>(), 2 * sys->order, sys->dW.as<double>(), sys->shift,
      sys->dWork.as<double2>());
  SYS_CK(cudaGetLastError());
  // the FP32 inverses for the iterations, inverted in place in FP32; the
  // FP64 blocks stay for the FP64 inverses, formed on the first FP64 apply
  c128ToC64FlatKernel<<<gridFor(tot, 256), 256, 0, s>>>(tot, sys->dWork.as<double2>(),
                                                        sys->dInv32.as<float2>());
  gaussJordan32Kernel<<<(unsigned)nb, 1024, 0, s>>>(
      sys->dOffsets.as<int64_t>(), sys->dBlkOff.as<int64_t>(), sys->dInv32.as<float2>(),
      sys->dPerm.as<int32_t>(), reinterpret_cast<float2 *>(sys->dColBuf.p), sys->dFlag.as<int32_t>());
  SYS_CK(cudaGetLastError());
  int32_t flag = 0;
  SYS_CK(cudaMemcpyAsync(&flag, sys->dFlag.p, 4, cudaMemcpyDeviceToHost, s));
  SYS_CK(cudaStreamSynchronize(s));
  if (flag) return sysFail(sys, BFG_ERROR_NUMERICAL, "block-Jacobi: a diagonal block is singular");
  sys->haveBj = true;
  sys->haveBj64 = false;
  return BFG_OK;
}

bfgStatus bfgSystemApplyBlockJacobi(bfgSystem sys, void const *R, void *Z) {
  if (!sys || !R || !Z) return BFG_ERROR_INVALID_ARGUMENTS;
  if (!sys->haveBj) return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "block-Jacobi not built");
  cudaStream_t s = sys->stream();
  int64_t const n = sys->n;
  if (!sys->haveBj64) {
    // the FP64 inverses, on first use (the FP64 blocks are consumed)
    int64_t const tot = sys->blkOff[sys->numCurves];
    SYS_CK(sys->dInv.alloc(tot * 16));
    SYS_CK(cudaMemsetAsync(sys->dFlag.p, 0, 4, s));
    gaussJordanKernel<<<(unsigned)sys->numCurves, 512, 0, s>>>(
        sys->dOffsets.as<int64_t>(), sys->dBlkOff.as<int64_t>(), sys->dWork.as<double2>(),
        sys->dInv.as<double2>(), sys->dColBuf.as<double2>(), sys->dFlag.as<int32_t>());
    SYS_CK(cudaGetLastError());
    int32_t flag = 0;
    SYS_CK(cudaMemcpyAsync(&flag, sys->dFlag.p, 4, cudaMemcpyDeviceToHost, s));
    SYS_CK(cudaStreamSynchronize(s));
    if (flag) return sysFail(sys, BFG_ERROR_NUMERICAL, "block-Jacobi: a diagonal block is singular");
    sys->haveBj64 = true;
  }
  blockDiagApplyKernel<<<(unsigned)((n + 7) / 8), 256, 0, s>>>(
      n, sys->dCurveOf.as<int64_t>(), sys->dOffsets.as<int64_t>(), sys->dBlkOff.as<int64_t>(),
      sys->dInv.as<double2>(), static_cast<double2 const *>(R), static_cast<double2 *>(Z));
  SYS_CK(cudaGetLastError());
  return BFG_OK;
}

namespace {
// z = M_bj (r - sub) + add from the FP32 inverses
void applyBj32(bfgSystem sys, double2 const *r, double2 *z, cudaStream_t s,
               double2 const *sub = nullptr, double2 const *add = nullptr) {
  bfg::launchAfter(blockDiagApply32Kernel, dim3((unsigned)sys->bjTiles), dim3(32 * kBjWarps), 0, s,
                   sys->dBjTiles.as<bfg::CurveTile>(), sys->dOffsets.as<int64_t>(),
                   sys->dBlkOff.as<int64_t>(), sys->dInv32.as<float2>(), r, sub, add, z);
}
}  // namespace

}  // extern "C"

namespace bfg {
bfgStatus systemApplyPrec(bfgSystem sys, bfgPrecision prec, void const *X, void *Y) {
  return systemApply(sys, prec, X, Y);
}
void applyBlockJacobi32(bfgSystem sys, double2 const *r, double2 const *sub, double2 const *add,
                        double2 *z, cudaStream_t s) {
  applyBj32(sys, r, z, s, sub, add);
}
}  // namespace bfg

extern "C" {

bfgStatus bfgSystemSetLearnedPreconditioner(bfgSystem sys, bfgMlp mlp, int32_t chunk) {
  if (!sys || !mlp || chunk < 1) return BFG_ERROR_INVALID_ARGUMENTS;
  if (!sys->haveBj) return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "learned: block-Jacobi not built");
  int32_t nIn = 0, nHid = 0, nOut = 0;
  bfgMlpGetShape(mlp, &nIn, &nHid, &nOut);
  if (nIn != 4 * chunk || nOut != 2 * chunk)
    return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "learned: network shape does not fit the chunk");
  std::vector<int64_t> st;
  std::vector<int32_t> ln;
  for (int64_t b = 0; b < sys->numCurves; ++b)
    for (int64_t a = sys->offsets[b]; a < sys->offsets[b + 1]; a += chunk) {
      st.push_back(a);
      ln.push_back((int32_t)std::min<int64_t>(chunk, sys->offsets[b + 1] - a));
    }
  cudaStream_t s = sys->stream();
  int64_t const nc = (int64_t)st.size();
  SYS_CK(sys->dChunkStart.alloc(std::max<int64_t>(1, nc) * 8));
  SYS_CK(sys->dChunkLen.alloc(std::max<int64_t>(1, nc) * 4));
  SYS_CK(sys->dFeat.alloc(std::max<int64_t>(1, nc) * 4 * chunk * 4));
  SYS_CK(sys->dOut.alloc(std::max<int64_t>(1, nc) * 2 * chunk * 4));
  SYS_CK(sys->dScale.alloc(std::max<int64_t>(1, nc) * 3 * 4));
  SYS_CK(sys->dZbj.alloc(sys->n * 16));
  SYS_CK(cudaMemcpyAsync(sys->dChunkStart.p, st.data(), nc * 8, cudaMemcpyHostToDevice, s));
  SYS_CK(cudaMemcpyAsync(sys->dChunkLen.p, ln.data(), nc * 4, cudaMemcpyHostToDevice, s));
  SYS_CK(cudaStreamSynchronize(s));
  sys->mlp = mlp;
  sys->chunk = chunk;
  sys->nChunks = nc;
  return BFG_OK;
}

bfgStatus bfgSystemLearnedNumChunks(bfgSystem sys, int64_t *numChunks) {
  if (!sys || !numChunks) return BFG_ERROR_INVALID_ARGUMENTS;
  *numChunks = sys->nChunks;
  return BFG_OK;
}

bfgStatus bfgSystemLearnedPairs(bfgSystem sys, void const *R, void const *E, void *features,
                                void *targets) {
  if (!sys || !R || !features || (E && !targets)) return BFG_ERROR_INVALID_ARGUMENTS;
  if (!sys->chunk) return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "learned: no chunks set");
  cudaStream_t s = sys->stream();
  double2 const *r = static_cast<double2 const *>(R);
  double2 *zbj = sys->dZbj.as<double2>();
  applyBj32(sys, r, zbj, s);
  learnedFeaturesKernel<<<(unsigned)sys->nChunks, 128, 0, s>>>(
      sys->chunk, sys->dChunkStart.as<int64_t>(), sys->dChunkLen.as<int32_t>(), r, zbj,
      static_cast<float *>(features), sys->dScale.as<float>());
  if (E)
    learnedTargetsKernel<<<(unsigned)sys->nChunks, 128, 0, s>>>(
        sys->chunk, sys->dChunkStart.as<int64_t>(), sys->dChunkLen.as<int32_t>(),
        static_cast<double2 const *>(E), zbj, sys->dScale.as<float>(), static_cast<float *>(targets));
  SYS_CK(cudaGetLastError());
  return BFG_OK;
}

bfgStatus bfgSolveGmres(bfgSystem sys, void const *B, void *X, double tol, int64_t maxIter,
                        int32_t precond, bfgPrecondFn userFn, void *userData,
                        bfgGmresResult *result) {
  if (!sys || !B || !X || !(tol > 0) || maxIter < 1) return BFG_ERROR_INVALID_ARGUMENTS;
  if (precond == BFG_PRECOND_BLOCK_JACOBI && !sys->haveBj)
    return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "block-Jacobi not built");
  if (precond == BFG_PRECOND_USER && !userFn)
    return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "user preconditioner missing");
  if (precond == BFG_PRECOND_LEARNED && !sys->mlp)
    return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "learned preconditioner not set");
  if (precond == BFG_PRECOND_TWO_LEVEL && !(sys->haveCoarse && sys->haveBj))
    return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS,
                   "two-level preconditioner: block-Jacobi and the coarse space not built");
  if (precond != BFG_PRECOND_NONE && precond != BFG_PRECOND_BLOCK_JACOBI &&
      precond != BFG_PRECOND_USER && precond != BFG_PRECOND_LEARNED &&
      precond != BFG_PRECOND_TWO_LEVEL)
    return sysFail(sys, BFG_ERROR_INVALID_ARGUMENTS, "unknown preconditioner");
  auto t0 = std::chrono::steady_clock::now();
  cudaStream_t s = sys->stream();
  int64_t const n = sys->n, m = maxIter;
  // one allocation: the basis V, Z = M V, w, r, the Hessenberg column's slots,
  // partial sums of the two reductions, their counters (m + 1 of dots, one of
  // the vector update) and the second pass's gate
  int const nChunks = dotChunks(n);
  size_t bytes = 0;
  auto place = [&](size_t b) {
    size_t const at = bytes;
    bytes += (b + 255) / 256 * 256;
    return at;
  };
  size_t const oV = place((size_t)(m + 1) * n * 16), oZ = place((size_t)m * n * 16);
  size_t const oW = place(n * 16), oR = place(n * 16), oH = place((size_t)(2 * m + 4) * 16);
  size_t const oPart =
      place(std::max<size_t>((size_t)nChunks * (m + 1), (size_t)axpyGrid(n)) * 16);
  size_t const oFlags = place((size_t)(m + 3) * 4);
  Dev work;
  SYS_CK(work.alloc(bytes));
  char *base = work.as<char>();
  double2 *part = reinterpret_cast<double2 *>(base + oPart);
  SYS_CK(cudaMemsetAsync(base + oFlags, 0, (size_t)(m + 3) * 4, s));
  uint32_t *counters = reinterpret_cast<uint32_t *>(base + oFlags), *axpyCounter = counters + m + 1;
  int32_t *gate = reinterpret_cast<int32_t *>(base + oFlags) + m + 2;
  // hOut[i] = (V_i, w) for i < k; self: ||w||^2
  auto dots = [&](double2 const *Vm, int k, double2 const *wv, double2 *hOut, double2 *self,
                  int32_t const *g = nullptr) {
    bool const apart = self && k >= 65535;   // the grid's limit in y
    if (apart)
      bfg::launchAfter(arnoldiDotsKernel, dim3((unsigned)nChunks, 1), dim3(kDotThreads), 0,
                       s, n, nullptr, n, 0, wv, part, counters, nullptr, self, g);
    bfg::launchAfter(arnoldiDotsKernel,
                     dim3((unsigned)nChunks, (unsigned)(k + (self && !apart ? 1 : 0))),
                     dim3(kDotThreads), 0, s, n, Vm, n, k, wv, part, counters, hOut, self, g);
  };
  double2 *Vp = reinterpret_cast<double2 *>(base + oV), *Zp = reinterpret_cast<double2 *>(base + oZ);
  double2 *wp = reinterpret_cast<double2 *>(base + oW), *rp = reinterpret_cast<double2 *>(base + oR);
  double2 *hp = reinterpret_cast<double2 *>(base + oH);
  double2 *xp = static_cast<double2 *>(X);
  double2 const *bp = static_cast<double2 const *>(B);

  auto norm = [&](double2 const *v, double *out) -> bfgStatus {
    dots(nullptr, 0, v, nullptr, hp);
    SYS_CK(cudaGetLastError());
    double2 hv;
    SYS_CK(cudaMemcpyAsync(&hv, hp, 16, cudaMemcpyDeviceToHost, s));
    SYS_CK(cudaStreamSynchronize(s));
    *out = std::sqrt(std::max(0.0, hv.x));
    return BFG_OK;
  };
  auto applyM = [&](double2 const *in, double2 *outv) -> bfgStatus {
    if (precond == BFG_PRECOND_NONE) {
      SYS_CK(cudaMemcpyAsync(outv, in, n * 16, cudaMemcpyDeviceToDevice, s));
      return BFG_OK;
    }
    if (precond == BFG_PRECOND_BLOCK_JACOBI) {
      applyBj32(sys, in, outv, s);
      SYS_CK(cudaGetLastError());
      return BFG_OK;
    }
    if (precond == BFG_PRECOND_TWO_LEVEL) return bfg::applyTwoLevel(sys, in, outv);
    if (precond == BFG_PRECOND_LEARNED) {
      applyBj32(sys, in, outv, s);
      int64_t const *cs = sys->dChunkStart.as<int64_t>();
      int32_t const *cl = sys->dChunkLen.as<int32_t>();
      learnedFeaturesKernel<<<(unsigned)sys->nChunks, 128, 0, s>>>(
          sys->chunk, cs, cl, in, outv, sys->dFeat.as<float>(), sys->dScale.as<float>());
      SYS_CK(cudaGetLastError());
      bfgStatus ms = (bfgStatus)bfg::mlpForwardOnStream(sys->mlp, sys->dFeat.as<float>(),
                                                        sys->nChunks, sys->dOut.as<float>(), s);
      if (ms != BFG_OK) return sysFail(sys, ms, "learned preconditioner: network failed");
      learnedApplyKernel<<<(unsigned)sys->nChunks, 128, 0, s>>>(
          sys->chunk, cs, cl, sys->dOut.as<float>(), sys->dScale.as<float>(), outv);
      SYS_CK(cudaGetLastError());
      return BFG_OK;
    }
    bfgStatus st = userFn(userData, in, outv, (void *)s);
    return st == BFG_OK ? st : sysFail(sys, st, "user preconditioner failed");
  };

  double bnorm = 0;
  bfgStatus st = norm(bp, &bnorm);
  if (st != BFG_OK) return st;
  if (bnorm == 0) {
    SYS_CK(cudaMemsetAsync(xp, 0, n * 16, s));
    if (result) *result = bfgGmresResult{0, 0.0, 0.0, 0.0, 1, 0};
    return BFG_OK;
  }
  // r0 = b - A x0
  if ((st = bfgSystemApply(sys, xp, rp)) != BFG_OK) return st;
  subFromKernel<<<gridFor(n, 256), 256, 0, s>>>(n, bp, rp);
  double beta = 0;
  if ((st = norm(rp, &beta)) != BFG_OK) return st;
  scaleCopyKernel<<<gridFor(n, 256), 256, 0, s>>>(n, 1.0 / beta, rp, Vp);

  // column j of the rotated Hessenberg matrix from entry j (j + 1) / 2 on; all
  // grow with the iterations, which are mostly far fewer than m
  std::vector<cd> H, g(1, cd(beta)), cs, sn, hcol;
  int64_t j = 0;
  double res = beta / bnorm, before = 0;   // residuals after this iteration, the one before
  bool converged = res < tol, ahead = false;
  auto product = [&](int64_t i) {   // w = A z_i, z_i = M v_i
    bfgStatus const e = applyM(Vp + i * n, Zp + i * n);
    return e != BFG_OK ? e : bfgSystemApply(sys, Zp + i * n, wp);
  };
  for (; j < m && !converged; ++j) {
    if (!ahead && (st = product(j)) != BFG_OK) return st;
    // classical Gram-Schmidt with a second pass where the DGKS criterion
    // asks for it, the norm and the next basis vector, all on the device;
    // one read of the Hessenberg column per iteration (h: passes 1 and 2 in
    // slots [0, k) and [k, 2k), ||w||^2 in slot 2k, before pass 1 in slot
    // 2k+1)
    int const k = (int)(j + 1);
    dots(Vp, k, wp, hp, hp + 2 * k + 1);
    bfg::launchAfter(arnoldiAxpyKernel, dim3(axpyGrid(n)),
                     dim3(kAxpyRows * kAxpySlices), 0, s,
        n, Vp, n, k, hp, -1.0, wp, nullptr, hp + 2 * k, part, axpyCounter,
        hp + 2 * k + 1, gate, hp + k);
    dots(Vp, k, wp, hp + k, nullptr, gate);
    bfg::launchAfter(arnoldiAxpyKernel, dim3(axpyGrid(n)),
                     dim3(kAxpyRows * kAxpySlices), 0, s,
        n, Vp, n, k, hp + k, -1.0, wp, gate, hp + 2 * k, part, axpyCounter, nullptr,
        nullptr, nullptr);
    bfg::launchAfter(scaleByNormKernel, dim3(gridFor(n, 256)), dim3(256), 0, s, n, hp + 2 * k, wp,
                     Vp + (j + 1) * n);
    SYS_CK(cudaGetLastError());
    double2 *hh = sys->column.ensure(2 * (size_t)k + 1);
    if (!hh) return sysFail(sys, BFG_ERROR_CUDA, "GMRES: no pinned memory");
    SYS_CK(cudaMemcpyAsync(hh, hp, (2 * k + 1) * 16, cudaMemcpyDeviceToHost, s));
    SYS_CK(cudaEventRecord(sys->column.ready, s));
    // The device waits ~30 us for the read, the rotations and the next
    // launches (99 us of kernels in a 130 us iteration at 2,073 unknowns), so
    // the next product is launched ahead of the read unless the residual's
    // last reduction, repeated, would end the solve here (within a factor of
    // 4; a product too many costs more than the wait saves).  A user's
    // preconditioner is called for the iterations only.
    ahead = precond != BFG_PRECOND_USER && j > 0 && j + 1 < m && res * (res / before) > 4 * tol;
    if (ahead && (st = product(j + 1)) != BFG_OK) return st;
    SYS_CK(cudaEventSynchronize(sys->column.ready));
    hcol.assign(k + 1, cd(0));
    for (int i = 0; i < k; ++i) hcol[i] = cd(hh[i].x + hh[k + i].x, hh[i].y + hh[k + i].y);
    double const wn = std::sqrt(std::max(0.0, hh[2 * k].x));
    hcol[k] = wn;
    // apply previous rotations, then a new one (linalg.c:202-227)
    for (int64_t i = 0; i < j; ++i) {
      cd const a = hcol[i], b = hcol[i + 1];
      hcol[i] = std::conj(cs[i]) * a + std::conj(sn[i]) * b;
      hcol[i + 1] = -sn[i] * a + cs[i] * b;
    }
    cd const a = hcol[j], b = hcol[j + 1];
    double const den = std::sqrt(std::norm(a) + std::norm(b));
    cs.push_back(den == 0 ? cd(1) : a / den);
    sn.push_back(den == 0 ? cd(0) : b / den);
    hcol[j] = std::conj(cs[j]) * a + std::conj(sn[j]) * b;
    hcol[j + 1] = 0;
    g.push_back(-sn[j] * g[j]);
    g[j] = std::conj(cs[j]) * g[j];
    H.insert(H.end(), hcol.begin(), hcol.begin() + k);
    before = res;
    res = std::abs(g[j + 1]) / bnorm;
    if (res < tol || wn == 0) converged = res < tol || wn == 0;
  }
  // y = R^-1 g, x += Z y
  std::vector<cd> yv(j, cd(0));
  for (int64_t i = j - 1; i >= 0; --i) {
    cd acc = g[i];
    for (int64_t q = i + 1; q < j; ++q) acc -= H[(size_t)q * (q + 1) / 2 + i] * yv[q];
    yv[i] = acc / H[(size_t)i * (i + 1) / 2 + i];
  }
  if (j > 0) {
    std::vector<double2> yd(j);
    for (int64_t i = 0; i < j; ++i) yd[i] = make_double2(yv[i].real(), yv[i].imag());
    SYS_CK(cudaMemcpyAsync(hp, yd.data(), j * 16, cudaMemcpyHostToDevice, s));
    bfg::launchAfter(arnoldiAxpyKernel, dim3(axpyGrid(n)),
                     dim3(kAxpyRows * kAxpySlices), 0, s,
        n, Zp, n, (int)j, hp, 1.0, xp, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
        nullptr);
    SYS_CK(cudaGetLastError());
  }
  // true residual, with the FP64 apply whatever the iterations used
  if ((st = systemApply(sys, BFG_PRECISION_FP64, xp, rp)) != BFG_OK) return st;
  subFromKernel<<<gridFor(n, 256), 256, 0, s>>>(n, bp, rp);
  double rn = 0;
  if ((st = norm(rp, &rn)) != BFG_OK) return st;
  double const secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  if (result) *result = bfgGmresResult{j, res, rn / bnorm, secs, converged ? 1 : 0, 0};
  return BFG_OK;
}

}  // extern "C"
