// FP64 apply of the butterfly factors (complex128 factors and vectors) with
// the products formed exactly from fixed-point parts: integer digits on the
// tensor cores for several right-hand sides (bfg_fixed.cuh), 31-bit halves on
// the integer units for one.  GB300's FP64 units (2 FMAs a clock and SM) made
// the plain form 3 to 40 times slower than HBM delivers the factors.  Same
// apply program and workspace as the other precisions
// (mat_block_dense.c:512-572, mat_product.c:211-245): one item = up to 32
// output rows of one block row, summing its blocks in order; no atomics on
// results, reproducible bit for bit.  Scales: one per (block row piece, row)
// of the factors, computed once when the factors are stored (rowExpKernel),
// and one per right-hand side of the input rows in hand, found as they are
// read.  Rows that fixed point does not cover (NaN, infinities, subnormals,
// products beyond the exponent range, operands graded in opposite directions:
// fixCovers, fixEven) are multiplied in plain FP64 by the same kernels.
//
// Measured (GB300; microseconds an apply; before: the FP64-unit kernels):
//   32,768 points, k = 256, 6.0e7 entries   R = 1: 526 -> 351
//     R = 2..4: 4,000 -> 571   R = 8: 4,018 -> 873   R = 16: 7,650 -> 1,647
//   65,536 points, k = 512, 2.1e8 entries   R = 1: 1,583 -> 905
//     R = 2..4: 1,467   R = 8: 2,302   R = 16: 23,853 -> 4,476
// Largest error against extended precision, in units of each result's sum of
// moduli, blocks of 20 to 120 columns: R = 1 5e-17 -> 1e-17, R = 2 1.6e-16 ->
// 4e-17, R = 16 8e-17 -> 4e-17 for entries of like size; operands graded in
// opposite directions by 2^10 5e-17 -> 6e-17, 2.3e-16 -> 1.9e-16, 8e-17 ->
// 1.3e-16 and by 2^30 5e-17 -> 5e-17, 1.7e-16 -> 9e-17, 7e-17 -> 1.2e-16.
//
// Why not `tcgen05` for the digits: a lane forms an entry's digits from the
// 16 bytes it loaded, in the registers `mma.sync` reads them from; `tcgen05`
// needs them in shared memory, and precomputed in HBM they would be 32 bytes
// an entry beside the stored 16.
//
// Complex to real: A (16 rows x 16) holds row m = Re a_m0, Im a_m0, Re a_m1,
// ...; B's rows 2c, 2c+1 are (Re x, -Im x) in the column of Re y and
// (Im x, Re x) in that of Im y.  In the fragment layouts of m16n8k16 a lane
// (g = lane / 4, t = lane % 4) holds the entries (g, t), (g + 8, t),
// (g, t + 4), (g + 8, t + 4) of A, one register each, and the results of rows
// g and g + 8 in columns 2t, 2t + 1: one complex value each.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "bfg_device.cuh"
#include "bfg_fixed.cuh"
#include "bfg_kernels.cuh"
#include "bfg_launch.cuh"

namespace bfg {
namespace {

static_assert(kItemRows == 32, "two 16-row MMA tiles per item");

// Row scales of every contribution of every item: rowExp[32 (contribution) +
// row], and the most small columns of a row (fixEven).  One CTA per item, the
// warps split a contribution's columns.  HBM bound: reads the stored factors
// once (a piece's second pass finds them in the caches).
__global__ void __launch_bounds__(256) rowExpKernel(ApplyItem const *__restrict__ items,
                                                    ApplyContrib *contribs,
                                                    double2 const *__restrict__ arena,
                                                    int16_t *__restrict__ rowExp) {
  __shared__ int red[8][32];
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ApplyItem const it = items[blockIdx.x];
  for (int c = 0; c < it.nContrib; ++c) {
    ApplyContrib const cb = contribs[it.contrib0 + c];
    double2 const *a = arena + cb.aOff + lane;
    int code = 0, small = 0;
    if (lane < it.rows)
      for (int j = warp; j < cb.n; j += 8) code = max(code, fixCode(a[(int64_t)j * cb.lda]));
    red[warp][lane] = code;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) code = max(code, red[w][lane]);
    __syncthreads();
    if (code > 0) {   // (a row of zeros is exact)
      int const least = code - fixRowGap(cb.n);
      for (int j = warp; j < cb.n; j += 8) small += fixCode(a[(int64_t)j * cb.lda]) < least;
    }
    red[warp][lane] = small;
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int w = 1; w < 8; ++w) small += red[w][lane];
      small = __reduce_max_sync(0xffffffffu, small);
      rowExp[(it.contrib0 + c) * 32 + lane] = (int16_t)fixScaleOf(code);
      if (lane == 0) contribs[it.contrib0 + c].graded = small;
    }
    __syncthreads();
  }
}

constexpr int kFixWarps = 4, kFixThreads = 32 * kFixWarps;

// What a warp of an item's CTA works on: rows 16 mt .. of the item and every
// ks-th k-step from kp on (two warps a row tile for items of more than 16
// rows, else all four on the one tile).
struct FixRole {
  int mt, kp, ks;
  int row0, row1;   // the lane's two rows (clamped into the item)
  __device__ __forceinline__ FixRole(int rows, int warp, int lane) {
    bool const two = rows > 16;
    mt = two ? warp & 1 : 0;
    kp = two ? warp >> 1 : warp;
    ks = two ? kFixWarps / 2 : kFixWarps;
    row0 = min(16 * mt + (lane >> 2), rows - 1);
    row1 = min(16 * mt + (lane >> 2) + 8, rows - 1);
  }
};

// The chunk being fetched: columns [j0, j0 + n) of contribution c of an item.
struct FixCursor {
  int c = 0, j0 = 0, n = 0;
  int ea0 = 1023, ea1 = 1023;   // scales of the lane's rows
  int eaMin = 1023, eaMax = 1023;
  double2 const *a = nullptr;   // item row 0, chunk column 0
  double2 const *x = nullptr;   // chunk row 0, right-hand side 0 of the tile
  int64_t lda = 0, xld = 0;
};

// the lane's four entries of k-step st; columns past the end re-read the last
// one (against zero inputs)
__device__ __forceinline__ void fixLoadA(double2 (&av)[4], FixCursor const &k, FixRole const &role,
                                         int st, int lane) {
  int64_t const c0 = (int64_t)min(8 * st + (lane & 3), k.n - 1) * k.lda;
  int64_t const c1 = (int64_t)min(8 * st + (lane & 3) + 4, k.n - 1) * k.lda;
  av[0] = k.a[c0 + role.row0];
  av[1] = k.a[c0 + role.row1];
  av[2] = k.a[c1 + role.row0];
  av[3] = k.a[c1 + role.row1];
}

__device__ __forceinline__ void fixNextBlock(FixCursor &k, ApplyItem const &it, ApplyContrib &cb,
                                             ApplyContrib const *__restrict__ contribs,
                                             int16_t const *__restrict__ rowExp,
                                             double2 const *arena, double2 const *X, int64_t ldx,
                                             double2 const *W, int64_t ldw, int64_t r0,
                                             FixRole const &role, int lane) {
  cb = contribs[it.contrib0 + k.c];
  int16_t const *e = rowExp + (it.contrib0 + k.c) * 32;
  k.ea0 = e[role.row0];
  k.ea1 = e[role.row1];
  int const mine = e[min(lane, it.rows - 1)];
  k.eaMin = __reduce_min_sync(0xffffffffu, mine);
  k.eaMax = __reduce_max_sync(0xffffffffu, mine);
  k.lda = cb.lda;
  k.xld = cb.inIsX ? ldx : ldw;
  k.x = (cb.inIsX ? X + cb.inRow * ldx : W + cb.inRow * ldw) + r0;
  k.a = arena + cb.aOff;
}

// Several right-hand sides: one CTA of 4 warps per (item, tile of 4 NT
// right-hand sides).  A block's columns are walked in chunks of 128 / NT: the
// chunk's input rows (fetched a chunk ahead, into registers) are split into
// digits in shared memory in the B fragments' order, the factor entries
// (fetched a k-step ahead) in the registers of the lane that loaded them.
// The digit sums are flushed into FP64 accumulators at the end of every chunk,
// whose inputs have a scale of their own, and a right-hand side that fixed point
// does not cover (fixCovers, fixEven) is summed in plain FP64 in that chunk: a
// right-hand side's result depends on nothing but its own entries.  The warps
// that share rows add their FP64 sums at the end, in order.
// Bound by instruction issue and latency, not by the tensor pipe: splitting the
// entries and the inputs takes about 50 instructions each.  So resident warps
// count.  (65,536 points, 8 and 16 right-hand sides: 2,302 and 4,476 us.  With
// seven digits, the gradings left out and the sums in registers 2,225 and
// 4,290.  The tiles' shape was chosen with seven digits and flushes a block:)
// 8 right-hand sides a tile with 168 registers and 3 CTAs an SM (16 of them: 255 and 2, the tensor pipe
// 30 % busy) took 2,076 us where 2 CTAs took 2,332, and two such tiles 3,980
// us for 16 where one of 16 took 4,782 although the entries are split twice;
// 32,768 points 882 -> 787 and 1,680 -> 1,455, 4,096 points 98 -> 100 and 187
// -> 155.
// 4 right-hand sides a tile at 4 CTAs an SM: 1,366 -> 1,330 us at 65,536 points,
// 69 -> 76 at 4,096.  Wider CTAs (8 warps on 128 rows, the next step split under
// the MMAs) were slower than tiles of 16, 2,330 against 1,650 us at 32,768 points and 16
// right-hand sides, and so was copying a chunk's inputs to shared memory
// (cp.async) during the chunk before, by 7 %.
template <int NT>
__global__ void __launch_bounds__(kFixThreads, 3) fixTileKernel(
    ApplyItem const *__restrict__ items, ApplyContrib const *__restrict__ contribs,
    int16_t const *__restrict__ rowExp, double2 const *__restrict__ arena, double2 const *X,
    int64_t ldx, double2 *W, int64_t R, unsigned tiles) {
  constexpr int RT = 4 * NT, KC = 128 / NT, D = kFixDigits;
  static_assert(KC / 8 / (kFixWarps / 2) <= kFixMaxSteps, "a chunk between flushes");
  // B fragments: word ((st D + digit) NT + n tile) 64 + 2 lane + register
  __shared__ __align__(16) uint32_t sB[(KC / 8) * D * NT * 64];
  __shared__ int sMax[2][RT], sBig[kFixWarps][RT];
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t = lane & 3;
  int const q = tid % RT, colX = tid / RT;   // the input entries this thread splits
  // the tiles of an item run side by side and read its blocks from HBM once
  ApplyItem const it = items[blockIdx.x / tiles];
  int64_t const r0 = (int64_t)(blockIdx.x % tiles) * RT;
  int const nr = (R - r0) < RT ? (int)(R - r0) : RT;
  FixRole const role(it.rows, warp, lane);

  // (row0 re, im, row1 re, im) of right-hand side 4 nt + t.  Eight right-hand
  // sides keep them in shared memory, where they are touched once a chunk: in
  // registers they were spilled with others (16 right-hand sides at 65,536 points
  // 4,824 -> 4,484 us; 4 a tile have the registers: 1,485 against 1,496)
  __shared__ double sAcc[NT * 4][kFixThreads];
  double rAcc[NT * 4];
  auto acc = [&](int u, int r) -> double & {
    if constexpr (NT > 1)
      return sAcc[4 * u + r][tid];
    else
      return rAcc[4 * u + r];
  };
  float sum[NT][kFixSums][4];
#pragma unroll
  for (int u = 0; u < NT; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      acc(u, r) = 0.0;
#pragma unroll
      for (int s = 0; s < kFixSums; ++s) sum[u][s][r] = 0.f;
    }

  FixCursor k;
  ApplyContrib cb{};
  double2 av[4], xv[4];
  auto fetch = [&](int buf) {
    if (k.j0 == 0) {
      fixNextBlock(k, it, cb, contribs, rowExp, arena, X, ldx, W, R, r0, role, lane);
    } else {
      k.a += KC * k.lda;
      k.x += KC * k.xld;
    }
    k.n = min(KC, cb.n - k.j0);
    int code = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int const col = colX + i * (kFixThreads / RT);
      xv[i] = (q < nr && col < k.n) ? k.x[col * k.xld + q] : make_double2(0.0, 0.0);
    }
    fixLoadA(av, k, role, role.kp, lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) code = max(code, fixCode(xv[i]));
#pragma unroll
    for (int o = RT; o < 32; o *= 2) code = max(code, __shfl_xor_sync(0xffffffffu, code, o));
    if (lane < RT && code) atomicMax(&sMax[buf][q], code);   // order does not matter
  };
  if (tid < 2 * RT) sMax[tid / RT][tid % RT] = 0;
  __syncthreads();

  int buf = 0;
  if (it.nContrib > 0) fetch(0);
  while (k.c < it.nContrib) {
    __syncthreads();
    // lane q: the scale code of right-hand side q's rows in hand
    int const code = lane < RT ? sMax[buf][lane] : 0;
    int const ex = fixScaleOf(code);
    int const exq = __shfl_sync(0xffffffffu, ex, q);
    int const leastq = __shfl_sync(0xffffffffu, code, q) - kFixInputGap;
    int const ea0 = k.ea0, ea1 = k.ea1;
    if (tid < RT) sMax[buf ^ 1][tid] = 0;   // read by every warp a chunk ago
    int big = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int const col = colX + i * (kFixThreads / RT);
      big += col < k.n && fixLarge(xv[i], leastq);
      uint32_t d[D];
      fixSplit(xv[i], exq, d);
      // column col = 8 st + c8: lane t = c8 % 4, register c8 / 4; result
      // columns 2 (q % 4) and 2 (q % 4) + 1 of n tile q / 4
      uint32_t *w = sB + ((col >> 3) * D * NT + (q >> 2)) * 64 +
                    2 * (8 * (q & 3) + (col & 3)) + ((col >> 2) & 1);
#pragma unroll
      for (int j = 0; j < D; ++j, w += NT * 64) {
        w[0] = d[j] ^ 0x80000000u;                   // (Re x, -Im x)
        w[8] = __byte_perm(d[j], 0, 0x1032);         // (Im x, Re x)
      }
    }
#pragma unroll
    for (int o = RT; o < 32; o *= 2) big += __shfl_xor_sync(0xffffffffu, big, o);
    if (lane < RT) sBig[warp][lane] = big;
    __syncthreads();
    // the right-hand sides that fixed point covers, each by its own rows alone
    // (bit q; every warp finds the same)
    bool ok = false;
    if (lane < RT) {
      int all = 0;
#pragma unroll
      for (int w = 0; w < kFixWarps; ++w) all += sBig[w][lane];
      ok = fixCovers(k.eaMin, k.eaMax, ex) && (code == 0 || fixEven(k.n, all, cb.graded));
    }
    unsigned const fixed = __ballot_sync(0xffffffffu, ok), rhs = (1u << nr) - 1u;
    int const nSteps = (k.n + 7) >> 3;
    if (fixed & rhs) {
#pragma unroll 1
      for (int st = role.kp; st < nSteps; st += role.ks) {
        uint32_t d[4][D];
#pragma unroll
        for (int e = 0; e < 4; ++e) fixSplit(av[e], e & 1 ? ea1 : ea0, d[e]);
        if (st + role.ks < nSteps) fixLoadA(av, k, role, st + role.ks, lane);
        uint2 const *b = reinterpret_cast<uint2 const *>(sB) + st * D * NT * 32 + lane;
#pragma unroll
        for (int j = 0; j < D; ++j) {
          uint2 bv[NT];
#pragma unroll
          for (int u = 0; u < NT; ++u) bv[u] = b[(j * NT + u) * 32];
#pragma unroll
          for (int i = 0; i < D && i + j < kFixSums; ++i)
#pragma unroll
            for (int u = 0; u < NT; ++u)
              fixMma(sum[u][i + j], d[0][i], d[1][i], d[2][i], d[3][i], bv[u].x, bv[u].y);
        }
      }
#pragma unroll
      for (int u = 0; u < NT; ++u) {
        int const exu = __shfl_sync(0xffffffffu, ex, 4 * u + t);
        bool const mine = (fixed >> (4 * u + t)) & 1u;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          double const v = fixAdd(acc(u, r), sum[u], r, (r < 2 ? ea0 : ea1) + exu);
          if (mine) acc(u, r) = v;
        }
      }
    }
    if (~fixed & rhs) {
      for (int st = role.kp; st < nSteps; st += role.ks)
        for (int col = 8 * st; col < min(8 * st + 8, k.n); ++col) {
          double2 const a0 = k.a[col * k.lda + role.row0], a1 = k.a[col * k.lda + role.row1];
#pragma unroll
          for (int u = 0; u < NT; ++u)
            if (((~fixed & rhs) >> (4 * u + t)) & 1u) {
              double2 const x = k.x[col * k.xld + 4 * u + t];
              cmacc(acc(u, 0), acc(u, 1), a0, x);
              cmacc(acc(u, 2), acc(u, 3), a1, x);
            }
        }
    }
    k.j0 += KC;
    if (k.j0 >= cb.n) {
      k.j0 = 0;
      ++k.c;
    }
    buf ^= 1;
    if (k.c < it.nContrib) fetch(buf);
  }
  if constexpr (NT == 1) {
#pragma unroll
    for (int r = 0; r < 4; ++r) sAcc[r][tid] = rAcc[r];
  }
  __syncthreads();
  if (role.kp != 0) return;
  int const warpStep = kFixWarps / role.ks;   // warps of one row tile
#pragma unroll
  for (int u = 0; u < NT; ++u) {
    double v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = sAcc[4 * u + r][tid];
    for (int w = 1; w < role.ks; ++w)
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] += sAcc[4 * u + r][tid + 32 * w * warpStep];
    int const rhs = 4 * u + t, row = 16 * role.mt + (lane >> 2);
    if (rhs < nr) {
      double2 *out = W + (it.outRow + row) * R + r0 + rhs;
      if (row < it.rows) out[0] = make_double2(v[0], v[1]);
      if (row + 8 < it.rows) out[8 * R] = make_double2(v[2], v[3]);
    }
  }
}

// ---------------------------------------------------------------------------
// One right-hand side.  A matrix tile of 8 columns would be nearly empty, so
// the products are formed from two 31-bit halves on the integer units
// instead: t (the scaled entry, rounded, |t| <= 2^61) = hi 2^31 + lo, and
//   t t' = 2^62 hi hi' + 2^31 (hi lo' + lo hi') + lo lo',
// of which the last, below 2^60 = 2^-60 of the largest t t', is left out: 12
// widening multiply-adds a complex entry (32 lanes of them a clock and SM,
// against 2 FP64 FMAs).  The sums of a batch of columns fit 64 bits; they are
// then added to wider ones.  A real product is off by less than 2^-59 of the
// largest (typically 2^-62).  An apply at 65,536 points: 936 us with 28-bit
// halves, whose four products a real one and 2^-55 were neither as fast nor
// as exact, 905 so; 866 with 30-bit halves, whose sums of a pass fit 64 bits,
// but which left opposite gradings of 2^12 with 8e-16 of the sum of moduli
// (FP64 sums 5e-17, these 9e-17).
//
// One CTA of 4 warps per item, lane = row.  A block's columns are walked in
// passes of at most 120: the pass's input rows are brought to one scale in
// shared memory, warp w multiplies columns w, w + 4, ..., splitting its factor
// entries in registers with the next three columns' loads in flight, and the
// warps' integer sums are added exactly before two threads a row turn them
// into FP64: one rounding a pass.  The next pass's input rows and first
// entries are fetched while a pass is multiplied, so a pass costs three
// barriers and no exposed latency.  A pass that fixed point does not cover
// (fixCovers, fixEven) is summed in plain FP64.
//
// Few items leave most of the chip idle while each walks its passes (4,096
// points: 264 items of 8 passes, 356 of 3): then a cluster of 2 or 4 CTAs
// shares an item's passes (kSplit), whose sums meet in rank 0 through
// distributed shared memory.  An apply from HBM: 2,048 points 44 -> 34 us,
// 4,096 65 -> 47, 8,192 94 -> 84, 16,384 184 -> 167, 32,768 unchanged (348).
// ---------------------------------------------------------------------------
constexpr int kGemvAhead = 3, kGemvWarps = 4;
constexpr int64_t kGemvCtas = 152 * 16;
static_assert(2 * kGemvAhead < 8, "two products of 2^60 a column and sum: below 2^63");
static_assert(kGemvCols <= 32 * kGemvWarps, "one input row per thread");
static_assert(kGemvCols % (kGemvWarps * kGemvAhead) == 0, "whole batches of columns");

__device__ __forceinline__ void fixUnpack(uint64_t v, uint32_t &lo, uint32_t &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
// (hi, lo) of v at scale E: t = v 2^(1083 - E) rounded, |hi|, |lo| <= 2^30
__device__ __forceinline__ int2 fixHalves(double v, int E) {
  uint32_t const h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
  uint32_t const mh = (h & 0xFFFFFu) | 0x100000u, sh = (uint32_t)E - ((h >> 20) & 0x7FFu);
  int32_t const s = (int32_t)h >> 31;
  // twice t, truncated (its last bit rounds lo); shr.u64 gives 0 from 64 on
  uint64_t y = ((uint64_t)__funnelshift_l(l, mh, 9) << 32) | (l << 9);
  asm("shr.u64 %0, %0, %1;" : "+l"(y) : "r"(sh));
  // 2 t + 1 + 2^31: the upper word is hi, the lower one 2 (lo + 2^30) and a bit
  // (unpacked by hand: a shift by 32 would be taken into 64-bit multiplications)
  uint32_t lo, hi;
  fixUnpack((y ^ (uint64_t)(int64_t)s) + (uint32_t)(0x80000001 - s), lo, hi);
  return make_int2((int32_t)hi, (int32_t)(lo >> 1) - (1 << 30));
}
__device__ __forceinline__ int4 fixHalves(double2 v, int E) {
  int2 const a = fixHalves(v.x, E), b = fixHalves(v.y, E);
  return make_int4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void fixMad(int64_t &acc, int32_t a, int32_t b) {
  acc += (int64_t)a * b;
}

// A sum of products in units of 2^62 (96 bits: low word and the rest) and of
// 2^39 (m).
struct FixWide {
  uint32_t low = 0;
  int64_t rest = 0, m = 0;
  __device__ __forceinline__ void add(int64_t hh, int64_t hl, int64_t lh) {
    uint32_t a, b, c, d;
    fixUnpack((uint64_t)hh, a, b);
    fixUnpack((uint64_t)rest, c, d);
    asm("add.cc.u32 %0, %0, %3; addc.cc.u32 %1, %1, %4; addc.u32 %2, %2, %5;"
        : "+&r"(low), "+&r"(c), "+&r"(d) : "r"(a), "r"(b), "r"((uint32_t)((int32_t)b >> 31)));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rest) : "r"(c), "r"(d));
    m += (hl >> 8) + (lh >> 8);
  }
  // m's whole units of 2^62 into the rest (rounded)
  __device__ __forceinline__ void settle() {
    int64_t const v = (int64_t)low + ((m + (1 << 22)) >> 23);
    low = (uint32_t)v;
    rest += v >> 32;
  }
};

template <int kSplit>
__global__ void __launch_bounds__(32 * kGemvWarps, 6)
fixGemvKernel(ApplyItem const *__restrict__ items, ApplyContrib const *__restrict__ contribs,
              int16_t const *__restrict__ rowExp, double2 const *__restrict__ arena,
              double2 const *X, int64_t ldx, double2 *W) {
  constexpr int S = kGemvWarps, U = kGemvAhead, KC = kGemvCols;
  __shared__ int4 sx[KC];
  __shared__ int sMax[2][S], sBig[S];
  // sums of the real and of the imaginary part: the rest and the low word
  __shared__ int64_t part[2][S][32];
  __shared__ uint32_t partLow[2][S][32];
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int const rank = blockIdx.x % kSplit;   // in the item's cluster
  ApplyItem const it = items[blockIdx.x / kSplit];
  bool const active = lane < it.rows;
  double acc = 0.0;   // the last two warps: real and imaginary part of row lane
  double spr = 0.0, spi = 0.0;   // plain FP64 sums of this lane's columns
  bool anySpecial = false;

  // the pass being fetched: columns [j0, j0 + n) of contribution c, of which
  // this CTA takes every kSplit-th pass: pass b of contribution c if b + c is
  // its rank modulo kSplit
  int c = 0, j0 = rank * KC, n = 0, last = 0, ea = 1023, have = -1;
  int const cols = kSplit > 1 && lane < it.nContrib ? contribs[it.contrib0 + lane].n : 0;
  auto seek = [&]() {   // from (c, j0) on to a pass that there is
    while (c < it.nContrib && j0 >= __shfl_sync(0xffffffffu, cols, c)) {
      ++c;
      j0 = ((rank - c) & (kSplit - 1)) * KC;
    }
  };
  if (kSplit > 1) seek();
  double2 const *a = nullptr, *x = nullptr;
  int64_t step = 0, xs = 0, lda = 0;
  ApplyContrib cb{};
  double2 av[U], xv;
  auto fetch = [&](int buf, bool first) {
    if (kSplit > 1 ? c != have : j0 == 0) {
      have = c;
      cb = contribs[it.contrib0 + c];
      ea = active ? rowExp[(it.contrib0 + c) * 32 + lane] : 1023;
      lda = cb.lda;
      step = (int64_t)S * lda;
      xs = cb.inIsX ? ldx : 1;
      x = cb.inIsX ? X + cb.inRow * ldx : W + cb.inRow;
      a = arena + cb.aOff + (active ? lane : 0);   // inactive lanes re-read row 0
      if (kSplit > 1) {
        x += j0 * xs;
        a += j0 * lda;
      }
    } else {
      x += kSplit * KC * xs;
      a += kSplit * KC * lda;
    }
    n = min(KC, cb.n - j0);
    // this warp's columns warp, warp + 4, ... in whole batches: a column past
    // the end re-reads the last one (or column 0) against a zero input
    last = (n - 1 - warp) / S;
    double2 const *aw = a + (n > warp ? warp * lda : 0);
#pragma unroll
    for (int u = 0; u < U; ++u) av[u] = aw[min(u, last) * step];
    // the inputs come from the kernel before; the factors and their scales were
    // complete before any apply (the host waited for them)
    if (first) afterPrevious();
    xv = tid < n ? x[(int64_t)tid * xs] : make_double2(0.0, 0.0);
    int const code = __reduce_max_sync(0xffffffffu, fixCode(xv));
    if (lane == 0) sMax[buf][warp] = code;
  };
  int buf = 0;
  if (c < it.nContrib) fetch(0, true);
  else afterPrevious();
  while (c < it.nContrib) {
    __syncthreads();
    int code = sMax[buf][0];
#pragma unroll
    for (int w = 1; w < S; ++w) code = max(code, sMax[buf][w]);
    int const ex = fixScaleOf(code);
    if (tid < KC) sx[tid] = tid < n ? fixHalves(xv, ex) : make_int4(0, 0, 0, 0);
    int const big =
        __popc(__ballot_sync(0xffffffffu, tid < n && fixLarge(xv, code - kFixInputGap)));
    if (lane == 0) sBig[warp] = big;
    __syncthreads();
    int all = 0;
#pragma unroll
    for (int w = 0; w < S; ++w) all += sBig[w];
    // the same in every warp: all hold the scales of the same 32 rows
    bool const special = !__all_sync(0xffffffffu, fixCovers(ea, ea, ex)) ||
                         !(code == 0 || fixEven(n, all, cb.graded));
    FixWide re, im;
    int const eaNow = ea;
    if (!special) {
      double2 const *aw = a + (n > warp ? warp * lda : 0);
      int4 const *xw = sx + warp;
#pragma unroll 1
      for (int i = 0; i <= last; i += U, xw += U * S) {
        double2 nv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) nv[u] = aw[min(i + U + u, last) * step];
        int64_t hr = 0, hlr = 0, lhr = 0, hi = 0, hli = 0, lhi = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          int4 const f = fixHalves(av[u], eaNow), y = xw[u * S];
          int const nh = -f.z, nl = -f.w;
          fixMad(hr, f.x, y.x);
          fixMad(hi, f.x, y.z);
          fixMad(hlr, f.x, y.y);
          fixMad(hli, f.x, y.w);
          fixMad(lhr, f.y, y.x);
          fixMad(lhi, f.y, y.z);
          fixMad(hr, nh, y.z);
          fixMad(hi, f.z, y.x);
          fixMad(hlr, nh, y.w);
          fixMad(hli, f.z, y.y);
          fixMad(lhr, nl, y.z);
          fixMad(lhi, f.w, y.x);
        }
        re.add(hr, hlr, lhr);
        im.add(hi, hli, lhi);
#pragma unroll
        for (int u = 0; u < U; ++u) av[u] = nv[u];
      }
      re.settle();
      im.settle();
      part[0][warp][lane] = re.rest;
      partLow[0][warp][lane] = re.low;
      part[1][warp][lane] = im.rest;
      partLow[1][warp][lane] = im.low;
    } else {
      anySpecial = true;
      for (int j = warp; j < n; j += S) cmacc(spr, spi, a[j * lda], x[j * xs]);
    }
    j0 += kSplit * KC;
    if (kSplit > 1) {
      seek();
    } else if (j0 >= cb.n) {
      j0 = 0;
      ++c;
    }
    buf ^= 1;
    if (c < it.nContrib) fetch(buf, false);
    if (!special) {
      __syncthreads();
      if (warp >= S - 2) {
        int const q = warp - (S - 2);
        // units of 2^62
        int64_t h = 0, l = 0;
#pragma unroll
        for (int w = 0; w < S; ++w) {
          h += part[q][w][lane];
          l += partLow[q][w][lane];
        }
        h += l >> 32;
        int const e = eaNow + ex;
        acc = fma((double)h, fixPow(e - 1049), fma((double)(uint32_t)l, fixPow(e - 1081), acc));
      }
    }
  }
  // rare: add the plain FP64 sums of the warps, in order
  if (anySpecial) {
    __syncthreads();
    double *const p = reinterpret_cast<double *>(part);
    p[warp * 32 + lane] = spr;
    p[(S + warp) * 32 + lane] = spi;
    __syncthreads();
    if (warp >= S - 2)
      for (int w = 0; w < S; ++w) acc += p[((warp - (S - 2)) * S + w) * 32 + lane];
  }
  if constexpr (kSplit > 1) {
    // the ranks' sums, in order, through the cluster's shared memory
    __shared__ double sums[2][32];
    auto cluster = cooperative_groups::this_cluster();
    if (warp >= S - 2) sums[warp - (S - 2)][lane] = acc;
    cluster.sync();
    if (rank == 0 && warp >= S - 2)
      for (int q = 1; q < kSplit; ++q)
        acc += *cluster.map_shared_rank(&sums[warp - (S - 2)][lane], q);
    cluster.sync();
    if (rank) return;
  }
  if (warp >= S - 2 && active) reinterpret_cast<double *>(W + it.outRow + lane)[warp - (S - 2)] = acc;
}

template <int NT>
cudaError_t launchTile(ApplyItem const *items, int64_t nItems, ApplyContrib const *contribs,
                       int16_t const *rowExp, double2 const *arena, double2 const *X, int64_t ldx,
                       double2 *W, int64_t R, cudaStream_t stream) {
  int64_t const tiles = (R + 4 * NT - 1) / (4 * NT);
  if (tiles > 0x7fffffff / nItems) return cudaErrorInvalidConfiguration;
  fixTileKernel<NT><<<(unsigned)(nItems * tiles), kFixThreads, 0, stream>>>(
      items, contribs, rowExp, arena, X, ldx, W, R, (unsigned)tiles);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launchRowExp(ApplyItem const *items, int64_t nItems, ApplyContrib *contribs,
                         double2 const *arena, int16_t *rowExp, cudaStream_t stream) {
  if (nItems == 0) return cudaSuccess;
  rowExpKernel<<<(unsigned)nItems, 256, 0, stream>>>(items, contribs, arena, rowExp);
  return cudaGetLastError();
}

cudaError_t launchApplyStageFixed(ApplyItem const *items, int64_t nItems,
                                  ApplyContrib const *contribs, int16_t const *rowExp,
                                  double2 const *arena, double2 const *X, int64_t ldx, double2 *W,
                                  int64_t R, cudaStream_t stream, int64_t nPasses) {
  if (nItems == 0) return cudaSuccess;
  if (R == 1) {
    // CTAs an item: as many as have two passes each, while the grid stays below
    // 16 CTAs an SM (6 are resident, but they end at different times: at
    // 4,096 points 57 us with a limit of 8, 46.5 with 12, 45 with 16, 53 with
    // 24; up to 8 CTAs an item or one and a half passes each gained nothing)
    int split = 1;
    while (split < 4 && nItems * split * 2 <= kGemvCtas && nPasses >= 2 * split * nItems) split *= 2;
    auto kernel = split == 4 ? fixGemvKernel<4> : split == 2 ? fixGemvKernel<2> : fixGemvKernel<1>;
    return launchAfterClusters(kernel, split, dim3((unsigned)(nItems * split)),
                               dim3(32 * kGemvWarps), 0, stream, items, contribs, rowExp, arena, X,
                               ldx, W);
  }
  // the narrowest tile that holds the right-hand sides (an empty column costs as
  // much as a full one: 32,768 points 571 us with 4 columns, 873 with 8,
  // whatever part of them is used), several of 8 for more
  if (R <= 4) return launchTile<1>(items, nItems, contribs, rowExp, arena, X, ldx, W, R, stream);
  return launchTile<2>(items, nItems, contribs, rowExp, arena, X, ldx, W, R, stream);
}

}  // namespace bfg
