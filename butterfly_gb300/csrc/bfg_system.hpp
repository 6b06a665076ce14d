// The boundary-integral system object shared by the solver (bfg_solver.cu)
// and the two-level preconditioner (bfg_coarse.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/bfg.h"
#include "bfg_kernels.cuh"

namespace bfg {

// an owned device allocation that only grows
struct Dev {
  void *p = nullptr;
  size_t bytes = 0;
  Dev() = default;
  Dev(Dev const &) = delete;
  Dev &operator=(Dev const &) = delete;
  ~Dev() { if (p) cudaFree(p); }
  cudaError_t alloc(size_t n) {
    if (n <= bytes) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    cudaError_t e = cudaMalloc(&p, std::max<size_t>(n, 16));
    if (e == cudaSuccess) bytes = n;
    return e;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  template <typename T> T *as() const { return static_cast<T *>(p); }
};

// a pinned landing place for device reads, with the event that says they are in
struct Landing {
  double2 *p = nullptr;
  size_t count = 0;
  cudaEvent_t ready = nullptr;
  Landing() = default;
  Landing(Landing const &) = delete;
  Landing &operator=(Landing const &) = delete;
  ~Landing() {
    if (p) cudaFreeHost(p);
    if (ready) cudaEventDestroy(ready);
  }
  // room for n entries (the old contents are lost; none may be in flight), null on failure
  double2 *ensure(size_t n) {
    if (!ready && cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) != cudaSuccess)
      return nullptr;
    if (n <= count) return p;
    if (p) cudaFreeHost(p);
    p = nullptr;
    count = 0;
    n = std::max<size_t>(2 * n, 256);
    if (cudaMallocHost(reinterpret_cast<void **>(&p), n * sizeof(double2)) != cudaSuccess)
      return p = nullptr;
    count = n;
    return p;
  }
};

// Pieces of `step` rows of the curves' ranges [start[b], start[b + 1]), one
// thread block each: their number follows the rows, however uneven the curves.
// (One curve of 2,000 points among 4,000 of 8, an iteration of GMRES with
// block-Jacobi: 1,256 us; with a grid of curves x the largest one's pieces,
// most of them empty, 1,734.)
struct CurveTile {
  int32_t curve, first;
};
inline std::vector<CurveTile> curveTiles(std::vector<int64_t> const &start, int step) {
  std::vector<CurveTile> t;
  for (size_t b = 0; b + 1 < start.size(); ++b)
    for (int64_t i = 0; i < start[b + 1] - start[b]; i += step)
      t.push_back(CurveTile{(int32_t)b, (int32_t)i});
  return t;
}

}  // namespace bfg

struct bfgSystem_s {
  using Dev = bfg::Dev;
  bfgContext ctx = nullptr;
  bfgFac fac = nullptr;
  int64_t n = 0, numCurves = 0;
  int32_t order = 0;
  double shift = 0.5;
  bfgPrecision applyPrec = BFG_PRECISION_FP64;   // of the butterfly part
  bfg::KernelParams kp{};
  std::vector<int64_t> offsets;
  std::vector<double> weights;                   // host copy (coarse mode counts)
  Dev dOffsets, dCurveOf, dX, dW, dKrVal, dKrCol;
  Dev tmpXw;
  bfg::Landing column;   // the solver's Hessenberg column
  // block-Jacobi
  bool haveBj = false, haveBj64 = false;   // the FP32 inverses; the FP64 ones (on first use)
  std::vector<int64_t> blkOff;
  int64_t bjTiles = 0;
  Dev dBjTiles;   // CurveTile
  Dev dBlkOff, dInv, dInv32, dWork, dColBuf, dPerm, dFlag;
  // learned preconditioner: chunks of consecutive points of a curve
  bfgMlp mlp = nullptr;
  int32_t chunk = 0;
  int64_t nChunks = 0;
  Dev dChunkStart, dChunkLen, dFeat, dOut, dScale, dZbj;
  // two-level preconditioner: per-curve Fourier coarse space Phi (curve b's
  // modes at coarse rows cStart[b] .. cStart[b+1], its basis table
  // n_b x M_b row-major complex64 at tabOff[b]), A_c = Phi^H A Phi and its
  // inverse (complex64, row-major)
  bool haveCoarse = false;
  int64_t coarseDim = 0;
  std::vector<int64_t> cStart, tabOff;
  int64_t modeTiles = 0, pointTiles = 0;
  Dev dModeTiles, dPointTiles;   // CurveTile
  Dev dCStart, dTabOff, dTab, dAc, dAcInv, dCoarseIn, dCoarseOut, dZ1, dT1, dT2;
  std::string err;
  cudaStream_t stream() const;
};

namespace bfg {
// one apply of a factorization inside a system (bfg_api.cpp)
bfgStatus facApplySystem(bfgFac f, bfgPrecision prec, SystemTerms const &sys, double2 *Y);
// A X for one device complex128 vector with the butterfly part in `prec`
bfgStatus systemApplyPrec(bfgSystem sys, bfgPrecision prec, void const *X, void *Y);
// z = M_bj (r - sub) + add from the FP32 block inverses (block-Jacobi built)
void applyBlockJacobi32(bfgSystem sys, double2 const *r, double2 const *sub, double2 const *add,
                        double2 *z, cudaStream_t s);
// the two-level preconditioner z = z1 + M_bj (r - A z1), z1 = Phi A_c^-1 Phi^H r
bfgStatus applyTwoLevel(bfgSystem sys, double2 const *r, double2 *z);
}  // namespace bfg
