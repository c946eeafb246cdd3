// The FP64-accurate BP3 operator and Gauss p+1 Laplacian in offset double-float arithmetic
// (mfgb_gaussfx.cuh).
#include "mfgb_gaussfx_launch.cuh"
#include "mfgb_internal.h"

namespace mfgb {

cudaError_t bp3_fx(int degree, int nq, int64_t n_cells, const uint32_t *map, const float2 *Gfx,
                   const int *gexp, const double *src, double *dst, const double *hB,
                   const double *hDG, cudaStream_t s, const int *done, const float2 *jxw,
                   bool after_start) {
  if (n_cells <= 0) return cudaSuccess;
  if (map == nullptr || (reinterpret_cast<uintptr_t>(Gfx) & 15u)) return cudaErrorInvalidValue;
  const int extra = nq - degree - 1;  // 1: BP3 (q = p + 2), 0: Gauss p + 1
  if (extra != 0 && extra != 1) return cudaErrorInvalidValue;
  if (jxw != nullptr)  // the Helmholtz form (Gauss p + 1 with the mass term)
    return extra == 0 ? helmholtz_fx(degree, n_cells, map, Gfx, gexp, jxw, src, dst, hB, hDG, s, done,
                                     after_start)
                      : cudaErrorInvalidValue;
  switch (degree * 2 + extra) {
#define MFGB_BP3FX(P, X)                                                                            \
  case 2 * P + X:                                                                                   \
    return gaussfx_pairs<P + 1, P + 1 + X, false>(n_cells, map, Gfx, gexp, src, dst, hB, hDG, s, done, \
                                                  nullptr, after_start);
    MFGB_BP3FX(1, 1) MFGB_BP3FX(2, 1) MFGB_BP3FX(3, 1) MFGB_BP3FX(4, 1) MFGB_BP3FX(5, 1)
    MFGB_BP3FX(6, 1) MFGB_BP3FX(7, 1) MFGB_BP3FX(8, 1)
    MFGB_BP3FX(1, 0) MFGB_BP3FX(2, 0) MFGB_BP3FX(3, 0) MFGB_BP3FX(4, 0) MFGB_BP3FX(5, 0)
    MFGB_BP3FX(6, 0) MFGB_BP3FX(7, 0) MFGB_BP3FX(8, 0)
#undef MFGB_BP3FX
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace mfgb
