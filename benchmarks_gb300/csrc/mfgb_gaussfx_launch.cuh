// mfgb_gaussfx_launch.cuh -- host side of the Gauss-point kernels (mfgb_gaussfx.cuh): thread-block
// shapes, matrix tables and launchers, shared by the Laplacian, Helmholtz and element-kernel
// translation units.
#pragma once
#include <algorithm>
#include <cmath>

#include "mfgb_gaussfx.cuh"
#include "mfgb_launch.cuh"

namespace mfgb {

// Cells per CTA and resident CTAs per SM, the fastest of two to four tried per size for the operators on
// pairs (1.5e7 DoFs, kernel ms; in brackets the best other one; BK3 on the caller's FP64 G takes the
// same, not tried for it).  NQ = NM: 2 1.89 [1.91], 3 0.79 [0.79], 4 0.52 [0.52], 5 0.467
// [0.469], 6 0.547 [0.550], 7 0.56 [0.63], 8 0.51 [0.52], 9 0.72 [0.74].  NQ = NM + 1: 3 5.22
// [5.43], 4 1.50 [1.55], 5 0.98 [1.00], 6 0.85 [0.92], 7 0.84 [0.87], 8 0.73 [0.74], 9 0.83 [0.88],
// 10 1.05 [1.13].
template <int E_, int MB_> struct GaussShapeIs {
  static constexpr int E = E_, MB = MB_;
};
template <int NM, int NQ> struct GaussShape;
template <> struct GaussShape<2, 2> : GaussShapeIs<32, 4> {};
template <> struct GaussShape<3, 3> : GaussShapeIs<14, 4> {};
template <> struct GaussShape<4, 4> : GaussShapeIs<4, 9> {};
template <> struct GaussShape<5, 5> : GaussShapeIs<5, 5> {};
template <> struct GaussShape<6, 6> : GaussShapeIs<3, 4> {};
template <> struct GaussShape<7, 7> : GaussShapeIs<4, 2> {};
template <> struct GaussShape<8, 8> : GaussShapeIs<2, 3> {};
template <> struct GaussShape<9, 9> : GaussShapeIs<1, 3> {};
template <> struct GaussShape<2, 3> : GaussShapeIs<14, 4> {};
template <> struct GaussShape<3, 4> : GaussShapeIs<8, 4> {};
template <> struct GaussShape<4, 5> : GaussShapeIs<5, 5> {};
template <> struct GaussShape<5, 6> : GaussShapeIs<5, 3> {};
template <> struct GaussShape<6, 7> : GaussShapeIs<4, 2> {};
template <> struct GaussShape<7, 8> : GaussShapeIs<2, 2> {};
template <> struct GaussShape<8, 9> : GaussShapeIs<2, 2> {};
template <> struct GaussShape<9, 10> : GaussShapeIs<1, 3> {};

// The tables of B[q*NM+i] and the derivative D[q*NQ+m] at the points (nullptr: none).  Returns
// false when SYM is asked for and a matrix lacks its mirror symmetry.
template <int NM, int NQ, bool SYM>
inline bool fill_gauss(const double *B, const double *D, GaussBasis<NM, NQ, SYM> &t) {
  constexpr int S = SYM ? 1 : 0, A = SYM ? -1 : 0;
  t = {};
  t.K = (float)(2.0 * (1.0 + 0x1p-20));
  double Bt[NM * NQ];
  for (int q = 0; q < NQ; ++q)
    for (int i = 0; i < NM; ++i) Bt[i * NQ + q] = B[q * NM + i];
  if (!fx_line_matrix<NM, NQ, S>(B, t.B) || !fx_line_matrix<NQ, NM, S>(Bt, t.Bt)) return false;
  if (!D) return true;
  double Dt[NQ * NQ];
  for (int q = 0; q < NQ; ++q)
    for (int m = 0; m < NQ; ++m) Dt[m * NQ + q] = D[q * NQ + m];
  if (!fx_line_matrix<NQ, NQ, A>(D, t.D) || !fx_line_matrix<NQ, NQ, A>(Dt, t.Dt)) return false;
  // D B from the symmetric parts (SYM), so that the product keeps the symmetry to rounding
  auto b = [&](int q, int i) {
    return SYM ? 0.5 * (B[q * NM + i] + B[(NQ - 1 - q) * NM + (NM - 1 - i)]) : B[q * NM + i];
  };
  auto d = [&](int q, int m) {
    return SYM ? 0.5 * (D[q * NQ + m] - D[(NQ - 1 - q) * NQ + (NQ - 1 - m)]) : D[q * NQ + m];
  };
  double DB[NQ * NM], DBt[NM * NQ];
  for (int q = 0; q < NQ; ++q)
    for (int i = 0; i < NM; ++i) {
      double s = 0.0, c = 0.0;  // sum with its rounding errors (two-sum and fma)
      for (int m = 0; m < NQ; ++m) {
        const double p = d(q, m) * b(m, i), e = std::fma(d(q, m), b(m, i), -p);
        const double n = s + p, r = n - s;
        c += ((s - (n - r)) + (p - r)) + e;
        s = n;
      }
      DB[q * NM + i] = DBt[i * NQ + q] = s + c;
    }
  return fx_line_matrix<NM, NQ, A>(DB, t.DB) && fx_line_matrix<NQ, NM, A>(DBt, t.DBt);
}

template <int NM, int NQ, class GT, bool EVEC, bool SYM, bool MASS, bool MT>
inline cudaError_t gaussfx_run(int64_t n_cells, const uint32_t *map, const GT *G, const int *gexp,
                               const double *src, double *dst, const GaussBasis<NM, NQ, SYM> &b,
                               cudaStream_t s, const int *done, const float2 *jxw,
                               bool after = false) {
  using Sh = GaussShape<NM, NQ>;
  constexpr int E = Sh::E, T = E * NQ * NQ;
  constexpr size_t smem = GaussLayout<NM, NQ, E, EVEC, 6, 2>::total;
  const auto kernel = gaussfx_kernel<NM, NQ, E, Sh::MB, GT, EVEC, SYM, MASS, MT>;
  static PerDevice found;
  const int per_sm = found([&] { return std::max(1, ctas_per_sm_beside(kernel, T, smem)); });
  const int64_t batches = (n_cells + E - 1) / E;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(batches, (int64_t)per_sm * num_sms()));
  return launch_after(after, kernel, grid, T, smem, s, n_cells, map, G, gexp, src, dst, b, done,
                      device_error_flag(), jxw);
}

// The library's own operators on L-vectors.  Bulk copies of the dof-map tiles need a 16-byte
// aligned map.
template <int NM, int NQ, bool MASS>
inline cudaError_t gaussfx_pairs(int64_t n_cells, const uint32_t *map, const float2 *G,
                                 const int *gexp, const double *src, double *dst, const double *hB,
                                 const double *hDG, cudaStream_t s, const int *done,
                                 const float2 *jxw, bool after) {
  GaussBasis<NM, NQ, true> b;
  if (!fill_gauss(hB, hDG, b)) return cudaErrorInvalidValue;  // GLL and Gauss points are symmetric
  if (reinterpret_cast<uintptr_t>(map) & 15u)
    return gaussfx_run<NM, NQ, float2, false, true, MASS, false>(n_cells, map, G, gexp, src, dst, b,
                                                                 s, done, jxw, after);
  return gaussfx_run<NM, NQ, float2, false, true, MASS, true>(n_cells, map, G, gexp, src, dst, b, s,
                                                              done, jxw, after);
}

}  // namespace mfgb
