// The CEED BK1 and BK3 element kernels in offset double-float arithmetic (mfgb_gaussfx.cuh) on the
// caller's arrays: matrices of points symmetric about the centre run in even-odd form, others and BK1's
// of degree 1 in the general one.
#include "mfgb_gaussfx_launch.cuh"
#include "mfgb_internal.h"

namespace mfgb {
namespace {

template <int NM, int NQ>
cudaError_t bk3(int64_t nelmt, const double *G, const double *in, double *out, const double *hB,
                const double *hDG, cudaStream_t s) {
  GaussBasis<NM, NQ, true> b;
  if (fill_gauss(hB, hDG, b))
    return gaussfx_run<NM, NQ, double, true, true, false, false>(nelmt, nullptr, G, nullptr, in, out,
                                                                 b, s, nullptr, nullptr);
  GaussBasis<NM, NQ, false> g;
  fill_gauss(hB, hDG, g);
  return gaussfx_run<NM, NQ, double, true, false, false, false>(nelmt, nullptr, G, nullptr, in, out,
                                                                g, s, nullptr, nullptr);
}

// Cells per CTA and resident CTAs per SM of the mass kernel, as the Laplacian's but where the missing
// geometry tile leaves room for more CTAs (ms on the mesh of the
// Laplacian's figures, against its shape: NQ = 7 0.434 / 0.496, 9 0.413 / 0.424, 10 0.459 / 0.502).
template <int NM, int NQ> struct Bk1Shape : GaussShape<NM, NQ> {};
template <> struct Bk1Shape<6, 7> : GaussShapeIs<3, 3> {};
template <> struct Bk1Shape<8, 9> : GaussShapeIs<1, 4> {};
template <> struct Bk1Shape<9, 10> : GaussShapeIs<1, 4> {};

template <int NM, int NQ, bool SYM>
cudaError_t bk1_run(int64_t nelmt, const double *in, const double *JxW, double *out,
                    const GaussBasis<NM, NQ, SYM> &b, cudaStream_t s) {
  using Sh = Bk1Shape<NM, NQ>;
  constexpr int E = Sh::E, T = E * NQ * NQ;
  constexpr size_t smem = sizeof(df) * E * GaussStride<NQ>::cell;
  const auto kernel = bk1fx_kernel<NM, NQ, E, Sh::MB, SYM>;
  static PerDevice found;
  const int per_sm = found([&] { return std::max(1, ctas_per_sm(kernel, T, smem)); });
  const int64_t batches = (nelmt + E - 1) / E;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(batches, (int64_t)per_sm * num_sms()));
  kernel<<<grid, T, smem, s>>>(nelmt, in, JxW, out, b.B, b.Bt, b.K);
  return cudaGetLastError();
}

template <int NM, int NQ>
cudaError_t bk1(int64_t nelmt, const double *in, const double *JxW, double *out, const double *hB,
                cudaStream_t s) {
  // (two nodes: the general form, whose error on smooth values is 0.96 of the plain kernel's against
  // 1.04 in even-odd form; 20.3 / 21.0 us at 1e5 values, 0.266 / 0.257 ms at 1.2e7)
  if constexpr (NM > 2) {
    GaussBasis<NM, NQ, true> b;
    if (fill_gauss(hB, nullptr, b)) return bk1_run(nelmt, in, JxW, out, b, s);
  }
  GaussBasis<NM, NQ, false> g;
  fill_gauss(hB, nullptr, g);
  return bk1_run(nelmt, in, JxW, out, g, s);
}

}  // namespace

cudaError_t bk3_fx(int degree, int64_t nelmt, const double *G, const double *in, double *out,
                   const double *hB, const double *hDG, cudaStream_t s) {
  if (nelmt <= 0) return cudaSuccess;
  if (reinterpret_cast<uintptr_t>(G) & 15u) return cudaErrorInvalidValue;  // bulk copies
  switch (degree) {
#define MFGB_BK3FX(P) \
  case P: return bk3<P + 1, P + 2>(nelmt, G, in, out, hB, hDG, s);
    MFGB_BK3FX(1) MFGB_BK3FX(2) MFGB_BK3FX(3) MFGB_BK3FX(4) MFGB_BK3FX(5) MFGB_BK3FX(6)
    MFGB_BK3FX(7) MFGB_BK3FX(8)
#undef MFGB_BK3FX
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t bk1_fx(int degree, int64_t nelmt, const double *in, const double *JxW, double *out,
                   const double *hB, cudaStream_t s) {
  if (nelmt <= 0) return cudaSuccess;
  switch (degree) {
#define MFGB_BK1FX(P) \
  case P: return bk1<P + 1, P + 2>(nelmt, in, JxW, out, hB, s);
    MFGB_BK1FX(1) MFGB_BK1FX(2) MFGB_BK1FX(3) MFGB_BK1FX(4) MFGB_BK1FX(5) MFGB_BK1FX(6)
    MFGB_BK1FX(7) MFGB_BK1FX(8)
#undef MFGB_BK1FX
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace mfgb
