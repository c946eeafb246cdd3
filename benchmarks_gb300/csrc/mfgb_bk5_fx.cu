// The FP64-accurate collocation operator with offset double-float accumulation
// (mfgb_bk5fx.cuh): its launcher, and the set-up of the per-cell scaled
// geometric factors it reads.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "mfgb_bk5fx.cuh"
#include "mfgb_internal.h"
#include "mfgb_launch.cuh"

namespace mfgb {

// Cells per CTA, resident CTAs per SM and work arrays of the two thread-block shapes (5 and 6 of
// the shape table).  Cells per CTA fill whole warps as far as they can (n = 5: 125 of 128 lanes,
// n = 6: 108 of 128, n = 7: 147 of 160); from n = 5 the two-array form buys one more resident CTA
// (n = 5: 44.8 KB a CTA, 96 registers, 5 CTAs).
// Kernel ms at 3e7 DoFs, shape 5 / 6: n = 2 3.07 / 3.12, 3 1.23 / 1.22, 4 0.745 / 0.745, 5 0.653 / 0.660,
// 6 0.708 / 0.706, 7 0.722 / 0.779, 8 0.629 / 0.652, 9 0.837 / 0.830 and at 8e6 DoFs 0.239 / 0.229 (its
// default is shape 6).  The kernel with one contraction output per thread and step that this one replaced,
// its better shape: 3.47, 1.85, 0.93, 0.92, 1.02, 1.20, 1.00, 1.45.  Measured for the scalar operator on
// pairs; BK6 (three components) and the seams on the caller's FP64 G take the cells per CTA of shape 5,
// which were not tried one by one for them.
template <int E_, int MB_, int NB_> struct FxShape {
  static constexpr int E = E_, MB = MB_, NB = NB_;
};
template <int N> struct FxDefault;
template <int N> struct FxAlt;
template <> struct FxDefault<2> : FxShape<32, 4, 3> {};
template <> struct FxDefault<3> : FxShape<7, 6, 3> {};
template <> struct FxDefault<4> : FxShape<4, 7, 3> {};
template <> struct FxDefault<5> : FxShape<5, 5, 2> {};
template <> struct FxDefault<6> : FxShape<3, 5, 2> {};
template <> struct FxDefault<7> : FxShape<3, 3, 2> {};
template <> struct FxDefault<8> : FxShape<2, 3, 2> {};
template <> struct FxDefault<9> : FxShape<1, 4, 2> {};
template <> struct FxAlt<2> : FxShape<16, 6, 3> {};
template <> struct FxAlt<3> : FxShape<14, 4, 3> {};
template <> struct FxAlt<4> : FxShape<8, 4, 3> {};
template <> struct FxAlt<5> : FxShape<5, 4, 3> {};
template <> struct FxAlt<6> : FxShape<5, 3, 2> {};
template <> struct FxAlt<7> : FxShape<2, 4, 2> {};
template <> struct FxAlt<8> : FxShape<1, 5, 2> {};
template <> struct FxAlt<9> : FxShape<2, 2, 2> {};

// test hook: applications left whose first copy wait is made to run out
static std::atomic<int> g_expire{0};

static bool take_expire() {
  for (int c = g_expire.load(); c > 0; c = g_expire.load())
    if (g_expire.compare_exchange_weak(c, c - 1)) return true;
  return false;
}

template <int N, int SYM>
static bool fx_basis(const double *D, FxBasis<N, SYM> &b) {
  double Dt[N * N];
  for (int i = 0; i < N; ++i)
    for (int m = 0; m < N; ++m) Dt[i * N + m] = D[m * N + i];
  b.K = (float)(2.0 * (1.0 + std::ldexp(1.0, -20)));
  return fx_line_matrix<N, N, SYM>(D, b.G) && fx_line_matrix<N, N, SYM>(Dt, b.T);
}

// one launch of the kernel: all resident CTAs, capped by the batches
template <int N, class Sh, class GT, bool EVEC, int NC, int SYM, bool MT, bool EXPIRE = false>
static cudaError_t fx_run(int64_t n_cells, const uint32_t *map, const GT *G, const int *gexp,
                          const double *src, double *dst, const FxBasis<N, SYM> &b, cudaStream_t s,
                          const int *done, bool after = false) {
  constexpr int E = Sh::E, T = E * N * N;
  constexpr size_t smem = FxLayout<N, E, GT, EVEC, Sh::NB>::total;
  const auto kernel = bk5fx_kernel<N, E, Sh::MB, Sh::NB, GT, EVEC, NC, SYM, MT, EXPIRE>;
  static PerDevice found;
  const int per_sm = found([&] { return std::max(1, ctas_per_sm_beside(kernel, T, smem)); });
  const int64_t nb = (n_cells + E - 1) / E;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(nb, (int64_t)per_sm * num_sms()));
  return launch_after(after, kernel, grid, T, smem, s, n_cells, map, G, gexp, src, dst, b, done,
                      device_error_flag());
}

// The kernel on the library's own scaled pairs.  Bulk copies of the dof-map tiles need a 16-byte
// aligned map.
template <int N, int NC>
static cudaError_t fx_pairs(int64_t n_cells, const uint32_t *map, const float2 *G, const int *gexp,
                            const double *src, double *dst, const double *D, cudaStream_t s,
                            const int *done, bool after) {
  FxBasis<N, -1> b;
  if (!fx_basis<N, -1>(D, b)) return cudaErrorInvalidValue;  // the GLL derivative has the symmetry
  using Sh = FxDefault<N>;
  const bool mt = (reinterpret_cast<uintptr_t>(map) & 15u) == 0;
  if (NC == 1 && take_expire())
    return fx_run<N, Sh, float2, false, 1, -1, false, true>(n_cells, map, G, gexp, src, dst, b, s,
                                                            done, after);
  if constexpr (NC == 1) {
    using Alt = FxAlt<N>;
    if (kernel_shape(ArithClass<ArithDF>::value, N) == SHAPE_FX_ALT)
      return mt ? fx_run<N, Alt, float2, false, 1, -1, true>(n_cells, map, G, gexp, src, dst, b, s, done, after)
                : fx_run<N, Alt, float2, false, 1, -1, false>(n_cells, map, G, gexp, src, dst, b, s, done, after);
  }
  return mt ? fx_run<N, Sh, float2, false, NC, -1, true>(n_cells, map, G, gexp, src, dst, b, s, done, after)
            : fx_run<N, Sh, float2, false, NC, -1, false>(n_cells, map, G, gexp, src, dst, b, s, done, after);
}

// The kernel on the caller's FP64 G (16-byte aligned): L-vectors through map, or element vectors
// (map == nullptr).  A derivative matrix without the mirror symmetry of symmetric points keeps
// the general form.
template <int N, int SYM>
static cudaError_t fx_seam(int64_t n_cells, const uint32_t *map, const double *G, const double *src,
                           double *dst, const FxBasis<N, SYM> &b, cudaStream_t s) {
  // (the general form keeps N^2 matrix entries live: its register cap is the wider one)
  using Sh = FxShape<FxDefault<N>::E, SYM == 0 ? (FxDefault<N>::MB + 1) / 2 : FxDefault<N>::MB,
                     FxDefault<N>::NB>;
  if (map == nullptr)
    return fx_run<N, Sh, double, true, 1, SYM, false>(n_cells, nullptr, G, nullptr, src, dst, b, s, nullptr);
  if (reinterpret_cast<uintptr_t>(map) & 15u)
    return fx_run<N, Sh, double, false, 1, SYM, false>(n_cells, map, G, nullptr, src, dst, b, s, nullptr);
  return fx_run<N, Sh, double, false, 1, SYM, true>(n_cells, map, G, nullptr, src, dst, b, s, nullptr);
}

template <int N>
static cudaError_t fx_seam_any(int64_t n_cells, const uint32_t *map, const double *G,
                               const double *src, double *dst, const double *D, cudaStream_t s) {
  FxBasis<N, -1> b;
  if (fx_basis<N, -1>(D, b)) return fx_seam<N, -1>(n_cells, map, G, src, dst, b, s);
  FxBasis<N, 0> general;
  fx_basis<N, 0>(D, general);
  return fx_seam<N, 0>(n_cells, map, G, src, dst, general, s);
}

#define MFGB_FX_DEGREES(CALL) \
  switch (N) {                \
    case 2: return CALL(2);   \
    case 3: return CALL(3);   \
    case 4: return CALL(4);   \
    case 5: return CALL(5);   \
    case 6: return CALL(6);   \
    case 7: return CALL(7);   \
    case 8: return CALL(8);   \
    case 9: return CALL(9);   \
    default: return cudaErrorInvalidValue; \
  }

cudaError_t bk5_fx_g64(int N, int64_t n_cells, const uint32_t *map, const double *G,
                       const double *src, double *dst, const double *D, cudaStream_t s) {
  if (n_cells <= 0) return cudaSuccess;
  if (map == nullptr || (reinterpret_cast<uintptr_t>(G) & 15u)) return cudaErrorInvalidValue;
#define MFGB_CALL(NN) (fx_seam_any<NN>(n_cells, map, G, src, dst, D, s))
  MFGB_FX_DEGREES(MFGB_CALL)
#undef MFGB_CALL
}

cudaError_t bk5_fx_evec(int N, int64_t nelmt, const double *G, const double *src, double *dst,
                        const double *D, cudaStream_t s) {
  if (nelmt <= 0) return cudaSuccess;
  if (reinterpret_cast<uintptr_t>(G) & 15u) return cudaErrorInvalidValue;  // bulk copies
#define MFGB_CALL(NN) (fx_seam_any<NN>(nelmt, nullptr, G, src, dst, D, s))
  MFGB_FX_DEGREES(MFGB_CALL)
#undef MFGB_CALL
}

// the BK6 vector Laplacian: 3 interleaved components per DoF on one scaled G
cudaError_t bk6_fx(int N, int64_t n_cells, const uint32_t *map, const float2 *G, const int *gexp,
                   const double *src, double *dst, const double *D, cudaStream_t s,
                   bool after_start) {
  if (n_cells <= 0) return cudaSuccess;
  if (map == nullptr || (reinterpret_cast<uintptr_t>(G) & 15u)) return cudaErrorInvalidValue;
#define MFGB_CALL(NN) (fx_pairs<NN, 3>(n_cells, map, G, gexp, src, dst, D, s, nullptr, after_start))
  MFGB_FX_DEGREES(MFGB_CALL)
#undef MFGB_CALL
}

cudaError_t bk5_fx(int N, int64_t n_cells, const uint32_t *map, const float2 *G, const int *gexp,
                   const double *src, double *dst, const double *D, cudaStream_t s,
                   const int *done, bool after_start) {
  if (n_cells <= 0) return cudaSuccess;
  if (map == nullptr || (reinterpret_cast<uintptr_t>(G) & 15u)) return cudaErrorInvalidValue;
#define MFGB_CALL(NN) (fx_pairs<NN, 1>(n_cells, map, G, gexp, src, dst, D, s, done, after_start))
  MFGB_FX_DEGREES(MFGB_CALL)
#undef MFGB_CALL
}

// Per-cell scaled split of the FP64 geometric factors: one warp per cell finds
// the largest biased exponent e among the cell's 6 n^3 values (and its per_j
// JxW values, when given) and writes them times 2^-(e - 1022) as float pairs
// (hi = nearest float, lo = nearest float of the remainder); gexp[cell] =
// e - 1022 (0 for an all-zero cell).  Values more than 2^126 below the cell's
// largest lose their low digits or flush to zero, far below the operator's
// accuracy bar relative to the cell's largest term.  nt > 0: the nt^3 points of
// every component are written with their first and last index exchanged (the
// order the Gauss-point kernel reads).
__global__ void g_to_fx_kernel(int64_t n_cells, int per_cell, const double *__restrict__ G,
                               float2 *__restrict__ out, int *__restrict__ gexp, int per_j,
                               const double *__restrict__ J, float2 *__restrict__ jout, int nt) {
  auto from = [=](int t) {
    if (nt == 0) return t;
    const int n2 = nt * nt, c = t / (n2 * nt), r = t - c * n2 * nt;
    const int a = r / n2, b = (r - a * n2) / nt, d = r - a * n2 - b * nt;
    return (c * nt + d) * n2 + b * nt + a;
  };
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  auto split = [](double x, int off) {
    const double y = scalbn(x, -off);
    const float hi = __double2float_rn(y);
    return make_float2(hi, __double2float_rn(y - (double)hi));
  };
  for (int64_t c = warp; c < n_cells; c += n_warps) {
    const double *g = G + c * per_cell;
    const double *j = J + c * per_j;
    int em = 0;
    for (int t = lane; t < per_cell; t += 32) {
      const int e = dexp(g[t]);
      em = max(em, e == 0x7FF ? 0 : e);
    }
    for (int t = lane; t < per_j; t += 32) {
      const int e = dexp(j[t]);
      em = max(em, e == 0x7FF ? 0 : e);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) em = max(em, __shfl_xor_sync(0xFFFFFFFFu, em, o));
    const int off = fx_offset(em);
    for (int t = lane; t < per_cell; t += 32) out[c * per_cell + t] = split(g[from(t)], off);
    for (int t = lane; t < per_j; t += 32) jout[c * per_j + t] = split(j[from(t)], off);
    if (lane == 0) gexp[c] = off;
  }
}

cudaError_t g_to_fx(int64_t n_cells, int per_cell, const double *G, float2 *Gfx, int *gexp,
                    cudaStream_t s, int per_cell_j, const double *J, float2 *Jfx, int nt) {
  if (n_cells <= 0) return cudaSuccess;
  if (per_cell_j > 0 && (!J || !Jfx)) return cudaErrorInvalidValue;
  const int64_t blocks = std::min<int64_t>((n_cells + 7) / 8, 152 * 32);
  g_to_fx_kernel<<<(int)blocks, 256, 0, s>>>(n_cells, per_cell, G, Gfx, gexp,
                                             per_cell_j > 0 ? per_cell_j : 0, J, Jfx, nt);
  return cudaGetLastError();
}

}  // namespace mfgb

extern "C" mfgb_status mfgb_test_expire_copy_wait(int n) {
  if (n < 0) {
    mfgb::set_error("mfgb_test_expire_copy_wait: n must be >= 0");
    return MFGB_ERR_INVALID_ARG;
  }
  mfgb::g_expire.store(n);
  return MFGB_OK;
}
