// mfgb_gaussfx.cuh -- operators with interpolation to NQ Gauss points per direction (NQ = NM or
// NM + 1) in offset double-float arithmetic: the BP5 Laplacian at p + 1 points
// (bakeoff_problems_dealii/include/bk3_kokkos_kernel.h:156-404), its Helmholtz form
// (bp5_kokkos/benchmark.cc:51-251), BP3 at p + 2 points (CEED_bp/include/bk3_kokkos_kernel.h:146-354)
// and the CEED BK3 / BK1 element kernels (CEED_BK/include/kernels/BK3/serial_kernels.hpp:29-188,
// BK1/serial_kernels.hpp:20-121).
//
// Scaling and accumulation as in mfgb_bk5fx.cuh (per-cell powers of two for the values and the
// geometric factors; offsets from the data), every contraction by whole lines (mfgb_fxline.cuh).
// The three directions are named by their part in the kernel:
//   F   first interpolated and last integrated: its lines are the gathered columns
//   M   the middle one
//   L   the last interpolated: the thread that owns an L-line at the points keeps its values, its
//       derivative and the metric's L-flux in registers, and the derivative along L is folded into
//       the interpolation (DB = D B, and its transpose on the way back), so that direction needs
//       no pass over shared memory of its own
// L-vectors use F, M, L = 0, 1, 2 (slowest to fastest node index: coalesced columns) with the
// geometric factors stored point-transposed, [cell][6][l][m][f]; element vectors use 2, 1, 0, so
// the caller's [e][6][point] order has the same meaning.
//
// What bounds it: multiply-adds, 195 a column at NM = NQ = 5 against 345 of the dense form with one
// output per thread and step, at 6 instructions each.
#pragma once
#include "mfgb_bk5fx.cuh"

namespace mfgb {

// SYM: every matrix in even-odd form (points symmetric about the centre), else general
template <int NM, int NQ, bool SYM>
struct GaussBasis {
  static constexpr int S = SYM ? 1 : 0, A = SYM ? -1 : 0;
  FxMat<NM, NQ, S> B;     // values at the points
  FxMat<NM, NQ, A> DB;    // derivatives at the points, D B
  FxMat<NQ, NQ, A> D, Dt;  // collocation derivative at the points
  FxMat<NQ, NM, S> Bt;
  FxMat<NQ, NM, A> DBt;
  float K;  // 2 (1 + 2^-20)
};

// Strides of a cell's work array (cell, l, m; f contiguous), padded so that the kernel's accesses
// spread over the 8-byte banks; wavefronts of one batch against the plain strides and the least
// possible, counted on the host for NM = NQ: 4 368 / 1040 (368), 5 1000 / 1210 (920),
// 6 1014 / 1542 (966), 8 1472 / 4672 (1472), 9 1422 / 1458 (1242).
template <int NQ> struct GaussStride;
#define MFGB_GSTRIDE(NN, CELL, L, M) \
  template <> struct GaussStride<NN> { static constexpr int cell = CELL, l = L, m = M; };
MFGB_GSTRIDE(2, 12, 6, 2) MFGB_GSTRIDE(3, 27, 9, 3) MFGB_GSTRIDE(4, 68, 17, 4)
MFGB_GSTRIDE(5, 153, 29, 5) MFGB_GSTRIDE(6, 260, 41, 6) MFGB_GSTRIDE(7, 369, 51, 7)
MFGB_GSTRIDE(8, 520, 65, 8) MFGB_GSTRIDE(9, 738, 82, 9) MFGB_GSTRIDE(10, 1030, 103, 10)
#undef MFGB_GSTRIDE

// work-array offsets of the lines each thread owns: M-lines at (point f, node l), M-lines at
// (point f, point l), F-lines at (point m, point l)
template <int NM, int NQ, int E>
struct GaussLines {
  unsigned short mn[E * NQ * NM], mq[E * NQ * NQ], f[E * NQ * NQ];
};
template <int NM, int NQ, int E>
constexpr GaussLines<NM, NQ, E> gauss_lines() {
  using S = GaussStride<NQ>;
  GaussLines<NM, NQ, E> r{};
  int a[E * NQ * NM] = {}, b[E * NQ * NQ] = {}, c[E * NQ * NQ] = {};
  for (int q = 0; q < E * NQ * NM; ++q) a[q] = q / (NQ * NM) * S::cell + q / NM % NQ + q % NM * S::l;
  for (int q = 0; q < E * NQ * NQ; ++q) {
    const int e = q / (NQ * NQ), i = q / NQ % NQ, l = q % NQ;
    b[q] = e * S::cell + i + l * S::l;
    c[q] = e * S::cell + i * S::m + l * S::l;
  }
  fx_deal(a, r.mn);
  fx_deal(b, r.mq);
  fx_deal(c, r.f);
  return r;
}
template <int NM, int NQ, int E>
__device__ const GaussLines<NM, NQ, E> gauss_line_table = gauss_lines<NM, NQ, E>();

// shared memory of one CTA: G tile (NG components), dof-map tile, NB work arrays, two mbarriers
template <int NM, int NQ, int E, bool EVEC, int NG, int NB>
struct GaussLayout {
  static constexpr size_t g_bytes = sizeof(double) * E * NG * NQ * NQ * NQ;
  static constexpr size_t map_bytes = EVEC ? 0 : ((size_t)E * NM * NM * NM * 4 + 12 + 15) / 16 * 16;
  static constexpr size_t work_bytes = sizeof(df) * NB * E * GaussStride<NQ>::cell;
  static constexpr size_t total = g_bytes + map_bytes + (work_bytes + 15) / 16 * 16 + 16;
};

// Lines x[n] at base + i * stride of a work array
template <int N>
__device__ __forceinline__ void load_line(df (&x)[N], const df *w, int stride) {
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = w[i * stride];
}
template <int N>
__device__ __forceinline__ void store_line(const df (&x)[N], df *w, int stride) {
#pragma unroll
  for (int i = 0; i < N; ++i) w[i * stride] = x[i];
}

// a gathered or loaded column to pairs on the common grid of its cell (largest exponent emax)
// (GRID = false: the pairs as they are)
template <bool GRID = true, int N>
__device__ __forceinline__ void fx_column(const double (&raw)[N], int emax, df (&x)[N]) {
  const int su = fx_offset(emax);
  if constexpr (!GRID) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = fx_from_double(raw[i], su);
  } else if ((unsigned)(emax - 1) < 0x7FEu) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = fx_from_double_grid(raw[i], su);
  } else {  // all zero or subnormal, or an inf or NaN among the values
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = fx_grid(fx_from_double(raw[i], su), 3.f);
  }
}

// largest |value| of a column as a biased exponent, into the cell's slot
template <int N>
__device__ __forceinline__ void fx_column_exp(const double (&raw)[N], int *slot) {
  unsigned em = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) em = max(em, (unsigned)(__double_as_longlong(raw[i]) >> 32) & 0x7FFFFFFFu);
  if (em >> 20) atomicMax(slot, (int)(em >> 20));
}

// Laplacian (MASS: plus the mass term JxW u, jxw as pairs on the cell's G scale, point-transposed
// like G).  E NQ^2 threads; the first E NM^2 own the node columns, thread (el, m, f) the L-line
// (m, f) of cell el.  G arrives a batch ahead by bulk copy, the dof map by the 16-byte aligned
// window around its tile (MAPTMA: the map array is 16-byte aligned), the gather a batch ahead in
// registers.  EVEC: contiguous element vectors, dst written; GT = double: the caller's FP64 G,
// scaled per element inside the kernel.
template <int NM, int NQ, int E, int MB, class GT, bool EVEC, bool SYM, bool MASS, bool MAPTMA>
__global__ void __launch_bounds__(E * NQ * NQ, MB)
    gaussfx_kernel(const int64_t n_cells, const uint32_t *__restrict__ map,
                   const GT *__restrict__ G, const int *__restrict__ gexp,
                   const double *__restrict__ src, double *__restrict__ dst,
                   const GaussBasis<NM, NQ, SYM> basis, const int *__restrict__ done_flag,
                   int *__restrict__ err_flag, const float2 *__restrict__ jxw) {
  if (done_flag != nullptr && *done_flag) return;
  using L = GaussLayout<NM, NQ, E, EVEC, 6, 2>;
  using S = GaussStride<NQ>;
  constexpr int M2 = NM * NM, M3 = M2 * NM, Q2 = NQ * NQ, Q3 = Q2 * NQ;
  constexpr bool G64 = std::is_same<GT, double>::value;
  extern __shared__ __align__(128) unsigned char smem[];
  GT *sG = reinterpret_cast<GT *>(smem);
  uint32_t *sMap = reinterpret_cast<uint32_t *>(smem + L::g_bytes);
  df *U = reinterpret_cast<df *>(smem + L::g_bytes + L::map_bytes);
  df *V = U + E * S::cell;
  uint64_t *mbar_g = reinterpret_cast<uint64_t *>(smem + L::total - 16), *mbar_m = mbar_g + 1;
  __shared__ int s_emax[2][E];
  __shared__ int s_gmax[E];  // G64: largest biased exponent of the element's G

  const int tid = threadIdx.x;
  const int el = tid / Q2, mf = tid - el * Q2;  // the owned L-line
  const int own = el * S::cell + mf / NQ * S::m + mf % NQ;
  const bool has_col = tid < E * M2;            // the owned node column
  const int gc = has_col ? tid / M2 : 0, jk = has_col ? tid - gc * M2 : 0;
  // column (m, l): L-vectors order the columns m-major as the map does, element vectors l-major
  const int col = gc * S::cell + (EVEC ? jk % NM * S::m + jk / NM * S::l : jk / NM * S::m + jk % NM * S::l);
  const bool has_mn = tid < E * NQ * NM;
  const int mn = has_mn ? gauss_line_table<NM, NQ, E>.mn[tid] : 0;
  const int mq = gauss_line_table<NM, NQ, E>.mq[tid], fq = gauss_line_table<NM, NQ, E>.f[tid];
  const int64_t n_batches = (n_cells + E - 1) / E;
  int64_t batch = blockIdx.x;
  if (batch >= n_batches) return;  // uniform across the CTA

  auto cells_of = [&](int64_t b) { return (int)min((int64_t)E, n_cells - b * E); };
  auto issue_g = [&](int64_t b) {
    const uint32_t bytes = (uint32_t)(sizeof(GT) * cells_of(b) * 6 * Q3);
    mbar_arrive_expect_tx(mbar_g, bytes);
    bulk_g2s(sG, G + b * E * 6 * Q3, bytes, mbar_g);
  };
  auto map_window = [&](int64_t b) -> uint32_t {  // bytes, 0: no bulk copy
    const int64_t first = b * E * M3, last = first + (int64_t)cells_of(b) * M3;
    const int64_t end = (last + 3) & ~(int64_t)3;
    return MAPTMA && end <= n_cells * M3 ? (uint32_t)(end - (first & ~(int64_t)3)) * 4u : 0u;
  };
  auto issue_map = [&](int64_t b) {
    const uint32_t bytes = map_window(b);
    mbar_arrive_expect_tx(mbar_m, bytes);
    if (bytes) bulk_g2s(sMap, map + ((b * E * M3) & ~(int64_t)3), bytes, mbar_m);
  };
  auto fail = [&](uint32_t pg, uint32_t pm) {
    if (tid == 0 && err_flag) atomicOr(err_flag, 1);
    mbar_wait(mbar_g, pg);  // bounded waits for copies still in flight
    if (!EVEC) mbar_wait(mbar_m, pm);
  };

  if (tid < 2 * E) (&s_emax[0][0])[tid] = 0;
  if (G64 && tid < E) s_gmax[tid] = 0;
  if (tid == 0) {
    mbar_init(mbar_g, 1);
    mbar_init(mbar_m, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (tid == 0) {
    issue_g(batch);
    if (!EVEC) issue_map(batch);
  }
  uint32_t ph_g = 0, ph_m = 0;
  uint32_t idx[NM];
  double raw[NM];
  int ge = 0;  // G exponent offset of the column's cell in the prefetched batch
  // dof indices of the column of batch b, from the map window or global
  auto indices = [&](int64_t b) {
    const bool ok = has_col && gc < cells_of(b);
    if (map_window(b)) {
      const uint32_t *m = sMap + ((b * E * M3) & 3) + gc * M3 + jk;
#pragma unroll
      for (int i = 0; i < NM; ++i) idx[i] = ok ? m[i * M2] : MFGB_INVALID_DOF;
    } else {
      const uint32_t *m = map + (b * E + gc) * M3 + jk;
#pragma unroll
      for (int i = 0; i < NM; ++i) idx[i] = ok ? __ldg(m + i * M2) : MFGB_INVALID_DOF;
    }
  };
  auto gather = [&](int64_t b) {
    if constexpr (EVEC) {
      const bool ok = has_col && gc < cells_of(b);
#pragma unroll
      for (int i = 0; i < NM; ++i) raw[i] = ok ? __ldg(src + (b * E + gc) * M3 + jk * NM + i) : 0.0;
    } else {
#pragma unroll
      for (int i = 0; i < NM; ++i) raw[i] = idx[i] != MFGB_INVALID_DOF ? __ldg(src + idx[i]) : 0.0;
    }
  };
  {
    if constexpr (!EVEC) {
      const bool ok = mbar_wait(mbar_m, ph_m);
      if (__syncthreads_or(!ok)) { fail(ph_g, ph_m); return; }
      ph_m ^= 1u;
      indices(batch);
    }
    gather(batch);
    if (has_col) fx_column_exp(raw, &s_emax[0][gc]);
    if (!G64 && has_col && gc < cells_of(batch)) ge = __ldg(gexp + batch * E + gc);
  }

  for (int it = 0; batch < n_batches; batch += gridDim.x, ++it) {
    const int slot = it & 1;
    const int64_t next = batch + gridDim.x;
    const bool has_next = next < n_batches;
    const bool okg = mbar_wait(mbar_g, ph_g);
    if (__syncthreads_or(!okg)) { fail(ph_g, ph_m); return; }  // barrier A
    ph_g ^= 1u;
    const GT *Gc = sG + el * 6 * Q3 + mf;
    if constexpr (G64) {  // the element's largest G exponent (read after barrier B)
      if (el < cells_of(batch)) {
        int eg = 0;
#pragma unroll 1
        for (int c = 0; c < 6; ++c)
#pragma unroll
          for (int l = 0; l < NQ; ++l) eg = max(eg, dexp(Gc[c * Q3 + l * Q2]));
        if (eg) atomicMax(&s_gmax[el], eg);
      }
    }
    // ---- interpolation: F on the gathered columns, then M, then L with the derivative along L
    const int su = fx_offset(s_emax[slot][gc]);
    if (has_col) {
      df x[NM], y[NQ];
      fx_column(raw, s_emax[slot][gc], x);
      fx_line_grid(basis.B, x, fx_line_max(x), y);
      store_line(y, U + col, 1);
    }
    __syncthreads();  // barrier B: s_emax[slot] read; the map tile is free
    if (tid < E) s_emax[slot][tid] = 0;  // next written two batches on
    int sg = 0;
    if constexpr (G64) {
      sg = fx_offset(s_gmax[el]);
      ge = fx_offset(s_gmax[gc]);
    }
    if (!EVEC && tid == 0 && has_next) {
      fence_proxy_async_smem();
      issue_map(next);
    }
    if (has_mn) {
      df x[NM], y[NQ];
      load_line(x, U + mn, S::m);
      fx_line(basis.B, x, y);
      store_line(y, U + mn, S::m);
    }
    __syncthreads();
    df ql[NQ], ul[MASS ? NQ : 1];
    {
      df x[NM], u[NQ];
      load_line(x, U + own, S::l);
      float mx = fx_line_max(x);
      if constexpr (SYM) {  // one grid for both contractions
        mx = __fmul_rn(mx, 1.0f + 0x1p-20f);
        const float C = __fmul_rn(mx, 3.f);
#pragma unroll
        for (int i = 0; i < NM; ++i)
          if (NM % 2 == 0 || i != NM / 2) x[i] = fx_grid(x[i], C);
      }
      fx_line_grid(basis.B, x, mx, u);
      store_line(u, U + own, S::l);
      fx_line_grid(basis.DB, x, mx, ql);
      if constexpr (MASS) {
#pragma unroll
        for (int l = 0; l < NQ; ++l) ul[l] = u[l];
      }
    }
    __syncthreads();
    // ---- gradient along the F- and M-lines
    {
      df x[NQ], y[NQ];
      load_line(x, U + fq, 1);
      fx_line(basis.D, x, y);
      store_line(y, V + fq, 1);
      load_line(x, U + mq, S::m);
      fx_line(basis.D, x, y);
      __syncthreads();  // U has been read
      store_line(y, U + mq, S::m);
    }
    __syncthreads();
    // ---- metric on the owned L-line, bound per point: max |q| times the row sums of |G|
#pragma unroll
    for (int l = 0; l < NQ; ++l) {
      const df qf = V[own + l * S::l], qm = U[own + l * S::l];
      auto g = [&](int q) {  // (a cell past the end reads a stale tile; nothing leaves it)
        if constexpr (G64) {  // converted to pairs scaled by 2^-sg as it is read
          const df d = fx_from_double(Gc[q * Q3 + l * Q2], sg);
          return make_float2(d.hi, d.lo);
        } else {
          return Gc[q * Q3 + l * Q2];
        }
      };
      const float2 gff = g(EVEC ? 5 : 0), gfm = g(EVEC ? 4 : 1), gfl = g(2), gmm = g(3),
                   gml = g(EVEC ? 1 : 4), gll = g(EVEC ? 0 : 5);
      const float kq = basis.K * fmaxf(fmaxf(fabsf(qf.hi), fabsf(qm.hi)), fabsf(ql[l].hi));
      const float Cf = (fabsf(gff.x) + fabsf(gfm.x) + fabsf(gfl.x)) * kq;
      const float Cm = (fabsf(gfm.x) + fabsf(gmm.x) + fabsf(gml.x)) * kq;
      const float Cl = (fabsf(gfl.x) + fabsf(gml.x) + fabsf(gll.x)) * kq;
      fxacc bf, bm, bl;
      fx_first(bf, gff.x, gff.y, qf.hi, qf.lo, Cf);
      fx_fma(bf, gfm.x, gfm.y, qm.hi, qm.lo);
      fx_fma(bf, gfl.x, gfl.y, ql[l].hi, ql[l].lo);
      fx_first(bm, gfm.x, gfm.y, qf.hi, qf.lo, Cm);
      fx_fma(bm, gmm.x, gmm.y, qm.hi, qm.lo);
      fx_fma(bm, gml.x, gml.y, ql[l].hi, ql[l].lo);
      fx_first(bl, gfl.x, gfl.y, qf.hi, qf.lo, Cl);
      fx_fma(bl, gml.x, gml.y, qm.hi, qm.lo);
      fx_fma(bl, gll.x, gll.y, ql[l].hi, ql[l].lo);
      V[own + l * S::l] = fx_finish(bf, Cf);
      U[own + l * S::l] = fx_finish(bm, Cm);
      ql[l] = fx_finish(bl, Cl);
    }
    __syncthreads();  // barrier C: the fluxes are in; G tile consumed, s_gmax read
    if (G64 && tid < E) s_gmax[tid] = 0;
    if (tid == 0 && has_next) {
      fence_proxy_async_smem();
      issue_g(next);
    }
    // this batch's scatter targets; then prefetch the next batch's gather
    const int sc = su + ge;  // the result scale of the column's cell
    uint32_t cur[NM];
#pragma unroll
    for (int i = 0; i < NM; ++i) cur[i] = EVEC ? 0u : idx[i];
    if (has_next) {
      if constexpr (!EVEC) {
        const bool okm = mbar_wait(mbar_m, ph_m);
        if (!okm && err_flag) atomicOr(err_flag, 1);  // the launch's result is void
        ph_m ^= 1u;
        if (okm) {
          indices(next);
        } else {
#pragma unroll
          for (int i = 0; i < NM; ++i) idx[i] = MFGB_INVALID_DOF;
        }
      }
      gather(next);
      if (!G64) ge = has_col && gc < cells_of(next) ? __ldg(gexp + next * E + gc) : 0;
    }
    float2 jw[MASS ? NQ : 1];
    if constexpr (MASS) {
      const float2 *j = jxw + (batch * E + el) * Q3 + mf;
      const bool ok = el < cells_of(batch);
#pragma unroll
      for (int l = 0; l < NQ; ++l) jw[l] = ok ? __ldg(j + l * Q2) : make_float2(0.f, 0.f);
    }
    // ---- integration: D^T along F and M in place, then L (both fluxes), M and F back to the nodes
    {
      df x[NQ], y[NQ];
      load_line(x, V + fq, 1);
      fx_line(basis.Dt, x, y);
      store_line(y, V + fq, 1);
      load_line(x, U + mq, S::m);
      fx_line(basis.Dt, x, y);
      store_line(y, U + mq, S::m);
    }
    __syncthreads();
    {
      df z[NQ], y[NM];
#pragma unroll
      for (int l = 0; l < NQ; ++l) {
        const df f = V[own + l * S::l], m = U[own + l * S::l];
        if constexpr (MASS) {
          const float C = basis.K * fabsf(jw[l].x) * fabsf(ul[l].hi);
          fxacc a;
          fx_first(a, jw[l].x, jw[l].y, ul[l].hi, ul[l].lo, C);
          z[l] = fx_sum3(f, m, fx_finish(a, C));
        } else {
          z[l] = fx_sum2(f, m);
        }
      }
      fx_line_joint(basis.Bt, basis.DBt, z, ql, y);
      store_line(y, U + own, S::l);
    }
    __syncthreads();
    if (has_mn) {
      df x[NQ], y[NM];
      load_line(x, U + mn, S::m);
      fx_line(basis.Bt, x, y);
      store_line(y, U + mn, S::m);
    }
    __syncthreads();
    if (has_col) {
      df x[NQ], y[NM];
      load_line(x, U + col, 1);
      fx_line(basis.Bt, x, y);
      if (!EVEC) cudaGridDependencySynchronize();  // dst has its start values
      auto put = [&](int i, double v) {
        if constexpr (EVEC) {  // the column's own place, written out below
          reinterpret_cast<double *>(U)[col + i] = v;
        } else {
          if (cur[i] != MFGB_INVALID_DOF) atomicAdd(dst + cur[i], v);
        }
      };
      if ((unsigned)(sc + 896) <= 1792u) {
        const unsigned kout = (unsigned)(896 + sc) << 20;
#pragma unroll
        for (int i = 0; i < NM; ++i) put(i, fx_f2d_fast(y[i].hi, kout) + fx_f2d_fast(y[i].lo, kout));
      } else {
#pragma unroll
        for (int i = 0; i < NM; ++i) put(i, fx_f2d(y[i].hi, sc) + fx_f2d(y[i].lo, sc));
      }
    }
    if constexpr (EVEC) {
      __syncthreads();
      double *out = dst + batch * E * M3;
      const int n = cells_of(batch) * M3;
      for (int t = tid; t < n; t += E * Q2) {
        const int c = t / M3, r = t - c * M3, lm = r / NM;
        out[t] = reinterpret_cast<const double *>(
            U)[c * S::cell + lm / NM * S::l + lm % NM * S::m + (r - lm * NM)];
      }
    }
    // the prefetched gather's largest exponent per cell (read after the next barrier A)
    if (has_next && has_col) fx_column_exp(raw, &s_emax[slot ^ 1][gc]);
  }
}

// CEED BK1: out_e = B^T (JxW_e o B in_e) on element vectors, directions F, M, L = 2, 1, 0.  The
// thread that owns an L-line interpolates it, multiplies by JxW and integrates it back without
// leaving its registers; each element's input and JxW are scaled by their own powers of two and
// loaded a batch ahead.
template <int NM, int NQ, int E, int MB, bool SYM>
__global__ void __launch_bounds__(E * NQ * NQ, MB)
    bk1fx_kernel(const int64_t nelmt, const double *__restrict__ in, const double *__restrict__ JxW,
                 double *__restrict__ out, const FxMat<NM, NQ, SYM ? 1 : 0> B,
                 const FxMat<NQ, NM, SYM ? 1 : 0> Bt, const float K) {
  using S = GaussStride<NQ>;
  constexpr bool SUMS = NM <= 4;  // short lines: by TwoSum (fx_line_sums)
  constexpr int M2 = NM * NM, M3 = M2 * NM, Q2 = NQ * NQ, Q3 = Q2 * NQ;
  extern __shared__ __align__(128) unsigned char smem[];
  df *U = reinterpret_cast<df *>(smem);
  __shared__ int s_emax[2][E], s_jmax[2][E];

  const int tid = threadIdx.x;
  const int el = tid / Q2, mf = tid - el * Q2;  // the owned L-line
  const int own = el * S::cell + mf / NQ * S::m + mf % NQ;
  const bool has_col = tid < E * M2;            // the owned column (m, l) of nodes
  const int gc = has_col ? tid / M2 : 0, jk = has_col ? tid - gc * M2 : 0;
  const int col = gc * S::cell + jk % NM * S::m + jk / NM * S::l;
  const bool has_mn = tid < E * NQ * NM;
  const int mn = has_mn ? gauss_line_table<NM, NQ, E>.mn[tid] : 0;
  const int64_t n_batches = (nelmt + E - 1) / E;
  int64_t batch = blockIdx.x;
  if (batch >= n_batches) return;  // uniform across the CTA
  auto cells_of = [&](int64_t b) { return (int)min((int64_t)E, nelmt - b * E); };
  if (tid < 2 * E) {
    (&s_emax[0][0])[tid] = 0;
    (&s_jmax[0][0])[tid] = 0;
  }
  __syncthreads();

  auto line = [](const auto &M, auto &x, auto &y) {
    if constexpr (SUMS)
      fx_line_sums(M, x, y);
    else
      fx_line(M, x, y);
  };
  double raw[NM], jraw[NQ];
  auto load = [&](int64_t b) {
    const bool okc = has_col && gc < cells_of(b), okl = el < cells_of(b);
#pragma unroll
    for (int i = 0; i < NM; ++i) raw[i] = okc ? __ldg(in + (b * E + gc) * M3 + jk * NM + i) : 0.0;
#pragma unroll
    for (int l = 0; l < NQ; ++l) jraw[l] = okl ? __ldg(JxW + (b * E + el) * Q3 + l * Q2 + mf) : 0.0;
  };
  auto reduce_exp = [&](int slot) {
    if (has_col) fx_column_exp(raw, &s_emax[slot][gc]);
    fx_column_exp(jraw, &s_jmax[slot][el]);
  };
  load(batch);
  reduce_exp(0);

  for (int it = 0; batch < n_batches; batch += gridDim.x, ++it) {
    const int slot = it & 1;
    const int64_t next = batch + gridDim.x;
    const bool has_next = next < n_batches;
    __syncthreads();  // the exponents of this batch are in; U is free
    const int sj = fx_offset(s_jmax[slot][el]);
    const int sc = fx_offset(s_emax[slot][gc]) + fx_offset(s_jmax[slot][gc]);  // the column's result scale
    df jx[NQ];
#pragma unroll
    for (int l = 0; l < NQ; ++l) jx[l] = fx_from_double(jraw[l], sj);
    if (has_col) {
      df x[NM], y[NQ];
      fx_column<!SUMS>(raw, s_emax[slot][gc], x);
      if constexpr (SUMS)
        fx_line_sums(B, x, y);
      else
        fx_line_grid(B, x, fx_line_max(x), y);
      store_line(y, U + col, 1);
    }
    __syncthreads();  // the exponents have been read
    if (tid < E) s_emax[slot][tid] = s_jmax[slot][tid] = 0;  // next written two batches on
    if (has_next) load(next);
    if (has_mn) {
      df x[NM], y[NQ];
      load_line(x, U + mn, S::m);
      line(B, x, y);
      store_line(y, U + mn, S::m);
    }
    __syncthreads();
    {
      df x[NM], u[NQ], y[NM];
      load_line(x, U + own, S::l);
      line(B, x, u);
#pragma unroll
      for (int l = 0; l < NQ; ++l) {
        const float C = K * fabsf(jx[l].hi) * fabsf(u[l].hi);
        fxacc a;
        fx_first(a, jx[l].hi, jx[l].lo, u[l].hi, u[l].lo, C);
        u[l] = fx_finish(a, C);
      }
      line(Bt, u, y);
      store_line(y, U + own, S::l);
    }
    __syncthreads();
    if (has_mn) {
      df x[NQ], y[NM];
      load_line(x, U + mn, S::m);
      line(Bt, x, y);
      store_line(y, U + mn, S::m);
    }
    __syncthreads();
    if (has_col) {
      df x[NQ], y[NM];
      load_line(x, U + col, 1);
      line(Bt, x, y);
      double *o = reinterpret_cast<double *>(U) + col;
      if ((unsigned)(sc + 896) <= 1792u) {
        const unsigned kout = (unsigned)(896 + sc) << 20;
#pragma unroll
        for (int i = 0; i < NM; ++i) o[i] = fx_f2d_fast(y[i].hi, kout) + fx_f2d_fast(y[i].lo, kout);
      } else {
#pragma unroll
        for (int i = 0; i < NM; ++i) o[i] = fx_f2d(y[i].hi, sc) + fx_f2d(y[i].lo, sc);
      }
    }
    __syncthreads();
    const int n = cells_of(batch) * M3;
    for (int t = tid; t < n; t += E * Q2) {
      const int c = t / M3, r = t - c * M3, lm = r / NM;
      out[batch * E * M3 + t] = reinterpret_cast<const double *>(
          U)[c * S::cell + lm / NM * S::l + lm % NM * S::m + (r - lm * NM)];
    }
    // the next batch's largest exponents per element (read after the next barrier)
    if (has_next) reduce_exp(slot ^ 1);
  }
}

}  // namespace mfgb
