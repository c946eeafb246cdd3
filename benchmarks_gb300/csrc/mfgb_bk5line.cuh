// mfgb_bk5line.cuh -- the BK5 collocation operator in plain FP32 or FP64 arithmetic with whole
// lines per thread: the pipeline of bk5fx_kernel (mfgb_bk5fx.cuh; bulk copies of G and the dof map
// a batch ahead, gather a batch ahead in registers, lines dealt to shared-memory banks, derivative
// in even-odd form) without scaling and offsets.  Reference: CEED_BK/include/kernels/BK5/
// templated_cuda_kernels.cuh:50-122 and bakeoff_problems_dealii/include/bk3_kokkos_kernel.h:129-151,
// 406-426.
#pragma once
#include "mfgb_bk5.cuh"
#include "mfgb_fxline.cuh"

namespace mfgb {

// Strides of a cell's work array (cell, i, j; k contiguous) by the size of a value; wavefronts of
// one batch of 4-byte values against the plain strides and the least possible, counted on the host:
// n = 3 204 / 276 (180), 4 304 / 736 (240), 5 640 / 865 (600), 6 474 / 696 (450), 8 512 / 1760 (480).
template <int N, int BYTES> struct LineStride;
#define MFGB_LSTRIDE(NN, BYTES, CELL, I, J) \
  template <> struct LineStride<NN, BYTES> { static constexpr int cell = CELL, i = I, j = J; };
MFGB_LSTRIDE(2, 4, 12, 5, 2) MFGB_LSTRIDE(3, 4, 41, 11, 3) MFGB_LSTRIDE(4, 4, 80, 19, 4)
MFGB_LSTRIDE(5, 4, 153, 29, 5) MFGB_LSTRIDE(6, 4, 228, 37, 6) MFGB_LSTRIDE(7, 4, 369, 52, 7)
MFGB_LSTRIDE(8, 4, 529, 66, 8) MFGB_LSTRIDE(9, 4, 785, 84, 9)
MFGB_LSTRIDE(2, 8, 12, 5, 2) MFGB_LSTRIDE(3, 8, 27, 9, 3) MFGB_LSTRIDE(4, 8, 68, 17, 4)
MFGB_LSTRIDE(5, 8, 153, 29, 5) MFGB_LSTRIDE(6, 8, 244, 39, 6) MFGB_LSTRIDE(7, 8, 369, 51, 7)
MFGB_LSTRIDE(8, 8, 568, 71, 8) MFGB_LSTRIDE(9, 8, 738, 82, 9)
#undef MFGB_LSTRIDE

// work-array offsets of the s-line (values j apart) and the t-line (contiguous) each thread owns
template <int N, int E, int BYTES>
struct LineOwners {
  unsigned short s[E * N * N], t[E * N * N];
};
template <int N, int E, int BYTES>
constexpr LineOwners<N, E, BYTES> line_owners() {
  using S = LineStride<N, BYTES>;
  LineOwners<N, E, BYTES> r{};
  int s[E * N * N] = {}, t[E * N * N] = {};
  for (int q = 0; q < E * N * N; ++q) {
    const int e = q / (N * N), a = q / N % N, b = q % N;
    s[q] = e * S::cell + a * S::i + b;
    t[q] = e * S::cell + a * S::i + b * S::j;
  }
  fx_deal<128 / BYTES>(s, r.s);
  fx_deal<128 / BYTES>(t, r.t);
  return r;
}
template <int N, int E, int BYTES>
__device__ const LineOwners<N, E, BYTES> line_owner_table = line_owners<N, E, BYTES>();

// shared memory of one CTA: G window, dof-map window (16 bytes of slack each: bulk copies take the
// aligned window around a tile), NB work arrays, two mbarriers
template <int N, int E, class R, int NB>
struct LineLayout {
  static constexpr int N3 = N * N * N;
  static constexpr size_t g_bytes = (sizeof(R) * E * 6 * N3 + 16 + 15) / 16 * 16;
  static constexpr size_t map_bytes = ((size_t)E * N3 * 4 + 12 + 15) / 16 * 16;
  static constexpr size_t work_bytes = sizeof(R) * NB * E * LineStride<N, sizeof(R)>::cell;
  static constexpr size_t total = g_bytes + map_bytes + (work_bytes + 15) / 16 * 16 + 16;
};

// G and map 16-byte aligned, basis in even-odd form.  NB = 3 work arrays, or 2 with the t-line
// results over u after one more barrier.
template <int N, int E, int MB, int NB, class A>
__global__ void __launch_bounds__(E * N * N, MB)
    bk5_line_kernel(const int64_t n_cells, const uint32_t *__restrict__ map,
                    const typename A::GType *__restrict__ G, const typename A::VecT *__restrict__ src,
                    typename A::VecT *__restrict__ dst, const Basis<N, A> basis,
                    const int *__restrict__ done_flag, int *__restrict__ err_flag) {
  if (done_flag != nullptr && *done_flag) return;
  using R = typename A::VecT;
  using L = LineLayout<N, E, R, NB>;
  using S = LineStride<N, sizeof(R)>;
  constexpr int N2 = N * N, N3 = N * N * N, AL = 16 / sizeof(R);  // AL: values in 16 bytes
  extern __shared__ __align__(128) unsigned char smem[];
  R *sG = reinterpret_cast<R *>(smem);
  uint32_t *sMap = reinterpret_cast<uint32_t *>(smem + L::g_bytes);
  R *s_u = reinterpret_cast<R *>(smem + L::g_bytes + L::map_bytes);
  R *s_s = s_u + E * S::cell;
  R *s_t = NB == 3 ? s_s + E * S::cell : s_u;
  uint64_t *mbar_g = reinterpret_cast<uint64_t *>(smem + L::total - 16), *mbar_m = mbar_g + 1;

  const int tid = threadIdx.x;
  const int el = tid / N2;
  const int jk = tid - el * N2;
  const int col = el * S::cell + jk / N * S::j + jk % N;      // own column u(., j, k): + i * S::i
  const int sline = line_owner_table<N, E, sizeof(R)>.s[tid];  // own line u(a, ., b): + m * S::j
  const int tline = line_owner_table<N, E, sizeof(R)>.t[tid];  // own line u(a, b, .): + m
  const int64_t n_batches = (n_cells + E - 1) / E;
  int64_t batch = blockIdx.x;
  if (batch >= n_batches) return;  // uniform across the CTA

  auto cells_of = [&](int64_t b) { return (int)min((int64_t)E, n_cells - b * E); };
  // The tile of `per` values a cell (al of them in 16 bytes) as the 16-byte aligned window around
  // it: its size in values, 0 when it would pass the array's end (the last batch: plain loads)
  auto window = [&](int64_t b, int per, int al) -> uint32_t {
    const int64_t first = b * E * per, last = first + (int64_t)cells_of(b) * per;
    const int64_t end = (last + al - 1) & ~(int64_t)(al - 1);
    return end <= n_cells * per ? (uint32_t)(end - (first & ~(int64_t)(al - 1))) : 0u;
  };
  auto issue = [&](int64_t b) {  // G of batch b
    const uint32_t n = window(b, 6 * N3, AL);
    mbar_arrive_expect_tx(mbar_g, n * (uint32_t)sizeof(R));
    if (n) bulk_g2s(sG, G + ((b * E * 6 * N3) & ~(int64_t)(AL - 1)), n * (uint32_t)sizeof(R), mbar_g);
  };
  auto issue_map = [&](int64_t b) {
    const uint32_t n = window(b, N3, 4);
    mbar_arrive_expect_tx(mbar_m, n * 4u);
    if (n) bulk_g2s(sMap, map + ((b * E * N3) & ~(int64_t)3), n * 4u, mbar_m);
  };
  auto fail = [&](uint32_t pg, uint32_t pm) {
    if (tid == 0 && err_flag) atomicOr(err_flag, 1);
    mbar_wait(mbar_g, pg);  // bounded waits for copies still in flight
    mbar_wait(mbar_m, pm);
  };
  if (tid == 0) {
    mbar_init(mbar_g, 1);
    mbar_init(mbar_m, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (tid == 0) {
    issue(batch);
    issue_map(batch);
  }
  uint32_t ph_g = 0, ph_m = 0;
  uint32_t idx[N];
  R raw[N];
  auto gather = [&](int64_t b) {
    const bool ok = el < cells_of(b);
    if (window(b, N3, 4)) {
      const uint32_t *m = sMap + ((b * E * N3) & 3) + el * N3 + jk;
#pragma unroll
      for (int i = 0; i < N; ++i) idx[i] = ok ? m[i * N2] : MFGB_INVALID_DOF;
    } else {
      const uint32_t *m = map + (b * E + el) * N3 + jk;
#pragma unroll
      for (int i = 0; i < N; ++i) idx[i] = ok ? __ldg(m + i * N2) : MFGB_INVALID_DOF;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) raw[i] = idx[i] != MFGB_INVALID_DOF ? __ldg(src + idx[i]) : R(0);
  };
  {
    const bool ok = mbar_wait(mbar_m, ph_m);
    if (__syncthreads_or(!ok)) { fail(ph_g, ph_m); return; }
    ph_m ^= 1u;
    gather(batch);
  }

  for (; batch < n_batches; batch += gridDim.x) {
    const int64_t next = batch + gridDim.x;
    const bool has_next = next < n_batches;
    const bool okg = mbar_wait(mbar_g, ph_g);
    if (__syncthreads_or(!okg)) { fail(ph_g, ph_m); return; }  // barrier A
    ph_g ^= 1u;
    const int shift = (int)((batch * E * 6 * N3) & (AL - 1));
    if (!window(batch, 6 * N3, AL)) {  // ordered before the metric by barrier B
      const int n = cells_of(batch) * 6 * N3;
      for (int t = tid; t < n; t += E * N2) sG[shift + t] = __ldg(G + batch * E * 6 * N3 + t);
    }
    // ---- own column to shared memory, its derivative in registers
    R x[N], y[N], qr[N];
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = s_u[col + i * S::i] = raw[i];
    even_odd_apply<N, A>(basis.Pg, basis.Qg, x, qr);
    __syncthreads();  // barrier B: s_u ready; the map tile is free
    if (tid == 0 && has_next) {
      fence_proxy_async_smem();
      issue_map(next);
    }
    // ---- derivative along the s- and t-lines
#pragma unroll
    for (int m = 0; m < N; ++m) x[m] = s_u[sline + m * S::j];
    even_odd_apply<N, A>(basis.Pg, basis.Qg, x, y);
#pragma unroll
    for (int m = 0; m < N; ++m) s_s[sline + m * S::j] = y[m];
#pragma unroll
    for (int m = 0; m < N; ++m) x[m] = s_u[tline + m];
    even_odd_apply<N, A>(basis.Pg, basis.Qg, x, y);
    if (NB == 2) __syncthreads();  // every line of u has been read
#pragma unroll
    for (int m = 0; m < N; ++m) s_t[tline + m] = y[m];
    __syncthreads();
    // ---- metric on the own column
    const R *Gc = sG + shift + el * 6 * N3 + jk;  // (past the last cell: a stale tile, nothing leaves it)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const R qs = s_s[col + i * S::i], qt = s_t[col + i * S::i], q = qr[i];
      const R grr = Gc[i * N2], grs = Gc[N3 + i * N2], grt = Gc[2 * N3 + i * N2],
              gss = Gc[3 * N3 + i * N2], gst = Gc[4 * N3 + i * N2], gtt = Gc[5 * N3 + i * N2];
      qr[i] = grr * q + grs * qs + grt * qt;
      s_s[col + i * S::i] = grs * q + gss * qs + gst * qt;
      s_t[col + i * S::i] = grt * q + gst * qs + gtt * qt;
    }
    __syncthreads();  // barrier C: fluxes ready, G tile consumed
    uint32_t cur[N];
#pragma unroll
    for (int i = 0; i < N; ++i) cur[i] = idx[i];
    if (has_next) {
      if (tid == 0) {
        fence_proxy_async_smem();
        issue(next);
      }
      const bool okm = mbar_wait(mbar_m, ph_m);
      if (!okm && err_flag) atomicOr(err_flag, 1);  // the launch's result is void
      ph_m ^= 1u;
      if (okm) {
        gather(next);
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) idx[i] = MFGB_INVALID_DOF, raw[i] = R(0);
      }
    }
    // ---- transposes along the lines, in place, and of the own column; sum and scatter
#pragma unroll
    for (int m = 0; m < N; ++m) x[m] = s_s[sline + m * S::j];
    even_odd_apply<N, A>(basis.Pt, basis.Qt, x, y);
#pragma unroll
    for (int m = 0; m < N; ++m) s_s[sline + m * S::j] = y[m];
#pragma unroll
    for (int m = 0; m < N; ++m) x[m] = s_t[tline + m];
    even_odd_apply<N, A>(basis.Pt, basis.Qt, x, y);
#pragma unroll
    for (int m = 0; m < N; ++m) s_t[tline + m] = y[m];
    even_odd_apply<N, A>(basis.Pt, basis.Qt, qr, y);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (cur[i] != MFGB_INVALID_DOF)
        atomicAdd(dst + cur[i], y[i] + (s_s[col + i * S::i] + s_t[col + i * S::i]));
  }
}

}  // namespace mfgb
