// mfgb_bk5fx.cuh -- FP64-accurate BK5 collocation operator on the FP32 pipes with
// offset ("fixed-exponent") double-float accumulation and per-cell exponent scaling.
//
// The operator is the one of bk5_tma_kernel (GLL collocation: gather through the
// dof map with the 0xFFFFFFFF mask, collocation gradient, symmetric metric G,
// transpose, atomic scatter; reference CEED_BK/include/kernels/BK5/
// templated_cuda_kernels.cuh:50-122 and bakeoff_problems_dealii/include/
// bk3_kokkos_kernel.h:129-151, 406-426) with the same bulk-TMA pipeline.  What
// differs is the arithmetic and the split of the contractions over the threads:
//
// * Scaling.  Every cell's gathered values are multiplied by 2^-su, su chosen
//   from the largest binary exponent among them so that |u| < 1, and the
//   geometric factors are stored pre-multiplied by a per-cell 2^-sg (|G| < 1;
//   sg in a per-cell int array).  The scalings are exact.  The cell's result is
//   multiplied by 2^(su + sg) when it is converted back to double, so any FP64
//   input range is carried (no float over- or underflow of the pairs).
//
// * Offset accumulation.  A dot product sum_k x_k y_k of double-float pairs is
//   accumulated as T + S with T started at an offset C >= 2 B, where B bounds
//   sum_k |x_k.hi y_k.hi|.  Every partial sum then keeps C/2 <= T <= 3C/2, so
//     T' = fma(x.hi, y.hi, T)     rounds the product into T,
//     d  = T' - T                 is exact (|T| >= |product|: Dekker's Fast2Sum),
//     r  = fma(x.hi, y.hi, -d)    is the rounding error of T' (to float precision),
//     S += (r + x.hi y.lo) + x.lo y.hi
//   and at the end hi = T - C is exact (Sterbenz), lo = S.  That is 6 FP32-pipe
//   instructions per multiply-add (5 for the first), against 12 for the
//   TwoSum-based form of ArithDF, with an error of about 2^-46 of C.  The bounds
//   B come from the data at hand: each line's maximum for the gradient and the
//   transpose, max |q| times the row sum of |G| per point for the metric.  (The
//   cell's bound |u| < 1 for the gradient was 0.6 to 1.8 % faster, but with the two sums
//   of the even-odd form its error exceeded the plain form's on values that are
//   not spread evenly: up to 1.5 times at p = 2 on a constant plus small changes,
//   1.1 to 1.35 on values over 60 binades.)
//
// * Line ownership (mfgb_fxline.cuh).  In every contraction a thread owns a whole
//   line, with the derivative matrix in even-odd form.
//
// What bounds it (p = 4, ncu at 8.5e6 DoFs): 1,299 warp-instructions a cell against 1,637 of the
// kernel with one output per thread and step, 69 % of the issue slots, 70 % of the shared-memory
// pipe, 5 CTAs an SM instead of 4.  67.6M DoFs: a vmult 2.22 -> 1.60 ms, 77 % of the measured copy
// bandwidth in the kernel; p = 6 and 8 (n^4 arithmetic per n^3 bytes) stay near 61 % and 49 %, bound by
// issue.
//
// Float32 restatements of this arithmetic with their error bounds are in
// tests/test_fx_arith.py and tests/test_fx_line.py.
#pragma once
#include <type_traits>

#include "mfgb_bk5.cuh"
#include "mfgb_fxline.cuh"

namespace mfgb {

// biased binary exponent of a double (0 for zero and subnormals, 2047 for inf/NaN)
__device__ __forceinline__ int dexp(double x) {
  return (int)(((unsigned)(__double_as_longlong(x) >> 32) >> 20) & 0x7FFu);
}

// x * 2^-off as a float pair by integer operations (off chosen so that the
// cell's largest value lands in [0.5, 1)): hi = the top 24 significant bits,
// lo = the next 29 bits rounded to float.  Values below 2^-126 after scaling
// (126 binades under the cell's largest), zeros and double subnormals flush to
// zero; inf and NaN give NaN.
__device__ __forceinline__ df fx_from_double(double x, int off) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hw = (unsigned)(b >> 32), lw = (unsigned)b;
  const unsigned sign = hw & 0x80000000u;
  const int e = (int)((hw >> 20) & 0x7FFu);
  df r;
  if (e == 0x7FF) { r.hi = __uint_as_float(0x7FC00000u); r.lo = 0.f; return r; }
  const int es = e - off;
  if (e == 0 || es <= 896) { r.hi = 0.f; r.lo = 0.f; return r; }
  const unsigned hm = ((hw & 0xFFFFFu) << 3) | (lw >> 29);
  r.hi = __uint_as_float(sign | ((unsigned)(es - 896) << 23) | hm);
  const unsigned rem = lw & 0x1FFFFFFFu;
  if (rem == 0u || es < 949) {
    r.lo = 0.f;
  } else {
    const unsigned fb = __float_as_uint(__uint2float_rn(rem));
    r.lo = __uint_as_float(sign | (fb + ((unsigned)(es - 1075) << 23)));
  }
  return r;
}

// f * 2^sc as a double by integer operations; float subnormals -> 0, results
// outside the double range -> 0 or +-inf, inf/NaN kept
__device__ __forceinline__ double fx_f2d(float f, int sc) {
  const unsigned u = __float_as_uint(f);
  const int ex = (int)((u >> 23) & 0xFFu);
  const unsigned long long sgn = (unsigned long long)(u & 0x80000000u) << 32;
  if (ex == 0) return 0.0;
  if (ex == 255)
    return __longlong_as_double((long long)(sgn | 0x7FF0000000000000ull |
                                            ((unsigned long long)(u & 0x7FFFFFu) << 29)));
  const int e2 = ex + 896 + sc;
  if (e2 <= 0) return __longlong_as_double((long long)sgn);
  if (e2 >= 2047) return __longlong_as_double((long long)(sgn | 0x7FF0000000000000ull));
  return __longlong_as_double((long long)(sgn | ((unsigned long long)e2 << 52) |
                                          ((unsigned long long)(u & 0x7FFFFFu) << 29)));
}

// The same for a cell whose scale keeps every result in the double range
// (|sc| <= 896, k = (896 + sc) << 20): the exponent is rebased on the high word
// by one integer addition; zero and subnormal floats give a signed zero,
// inf and NaN stay inf and NaN.
__device__ __forceinline__ double fx_f2d_fast(float f, unsigned k) {
  const unsigned u = __float_as_uint(f);
  const unsigned a = u & 0x7FFFFFFFu, sgn = u & 0x80000000u;
  unsigned hi = ((a >> 3) + k) | sgn;
  unsigned lo = u << 29;
  if (a < 0x00800000u) hi = sgn, lo = 0u;
  if (a >= 0x7F800000u) hi = sgn | 0x7FF00000u | ((a & 0x7FFFFFu) >> 3);
  return __hiloint2double((int)hi, (int)lo);
}

// the scale offset of a cell from its largest biased exponent
__device__ __forceinline__ int fx_offset(int emax) { return emax > 0 ? emax - 1022 : 0; }

// The same for the gathered values of a cell whose largest exponent is that of a
// normal finite number (0 < emax < 0x7FF), without branches: values more than 126
// binades below the cell's largest come out as denormal floats instead of zeros,
// which the rounding to the grid of 2^-23 removes.  Returns the pair on that grid:
// 1 + |x| lies in one binade, so it is twice as fine as the grid of signed values,
// and sums and differences of two (at most 2 = 2^24 steps) are exact.
__device__ __forceinline__ df fx_from_double_grid(double x, int off) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hw = (unsigned)(b >> 32), lw = (unsigned)b;
  const unsigned sign = hw & 0x80000000u;
  const int f = max((int)((hw >> 20) & 0x7FFu) - (off + 896), 0);  // float exponent field
  const unsigned hm = __funnelshift_l(lw, hw, 3) & 0x7FFFFFu;
  const float scale = __uint_as_float((unsigned)(max(f, 53) - 52) << 23);  // 2^-23 ulp units of lo
  const float x24 = __uint_as_float(((unsigned)f << 23) | hm);             // 24 bits of |x|
  const float h = __fsub_rn(__fadd_rn(1.f, x24), 1.f);
  const float l = __fmaf_rn(__uint2float_rn(lw & 0x1FFFFFFFu), scale, __fsub_rn(x24, h));
  df r;
  r.hi = __uint_as_float(__float_as_uint(h) ^ sign);
  r.lo = __uint_as_float(__float_as_uint(l) ^ sign);
  return r;
}

// The derivative matrix in both directions: G for the gradient, T transposed.
// SYM = -1: even-odd form (the GLL derivative), 0: a caller's general matrix.
template <int N, int SYM>
struct FxBasis {
  FxMat<N, N, SYM> G, T;
  float K;  // 2 (1 + 2^-20): the factor 2 of the offset, plus a margin for the bound's rounding
};

// Strides of a cell's work array (cell, i, j; k contiguous) and the lines' owners.  A column
// is owned by the thread that gathered it; which thread owns which s- or t-line is free, so the
// lines are dealt to half-warps with different 8-byte banks each (fx_lines), after a small padding
// where the plain strides leave too few banks.  Shared-memory wavefronts of a batch's work-array
// accesses, counted on the host, against lines dealt in order over the plain array (and the least
// possible): n = 4 240 / 624 (240), 5 600 / 900 (600), 6 654 / 1050 (630), 8 512 / 1504 (480),
// 9 882 / 990 (810).
template <int N> struct FxStride;
#define MFGB_FXSTRIDE(NN, CELL, I, J) \
  template <> struct FxStride<NN> { static constexpr int cell = CELL, i = I, j = J; };
MFGB_FXSTRIDE(2, 12, 5, 2) MFGB_FXSTRIDE(3, 27, 9, 3) MFGB_FXSTRIDE(4, 68, 17, 4)
MFGB_FXSTRIDE(5, 153, 29, 5) MFGB_FXSTRIDE(6, 244, 39, 6) MFGB_FXSTRIDE(7, 369, 51, 7)
MFGB_FXSTRIDE(8, 568, 71, 8) MFGB_FXSTRIDE(9, 738, 82, 9)
#undef MFGB_FXSTRIDE

// work-array offsets of the s-line (values j apart) and the t-line (contiguous) each thread owns
template <int N, int E>
struct FxLines {
  unsigned short s[E * N * N], t[E * N * N];
};

template <int N, int E>
constexpr FxLines<N, E> fx_lines() {
  using S = FxStride<N>;
  FxLines<N, E> r{};
  int s[E * N * N] = {}, t[E * N * N] = {};
  for (int q = 0; q < E * N * N; ++q) {
    const int e = q / (N * N), a = q / N % N, b = q % N;
    s[q] = e * S::cell + a * S::i + b;
    t[q] = e * S::cell + a * S::i + b * S::j;
  }
  fx_deal(s, r.s);
  fx_deal(t, r.t);
  return r;
}
template <int N, int E>
__device__ const FxLines<N, E> fx_line_table = fx_lines<N, E>();

// shared memory of one CTA: G tile, dof-map tile (L-vectors), NB work arrays, two mbarriers
template <int N, int E, class GT, bool EVEC, int NB>
struct FxLayout {
  static constexpr int N3 = N * N * N;
  static constexpr size_t g_bytes = sizeof(GT) * E * 6 * N3;
  static constexpr size_t map_bytes = EVEC ? 0 : ((size_t)E * N3 * 4 + 12 + 15) / 16 * 16;
  static constexpr size_t work_bytes = sizeof(df) * NB * E * FxStride<N>::cell;
  static constexpr size_t total = g_bytes + map_bytes + (work_bytes + 15) / 16 * 16 + 16;
};

template <class GT> struct FxGArith;
template <> struct FxGArith<float2> { using type = ArithDF; };
template <> struct FxGArith<double> { using type = ArithF64; };

// One CTA works on E cells at a time with N^2 threads per cell.  Per batch:
//   barrier A   G(b) has landed; u(b) was gathered into registers during batch b-1, its
//               largest exponent per cell reduced into s_emax by shared atomics
//   column      thread (j, k) converts its column u(., j, k) to pairs on a common grid, writes
//               it to shared memory and contracts it: q_r stays in registers
//   barrier B   map(b+next) is requested (bulk TMA)
//   lines       thread (a, b) owns the line u(a, ., b), then u(a, b, .): q_s, q_t to shared
//               memory (NB = 2: q_t over u, after one more barrier)
//   barrier     thread (j, k) applies the metric to its column: v_r in registers, v_s, v_t over
//               q_s, q_t
//   barrier C   G(b+next) is requested, u(b+next) gathered into registers
//   lines       the transposed contractions of the s- and t-lines, in place
//   barrier     thread (j, k) contracts v_r and adds the shares of the three directions;
//               conversion to double and atomic scatter
// GT = float2: G as scaled pairs with the exponent offset gexp[cell] (operators); double: the
// caller's FP64 G, whose largest exponent per cell is reduced in shared memory and which the
// metric converts as it reads it (kernel seams).  EVEC: contiguous element vectors, dst is
// written, not added to; otherwise through the dof map.  NC interleaved components share one G
// tile, each with its own exponent per cell (the slots of s_emax alternate with the component).
// MAPTMA = false loads the dof map with plain loads (a map array that is not 16-byte aligned).
// EXPIRE (test hook): the first G copy is armed but not issued, and every wait gives up after
// 1 ms, so the timeout path runs with no copy in flight.
template <int N, int E, int MB, int NB, class GT, bool EVEC, int NC, int SYM, bool MAPTMA,
          bool EXPIRE = false>
__global__ void __launch_bounds__(E * N * N, MB)
    bk5fx_kernel(const int64_t n_cells, const uint32_t *__restrict__ map,
                 const GT *__restrict__ G, const int *__restrict__ gexp,
                 const double *__restrict__ src, double *__restrict__ dst,
                 const FxBasis<N, SYM> basis, const int *__restrict__ done_flag,
                 int *__restrict__ err_flag) {
  if (done_flag != nullptr && *done_flag) return;
  using L = FxLayout<N, E, GT, EVEC, NB>;
  using S = FxStride<N>;
  constexpr int N2 = N * N, N3 = N * N * N;
  constexpr bool G64 = std::is_same<GT, double>::value;
  extern __shared__ __align__(128) unsigned char smem[];
  GT *sG = reinterpret_cast<GT *>(smem);
  uint32_t *sMap = reinterpret_cast<uint32_t *>(smem + L::g_bytes);
  df *s_u = reinterpret_cast<df *>(smem + L::g_bytes + L::map_bytes);
  df *s_s = s_u + E * S::cell;
  df *s_t = NB == 3 ? s_s + E * S::cell : s_u;
  uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + L::total - 16);
  uint64_t *mbar_g = mbar, *mbar_m = mbar + 1;
  __shared__ int s_emax[2][E];
  __shared__ int s_gmax[E];  // G64: largest biased exponent of the cell's G

  const int tid = threadIdx.x;
  const int el = tid / N2;
  const int jk = tid - el * N2;
  const int j = jk / N;
  const int k = jk - j * N;
  const int col = el * S::cell + j * S::j + k;     // own column u(., j, k): + i * S::i
  const int sline = fx_line_table<N, E>.s[tid];    // own line u(a, ., b) of some cell: + m * S::j
  const int tline = fx_line_table<N, E>.t[tid];    // own line u(a, b, .) of some cell: + m
  const int64_t n_batches = (n_cells + E - 1) / E;
  int64_t batch = blockIdx.x;
  if (batch >= n_batches) return;  // uniform across the CTA

  TmaTiles<N, E, typename FxGArith<GT>::type> T{n_cells, map, G, src, sG, sMap, mbar_g, mbar_m};
  // the dof-map tile of batch b arrives as the 16-byte aligned window around it, which starts
  // (b E N^3) mod 4 entries before the tile; the last one by plain loads when its window would
  // pass the map's end
  auto map_window = [&](int64_t b) -> uint32_t {  // bytes, 0: no bulk copy
    const int64_t first = b * E * N3, last = first + (int64_t)T.cells_of(b) * N3;
    const int64_t end = (last + 3) & ~(int64_t)3;
    return MAPTMA && end <= n_cells * N3 ? (uint32_t)(end - (first & ~(int64_t)3)) * 4u : 0u;
  };
  auto issue_map = [&](int64_t b) {
    const uint32_t bytes = map_window(b);
    mbar_arrive_expect_tx(mbar_m, bytes);
    if (bytes) bulk_g2s(sMap, map + ((b * E * N3) & ~(int64_t)3), bytes, mbar_m);
  };
  constexpr uint64_t wlim = EXPIRE ? 1000000ull : MFGB_WAIT_LIMIT_NS;
  auto fail = [&](uint32_t pg, uint32_t pm) {
    if (tid == 0 && err_flag) atomicOr(err_flag, 1);
    mbar_wait(mbar_g, pg, wlim);  // bounded waits for copies still in flight
    if (!EVEC) mbar_wait(mbar_m, pm, wlim);
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
    if (EXPIRE)
      mbar_arrive_expect_tx(mbar_g, 16u);
    else
      T.issue_g(batch);
    if (!EVEC) issue_map(batch);
  }
  uint32_t ph_g = 0, ph_m = 0;
  uint32_t idx[N];
  double raw[N];
  int ge = 0;  // G exponent offset of this thread's cell in the prefetched batch
  // dof indices of column (el, jk) of batch b, from the map tile or global
  auto indices = [&](int64_t b) {
    const bool ok = el < T.cells_of(b);
    if (map_window(b)) {
      const uint32_t *m = sMap + ((b * E * N3) & 3) + el * N3 + jk;
#pragma unroll
      for (int i = 0; i < N; ++i) idx[i] = ok ? m[i * N2] : MFGB_INVALID_DOF;
    } else {
      const uint32_t *m = map + (b * E + el) * N3 + jk;
#pragma unroll
      for (int i = 0; i < N; ++i) idx[i] = ok ? __ldg(m + i * N2) : MFGB_INVALID_DOF;
    }
  };
  // component c of the column's values (EVEC: of batch b), and the cell's G exponent
  auto gather = [&](int64_t b, int c) {
    if constexpr (EVEC) {
      const bool ok = el < T.cells_of(b);
#pragma unroll
      for (int i = 0; i < N; ++i)
        raw[i] = ok ? __ldg(src + (b * E + el) * N3 + i * N2 + jk) : 0.0;
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i)
        raw[i] = idx[i] != MFGB_INVALID_DOF ? __ldg(src + (size_t)NC * idx[i] + c) : 0.0;
    }
  };
  // gathered column -> its largest exponent into the cell's slot
  auto reduce_exp = [&](int slot) {
    unsigned em = 0;
#pragma unroll
    for (int i = 0; i < N; ++i)
      em = max(em, (unsigned)(__double_as_longlong(raw[i]) >> 32) & 0x7FFFFFFFu);
    if (em >> 20) atomicMax(&s_emax[slot][el], (int)(em >> 20));
  };
  {
    if constexpr (!EVEC) {
      const bool ok = mbar_wait(mbar_m, ph_m, wlim);
      if (__syncthreads_or(!ok)) { fail(ph_g, ph_m); return; }
      ph_m ^= 1u;
      indices(batch);
    }
    gather(batch, 0);
    reduce_exp(0);
    if (!G64 && el < T.cells_of(batch)) ge = __ldg(gexp + batch * E + el);
  }

  int cnt = 0;  // components run so far: the exponent slot alternates with it
  for (; batch < n_batches; batch += gridDim.x) {
    const int64_t next = batch + gridDim.x;
    const bool has_next = next < n_batches;
    const bool okg = mbar_wait(mbar_g, ph_g, wlim);
    if (__syncthreads_or(!okg)) { fail(ph_g, ph_m); return; }  // barrier A
    ph_g ^= 1u;
    const bool valid = el < T.cells_of(batch);
    const GT *Gc = sG + el * 6 * N3 + jk;
    if constexpr (G64) {  // the cell's largest G exponent (read after barrier B)
      if (valid) {
        int eg = 0;
#pragma unroll 1
        for (int c = 0; c < 6; ++c)
#pragma unroll
          for (int i = 0; i < N; ++i) eg = max(eg, dexp(Gc[c * N3 + i * N2]));
        if (eg) atomicMax(&s_gmax[el], eg);
      }
    }
    int sg = ge;  // G64: set after barrier B
#pragma unroll 1
    for (int c = 0; c < NC; ++c, ++cnt) {
      const int slot = cnt & 1;
      if (NC > 1 && c > 0) __syncthreads();  // this component's exponents are in; work arrays free
      const int emax = s_emax[slot][el];
      const int su = fx_offset(emax);
      df x[N], qr[N];
      if ((unsigned)(emax - 1) < 0x7FEu) {
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = fx_from_double_grid(raw[i], su);
      } else {  // all zero or subnormal, or an inf or NaN among the values
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = fx_grid(fx_from_double(raw[i], su), 3.f);
      }
#pragma unroll
      for (int i = 0; i < N; ++i) s_u[col + i * S::i] = x[i];
      fx_line_grid(basis.G, x, fx_line_max(x), qr);
      __syncthreads();  // barrier B: s_u ready, s_emax[slot] read (c = 0: the map tile is free)
      if (jk == 0) s_emax[slot][el] = 0;  // next written two components on
      if constexpr (G64)
        if (c == 0) sg = fx_offset(s_gmax[el]);
      if (!EVEC && c == 0 && tid == 0 && has_next) {
        fence_proxy_async_smem();
        issue_map(next);
      }
      // ---- gradient along the s- and t-lines
      {
        df y[N];
#pragma unroll
        for (int m = 0; m < N; ++m) x[m] = s_u[sline + m * S::j];
        fx_line_grid(basis.G, x, fx_line_max(x), y);
#pragma unroll
        for (int m = 0; m < N; ++m) s_s[sline + m * S::j] = y[m];
#pragma unroll
        for (int m = 0; m < N; ++m) x[m] = s_u[tline + m];
        fx_line_grid(basis.G, x, fx_line_max(x), y);
        if (NB == 2) __syncthreads();  // every s-line has been read
#pragma unroll
        for (int m = 0; m < N; ++m) s_t[tline + m] = y[m];
      }
      __syncthreads();
      // ---- metric, bound per point: max |q| times the row sums of |G|
      df vr[N];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const df qs = s_s[col + i * S::i], qt = s_t[col + i * S::i];
        auto g = [&](int q) {  // (a cell past the end reads a stale tile; nothing leaves it)
          if constexpr (G64) {  // converted to pairs scaled by 2^-sg as it is read
            const df d = fx_from_double(Gc[q * N3 + i * N2], sg);
            return make_float2(d.hi, d.lo);
          } else {
            return Gc[q * N3 + i * N2];
          }
        };
        const float2 grr = g(0), grs = g(1), grt = g(2), gss = g(3), gst = g(4), gtt = g(5);
        const float kq = basis.K * fmaxf(fmaxf(fabsf(qr[i].hi), fabsf(qs.hi)), fabsf(qt.hi));
        const float Cr = (fabsf(grr.x) + fabsf(grs.x) + fabsf(grt.x)) * kq;
        const float Cs = (fabsf(grs.x) + fabsf(gss.x) + fabsf(gst.x)) * kq;
        const float Ct = (fabsf(grt.x) + fabsf(gst.x) + fabsf(gtt.x)) * kq;
        fxacc br, bs, bt;
        fx_first(br, grr.x, grr.y, qr[i].hi, qr[i].lo, Cr);
        fx_fma(br, grs.x, grs.y, qs.hi, qs.lo);
        fx_fma(br, grt.x, grt.y, qt.hi, qt.lo);
        fx_first(bs, grs.x, grs.y, qr[i].hi, qr[i].lo, Cs);
        fx_fma(bs, gss.x, gss.y, qs.hi, qs.lo);
        fx_fma(bs, gst.x, gst.y, qt.hi, qt.lo);
        fx_first(bt, grt.x, grt.y, qr[i].hi, qr[i].lo, Ct);
        fx_fma(bt, gst.x, gst.y, qs.hi, qs.lo);
        fx_fma(bt, gtt.x, gtt.y, qt.hi, qt.lo);
        vr[i] = fx_finish(br, Cr);
        s_s[col + i * S::i] = fx_finish(bs, Cs);
        s_t[col + i * S::i] = fx_finish(bt, Ct);
      }
      __syncthreads();  // barrier C: v_s, v_t ready (last component: G tile consumed)
      if (c == NC - 1) {
        if (G64 && jk == 0) s_gmax[el] = 0;
        if (tid == 0 && has_next) {
          fence_proxy_async_smem();
          T.issue_g(next);
        }
      }
      // this component's scatter targets; then prefetch the next component
      // (the next batch's first one after the last)
      const int64_t out_cell = batch * E + el;
      const int sc = su + sg;  // the cell's result scale
      uint32_t cur[N];
#pragma unroll
      for (int i = 0; i < N; ++i) cur[i] = EVEC ? 0u : idx[i];
      if (c + 1 < NC) {
        gather(batch, c + 1);
      } else if (has_next) {
        if constexpr (!EVEC) {
          const bool okm = mbar_wait(mbar_m, ph_m, wlim);
          if (!okm && err_flag) atomicOr(err_flag, 1);  // the launch's result is void
          ph_m ^= 1u;
          if (okm) {
            indices(next);
          } else {
#pragma unroll
            for (int i = 0; i < N; ++i) idx[i] = MFGB_INVALID_DOF;
          }
        }
        gather(next, 0);
        if (!G64) ge = el < T.cells_of(next) ? __ldg(gexp + next * E + el) : 0;
      }
      // ---- transpose along the s- and t-lines, in place
      {
        df y[N];
#pragma unroll
        for (int m = 0; m < N; ++m) x[m] = s_s[sline + m * S::j];
        fx_line(basis.T, x, y);
#pragma unroll
        for (int m = 0; m < N; ++m) s_s[sline + m * S::j] = y[m];
#pragma unroll
        for (int m = 0; m < N; ++m) x[m] = s_t[tline + m];
        fx_line(basis.T, x, y);
#pragma unroll
        for (int m = 0; m < N; ++m) s_t[tline + m] = y[m];
      }
      fx_line(basis.T, vr, qr);  // the r-share of the own column
      __syncthreads();
      if (!EVEC) cudaGridDependencySynchronize();  // dst has its start values
      auto put = [&](int i, double v) {
        if constexpr (EVEC) {
          if (valid) dst[out_cell * N3 + i * N2 + jk] = v;
        } else {
          if (cur[i] != MFGB_INVALID_DOF) atomicAdd(dst + (size_t)NC * cur[i] + c, v);
        }
      };
      if ((unsigned)(sc + 896) <= 1792u) {
        const unsigned kout = (unsigned)(896 + sc) << 20;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const df y = fx_sum3(qr[i], s_s[col + i * S::i], s_t[col + i * S::i]);
          put(i, fx_f2d_fast(y.hi, kout) + fx_f2d_fast(y.lo, kout));
        }
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const df y = fx_sum3(qr[i], s_s[col + i * S::i], s_t[col + i * S::i]);
          put(i, fx_f2d(y.hi, sc) + fx_f2d(y.lo, sc));
        }
      }
      // the prefetched gather's largest exponent per cell, once its loads have landed (read
      // after the next component's first barrier, or the next batch's barrier A)
      if (c + 1 < NC || has_next) reduce_exp(slot ^ 1);
    }
  }
}

}  // namespace mfgb
