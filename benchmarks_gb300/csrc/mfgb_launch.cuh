// mfgb_launch.cuh -- host-side launch helpers for the BK5 kernels.
#pragma once
#include <algorithm>
#include "mfgb_bk5.cuh"
#include "mfgb_bk5line.cuh"
#include "mfgb_internal.h"

namespace mfgb {

// elements per CTA for each N = p + 1 (CTA = E * N^2 threads)
template <int N> struct ElemsPerCta;
template <> struct ElemsPerCta<2> { static constexpr int value = 32; };
template <> struct ElemsPerCta<3> { static constexpr int value = 16; };
template <> struct ElemsPerCta<4> { static constexpr int value = 8; };
template <> struct ElemsPerCta<5> { static constexpr int value = 8; };
template <> struct ElemsPerCta<6> { static constexpr int value = 4; };
template <> struct ElemsPerCta<7> { static constexpr int value = 4; };
template <> struct ElemsPerCta<8> { static constexpr int value = 2; };
template <> struct ElemsPerCta<9> { static constexpr int value = 2; };

// bulk-TMA column kernel: elements per CTA, per arithmetic (default: as the
// column kernel)
template <int N, class A> struct ElemsPerCtaTma { static constexpr int value = ElemsPerCta<N>::value; };
template <> struct ElemsPerCtaTma<5, ArithDF> { static constexpr int value = 5; };

// Alternative cells per CTA for the autotuner's shapes 3 (column) and 4 (bulk
// TMA): a CTA of (nearly) whole warps, smaller or larger than the default.  Their
// residency cap follows the register budget of the arithmetic (about 128
// registers a thread for FP64 and double-float, 64 for FP32).  Offered (value
// > 0) for FP32 at every N and for FP64 / double-float up to N = 5; above that
// a 128-register cap spills, and the alternative shapes run as shapes 0 / 2.
template <int N> struct AltElemsN;
template <> struct AltElemsN<2> { static constexpr int value = 16; };  // 64 threads
template <> struct AltElemsN<3> { static constexpr int value = 14; };  // 126
template <> struct AltElemsN<4> { static constexpr int value = 4; };   // 64
template <> struct AltElemsN<5> { static constexpr int value = 10; };  // 250
template <> struct AltElemsN<6> { static constexpr int value = 3; };   // 108
template <> struct AltElemsN<7> { static constexpr int value = 6; };   // 294
template <> struct AltElemsN<8> { static constexpr int value = 1; };   // 64
template <> struct AltElemsN<9> { static constexpr int value = 4; };   // 324
template <int N, class A> struct AltElems { static constexpr int value = 0; };
template <int N> struct AltElems<N, ArithF32> { static constexpr int value = AltElemsN<N>::value; };
template <int N> struct AltElems<N, ArithF64> {
  static constexpr int value = N <= 5 ? AltElemsN<N>::value : 0;
};
template <int N> struct AltElems<N, ArithDF> {
  static constexpr int value = N <= 5 ? AltElemsN<N>::value : 0;
};
template <class A> struct RegThreads { static constexpr int value = 512; };
template <> struct RegThreads<ArithF32> { static constexpr int value = 1024; };
template <int N, int E, class A> struct AltMinBlocks {
  static constexpr int threads = (E * N * N + 31) / 32 * 32;
  static constexpr int raw = RegThreads<A>::value / (threads > 0 ? threads : 1);
  static constexpr int value = raw < 1 ? 1 : (raw > 8 ? 8 : raw);
};

// point-per-thread kernel: elements per CTA (CTA = E * N^3 threads)
template <int N> struct ElemsPerCtaPt;
template <> struct ElemsPerCtaPt<2> { static constexpr int value = 32; };
template <> struct ElemsPerCtaPt<3> { static constexpr int value = 8; };
template <> struct ElemsPerCtaPt<4> { static constexpr int value = 4; };
template <> struct ElemsPerCtaPt<5> { static constexpr int value = 2; };
template <> struct ElemsPerCtaPt<6> { static constexpr int value = 2; };
template <> struct ElemsPerCtaPt<7> { static constexpr int value = 1; };
template <> struct ElemsPerCtaPt<8> { static constexpr int value = 1; };
template <> struct ElemsPerCtaPt<9> { static constexpr int value = 1; };

// Kernel shape: 0 = column (thread owns an i-column), 1 = point-per-thread,
// 2 = column with TMA-prefetched geometric factors.  Default per
// (arithmetic, N); overridable at run time (autotuner).
// 5 and 6 (double-float only, GLL operators): the offset-accumulation kernel of
// mfgb_bk5fx.cuh at its two cells per CTA (FxDefault, FxAlt); elsewhere they run as 2 / 4.
enum { SHAPE_COLUMN = 0, SHAPE_POINT = 1, SHAPE_TMA = 2, SHAPE_COLUMN_ALT = 3, SHAPE_TMA_ALT = 4,
       SHAPE_FX = 5, SHAPE_FX_ALT = 6,
       SHAPE_LINE = 7, SHAPE_LINE_ALT = 8 };  // what shapes 2 and 4 become (bk5_shape)
int kernel_shape(int arith_class, int N);  // mfgb_api.cu
int *device_error_flag();                  // mfgb_api.cu

template <class A> struct ArithClass { static constexpr int value = 0; };  // FP64
template <> struct ArithClass<ArithDF> { static constexpr int value = 1; };
template <> struct ArithClass<ArithDFG64> { static constexpr int value = 1; };
template <> struct ArithClass<ArithF32> { static constexpr int value = 2; };

inline int num_sms() {
  static int sms = -1;
  if (sms < 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 152;
  }
  return sms;
}

// CTAs per SM of one kernel instantiation (queried once).  Sets the kernel's
// dynamic shared-memory limit to smem: without it, dynamic plus static shared
// memory above 48 KB fails at launch.
template <class K>
int ctas_per_sm(K kernel, int threads, size_t smem) {
  int ps = 0;
  if (smem > 0) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, kernel, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    ps = 0;
  }
  return ps;
}

// The same for a kernel that starts beside the one before it (launch_after): shared memory at its
// largest share of the SM, so that a first CTA placed while the other kernel runs does not leave the SM
// a split into which the second one does not fit (vmult at 0.4M DoFs, us without / with: collocation
// p = 4 18.0 / 14.7, Gauss p = 4 22.7 / 18.7, BP3 p = 8 35.1 / 29.1).
template <class K>
int ctas_per_sm_beside(K kernel, int threads, size_t smem) {
  const int ps = ctas_per_sm(kernel, threads, smem);
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  return ps;
}

// One launch; after = true: it may begin while the kernel before it on the stream (which must let it,
// start_vmult) still runs, and waits for that one's end inside (cudaGridDependencySynchronize).
template <class... P, class... Q>
cudaError_t launch_after(bool after, void (*kernel)(P...), int grid, int threads, size_t smem,
                         cudaStream_t s, Q... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = after ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Shapes 2 and 4 of the plain arithmetics as the line kernel (mfgb_bk5line.cuh): cells per CTA,
// resident CTAs and work arrays.  FP32 at every degree, FP64 from N = 6 (below, the column kernel's
// 4.05 / 3.82 ms at N = 4, 5 are not beaten: 4.62 / 3.86; the FP64 pipe is the bound and the even-odd
// additions cost as much as the multiply-adds they save).  One application (clearing, kernel, identity
// rows) at 3e7 DoFs in ms against the same with the best earlier shape: FP32, N = 3..9 0.68 / 0.75, 0.42 /
// 0.50, 0.36 / 0.51, 0.32 / 0.36, 0.30 / 0.51, 0.27 / 0.28, 0.28 / 0.42; FP64, N = 6..9 4.28 / 4.49, 4.21 /
// 4.63, 3.91 / 4.34, 4.71 / 5.00.
template <int E_, int MB_, int NB_> struct LineShapeIs {
  static constexpr int E = E_, MB = MB_, NB = NB_;
};
template <int N, class A> struct LineShape : LineShapeIs<0, 0, 0> {};
template <> struct LineShape<2, ArithF32> : LineShapeIs<64, 6, 2> {};
template <> struct LineShape<3, ArithF32> : LineShapeIs<28, 5, 2> {};
template <> struct LineShape<4, ArithF32> : LineShapeIs<16, 4, 3> {};
template <> struct LineShape<5, ArithF32> : LineShapeIs<10, 4, 2> {};
template <> struct LineShape<6, ArithF32> : LineShapeIs<7, 4, 3> {};
template <> struct LineShape<7, ArithF32> : LineShapeIs<5, 4, 2> {};
template <> struct LineShape<8, ArithF32> : LineShapeIs<3, 4, 3> {};
template <> struct LineShape<9, ArithF32> : LineShapeIs<3, 3, 3> {};
template <> struct LineShape<6, ArithF64> : LineShapeIs<5, 3, 2> {};
template <> struct LineShape<7, ArithF64> : LineShapeIs<3, 3, 2> {};
template <> struct LineShape<8, ArithF64> : LineShapeIs<2, 3, 2> {};
template <> struct LineShape<9, ArithF64> : LineShapeIs<1, 4, 2> {};
// fewer cells per CTA: shape 4, and shape 2 on meshes too small for one batch per resident CTA
template <int N, class A> struct LineAlt : LineShape<N, A> {};
template <> struct LineAlt<2, ArithF32> : LineShapeIs<32, 8, 3> {};
template <> struct LineAlt<3, ArithF32> : LineShapeIs<14, 8, 3> {};
template <> struct LineAlt<4, ArithF32> : LineShapeIs<8, 8, 3> {};
template <> struct LineAlt<5, ArithF32> : LineShapeIs<5, 8, 3> {};
template <> struct LineAlt<6, ArithF32> : LineShapeIs<3, 8, 3> {};
template <> struct LineAlt<7, ArithF32> : LineShapeIs<3, 6, 2> {};
template <> struct LineAlt<8, ArithF32> : LineShapeIs<1, 12, 3> {};
template <> struct LineAlt<9, ArithF32> : LineShapeIs<1, 8, 3> {};
template <> struct LineAlt<6, ArithF64> : LineShapeIs<3, 5, 2> {};

// The shape of degrees with a line kernel where that one does not apply: element vectors, arrays that
// are not 16-byte aligned, a caller's matrix without the mirror symmetry.  FP64, ms at 6e6 values as
// this shape / the column kernel: element vectors N = 7 0.585 / 0.659, 9 0.699 / 0.916 (N = 6 and 8 run
// the column kernel: no bulk copies there); L-vectors with a general matrix N = 6..9 0.973 / 0.999,
// 0.988 / 1.149, 1.029 / 1.052, 1.047 / 1.319.
template <int N, class A> struct LineFallback { static constexpr int value = SHAPE_COLUMN; };
template <> struct LineFallback<6, ArithF64> { static constexpr int value = SHAPE_TMA; };
template <> struct LineFallback<7, ArithF64> { static constexpr int value = SHAPE_POINT; };
template <> struct LineFallback<8, ArithF64> { static constexpr int value = SHAPE_TMA; };
template <> struct LineFallback<9, ArithF64> { static constexpr int value = SHAPE_POINT; };
// whether the column kernel with bulk copies can be chosen
template <int N, class A, bool EVEC>
constexpr bool has_tma() {
  return !EVEC && (LineShape<N, A>::E == 0 || LineFallback<N, A>::value == SHAPE_TMA);
}

// The kernel a launch takes, from the shape table's entry: aligned: G and the map on 16 bytes, mirror:
// the matrix has the mirror symmetry of symmetric points (Basis::eo).  Shapes 5 / 6 are the
// double-float operators' own and run as 2 / 4 here; without an alternative cells-per-CTA
// instantiation (E-vectors, other arithmetic, large N) 3 / 4 run as 0 / 2; bulk copies need aligned
// tiles of L-vectors.
template <int N, class A, bool EVEC>
int bk5_shape(bool aligned, bool mirror) {
  int shape = kernel_shape(ArithClass<A>::value, N);
  if (shape == SHAPE_FX) shape = SHAPE_TMA;
  if (shape == SHAPE_FX_ALT) shape = SHAPE_TMA_ALT;
  if (LineShape<N, A>::E > 0 && (shape == SHAPE_TMA || shape == SHAPE_TMA_ALT)) {
    if (!EVEC && aligned && mirror) return shape == SHAPE_TMA ? SHAPE_LINE : SHAPE_LINE_ALT;
    shape = LineFallback<N, A>::value;
  }
  if (EVEC || AltElems<N, A>::value == 0) {
    if (shape == SHAPE_COLUMN_ALT) shape = SHAPE_COLUMN;
    if (shape == SHAPE_TMA_ALT) shape = SHAPE_TMA;
  }
  if ((shape == SHAPE_TMA || shape == SHAPE_TMA_ALT) && (EVEC || !aligned)) shape = SHAPE_COLUMN;
  return shape;
}

// one launch of the line kernel
template <int N, class A, class Sh>
cudaError_t line_run(int64_t n_cells, const uint32_t *map, const typename A::GType *G,
                     const typename A::VecT *src, typename A::VecT *dst, const Basis<N, A> &basis,
                     int *grid_used, cudaStream_t stream, const int *done) {
  constexpr int E = Sh::E, T = E * N * N;
  constexpr size_t smem = LineLayout<N, E, typename A::VecT, Sh::NB>::total;
  const auto kernel = bk5_line_kernel<N, E, Sh::MB, Sh::NB, A>;
  static PerDevice found;
  const int per_sm = found([&] { return std::max(1, ctas_per_sm(kernel, T, smem)); });
  const int64_t nb = (n_cells + E - 1) / E;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(nb, (int64_t)per_sm * num_sms()));
  if (grid_used) *grid_used = grid;
  if (n_cells <= 0) return cudaSuccess;
  kernel<<<grid, T, smem, stream>>>(n_cells, map, G, src, dst, basis, done, device_error_flag());
  return cudaGetLastError();
}

// grid for a persistent launch: all resident CTAs, capped by the work
template <int N, class A, bool EVEC, bool EN>
int bk5_grid(int64_t n_cells, int shape) {
  static int per_sm[5] = {-1, -1, -1, -1, -1};
  int &ps = per_sm[shape];
  int E = 1;
  constexpr int EA = AltElems<N, A>::value;
  if (shape == SHAPE_COLUMN_ALT) {
    if constexpr (EA > 0 && !EVEC) {
      E = EA;
      if (ps < 0)
        ps = ctas_per_sm(bk5_kernel_mb<N, EA, A, EVEC, EN, AltMinBlocks<N, EA, A>::value>,
                         EA * N * N, 0);
    }
  } else if (shape == SHAPE_TMA_ALT) {
    if constexpr (EA > 0 && has_tma<N, A, EVEC>()) {
      E = EA;
      if (ps < 0)
        ps = ctas_per_sm(bk5_tma_kernel<N, EA, A, EN, AltMinBlocks<N, EA, A>::value>, EA * N * N,
                         TmaLayout<N, EA, A>::total);
    }
  } else if (shape == SHAPE_POINT) {
    E = ElemsPerCtaPt<N>::value;
    if (ps < 0) ps = ctas_per_sm(bk5_pt_kernel<N, ElemsPerCtaPt<N>::value, A, EVEC, EN>, E * N * N * N, 0);
  } else if (shape == SHAPE_TMA) {
    if constexpr (has_tma<N, A, EVEC>()) {
      constexpr int ET = ElemsPerCtaTma<N, A>::value;
      E = ET;
      if (ps < 0)
        ps = ctas_per_sm(bk5_tma_kernel<N, ET, A, EN>, ET * N * N, TmaLayout<N, ET, A>::total);
    }
  } else {
    E = ElemsPerCta<N>::value;
    if (ps < 0) {
      if constexpr (ColumnMinBlocks<N, A>::value > 0)
        ps = ctas_per_sm(bk5_kernel_capped<N, ElemsPerCta<N>::value, A, EVEC, EN>, E * N * N, 0);
      else
        ps = ctas_per_sm(bk5_kernel<N, ElemsPerCta<N>::value, A, EVEC, EN>, E * N * N, 0);
    }
  }
  if (ps < 1) ps = 1;
  const int64_t n_batches = (n_cells + E - 1) / E;
  const int64_t full = (int64_t)ps * num_sms();
  return (int)std::max<int64_t>(1, std::min<int64_t>(n_batches, full));
}

template <int N, class A, bool EVEC, bool EN>
cudaError_t bk5_launch(int64_t n_cells, const uint32_t *map, const typename A::GType *G,
                       const typename A::VecT *src, typename A::VecT *dst,
                       const Basis<N, A> &basis, double *partials, int *grid_used,
                       cudaStream_t stream, const int *done_flag = nullptr) {
  const bool aligned = !((reinterpret_cast<uintptr_t>(G) | reinterpret_cast<uintptr_t>(map)) & 15u);
  const int shape = bk5_shape<N, A, EVEC>(aligned, basis.eo);
  if constexpr (!EVEC && LineShape<N, A>::E > 0) {
    using Sh = LineShape<N, A>;
    if (shape == SHAPE_LINE_ALT || (shape == SHAPE_LINE && n_cells <= (int64_t)Sh::E * Sh::MB * num_sms()))
      return line_run<N, A, LineAlt<N, A>>(n_cells, map, G, src, dst, basis, grid_used, stream, done_flag);
    if (shape == SHAPE_LINE)
      return line_run<N, A, Sh>(n_cells, map, G, src, dst, basis, grid_used, stream, done_flag);
  }
  const int grid = bk5_grid<N, A, EVEC, EN>(n_cells, shape);
  if (grid_used) *grid_used = grid;
  if (n_cells <= 0) return cudaSuccess;
  constexpr int EA = AltElems<N, A>::value;
  constexpr int MBA = AltMinBlocks<N, EA, A>::value;
  constexpr bool TMA = has_tma<N, A, EVEC>();
  if (shape == SHAPE_COLUMN_ALT) {
    if constexpr (EA > 0 && !EVEC)
      bk5_kernel_mb<N, EA, A, EVEC, EN, MBA><<<grid, EA * N * N, 0, stream>>>(
          n_cells, map, G, src, dst, basis, partials, done_flag);
  } else if (shape == SHAPE_TMA_ALT) {
    if constexpr (EA > 0 && TMA)
      bk5_tma_kernel<N, EA, A, EN, MBA><<<grid, EA * N * N, TmaLayout<N, EA, A>::total, stream>>>(
          n_cells, map, G, src, dst, basis, partials, done_flag, device_error_flag());
  } else if (shape == SHAPE_POINT) {
    constexpr int E = ElemsPerCtaPt<N>::value;
    bk5_pt_kernel<N, E, A, EVEC, EN><<<grid, E * N * N * N, 0, stream>>>(
        n_cells, map, G, src, dst, basis, partials, done_flag);
  } else if (shape == SHAPE_TMA) {
    if constexpr (TMA) {
      constexpr int E = ElemsPerCtaTma<N, A>::value;
      bk5_tma_kernel<N, E, A, EN><<<grid, E * N * N, TmaLayout<N, E, A>::total, stream>>>(
          n_cells, map, G, src, dst, basis, partials, done_flag, device_error_flag());
    }
  } else {
    constexpr int E = ElemsPerCta<N>::value;
    if constexpr (ColumnMinBlocks<N, A>::value > 0)
      bk5_kernel_capped<N, E, A, EVEC, EN><<<grid, E * N * N, 0, stream>>>(
          n_cells, map, G, src, dst, basis, partials, done_flag);
    else
      bk5_kernel<N, E, A, EVEC, EN><<<grid, E * N * N, 0, stream>>>(n_cells, map, G, src, dst,
                                                                     basis, partials, done_flag);
  }
  return cudaGetLastError();
}

}  // namespace mfgb
