// mfgb_fxline.cuh -- 1D contractions of whole lines in offset double-float arithmetic.
//
// A tensor-product operator is a sequence of products of small 1D matrices with the
// lines of a cell.  Here one thread owns a whole line: it reads the line's values
// once, keeps them in registers and computes every output of the line, so the
// matrix entries are compile-time indexed (constant operands), each value is read
// once per direction instead of once per output, and the matrix's mirror symmetry
// can be used.
//
// Even-odd form.  The matrices of points symmetric about the cell centre satisfy
// M[NO-1-o][NI-1-i] = +M[o][i] (interpolation) or -M[o][i] (derivative).  With
// e_i = x_i + x_{NI-1-i}, f_i = x_i - x_{NI-1-i} and the half-size matrices
// P = (M[o][i] + M[o][NI-1-i]) / 2, Q = (M[o][i] - M[o][NI-1-i]) / 2,
//   A_o = sum_i P[o][i] e_i (+ the centre column),  B_o = sum_i Q[o][i] f_i,
//   y_o = A_o + B_o,   y_{NO-1-o} = +-(A_o - B_o)
// which halves the multiply-adds.  In the offset form a multiply-add costs 6
// instructions, while the additions here are exact on the high parts and cost one
// instruction per part:
//   * the inputs are first rounded to a common grid (T = fl(3 m + x), h = T - 3 m
//     exact, the remainder joins the low part; m >= max |x|): 2 m <= T <= 4 m, so h
//     is a multiple of g = ulp(2 m) and |h_a +- h_b| <= 2 m <= 2^24 g is exact;
//   * A and B share the offset C = b + R, b the larger of their bounds and R >= b the
//     bound of A +- B (the row sum of |M|): every T is at least C - b = R, so the high
//     parts T - C are multiples of g = ulp(R) and |A +- B| <= R <= 2^24 g is exact.
// For R near b this is the plain form's offset 2 b, and the rounding error stays at
// about 2^-46 of the bound; tests/test_fx_line.py restates the arithmetic and checks
// the exact steps.
#pragma once
#include "mfgb_common.cuh"

namespace mfgb {

// offset accumulator: value = (T - C) + S
struct fxacc {
  float T, S;
};

__device__ __forceinline__ void fx_first(fxacc &a, float xh, float xl, float yh, float yl,
                                         float C) {
  a.T = __fmaf_rn(xh, yh, C);
  const float d = __fsub_rn(a.T, C);
  const float r = __fmaf_rn(xh, yh, -d);
  a.S = __fmaf_rn(xl, yh, __fmaf_rn(xh, yl, r));
}

// the low-order terms of one product (its rounding error and the two cross
// products) are summed first and join S with one addition: the two chains a
// sum carries (T and S) advance by one dependent instruction per term
__device__ __forceinline__ void fx_fma(fxacc &a, float xh, float xl, float yh, float yl) {
  const float t = __fmaf_rn(xh, yh, a.T);
  const float d = __fsub_rn(t, a.T);
  const float r = __fmaf_rn(xh, yh, -d);
  const float e = __fmaf_rn(xl, yh, __fmaf_rn(xh, yl, r));
  a.S = __fadd_rn(a.S, e);
  a.T = t;
}

__device__ __forceinline__ df fx_finish(const fxacc &a, float C) {
  df r;
  r.hi = __fsub_rn(a.T, C);
  r.lo = a.S;
  return r;
}

// x rounded to the grid of offset C = 3 m, m >= |x|; the remainder joins the low part
__device__ __forceinline__ df fx_grid(df x, float C) {
  df r;
  r.hi = __fsub_rn(__fadd_rn(C, x.hi), C);
  r.lo = __fadd_rn(__fsub_rn(x.hi, r.hi), x.lo);
  return r;
}

__device__ __forceinline__ df fx_add_exact(df a, df b) {  // both on one grid
  return df{__fadd_rn(a.hi, b.hi), __fadd_rn(a.lo, b.lo)};
}
__device__ __forceinline__ df fx_sub_exact(df a, df b) {
  return df{__fsub_rn(a.hi, b.hi), __fsub_rn(a.lo, b.lo)};
}

// a + b: TwoSum of the high parts, the error joins the low parts
__device__ __forceinline__ df fx_sum2(df a, df b) {
  const float s = __fadd_rn(a.hi, b.hi);
  const float bb = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
  return df{s, __fadd_rn(__fadd_rn(a.lo, b.lo), e)};
}

// a + b + c: TwoSum of the high parts, the errors join the low parts
__device__ __forceinline__ df fx_sum3(df a, df b, df c) {
  const float s = __fadd_rn(a.hi, b.hi);
  const float bb = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
  const float t = __fadd_rn(s, c.hi);
  const float cc = __fsub_rn(t, s);
  const float f = __fadd_rn(__fsub_rn(s, __fsub_rn(t, cc)), __fsub_rn(c.hi, cc));
  return df{t, __fadd_rn(__fadd_rn(__fadd_rn(a.lo, b.lo), __fadd_rn(e, f)), c.lo)};
}

// 1D matrix M[NO][NI] for line contractions.  SYM: +1 / -1 mirror (anti)symmetric
// in even-odd form, 0 general (dense).  c[o]: the offset per unit of the largest
// |input| (host: fx_line_matrix).
template <int NI, int NO, int SYM>
struct FxMat {
  static constexpr int ni = NI, no = NO, sym = SYM;
  static constexpr int HI = NI / 2, CI = (NI + 1) / 2, CO = (NO + 1) / 2;
  float Ph[CO][CI], Pl[CO][CI];  // the centre column (odd NI) is Ph[.][HI]
  float Qh[CO][HI], Ql[CO][HI];
  float c[CO];
};
template <int NI, int NO>
struct FxMat<NI, NO, 0> {
  static constexpr int ni = NI, no = NO, sym = 0;
  float h[NO][NI], l[NO][NI];
  float c[NO];
};

// y = M x from the sums e and differences f of the mirrored inputs (SYM != 0; the centre input, odd
// NI, in xc), mx >= max |x.hi|
template <int NI, int NO, int SYM>
__device__ __forceinline__ void fx_line_ef(const FxMat<NI, NO, SYM> &M, const df *e, const df *f,
                                           df xc, float mx, df (&y)[NO]) {
  constexpr int HI = NI / 2;
#pragma unroll
  for (int o = 0; o < (NO + 1) / 2; ++o) {
    const bool centre = (NO % 2) && o == NO / 2;
    const float C = M.c[o] * mx;
    df A{0.f, 0.f}, B{0.f, 0.f};
    if (!(centre && SYM < 0)) {
      fxacc a;
      fx_first(a, M.Ph[o][0], M.Pl[o][0], e[0].hi, e[0].lo, C);
#pragma unroll
      for (int i = 1; i < HI; ++i) fx_fma(a, M.Ph[o][i], M.Pl[o][i], e[i].hi, e[i].lo);
      if constexpr (NI % 2) fx_fma(a, M.Ph[o][HI], M.Pl[o][HI], xc.hi, xc.lo);
      A = fx_finish(a, C);
    }
    if (!(centre && SYM > 0)) {
      fxacc b;
      fx_first(b, M.Qh[o][0], M.Ql[o][0], f[0].hi, f[0].lo, C);
#pragma unroll
      for (int i = 1; i < HI; ++i) fx_fma(b, M.Qh[o][i], M.Ql[o][i], f[i].hi, f[i].lo);
      B = fx_finish(b, C);
    }
    if (centre) {
      y[o] = SYM < 0 ? B : A;
    } else {
      y[o] = fx_add_exact(A, B);
      y[NO - 1 - o] = SYM < 0 ? fx_sub_exact(B, A) : fx_sub_exact(A, B);
    }
  }
}

// y = M x for inputs already on the grid of offset 3 mx, mx >= max |x.hi| (SYM != 0)
template <int NI, int NO, int SYM>
__device__ __forceinline__ void fx_line_grid(const FxMat<NI, NO, SYM> &M, const df (&x)[NI], float mx,
                                             df (&y)[NO]) {
  if constexpr (SYM == 0) {
#pragma unroll
    for (int o = 0; o < NO; ++o) {
      const float C = M.c[o] * mx;
      fxacc a;
      fx_first(a, M.h[o][0], M.l[o][0], x[0].hi, x[0].lo, C);
#pragma unroll
      for (int i = 1; i < NI; ++i) fx_fma(a, M.h[o][i], M.l[o][i], x[i].hi, x[i].lo);
      y[o] = fx_finish(a, C);
    }
  } else {
    df e[NI / 2], f[NI / 2];
#pragma unroll
    for (int i = 0; i < NI / 2; ++i) {
      e[i] = fx_add_exact(x[i], x[NI - 1 - i]);
      f[i] = fx_sub_exact(x[i], x[NI - 1 - i]);
    }
    fx_line_ef(M, e, f, x[NI / 2], mx, y);
  }
}

template <int N>
__device__ __forceinline__ float fx_line_max(const df (&x)[N]) {
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) m = fmaxf(m, fabsf(x[i].hi));
  return m;
}

// y = M x for any inputs: the line's largest |value| sets the grid and the offsets
template <int NI, int NO, int SYM>
__device__ __forceinline__ void fx_line(const FxMat<NI, NO, SYM> &M, df (&x)[NI], df (&y)[NO]) {
  float mx = fx_line_max(x);
  if constexpr (SYM != 0) {
    mx = __fmul_rn(mx, 1.0f + 0x1p-20f);  // the rounded values may exceed it by half a grid step
    const float C = __fmul_rn(mx, 3.f);
#pragma unroll
    for (int i = 0; i < NI / 2; ++i) {
      x[i] = fx_grid(x[i], C);
      x[NI - 1 - i] = fx_grid(x[NI - 1 - i], C);
    }
  }
  fx_line_grid(M, x, mx, y);
}

// The same with the sums and differences by TwoSum instead of a common grid: 4 instructions a pair
// more, and no rounding of the inputs' low parts to the grid.  For interpolation of short lines,
// where that rounding is what is left (relative error of one line, NI -> NO = 2 -> 3: plain form
// 8.6e-15, grid 10.2e-15, TwoSum 8.4e-15; 4 -> 5: 16.4, 15.6, 13.9; 5 -> 4: 11.5, 12.8, 10.6).
template <int NI, int NO, int SYM>
__device__ __forceinline__ void fx_line_sums(const FxMat<NI, NO, SYM> &M, const df (&x)[NI],
                                             df (&y)[NO]) {
  const float mx = fx_line_max(x);
  if constexpr (SYM == 0) {
    fx_line_grid(M, x, mx, y);
  } else {
    df e[NI / 2], f[NI / 2];
#pragma unroll
    for (int i = 0; i < NI / 2; ++i) {
      const df a = x[i], b = x[NI - 1 - i];
      e[i] = fx_sum2(a, b);
      f[i] = fx_sum2(a, df{-b.hi, -b.lo});
    }
    fx_line_ef(M, e, f, x[NI / 2], __fmul_rn(mx, 1.0f + 0x1p-20f), y);
  }
}

// y = P z + R v with P symmetric and R antisymmetric (SYM) or both general: the two products share
// their accumulators, y_o = X + Y, y_{NO-1-o} = X - Y with X = A_P + B_R, Y = B_P + A_R
template <int NI, int NO, int SP, int SR>
__device__ __forceinline__ void fx_line_joint(const FxMat<NI, NO, SP> &P, const FxMat<NI, NO, SR> &R,
                                              df (&z)[NI], df (&v)[NI], df (&y)[NO]) {
  float mz = fx_line_max(z), mv = fx_line_max(v);
  if constexpr (SP == 0) {
    static_assert(SR == 0, "both general or P symmetric and R antisymmetric");
#pragma unroll
    for (int o = 0; o < NO; ++o) {
      const float C = __fmaf_rn(P.c[o], mz, R.c[o] * mv);
      fxacc a;
      fx_first(a, P.h[o][0], P.l[o][0], z[0].hi, z[0].lo, C);
      fx_fma(a, R.h[o][0], R.l[o][0], v[0].hi, v[0].lo);
#pragma unroll
      for (int i = 1; i < NI; ++i) {
        fx_fma(a, P.h[o][i], P.l[o][i], z[i].hi, z[i].lo);
        fx_fma(a, R.h[o][i], R.l[o][i], v[i].hi, v[i].lo);
      }
      y[o] = fx_finish(a, C);
    }
  } else {
    static_assert(SP == 1 && SR == -1, "both general or P symmetric and R antisymmetric");
    constexpr int HI = NI / 2;
    mz = __fmul_rn(mz, 1.0f + 0x1p-20f);
    mv = __fmul_rn(mv, 1.0f + 0x1p-20f);
    const float Cz = __fmul_rn(mz, 3.f), Cv = __fmul_rn(mv, 3.f);
    df ez[HI], fz[HI], ev[HI], fv[HI];
#pragma unroll
    for (int i = 0; i < HI; ++i) {
      const df a = fx_grid(z[i], Cz), b = fx_grid(z[NI - 1 - i], Cz);
      ez[i] = fx_add_exact(a, b), fz[i] = fx_sub_exact(a, b);
      const df c = fx_grid(v[i], Cv), d = fx_grid(v[NI - 1 - i], Cv);
      ev[i] = fx_add_exact(c, d), fv[i] = fx_sub_exact(c, d);
    }
#pragma unroll
    for (int o = 0; o < (NO + 1) / 2; ++o) {
      const bool centre = (NO % 2) && o == NO / 2;
      const float C = __fmaf_rn(P.c[o], mz, R.c[o] * mv);
      fxacc a;
      fx_first(a, P.Ph[o][0], P.Pl[o][0], ez[0].hi, ez[0].lo, C);
      fx_fma(a, R.Qh[o][0], R.Ql[o][0], fv[0].hi, fv[0].lo);
#pragma unroll
      for (int i = 1; i < HI; ++i) {
        fx_fma(a, P.Ph[o][i], P.Pl[o][i], ez[i].hi, ez[i].lo);
        fx_fma(a, R.Qh[o][i], R.Ql[o][i], fv[i].hi, fv[i].lo);
      }
      if constexpr (NI % 2) fx_fma(a, P.Ph[o][HI], P.Pl[o][HI], z[HI].hi, z[HI].lo);
      const df X = fx_finish(a, C);
      if (centre) {
        y[o] = X;
      } else {
        fxacc b;
        fx_first(b, P.Qh[o][0], P.Ql[o][0], fz[0].hi, fz[0].lo, C);
        fx_fma(b, R.Ph[o][0], R.Pl[o][0], ev[0].hi, ev[0].lo);
#pragma unroll
        for (int i = 1; i < HI; ++i) {
          fx_fma(b, P.Qh[o][i], P.Ql[o][i], fz[i].hi, fz[i].lo);
          fx_fma(b, R.Ph[o][i], R.Pl[o][i], ev[i].hi, ev[i].lo);
        }
        if constexpr (NI % 2) fx_fma(b, R.Ph[o][HI], R.Pl[o][HI], v[HI].hi, v[HI].lo);
        const df Y = fx_finish(b, C);
        y[o] = fx_add_exact(X, Y);
        y[NO - 1 - o] = fx_sub_exact(X, Y);
      }
    }
  }
}

// deals the lines a[0..T) over groups of W lanes that access shared memory together (16 for 8-byte
// values, 32 for 4-byte ones): each takes lines from the banks (offset mod W) that have most left, a
// bank twice only when every other one is used up
template <int W = 16, int T>
constexpr void fx_deal(const int (&a)[T], unsigned short (&out)[T]) {
  bool used[T] = {};
  int left[W] = {};
  for (int v : a) ++left[v % W];
  for (int h = 0; h < T; h += W) {
    bool bank[W] = {};
    for (int t = h; t < T && t < h + W; ++t) {
      int best = -1;
      for (int b = 0; b < W; ++b)
        if (left[b] > 0 && !bank[b] && (best < 0 || left[b] > left[best])) best = b;
      if (best < 0)
        for (int b = 0; b < W; ++b)
          if (left[b] > 0 && (best < 0 || left[b] > left[best])) best = b;
      bank[best] = true;
      --left[best];
      for (int q = 0; q < T; ++q)
        if (!used[q] && a[q] % W == best) {
          used[q] = true;
          out[t] = (unsigned short)a[q];
          break;
        }
    }
  }
}

// host: the tables of M[o*NI + i].  Returns false when SYM != 0 and M lacks that
// mirror symmetry (to 2^-49 of its largest entry, the precision of the pairs).
template <int NI, int NO, int SYM>
inline bool fx_line_matrix(const double *M, FxMat<NI, NO, SYM> &t) {
  auto split = [](double v, float &h, float &l) {
    h = (float)v;
    l = (float)(v - (double)h);
  };
  auto mag = [](double v) { return v < 0 ? -v : v; };
  if constexpr (SYM == 0) {
    for (int o = 0; o < NO; ++o) {
      double s = 0.0;
      for (int i = 0; i < NI; ++i) {
        split(M[o * NI + i], t.h[o][i], t.l[o][i]);
        s += mag(t.h[o][i]);
      }
      t.c[o] = (float)(2.0 * (1.0 + 0x1p-20) * s);
    }
    return true;
  } else {
    double big = 0.0, off = 0.0;
    for (int q = 0; q < NI * NO; ++q) {
      const double a = mag(M[q]), d = mag(M[q] - SYM * M[NI * NO - 1 - q]);
      big = a > big ? a : big;
      off = d > off ? d : off;
    }
    if (!(off <= 0x1p-49 * big)) return false;
    constexpr int HI = NI / 2;
    for (int o = 0; o < (NO + 1) / 2; ++o) {
      // the mirrored row averaged in: the symmetric part of M, exactly
      auto m = [&](int i) {
        return 0.5 * (M[o * NI + i] + SYM * M[(NO - 1 - o) * NI + (NI - 1 - i)]);
      };
      double bp = 0.0, bq = 0.0, row = 0.0;
      for (int i = 0; i < HI; ++i) {
        split(0.5 * (m(i) + m(NI - 1 - i)), t.Ph[o][i], t.Pl[o][i]);
        split(0.5 * (m(i) - m(NI - 1 - i)), t.Qh[o][i], t.Ql[o][i]);
        bp += 2.0 * mag(t.Ph[o][i]);  // |e|, |f| <= 2 max |x|
        bq += 2.0 * mag(t.Qh[o][i]);
        row += 2.0 * (mag(t.Ph[o][i]) > mag(t.Qh[o][i]) ? mag(t.Ph[o][i]) : mag(t.Qh[o][i]));
      }
      if (NI % 2) {
        split(m(HI), t.Ph[o][HI], t.Pl[o][HI]);
        bp += mag(t.Ph[o][HI]);
        row += mag(t.Ph[o][HI]);
      }
      t.c[o] = (float)((1.0 + 0x1p-18) * ((bp > bq ? bp : bq) + row));
    }
    return true;
  }
}

}  // namespace mfgb
