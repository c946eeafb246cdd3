// mfgb_mg_kernels.cuh -- element-wise, Chebyshev and transfer kernels shared
// by the single-problem multigrid (mfgb_mg.cu) and the batched solver
// (mfgb_batch.cu).  Internal to the library.
#pragma once
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "mfgb_common.cuh"
#include "mfgb_internal.h"

namespace mfgb {
namespace {

constexpr int T256 = 256;

inline unsigned grid1d(int64_t n) {
  const int64_t g = (n + T256 - 1) / T256;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(g, 152 * 32));
}

#define GRID_STRIDE(t, n)                                                             \
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < (n); \
       t += (int64_t)gridDim.x * blockDim.x)

// Start vector of the lambda_max power iterations, entry i of a level:
// 0.5 + U[0, 1) from SplitMix64 (Steele, Lea, Flood 2014) of i, so that the
// batched set-up can generate every problem's start on the GPU in parallel.
__device__ __forceinline__ double power_start_value(uint64_t i) {
  uint64_t z = (i + 1) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return 0.5 + (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

__global__ void k_power_start(int64_t n, double *v) {
  GRID_STRIDE(t, n) v[t] = power_start_value((uint64_t)t);
}

template <class T>
__global__ void k_fill(int64_t n, T *x, T v) {
  GRID_STRIDE(t, n) x[t] = v;
}

template <class T>
__global__ void k_copy_constrained(int64_t nc, const int64_t *__restrict__ c,
                                   const T *__restrict__ src, T *__restrict__ dst) {
  GRID_STRIDE(t, nc) dst[c[t]] = src[c[t]];
}

template <class T>
__global__ void k_set_constrained(int64_t nc, const int64_t *__restrict__ c, T *__restrict__ v,
                                  T val) {
  GRID_STRIDE(t, nc) v[c[t]] = val;
}

template <class TO, class TI>
__global__ void k_convert(int64_t n, const TI *__restrict__ a, TO *__restrict__ b) {
  GRID_STRIDE(t, n) b[t] = (TO)a[t];
}

// Smoothing works on an operator result t that every consumer zeroes again after reading it, so
// that the next application can accumulate into it: no clearing pass and launch of its own.  The
// identity rows of the constrained DoFs are taken from the operator's input instead of being copied
// into its result: `bits` has one bit per DoF, set where it is constrained.
__device__ __forceinline__ bool bit_at(const uint32_t *__restrict__ bits, int64_t t) {
  return (__ldg(bits + (t >> 5)) >> (t & 31)) & 1u;
}

// 16-byte packs: the level vectors are whole allocations, so every pack of W values is aligned and
// lies in one word of bits; the last n % W values go one at a time
template <class T> struct alignas(16) Pack {
  static constexpr int W = 16 / sizeof(T);
  T v[W];
};
template <class T> __device__ __forceinline__ Pack<T> pack_at(const T *p, int64_t t) {
  return *reinterpret_cast<const Pack<T> *>(p + t);
}
template <class T> __device__ __forceinline__ void put_pack(T *p, int64_t t, const Pack<T> &v) {
  *reinterpret_cast<Pack<T> *>(p + t) = v;
}

// The smoother's vector passes are bound by their bytes, so they move no value twice: after the first
// step from x0 = 0, d is x and r is b (none is written), and the last step writes neither (8.5e6 DoFs
// of degree 4 to 1e-10: 28.8 -> 28.4 ms).
// A finite value on a constrained row that stays finite in the smoother's recurrence (coefficients of
// a few units a step); past it, and for infinities and NaN, Q1 levels select those values away (q1_row)
__device__ __forceinline__ bool q1_large(float v) { return !(fabsf(v) <= 1e30f); }

// Chebyshev first step from x0 = 0: x = d = (1/theta) Dinv b ; r = b ; t = 0 (d, r: null where x and b
// are read in their place); *large (where given) is set if b is q1_large on a constrained row
template <class T>
__global__ void k_cheb_first_zero(int64_t n, const T *__restrict__ b, const T *__restrict__ dinv,
                                  T *__restrict__ x, T *__restrict__ d, T *__restrict__ r,
                                  T *__restrict__ tz, T inv_theta,
                                  const uint32_t *__restrict__ bits = nullptr, int *large = nullptr) {
  constexpr int W = Pack<T>::W;
  GRID_STRIDE(q, n / W) {
    const int64_t t = q * W;
    const Pack<T> pb = pack_at(b, t), pd = pack_at(dinv, t);
    Pack<T> o, z;
    if (large) {
#pragma unroll
      for (int k = 0; k < W; ++k)
        if (q1_large((float)pb.v[k]) && bit_at(bits, t + k)) *large = 1;
    }
#pragma unroll
    for (int k = 0; k < W; ++k) o.v[k] = inv_theta * pd.v[k] * pb.v[k], z.v[k] = T(0);
    if (r) put_pack(r, t, pb);
    if (d) put_pack(d, t, o);
    put_pack(x, t, o);
    put_pack(tz, t, z);
  }
  GRID_STRIDE(q, n % W) {
    const int64_t t = n / W * W + q;
    const T v = inv_theta * dinv[t] * b[t];
    if (large && q1_large((float)b[t]) && bit_at(bits, t)) *large = 1;
    if (r) r[t] = b[t];
    if (d) d[t] = v;
    x[t] = v;
    tz[t] = T(0);
  }
}

// Chebyshev first step from x0: r = b - A x (A x in ax, zeroed); d = (1/theta) Dinv r; x += d
template <class T>
__global__ void k_cheb_first(int64_t n, const T *__restrict__ b, T *__restrict__ ax,
                             const T *__restrict__ dinv, T *__restrict__ x, T *__restrict__ d,
                             T *__restrict__ r, const uint32_t *__restrict__ bits, T inv_theta) {
  constexpr int W = Pack<T>::W;
  GRID_STRIDE(q, n / W) {
    const int64_t t = q * W;
    const Pack<T> pb = pack_at(b, t), pa = pack_at(ax, t), pd = pack_at(dinv, t);
    Pack<T> px = pack_at(x, t), od, orr, z;
    const uint32_t m = __ldg(bits + (t >> 5)) >> (t & 31);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      orr.v[k] = pb.v[k] - ((m >> k) & 1u ? px.v[k] : pa.v[k]);
      od.v[k] = inv_theta * pd.v[k] * orr.v[k];
      px.v[k] += od.v[k];
      z.v[k] = T(0);
    }
    put_pack(r, t, orr);
    put_pack(d, t, od);
    put_pack(x, t, px);
    put_pack(ax, t, z);
  }
  GRID_STRIDE(q, n % W) {
    const int64_t t = n / W * W + q;
    const T rt = b[t] - (bit_at(bits, t) ? x[t] : ax[t]);
    const T dt = inv_theta * dinv[t] * rt;
    r[t] = rt;
    d[t] = dt;
    x[t] += dt;
    ax[t] = T(0);
  }
}

// r = r0 - A d0 (A d0 in ad, zeroed); d = c1 d0 + c2 Dinv r; x += d (d0 may be x; d, r: null in the
// last step)
template <class T>
__global__ void k_cheb_step(int64_t n, T *__restrict__ ad, const T *__restrict__ dinv, T *x,
                            const T *d0, T *d, const T *r0, T *r, const uint32_t *__restrict__ bits,
                            T c1, T c2) {
  constexpr int W = Pack<T>::W;
  GRID_STRIDE(q, n / W) {
    const int64_t t = q * W;
    const Pack<T> pa = pack_at(ad, t), pi = pack_at(dinv, t);
    Pack<T> px = pack_at(x, t), pd = pack_at(d0, t), pr = pack_at(r0, t), z;
    const uint32_t m = __ldg(bits + (t >> 5)) >> (t & 31);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      pr.v[k] -= (m >> k) & 1u ? pd.v[k] : pa.v[k];
      pd.v[k] = c1 * pd.v[k] + c2 * pi.v[k] * pr.v[k];
      px.v[k] += pd.v[k];
      z.v[k] = T(0);
    }
    if (r) put_pack(r, t, pr);
    if (d) put_pack(d, t, pd);
    put_pack(x, t, px);
    put_pack(ad, t, z);
  }
  GRID_STRIDE(q, n % W) {
    const int64_t t = n / W * W + q;
    const T dv = d0[t], rt = r0[t] - (bit_at(bits, t) ? dv : ad[t]);
    const T dt = c1 * dv + c2 * dinv[t] * rt;
    if (r) r[t] = rt;
    if (d) d[t] = dt;
    x[t] += dt;
    ad[t] = T(0);
  }
}

// r = b - A x (A x in ax, zeroed)
template <class T>
__global__ void k_level_residual(int64_t n, const T *__restrict__ b, T *__restrict__ ax,
                                 const T *__restrict__ x, const uint32_t *__restrict__ bits,
                                 T *__restrict__ r) {
  constexpr int W = Pack<T>::W;
  GRID_STRIDE(q, n / W) {
    const int64_t t = q * W;
    const Pack<T> pb = pack_at(b, t), pa = pack_at(ax, t);
    Pack<T> o, z;
    const uint32_t m = __ldg(bits + (t >> 5)) >> (t & 31);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      o.v[k] = pb.v[k] - ((m >> k) & 1u ? x[t + k] : pa.v[k]);
      z.v[k] = T(0);
    }
    put_pack(r, t, o);
    put_pack(ax, t, z);
  }
  GRID_STRIDE(q, n % W) {
    const int64_t t = n / W * W + q;
    r[t] = b[t] - (bit_at(bits, t) ? x[t] : ax[t]);
    ax[t] = T(0);
  }
}

// x += t ; t = 0
template <class T>
__global__ void k_add_clear(int64_t n, T *__restrict__ tv, T *__restrict__ x) {
  constexpr int W = Pack<T>::W;
  GRID_STRIDE(q, n / W) {
    const int64_t t = q * W;
    Pack<T> px = pack_at(x, t), z;
    const Pack<T> pt = pack_at(tv, t);
#pragma unroll
    for (int k = 0; k < W; ++k) px.v[k] += pt.v[k], z.v[k] = T(0);
    put_pack(x, t, px);
    put_pack(tv, t, z);
  }
  GRID_STRIDE(q, n % W) {
    const int64_t t = n / W * W + q;
    x[t] += tv[t];
    tv[t] = T(0);
  }
}

// r = b - ax
template <class T>
__global__ void k_residual(int64_t n, const T *__restrict__ b, const T *__restrict__ ax,
                           T *__restrict__ r) {
  GRID_STRIDE(t, n) r[t] = b[t] - ax[t];
}

template <class T>
__global__ void k_scale_by(int64_t n, const T *__restrict__ s, T *__restrict__ v) {
  GRID_STRIDE(t, n) v[t] *= s[t];
}

// ---- Q1 levels as assembled stencils (FP32 V-cycle) ------------------------
// A Q1 level's operator has 27 entries a row.  Assembled (in FP64 from the FP64 geometric factors,
// rounded once), its application is a gather that can be fused with the smoother's vector update: one
// launch a step instead of two, no atomics, 108 bytes a row instead of 192 of geometric factors a
// cell.  The input must not be overwritten while neighbours read it, so d alternates between two
// arrays and a smoother that starts from x leaves x in a third until its last step.
// Bound by launches and latency: per multigrid iteration at 8.5e6 DoFs and degree 4 (three such levels)
// 2.86 -> 2.67 ms, 24 mixed problems solved together 46.5 -> 44.6 ms.
// S[s][row], s = (dk+1)*9 + (dj+1)*3 + (di+1); rows of constrained nodes are not read.  A constrained
// neighbour's coefficient is -0 (no other one is).

// One row per thread: the rows of the up to 8 cells around node (i, j, k) that belong to it.
__global__ void __launch_bounds__(T256)
    k_q1_assemble(int nx, int ny, int nz, const double *__restrict__ G, double d0, double d1,
                  float *__restrict__ S, int64_t stride) {
  const int fx = nx + 1, fy = ny + 1, fz = nz + 1;
  const double D[2][2] = {{d0, d1}, {d0, d1}};  // both GLL points of a linear function
  GRID_STRIDE(row, (int64_t)fx * fy * fz) {
    const int i = (int)(row % fx), j = (int)(row / fx % fy), k = (int)(row / ((int64_t)fx * fy));
    double acc[27];
    for (int s = 0; s < 27; ++s) acc[s] = 0.0;
    for (int c = 0; c < 8; ++c) {  // the cell at (i, j, k) - (c bits); node is its corner a = c bits
      const int ai = c & 1, aj = (c >> 1) & 1, ak = c >> 2;
      const int ci = i - ai, cj = j - aj, ck = k - ak;
      if (ci < 0 || cj < 0 || ck < 0 || ci >= nx || cj >= ny || ck >= nz) continue;
      const double *g = G + (ci + (int64_t)nx * (cj + (int64_t)ny * ck)) * 48;  // [6][8], k slowest
      for (int q = 0; q < 8; ++q) {
        const int qi = q & 1, qj = (q >> 1) & 1, qk = q >> 2;
        // derivatives of the corner's basis function at the point along r (k), s (j), t (i)
        const double br = qj == aj && qi == ai ? D[qk][ak] : 0.0;
        const double bs = qk == ak && qi == ai ? D[qj][aj] : 0.0;
        const double bt = qk == ak && qj == aj ? D[qi][ai] : 0.0;
        if (br == 0.0 && bs == 0.0 && bt == 0.0) continue;
        const double vr = g[q] * br + g[8 + q] * bs + g[16 + q] * bt;
        const double vs = g[8 + q] * br + g[24 + q] * bs + g[32 + q] * bt;
        const double vt = g[16 + q] * br + g[32 + q] * bs + g[40 + q] * bt;
        for (int b = 0; b < 2; ++b) {  // its flux against the functions that vary there
          acc[(b - ak + 1) * 9 + (qj - aj + 1) * 3 + (qi - ai + 1)] += D[qk][b] * vr;
          acc[(qk - ak + 1) * 9 + (b - aj + 1) * 3 + (qi - ai + 1)] += D[qj][b] * vs;
          acc[(qk - ak + 1) * 9 + (qj - aj + 1) * 3 + (b - ai + 1)] += D[qi][b] * vt;
        }
      }
    }
    for (int s = 0; s < 27; ++s) {
      const int ni = i + s % 3 - 1, nj = j + s / 3 % 3 - 1, nk = k + s / 9 - 1;
      const bool in = ni > 0 && nj > 0 && nk > 0 && ni < fx - 1 && nj < fy - 1 && nk < fz - 1;
      S[s * stride + row] = in ? __fadd_rn((float)acc[s], 0.f) : -0.f;  // (-0 + 0 = 0)
    }
  }
}

// (A v)[t] for an unconstrained row t; S at the part's first row, v at its first value.  -0 times a
// finite value on a constrained row adds nothing, but an infinity or NaN there must stay there as in the
// operators' masked gather: MASK selects it away.  Only the finest level can have such values (the
// restriction writes 0 on those rows), and selecting in every pass cost p = 1 at 8e6 DoFs 41.4 -> 46.4
// ms a solve, so the first smoothing pass looks at them and the others run one of two loops (37.5 ms).
template <bool MASK>
__device__ __forceinline__ float q1_row(const float *__restrict__ S, int64_t stride, int fx, int fxy,
                                        int64_t t, const float *__restrict__ v) {
  const float *c = S + t, *p = v + t;
  float plane[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    plane[k] = 0.f;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float a = __ldg(c + (k * 9 + j * 3 + i) * stride);
        const float x = p[(k - 1) * fxy + (j - 1) * fx + i - 1];
        plane[k] += a * (MASK && __float_as_uint(a) == 0x80000000u ? 0.f : x);
      }
  }
  return plane[0] + plane[1] + plane[2];
}

// What a Q1 pass does with (A v)[t]: the values of one row
struct Q1Row {
  const float *b, *dinv;
  float *r;
};

// r = b - A x
template <bool MASK>
__device__ __forceinline__ void q1_residual(const float *S, int64_t stride, int fx, int fxy, bool fixed,
                                            int64_t t, const float *x, const Q1Row &q) {
  q.r[t] = q.b[t] - (fixed ? x[t] : q1_row<MASK>(S, stride, fx, fxy, t, x));
}
// r = b - A x; d = c2 Dinv r; y = x + d
template <bool MASK>
__device__ __forceinline__ void q1_first(const float *S, int64_t stride, int fx, int fxy, bool fixed,
                                         int64_t t, const float *x, const Q1Row &q, float *d, float *y,
                                         float c2) {
  const float xt = x[t], rt = q.b[t] - (fixed ? xt : q1_row<MASK>(S, stride, fx, fxy, t, x));
  const float dt = c2 * q.dinv[t] * rt;
  q.r[t] = rt;
  d[t] = dt;
  y[t] = xt + dt;
}
// r -= A d; dn = c1 d + c2 Dinv r; y = x + dn
template <bool MASK>
__device__ __forceinline__ void q1_step(const float *S, int64_t stride, int fx, int fxy, bool fixed,
                                        int64_t t, const float *d, const Q1Row &q, float *dn,
                                        const float *x, float *y, float c1, float c2) {
  const float dv = d[t], rt = q.r[t] - (fixed ? dv : q1_row<MASK>(S, stride, fx, fxy, t, d));
  const float dt = c1 * dv + c2 * q.dinv[t] * rt;
  q.r[t] = rt;
  dn[t] = dt;
  y[t] = x[t] + dt;
}

// f(mask) with mask = true_type where *large is set (nullptr: never)
template <class F>
__device__ __forceinline__ void q1_masked(const int *large, F f) {
  if (large != nullptr && *large)
    f(std::true_type());
  else
    f(std::false_type());
}

__global__ void __launch_bounds__(T256)
    k_q1_residual(int64_t n, const float *__restrict__ S, int fx, int fxy,
                  const uint32_t *__restrict__ bits, const float *__restrict__ x, Q1Row q,
                  const int *large) {
  q1_masked(large, [&](auto m) {
    GRID_STRIDE(t, n) q1_residual<decltype(m)::value>(S, n, fx, fxy, bit_at(bits, t), t, x, q);
  });
}
__global__ void __launch_bounds__(T256)
    k_q1_first(int64_t n, const float *__restrict__ S, int fx, int fxy,
               const uint32_t *__restrict__ bits, const float *__restrict__ x, Q1Row q,
               float *__restrict__ d, float *__restrict__ y, float c2, const int *large) {
  q1_masked(large, [&](auto m) {
    GRID_STRIDE(t, n) q1_first<decltype(m)::value>(S, n, fx, fxy, bit_at(bits, t), t, x, q, d, y, c2);
  });
}
__global__ void __launch_bounds__(T256)
    k_q1_step(int64_t n, const float *__restrict__ S, int fx, int fxy,
              const uint32_t *__restrict__ bits, const float *__restrict__ d, Q1Row q,
              float *__restrict__ dn, const float *x, float *y, float c1, float c2, const int *large) {
  q1_masked(large, [&](auto m) {
    GRID_STRIDE(t, n)
      q1_step<decltype(m)::value>(S, n, fx, fxy, bit_at(bits, t), t, d, q, dn, x, y, c1, c2);
  });
}

// ---- p-transfer: fine degree pf, coarse degree pc, same cells ------------
struct PTransferParams {
  float B32[81];
  double B64[81];  // B[a*(pc+1) + b] = l^c_b(x^f_a)
  int nf, nc;      // points per direction (fine, coarse)
};

template <class T>
__device__ __forceinline__ T bval(const PTransferParams &P, int idx);
template <>
__device__ __forceinline__ float bval<float>(const PTransferParams &P, int idx) {
  return P.B32[idx];
}
template <>
__device__ __forceinline__ double bval<double>(const PTransferParams &P, int idx) {
  return P.B64[idx];
}

// Sum-factorised p-transfers: one CTA per cell, three 1D passes through
// shared memory (nc^3 -> nc*nc*nf -> nc*nf*nf -> nf^3 and back).
template <class T>
__global__ void __launch_bounds__(128)
    k_p_prolongate_sf(int64_t n_cells, const uint32_t *__restrict__ map_f,
                      const uint32_t *__restrict__ map_c, const T *__restrict__ xc,
                      T *__restrict__ tf, PTransferParams P) {
  __shared__ T s0[729], s1[729];
  const int nf = P.nf, nc = P.nc, nf3 = nf * nf * nf, nc3 = nc * nc * nc;
  for (int64_t e = blockIdx.x; e < n_cells; e += gridDim.x) {
    for (int t = threadIdx.x; t < nc3; t += blockDim.x) {
      const uint32_t dc = map_c[e * nc3 + t];
      s0[t] = dc != MFGB_INVALID_DOF ? xc[dc] : T(0);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nc * nc * nf; t += blockDim.x) {  // along k: [a][b][kf]
      const int a = t / (nc * nf), b = (t / nf) % nc, kf = t % nf;
      T s = 0;
      for (int c = 0; c < nc; ++c) s += bval<T>(P, kf * nc + c) * s0[(a * nc + b) * nc + c];
      s1[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nc * nf * nf; t += blockDim.x) {  // along j: [a][jf][kf]
      const int a = t / (nf * nf), jf = (t / nf) % nf, kf = t % nf;
      T s = 0;
      for (int b = 0; b < nc; ++b) s += bval<T>(P, jf * nc + b) * s1[(a * nc + b) * nf + kf];
      s0[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nf3; t += blockDim.x) {  // along i: [if][jf][kf]
      const int i = t / (nf * nf), jk = t % (nf * nf);
      const uint32_t df = map_f[e * nf3 + t];
      if (df == MFGB_INVALID_DOF) continue;
      T s = 0;
      for (int a = 0; a < nc; ++a) s += bval<T>(P, i * nc + a) * s0[a * nf * nf + jk];
      tf[df] = s;
    }
    __syncthreads();
  }
}

template <class T>
__global__ void __launch_bounds__(128)
    k_p_restrict_sf(int64_t n_cells, const uint32_t *__restrict__ map_f,
                    const uint32_t *__restrict__ map_c, const T *__restrict__ rf,
                    const T *__restrict__ inv_val_f, T *__restrict__ rc, PTransferParams P) {
  __shared__ T s0[729], s1[729];
  const int nf = P.nf, nc = P.nc, nf3 = nf * nf * nf, nc3 = nc * nc * nc;
  for (int64_t e = blockIdx.x; e < n_cells; e += gridDim.x) {
    for (int t = threadIdx.x; t < nf3; t += blockDim.x) {
      const uint32_t df = map_f[e * nf3 + t];
      s0[t] = df != MFGB_INVALID_DOF ? rf[df] * inv_val_f[df] : T(0);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nc * nf * nf; t += blockDim.x) {  // along i: [a][jf][kf]
      const int a = t / (nf * nf), jk = t % (nf * nf);
      T s = 0;
      for (int i = 0; i < nf; ++i) s += bval<T>(P, i * nc + a) * s0[i * nf * nf + jk];
      s1[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nc * nc * nf; t += blockDim.x) {  // along j: [a][b][kf]
      const int a = t / (nc * nf), b = (t / nf) % nc, kf = t % nf;
      T s = 0;
      for (int j = 0; j < nf; ++j) s += bval<T>(P, j * nc + b) * s1[(a * nf + j) * nf + kf];
      s0[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nc3; t += blockDim.x) {  // along k: [a][b][c]
      const int a = t / (nc * nc), b = (t / nc) % nc, c = t % nc;
      const uint32_t dc = map_c[e * nc3 + t];
      if (dc == MFGB_INVALID_DOF) continue;
      T s = 0;
      for (int k = 0; k < nf; ++k) s += bval<T>(P, k * nc + c) * s0[(a * nc + b) * nf + k];
      atomicAdd(rc + dc, s);
    }
    __syncthreads();
  }
}

// Column-layout p-transfers: a CTA holds E cells and thread (e, j, k) owns the
// fine column i = 0..NF-1 of cell e in registers.  Prolongation reads the
// cell's NC^3 coarse values from shared memory and writes its fine column
// (plain writes: shared fine DoFs get the same value from every cell);
// restriction forms s[a] = sum_i B[i][a] r_i in registers, then one thread per
// coarse DoF sums B[j][b] B[k][c] s[a][j][k] over the cell and adds atomically.
template <int NF> struct PtCells {
  static constexpr int value = NF <= 3 ? 16 : NF <= 5 ? 8 : NF <= 7 ? 4 : 2;
};

template <class T, int NF, int NC>
__global__ void __launch_bounds__(NF * NF * PtCells<NF>::value)
    k_p_prolongate_col(int64_t n_cells, const uint32_t *__restrict__ map_f,
                       const uint32_t *__restrict__ map_c, const T *__restrict__ xc,
                       T *__restrict__ tf, PTransferParams P) {
  constexpr int E = PtCells<NF>::value, NF2 = NF * NF, NF3 = NF2 * NF, NC3 = NC * NC * NC;
  __shared__ T sB[NF * NC];
  __shared__ T sc[E * NC3];
  const int tid = threadIdx.x, el = tid / NF2, jk = tid - el * NF2, j = jk / NF, k = jk - j * NF;
  for (int t = tid; t < NF * NC; t += blockDim.x) sB[t] = bval<T>(P, t);
  const int64_t n_batches = (n_cells + E - 1) / E;
  for (int64_t batch = blockIdx.x; batch < n_batches; batch += gridDim.x) {
    for (int t = tid; t < E * NC3; t += blockDim.x) {
      const int64_t c = batch * E + t / NC3;
      const uint32_t d = c < n_cells ? map_c[c * NC3 + t % NC3] : MFGB_INVALID_DOF;
      sc[t] = d != MFGB_INVALID_DOF ? xc[d] : T(0);
    }
    __syncthreads();
    const int64_t cell = batch * E + el;
    if (cell < n_cells) {
      const T *x = sc + el * NC3;
      T t2[NC];
#pragma unroll
      for (int a = 0; a < NC; ++a) {
        T acc = 0;
#pragma unroll
        for (int b = 0; b < NC; ++b) {
          T in = 0;
#pragma unroll
          for (int c = 0; c < NC; ++c) in += sB[k * NC + c] * x[(a * NC + b) * NC + c];
          acc += sB[j * NC + b] * in;
        }
        t2[a] = acc;
      }
#pragma unroll
      for (int i = 0; i < NF; ++i) {
        const uint32_t d = map_f[cell * NF3 + i * NF2 + jk];
        if (d == MFGB_INVALID_DOF) continue;
        T v = 0;
#pragma unroll
        for (int a = 0; a < NC; ++a) v += sB[i * NC + a] * t2[a];
        tf[d] = v;
      }
    }
    __syncthreads();
  }
}

template <class T, int NF, int NC>
__global__ void __launch_bounds__(NF * NF * PtCells<NF>::value)
    k_p_restrict_col(int64_t n_cells, const uint32_t *__restrict__ map_f,
                     const uint32_t *__restrict__ map_c, const T *__restrict__ rf,
                     const T *__restrict__ inv_val_f, T *__restrict__ rc, PTransferParams P) {
  constexpr int E = PtCells<NF>::value, NF2 = NF * NF, NF3 = NF2 * NF, NC3 = NC * NC * NC;
  __shared__ T sB[NF * NC];
  __shared__ T ss[E * NC * NF2];
  const int tid = threadIdx.x, el = tid / NF2, jk = tid - el * NF2;
  for (int t = tid; t < NF * NC; t += blockDim.x) sB[t] = bval<T>(P, t);
  const int64_t n_batches = (n_cells + E - 1) / E;
  for (int64_t batch = blockIdx.x; batch < n_batches; batch += gridDim.x) {
    __syncthreads();  // sB ready / previous batch's ss consumed
    const int64_t cell = batch * E + el;
    T r[NF];
#pragma unroll
    for (int i = 0; i < NF; ++i) {
      const uint32_t d = cell < n_cells ? map_f[cell * NF3 + i * NF2 + jk] : MFGB_INVALID_DOF;
      r[i] = d != MFGB_INVALID_DOF ? rf[d] * inv_val_f[d] : T(0);
    }
#pragma unroll
    for (int a = 0; a < NC; ++a) {
      T acc = 0;
#pragma unroll
      for (int i = 0; i < NF; ++i) acc += sB[i * NC + a] * r[i];
      ss[(el * NC + a) * NF2 + jk] = acc;
    }
    __syncthreads();
    for (int t = tid; t < E * NC3; t += blockDim.x) {
      const int e2 = t / NC3, l = t - e2 * NC3;
      const int64_t c2 = batch * E + e2;
      if (c2 >= n_cells) continue;
      const uint32_t d = map_c[c2 * NC3 + l];
      if (d == MFGB_INVALID_DOF) continue;
      const int a = l / (NC * NC), b = (l / NC) % NC, c = l % NC;
      const T *sa = ss + (e2 * NC + a) * NF2;
      T acc = 0;
#pragma unroll
      for (int jj = 0; jj < NF; ++jj) {
        T in = 0;
#pragma unroll
        for (int kk = 0; kk < NF; ++kk) in += sB[kk * NC + c] * sa[jj * NF + kk];
        acc += sB[jj * NC + b] * in;
      }
      atomicAdd(rc + d, acc);
    }
  }
}

// launch helpers: the (NF, NC) pairs of the halving rule p -> max(1, p/2)
template <class T, int NF, int NC>
void p_transfer_col(bool restrict_, int64_t n_cells, const uint32_t *map_f, const uint32_t *map_c,
                    const T *x, const T *inv_val, T *y, const PTransferParams &P, cudaStream_t s) {
  constexpr int E = PtCells<NF>::value;
  const int64_t n_batches = (n_cells + E - 1) / E;
  const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(n_batches, 152 * 8));
  if (restrict_)
    k_p_restrict_col<T, NF, NC><<<grid, E * NF * NF, 0, s>>>(n_cells, map_f, map_c, x, inv_val, y, P);
  else
    k_p_prolongate_col<T, NF, NC><<<grid, E * NF * NF, 0, s>>>(n_cells, map_f, map_c, x, y, P);
}

// y = P x (prolongation into a zeroed y) or y += R x (restriction), any (nf, nc)
template <class T>
void p_transfer(bool restrict_, int64_t n_cells, const uint32_t *map_f, const uint32_t *map_c,
                const T *x, const T *inv_val, T *y, const PTransferParams &P, cudaStream_t s) {
  if (n_cells <= 0) return;
  const int key = P.nf * 16 + P.nc;
  switch (key) {
#define MFGB_PT(NF, NC)                                                              \
  case NF * 16 + NC:                                                                 \
    p_transfer_col<T, NF, NC>(restrict_, n_cells, map_f, map_c, x, inv_val, y, P, s); \
    return;
    MFGB_PT(3, 2) MFGB_PT(4, 2) MFGB_PT(5, 3) MFGB_PT(6, 3) MFGB_PT(7, 4) MFGB_PT(8, 4)
    MFGB_PT(9, 5)
#undef MFGB_PT
    default: break;
  }
  const unsigned grid = (unsigned)std::min<int64_t>(n_cells, 152 * 16);
  if (restrict_)
    k_p_restrict_sf<T><<<grid, 128, 0, s>>>(n_cells, map_f, map_c, x, inv_val, y, P);
  else
    k_p_prolongate_sf<T><<<grid, 128, 0, s>>>(n_cells, map_f, map_c, x, y, P);
}

// ---- h-transfer between nested structured Q1 grids -----------------------
// Level nodes of an axis sit at fine mesh nodes min(k s, nf) (BoxStride); the
// coarse level (stride 2s) keeps every other node and the last one.  x fastest.
struct HGrid {
  int fx, fy, fz, cx, cy, cz;      // node counts
  int nf[3];                       // cells of the uniform mesh the strides refer to
  int s;                           // stride of the fine level
};

// Weight of the right-hand coarse neighbour (I+1)/2 of an odd fine node I (its left-hand one has the
// rest): the fraction of their distance the node's position gives, 1/2 unless the last coarse cell is
// narrower.  An even node is coarse node I/2.
__host__ __device__ __forceinline__ double h_right(int I, int nf, int s) {
  const int A = (I - 1) * s, P = min(I * s, nf), B = min((I + 1) * s, nf);
  return B - A == 2 * s ? 0.5 : (double)(P - A) / (double)(B - A);
}

// a * b of pairs, the sum of h and l rounded once and not contracted
__host__ __device__ __forceinline__ float h_sum(float h, float l) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(h, l);
#else
  const volatile float s = h + l;
  return s;
#endif
}
__host__ __device__ __forceinline__ df h_mul(df a, df b) {
  const float h = a.hi * b.hi;
  const float l = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, fmaf(a.hi, b.hi, -h))), s = h_sum(h, l);
  return df{s, h_sum(l, -h_sum(s, -h))};
}

// Both transfers go one axis at a time with the axis weights found once per node, and 32-bit indices
// (Q1 levels are below 2^31 nodes): with three FP64 weights, a division among them, for each of the
// 27 neighbours and 64-bit index divisions, a restriction of 8e4 nodes took 70 us.  In FP32 that loses
// nothing where at most one weight is not a half or 1 (error against 64 bits 0.97 of the form with
// products of weights), nor in the restriction (0.71, and 0.76 at other nodes: 27 terms in a row are
// rounded more often); a prolongation between two or three narrower cells had 1.44 of it, so those few
// nodes take the products, rounded once, from pairs.

// x_f[t] += (P x_c)[t] for fine node t (interior nodes only)
template <class T>
__host__ __device__ __forceinline__ void h_prolongate_node(const HGrid &g, int64_t node,
                                                           const T *__restrict__ xc,
                                                           T *__restrict__ xf) {
  const unsigned t = (unsigned)node, row = t / (unsigned)g.fx;
  const int I = (int)(t - row * g.fx), K = (int)(row / (unsigned)g.fy), J = (int)(row - (unsigned)K * g.fy);
  if (I == 0 || J == 0 || K == 0 || I == g.fx - 1 || J == g.fy - 1 || K == g.fz - 1) return;
  T w[3][2] = {{T(1), T(0)}, {T(1), T(0)}, {T(1), T(0)}};
  const int at[3] = {I, J, K};
  int uneven = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    if (at[a] & 1) {
      const double r = h_right(at[a], g.nf[a], g.s);
      w[a][0] = (T)(1.0 - r);
      w[a][1] = (T)r;
      uneven += w[a][1] != T(0.5);
    }
  const T *x0 = xc + I / 2 + (int64_t)g.cx * (J / 2 + (int64_t)g.cy * (K / 2));
  T acc = 0;
  if (sizeof(T) == 4 && uneven > 1) {
    df p[3][2];  // the axis weights as pairs
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      p[a][0] = p[a][1] = df{1.f, 0.f};
      if (at[a] & 1) {
        const int A = (at[a] - 1) * g.s, P = min(at[a] * g.s, g.nf[a]), B = min((at[a] + 1) * g.s, g.nf[a]);
        const float den = (float)(B - A), inv = 1.f / den, l = (float)w[a][0], r = (float)w[a][1];
        p[a][0] = df{l, fmaf(-l, den, (float)(B - P)) * inv};
        p[a][1] = df{r, fmaf(-r, den, (float)(P - A)) * inv};
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (k > (K & 1) || j > (J & 1)) continue;
        const T *x = x0 + (int64_t)g.cx * (j + (int64_t)g.cy * k);
        const df q = h_mul(p[2][k], p[1][j]);
        acc += (T)h_mul(q, p[0][0]).hi * x[0];
        if (I & 1) acc += (T)h_mul(q, p[0][1]).hi * x[1];
      }
    xf[node] += acc;
    return;
  }
  for (int k = 0; k <= (K & 1); ++k) {
    T plane = 0;
    for (int j = 0; j <= (J & 1); ++j) {
      const T *x = x0 + (int64_t)g.cx * (j + (int64_t)g.cy * k);
      T line = w[0][0] * x[0];
      if (I & 1) line += w[0][1] * x[1];
      plane += w[1][j] * line;
    }
    acc += w[2][k] * plane;
  }
  xf[node] += acc;
}

// r_c[t] = (P^T r_f)[t] for coarse node t (boundary nodes -> 0)
template <class T>
__device__ __forceinline__ void h_restrict_node(const HGrid &g, int64_t node,
                                                const T *__restrict__ rf, T *__restrict__ rc) {
  const unsigned t = (unsigned)node, row = t / (unsigned)g.cx;
  const int i = (int)(t - row * g.cx), k = (int)(row / (unsigned)g.cy), j = (int)(row - (unsigned)k * g.cy);
  if (i == 0 || j == 0 || k == 0 || i == g.cx - 1 || j == g.cy - 1 || k == g.cz - 1) {
    rc[node] = 0;
    return;
  }
  // fine neighbours 2i-1 .. 2i+1 exist for every interior coarse node
  T w[3][2];
  const int at[3] = {i, j, k};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    w[a][0] = (T)h_right(2 * at[a] - 1, g.nf[a], g.s);
    w[a][1] = (T)(1.0 - h_right(2 * at[a] + 1, g.nf[a], g.s));
  }
  const T *r0 = rf + 2 * i + (int64_t)g.fx * (2 * j + (int64_t)g.fy * (2 * k));
  T acc = 0;
#pragma unroll
  for (int K = -1; K <= 1; ++K) {
    T plane = 0;
#pragma unroll
    for (int J = -1; J <= 1; ++J) {
      const T *r = r0 + (int64_t)g.fx * (J + (int64_t)g.fy * K);
      const T line = w[0][0] * r[-1] + r[0] + w[0][1] * r[1];
      plane += J < 0 ? w[1][0] * line : J > 0 ? w[1][1] * line : line;
    }
    acc += K < 0 ? w[2][0] * plane : K > 0 ? w[2][1] * plane : plane;
  }
  rc[node] = acc;
}

template <class T>
__global__ void k_h_prolongate_add(HGrid g, const T *__restrict__ xc, T *__restrict__ xf) {
  GRID_STRIDE(t, (int64_t)g.fx * g.fy * g.fz) h_prolongate_node(g, t, xc, xf);
}

template <class T>
__global__ void k_h_restrict(HGrid g, const T *__restrict__ rf, T *__restrict__ rc) {
  GRID_STRIDE(t, (int64_t)g.cx * g.cy * g.cz) h_restrict_node(g, t, rf, rc);
}

// ---- valence (number of cells sharing a DoF) ----------------------------
template <class T>
__global__ void k_count_valence(int64_t n, const uint32_t *__restrict__ map, T *__restrict__ val) {
  GRID_STRIDE(t, n) {
    const uint32_t d = map[t];
    if (d != MFGB_INVALID_DOF) atomicAdd(val + d, (T)1);
  }
}

template <class T>
__global__ void k_invert_pos(int64_t n, T *__restrict__ v) {
  GRID_STRIDE(t, n) v[t] = v[t] > 0 ? (T)1 / v[t] : (T)0;
}

// ---- host helpers ---------------------------------------------------------
HGrid hgrid(const mfgb_box_desc &fb, const BoxStride &fs, const mfgb_box_desc &cb) {
  return HGrid{fb.nx + 1, fb.ny + 1, fb.nz + 1, cb.nx + 1, cb.ny + 1, cb.nz + 1,
               {fs.nf[0], fs.nf[1], fs.nf[2]}, fs.s};
}

PTransferParams ptransfer(const mfgb_operator *fine, const mfgb_operator *coarse) {
  PTransferParams P{};
  P.nf = fine->n;
  P.nc = coarse->n;
  for (int a = 0; a < P.nf; ++a)
    for (int b = 0; b < P.nc; ++b) {
      const double v = lagrange_value(P.nc, coarse->gll_x, b, fine->gll_x[a]);
      P.B64[a * P.nc + b] = v;
      P.B32[a * P.nc + b] = (float)v;
    }
  return P;
}

}  // namespace
}  // namespace mfgb
