// Point formulas shared by the multigrid kernels (per-level grid kernels,
// single-block tail, cluster and cooperative forms).  Every form goes through
// the same functions, with the multiply-adds written out, so a level gives the
// same bits wherever it runs.
#pragma once

#include <cuda_fp16.h>

#include <cmath>

namespace pfgpu {

__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// r = b - A x of one point in ParFlow's Matvec order (alpha = -1, beta = 1):
// C W E S N L U
template <typename T>
__device__ __forceinline__ T residual_value(T b, T d, T x, T w, T xw, T e, T xe, T s, T xs, T n,
                                            T xn, T l, T xl, T u, T xu) {
  T y = fma(d, x, -b);
  y = fma(w, xw, y);
  y = fma(e, xe, y);
  y = fma(s, xs, y);
  y = fma(n, xn, y);
  y = fma(l, xl, y);
  y = fma(u, xu, y);
  return -y;
}

// coarse right-hand side of one coarse point: r_f(c) + (p2(f-1) r_f(f-1) +
// p1(f+1) r_f(f+1)) (mg_semi_restrict.c:161-169); H: the scaled form, whose
// weight w at the coarse point itself is s_c
template <typename T, bool H>
__device__ __forceinline__ T restrict_value(T w, T rc, T w2m, T rm, T w1p, T rp) {
  const T side = fma(w2m, rm, mul_rn(w1p, rp));
  if constexpr (H)
    return fma(w, rc, side);
  else
    return add_rn(rc, side);
}

// correction of one fine point from the coarse points below and above it
// (mg_semi_prolong.c:119-124, 191-197): the coarse value itself at a coarse
// point (times s_c when H), else p1 e(below) + p2 e(above)
template <typename T, bool H>
__device__ __forceinline__ T prolong_value(bool fine_point, T w1, T w2, T el, T eh) {
  const T coarse = H ? mul_rn(w1, el) : el;
  return fine_point ? fma(w1, el, mul_rn(w2, eh)) : coarse;
}

// ---- scaled FP16 operator -----------------------------------------------------
// 1/S for S = sqrt(|c|), 1 where c is 0 or not finite (hardware reciprocal
// square root: the scaled values are stored as 11-bit FP16 significands)
__device__ __forceinline__ float inv_scale_of(float c) {
  const float a = fabsf(c);
  return (a > 0.0f && isfinite(a)) ? rsqrtf(a) : 1.0f;
}
// S from c and 1/S without a division
__device__ __forceinline__ float scale_from(float c, float inv) {
  const float a = fabsf(c);
  return (a > 0.0f && isfinite(a)) ? a * inv : 1.0f;
}

// A divisor with its float reciprocal: t / d from one multiplication and a
// one-step correction (exact while the float product errs by less than one,
// i.e. for t < 2^22; larger t take the integer division).  The single-block
// tail splits a linear index per cell and phase, where integer division
// would dominate its instruction count.
struct FastDiv {
  int d;
  float inv;
};
__device__ __forceinline__ FastDiv fast_div(int d) { return FastDiv{d, 1.0f / (float)d}; }
__device__ __forceinline__ int quot(int t, FastDiv f) {
  if (t >= (1 << 22)) return t / f.d;
  int q = (int)((float)t * f.inv);
  if ((q + 1) * f.d <= t) q++;
  if (q * f.d > t) q--;
  return q;
}
__device__ __forceinline__ void split_ijk(int t, FastDiv fx, FastDiv fy, int &i, int &j,
                                          int &k) {
  const int r = quot(t, fx);
  i = t - r * fx.d;
  k = quot(r, fy);
  j = r - k * fy.d;
}

}  // namespace pfgpu
