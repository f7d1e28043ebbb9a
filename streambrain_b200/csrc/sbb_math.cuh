// Device arithmetic shared by every kernel that touches a trace or a weight, so
// that the general-shape kernels and the tensor-core kernels produce the same
// values from the same batch sums.
#pragma once
#include "sbb_kernels.cuh"

#include <math.h>

namespace sbb {

__device__ __forceinline__ float sbb_log(float x) { return logf(x); }
__device__ __forceinline__ double sbb_log(double x) { return log(x); }
__device__ __forceinline__ float sbb_exp(float x) { return expf(x); }
__device__ __forceinline__ double sbb_exp(double x) { return exp(x); }

// One moving-average step from a batch sum: sum/B, *taupdt, old*(1-taupdt), add,
// clamp at zero (a NaN clamps to zero, as std::max(0, NaN) does).
template <typename T>
__device__ __forceinline__ T trace_ema(T old, T sum, const TraceParams<T> &p) {
  T tmp = sum / p.batch;
  tmp = tmp * p.taupdt;
  T c = old * p.one_minus;
  c = c + tmp;
  return c > (T)0 ? c : (T)0;
}

template <typename T>
__device__ __forceinline__ T log_ratio(T cij, T ci, T cj, T cthr4) {
  const T num = cij < cthr4 ? cthr4 : cij;
  return sbb_log(num / (ci * cj));
}

// v / d for many v in [0, 1] and one d in [1, 2^20], correctly rounded, from the rounded reciprocal of d: Markstein's method
// (IBM J. Res. Dev. 34, 1990): with y = RN(1/d), q = RN(v y) and the remainder r = v - q d, RN(q + r y) is RN(v / d) unless
// d's significand is all ones; nothing underflows on the way for v >= MIN.  Three instructions for the division's dozen or
// more.
template <typename T>
struct DivideBy {
  static constexpr T MIN = sizeof(T) == 4 ? (T)0x1p-100 : (T)0x1p-900;
  T d, y;
  bool plain;   // the one significand the method does not cover
  __device__ __forceinline__ explicit DivideBy(T divisor) : d(divisor) {
    if constexpr (sizeof(T) == 4) {
      y = __frcp_rn(divisor);
      plain = (__float_as_uint(divisor) & 0x7FFFFFu) == 0x7FFFFFu;
    } else {
      y = __drcp_rn(divisor);
      plain = (__double_as_longlong(divisor) & 0xFFFFFFFFFFFFFll) == 0xFFFFFFFFFFFFFll;
    }
  }
  __device__ __forceinline__ bool covers(T v) const { return !(plain || (v < MIN && v > (T)0)); }
  __device__ __forceinline__ T quotient(T v) const {   // (a NaN divisor: the method's NaN is the division's)
    const T q = v * y;
    return fma(fma(-q, d, v), y, q);
  }
  __device__ __forceinline__ T operator()(T v) const { return covers(v) ? quotient(v) : v / d; }
};

// One unit's gain and bias from its new trace (kernels_openmp_internal.cc:221-246); k = (khalf - 1) pmin4^2.
template <typename T>
__device__ __forceinline__ void bias_regularized(T &bias, T &kbi, T pj, T cthr, T khalf, T pmin4, T k, T taubdt) {
  T kb = (T)1 + k / ((pj - pmin4) * (pj - pmin4));
  if (pj < pmin4 || kb < khalf) kb = khalf;
  const T g = ((T)1 - taubdt) * kbi + taubdt * kb;
  kbi = g;
  bias = pj < cthr ? g * sbb_log((T)2 * cthr) : g * sbb_log(pj);
}

// The arithmetic of the tensor-core path (fused epilogue, and the element-wise tail of the
// data-parallel step when that path is selected): the batch mean and the moving-average weight
// folded into one factor taupdt / batch, the ratio by IEEE reciprocals of Ci and Cj formed once per
// row / column, the logarithm by lg2.approx (relative error below 2^-22) -- about a quarter of the
// instructions of the IEEE forms above, and well inside the tolerance of the weights (which are a
// logarithm of a ratio of noisy traces).
__device__ __forceinline__ float trace_ema_fast(float old, float sum, float one_minus, float ema_scale) {
  return fmaxf(fmaf(old, one_minus, sum * ema_scale), 0.f);
}
__device__ __forceinline__ float log_ratio_fast(float cij, float rci, float rcj, float cthr4) {
  return __log2f(fmaxf(cij, cthr4) * (rci * rcj)) * 0.693147180559945309f;
}

// The "lo" part of a float32 value v for a product carried by TF32 tensor cores.  The tensor core reads
// only the upper 19 bits of a 32-bit operand, so the untouched value already acts as hi = v truncated to TF32
// and only lo = v - hi (exact) has to be produced; it is rounded to the 11 significant bits of TF32 (Veltkamp
// split with 2^13 + 1, all on the FMA pipe), so that what the tensor core drops of it is zero.  hi + lo then
// differs from v by at most 2^-22 |v|.  Inf / NaN give a NaN lo.
__device__ __forceinline__ float tf32_lo(float v) {
  const float hi = __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
  const float lo = __fsub_rn(v, hi);
  const float c = __fmul_rn(lo, 8193.f);
  return __fsub_rn(c, __fsub_rn(c, lo));
}
__device__ __forceinline__ double tf32_lo(double v) { return v; }   // never used: float64 has no tensor path

}  // namespace sbb
