// Elementwise math shared by the Sinkhorn kernels.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "wdl_internal.cuh"

namespace wdl {

// log(x) of a positive FP32 value returned in FP64 with an absolute error of a
// few 1e-8 instead of logf's one ulp of |log x| (~1e-6 at |log x| ~ 10): x is
// split as m * 2^e with m in [sqrt(1/2), sqrt(2)), e*ln2 is formed in FP64 and
// only log(m), which is small, comes from logf.  Used where FP32 logarithms are
// summed in FP64 over a whole grid (weight-gradient dot products, the weighted
// geometric mean), so that the sums keep FP32-level relative accuracy.
// A saturated x = inf stays inf: callers find overflows by it.
__device__ __forceinline__ double log_f32_precise(float x) {
  const int i = __float_as_int(x);
  if ((unsigned)(i - 0x00800000) >= 0x7f000000u) {  // not a positive normal number
    int e;
    float m = frexpf(x, &e);  // subnormal: x = m * 2^e, m in [0.5, 1)
    if (!(m < INFINITY)) return (double)m;
    if (m < 0.70710678f) {
      m *= 2.0f;
      e -= 1;
    }
    return (double)e * 0.6931471805599453 + (double)logf(m);
  }
  const int e = (i - 0x3f3504f3) >> 23;  // sqrt(1/2) = 0x3f3504f3
  const float m = __int_as_float(i - (int)((unsigned)e << 23));
  return (double)e * 0.6931471805599453 + (double)logf(m);
}

// exp(s) for an FP64 exponent returned in FP32: s = n*ln2 + r with |r| <= ln2/2,
// exp(s) = 2^n * expf(r); relative error ~1e-7 for the whole FP32 range.
__device__ __forceinline__ float exp_to_f32(double s) {
  if (s < -110.0) return 0.0f;
  if (s > 89.0) return INFINITY;
  const double n = rint(s * 1.4426950408889634);
  const float r = (float)(s - n * 0.6931471805599453);
  return ldexpf(expf(r), (int)n);
}

template <typename T>
__device__ __forceinline__ T d_exp(T x);
template <>
__device__ __forceinline__ float d_exp<float>(float x) { return expf(x); }
template <>
__device__ __forceinline__ double d_exp<double>(double x) { return exp(x); }
template <typename T>
__device__ __forceinline__ T d_log(T x);
template <>
__device__ __forceinline__ float d_log<float>(float x) { return logf(x); }
template <>
__device__ __forceinline__ double d_log<double>(double x) { return log(x); }
// Natural log of a magnitude feeding a log-domain operand: FP32 takes the
// hardware base-2 logarithm times ln 2 (absolute error ~2e-7, i.e. ~2e-7
// relative on the scaling it encodes; a log-domain value of magnitude >= 2 is
// rounded more coarsely than that anyway); FP64 the library log.
template <typename T>
__device__ __forceinline__ T d_log_mag(T x);
template <>
__device__ __forceinline__ float d_log_mag<float>(float x) {
  float y;
  asm("lg2.approx.f32 %0, %1;" : "=f"(y) : "f"(fabsf(x)));
  return y * 0.6931471805599453f;
}
template <>
__device__ __forceinline__ double d_log_mag<double>(double x) { return log(fabs(x)); }

// safe_log = log(max(EPSILON, x)) (cpp/loss.h:3-5).
template <typename T>
__device__ __forceinline__ T safe_log(T x);
template <>
__device__ __forceinline__ double safe_log<double>(double x) {
  return log(x > kEpsilon ? x : kEpsilon);
}
template <>
__device__ __forceinline__ float safe_log<float>(float x) {
  return x > 0.f ? logf(x) : float(kLogEpsilon);
}

// Logarithms that are summed in FP64 (grid reductions, the geometric mean over
// atoms): FP64 mode uses log directly; FP32 mode uses the split form of
// log_f32_precise so the FP64 sum is not limited by logf's absolute error.
template <typename T>
__device__ __forceinline__ double acc_log(T x);
template <>
__device__ __forceinline__ double acc_log<double>(double x) { return log(x); }
template <>
__device__ __forceinline__ double acc_log<float>(float x) {
  return x > 0.f ? log_f32_precise(x) : (double)logf(x);
}
template <typename T>
__device__ __forceinline__ double acc_safe_log(T x);
template <>
__device__ __forceinline__ double acc_safe_log<double>(double x) {
  return log(x > kEpsilon ? x : kEpsilon);
}
template <>
__device__ __forceinline__ double acc_safe_log<float>(float x) {
  return x > 0.f ? log_f32_precise(x) : kLogEpsilon;
}
template <typename T>
__device__ __forceinline__ T exp_from(double s);
template <>
__device__ __forceinline__ double exp_from<double>(double s) { return exp(s); }
template <>
__device__ __forceinline__ float exp_from<float>(double s) { return exp_to_f32(s); }

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < nw ? sh[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  return t;  // valid in thread 0
}

}  // namespace wdl
