// The number type of the point functions: double, and the operations they are
// written in.
#pragma once

#include "rc_div.cuh"
#include "rc_math.h"

namespace rc {

__device__ __forceinline__ double val(double x) { return x; }
__device__ __forceinline__ double n_abs(double x) { return fabs(x); }
__device__ __forceinline__ double n_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ double n_exp(double x) { return rcm::exp(x); }
__device__ __forceinline__ double n_log(double x) { return rcm::log(x); }
// x^y with log x given
__device__ __forceinline__ double n_pow(double x, double y, double logx) {
  return rcm::pow_log<rcm::HwMul>(x, y, logx);
}
__device__ __forceinline__ double n_pow(double x, double y) { return n_pow(x, y, n_log(x)); }
// a / b for a divisor fixed in advance
__device__ __forceinline__ double div_fixed(double a, double b, const double* r) { return div_rn(a, b, r); }
// x < 0.0
__device__ __forceinline__ bool negative(double x) { return less(x, 0.0); }
// the reciprocal pair of b, to be stored
__device__ __forceinline__ Recip recip(double b) { return recip_of(b); }
// the reciprocal pair of b for div_by
__device__ __forceinline__ Recip pair_of(double b) { return recip_of(b); }
__device__ __forceinline__ double div_by(double a, double b, Recip r) { return div_rn(a, b, r.h, r.l); }

}  // namespace rc
