// The number types of the point functions, double and Num (rc_soft.cuh), and
// the operations they are written in.
#pragma once

#include "rc_div.cuh"
#include "rc_math.h"
#include "rc_soft.cuh"

namespace rc {

// The operations that double and Num spell differently.
__device__ __forceinline__ double val(double x) { return x; }
__device__ __forceinline__ double n_abs(double x) { return fabs(x); }
__device__ __forceinline__ double n_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ double n_exp(double x) { return rcm::exp(x); }
__device__ __forceinline__ double n_log(double x) { return rcm::log(x); }
__device__ __forceinline__ double n_pow(double x, double y, double logx) {
  return rcm::pow_log<rcm::HwMul>(x, y, logx);
}
__device__ __forceinline__ double div_fixed(double a, double b, const double* r) { return div_rn(a, b, r); }
template <bool M>
__device__ __forceinline__ double val(Num<M> x) { return x.v; }
template <bool M>
__device__ __forceinline__ bool less(Num<M> a, Num<M> b) { return less(a.v, b.v); }
template <bool M>
__device__ __forceinline__ Num<M> plus_zero(Num<M> x) { return plus_zero(x.v); }
template <bool M>
__device__ __forceinline__ Num<M> half_of(Num<M> x) { return half_of(x.v); }
template <bool M>
__device__ __forceinline__ Num<M> twice_of(Num<M> x) { return twice_of(x.v); }
template <bool M>
__device__ __forceinline__ Num<M> n_abs(Num<M> x) {
  return __hiloint2double(__double2hiint(x.v) & 0x7fffffff, __double2loint(x.v));
}
template <bool M>
__device__ __forceinline__ Num<M> n_sqrt(Num<M> x) { return soft_sqrt(x.v); }
template <bool M>
__device__ __forceinline__ Num<M> n_exp(Num<M> x) { return M ? soft_exp(x.v) : rcm::exp(x.v); }
template <bool M>
__device__ __forceinline__ Num<M> n_log(Num<M> x) { return M ? soft_log(x.v) : rcm::log(x.v); }
template <bool M>
__device__ __forceinline__ Num<M> n_pow(Num<M> x, double y, Num<M> logx) {
  return M ? soft_pow(x.v, y, logx.v) : rcm::pow_log<rcm::HwMul>(x.v, y, logx.v);
}
template <class N>
__device__ __forceinline__ N n_pow(N x, double y) { return n_pow(x, y, n_log(x)); }
// a / b for a divisor fixed in advance: with the FP64 unit busy the integer
// division (104 cycles) is cheaper than the pair's four operations (308); a
// single warp's chain is shorter through the pair (250 against 278 cycles)
template <bool M>
__device__ __forceinline__ Num<M> div_fixed(Num<M> a, Num<M> b, const double* r) {
  return M ? soft_div(a.v, b.v) : div_rn(a.v, b.v, r);
}
// x < 0.0
template <class N>
__device__ __forceinline__ bool negative(N x) { return less(val(x), 0.0); }
// the reciprocal pair of b, to be stored
template <class N>
__device__ __forceinline__ Recip recip(N b) {
  const N h = 1.0 / b;
  return {val(h), val(N(fma(-val(b), val(h), 1.0)) * h)};
}
// the reciprocal pair of b for div_by, where div_by uses one
template <class N>
__device__ __forceinline__ Recip pair_of(N b) { return recip_of(val(b)); }
template <>
__device__ __forceinline__ Recip pair_of(Num<true>) { return {0.0, 0.0}; }
template <class N>
__device__ __forceinline__ N div_by(N a, N b, Recip r) {
  const double p[2] = {r.h, r.l};
  return div_fixed(a, b, p);
}

}  // namespace rc
