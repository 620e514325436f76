// The number types of the point functions, double and Num (rc_soft.cuh), and
// the operations they are written in.
#pragma once

#include "rc_div.cuh"
#include "rc_math.h"
#include "rc_soft.cuh"

namespace rc {

// The operations that double and Num spell differently.
__device__ __forceinline__ double n_abs(double x) { return fabs(x); }
__device__ __forceinline__ double n_exp(double x) { return rcm::exp(x); }
__device__ __forceinline__ double n_log(double x) { return rcm::log(x); }
__device__ __forceinline__ double n_pow(double x, double y, double logx) {
  return rcm::pow_log<rcm::HwMul>(x, y, logx);
}
// a / b with V = rcs::recip32(b) known: a divisor fixed in advance, or shared.
// The FP64 unit has no part in it; through a pair of reciprocals in FP64 it
// took four operations (250 cycles of a warp alone, 308 of many).
__device__ __forceinline__ double div_fixed(double a, double b, unsigned V) { return soft_div_by(a, b, V); }
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
template <bool M>
__device__ __forceinline__ Num<M> div_fixed(Num<M> a, Num<M> b, unsigned V) { return soft_div_by(a.v, b.v, V); }
// x < 0.0
template <class N>
__device__ __forceinline__ bool negative(N x) { return less(val(x), 0.0); }
}  // namespace rc
