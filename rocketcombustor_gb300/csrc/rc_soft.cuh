// FP64 multiplication, division and square root on the integer pipes,
// correctly rounded (round to nearest even): the IEEE results bit for bit.
//
// Why: a GB300 SM sub-partition holds its FP64 unit for 64-77 cycles per warp
// instruction, so the FP64 kernels of this library run at the FP64 issue rate
// while the integer and FP32 pipes idle.  Measured (8 warps per sub-partition,
// cycles of a sub-partition per warp operation, hardware / here):
// multiplication 77 / 65, division 573 / 104, square root 574 / 131, and a
// hardware addition with a multiplication here 98 for both against 154.  With
// one warp per sub-partition (latency, one dependent chain) 55 / 216, 574 /
// 278, 608 / 302: only division and square root gain there.  An addition done
// this way takes 102 cycles and stays on the FP64 unit.
//
// Methods (software floating point on integers as in J.-M. Muller et al., Handbook
// of Floating-Point Arithmetic, Birkhaeuser 2010, chapter 10; quotient digits
// from a truncated reciprocal and a correction, N. Moeller and T. Granlund,
// "Improved division by invariant integers", IEEE Trans. Computers 60(2), 2011):
// significands as 53-bit integers.  Multiplication: the 106-bit
// product from four 32 x 32 products, normalised and rounded on the bits
// below.  Division: digit by digit with a 32-bit reciprocal (hardware FP32
// reciprocal and one Newton step in integers, kept below the true value), two
// quotient digits of 31 and 23 bits with exact remainders modulo 2^64, one
// correction; the quotient of two 53-bit significands never lies half way
// between two doubles, so its 54 leading bits round it.  Square root: the same
// with an FP32 reciprocal square root and one exact remainder.  Operands with
// exponents outside -400..400, infinities and NaNs take the hardware operation;
// zero times, or over, a finite number is a signed zero.  Works on the host too (tests compare it there with the
// processor's own operations).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define RCS_HD __host__ __device__ __forceinline__
#else
#define RCS_HD inline
#endif

namespace rcs {

#ifndef __CUDA_ARCH__
inline int seed_ulps = 0;  // host tests: error added to the seeds, in ulps
#endif

RCS_HD uint32_t hi32(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2hiint(x);
#else
  uint64_t b; std::memcpy(&b, &x, 8); return (uint32_t)(b >> 32);
#endif
}
RCS_HD uint32_t lo32(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2loint(x);
#else
  uint64_t b; std::memcpy(&b, &x, 8); return (uint32_t)b;
#endif
}
RCS_HD double make(uint32_t h, uint32_t l) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)h, (int)l);
#else
  const uint64_t b = ((uint64_t)h << 32) | l; double x; std::memcpy(&x, &b, 8); return x;
#endif
}
RCS_HD double make64(uint64_t b) { return make((uint32_t)(b >> 32), (uint32_t)b); }
RCS_HD uint32_t umulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
RCS_HD int32_t smulhi(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
RCS_HD uint32_t umax(uint32_t a, uint32_t b) { return a > b ? a : b; }
RCS_HD uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }
// the bits of an approximation of 1/f, 1/sqrt(f) (relative error below 2^-21)
RCS_HD uint32_t rcp_bits(uint32_t f) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  return __float_as_uint(r);
#else
  float x; std::memcpy(&x, &f, 4); x = 1.0f / x; uint32_t r; std::memcpy(&r, &x, 4); return r + seed_ulps;
#endif
}
RCS_HD uint32_t rsqrt_bits(uint32_t f) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  return __float_as_uint(r);
#else
  float x; std::memcpy(&x, &f, 4); x = 1.0f / std::sqrt(x); uint32_t r; std::memcpy(&r, &x, 4); return r + seed_ulps;
#endif
}

constexpr uint32_t EXP_MASK = 0x7ff00000u, SIGN_BIT = 0x80000000u;
// fields of exponents -400 .. 400
constexpr uint32_t EXP_LO = (1023u - 400u) << 20, EXP_SPAN = 800u << 20;

// one of the two is zero and neither is infinite or NaN
RCS_HD bool zero_times_finite(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl) {
  const bool za = ((ah << 1) | al) == 0u, zb = ((bh << 1) | bl) == 0u;
  return (za || zb) && umax(ah & EXP_MASK, bh & EXP_MASK) != EXP_MASK;
}

RCS_HD double mul(double a, double b) {
  const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), bl = lo32(b);
  const uint32_t ea = (ah & EXP_MASK) - EXP_LO, eb = (bh & EXP_MASK) - EXP_LO;
  if (umax(ea, eb) > EXP_SPAN) {
    if (zero_times_finite(ah, al, bh, bl)) return make((ah ^ bh) & SIGN_BIT, 0u);
    return a * b;
  }
  const uint32_t mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
  const uint32_t A1 = (mah << 11) | (al >> 21), A0 = al << 11;  // a's significand from bit 63 down
  const uint64_t p00 = (uint64_t)A0 * bl;
  const uint64_t p01 = (uint64_t)A0 * mbh + (p00 >> 32);
  const uint64_t p10 = (uint64_t)A1 * bl + (uint32_t)p01;
  uint64_t h = (uint64_t)A1 * mbh + (p01 >> 32);
  h += p10 >> 32;
  uint32_t l1 = (uint32_t)p10, l0 = (uint32_t)p00;  // the 64 bits below h
  uint32_t e = ea + eb + (2u * EXP_LO - (1023u << 20));
  if (!(h >> 52)) {  // product of the significands below 2: one more bit
    h = (h << 1) | (l1 >> 31);
    l1 = (l1 << 1) | (l0 >> 31);
    l0 <<= 1;
    e -= 1u << 20;
  }
  h += l1 >> 31;
  if (((l1 << 1) | l0) == 0u && (l1 >> 31)) h &= ~(uint64_t)1;  // a tie goes to the even one
  const uint32_t rh = (uint32_t)(h >> 32) + e;
  return make(rh | ((ah ^ bh) & SIGN_BIT), (uint32_t)h);
}

// The reciprocal that div_by needs, from b's significand alone: 2^63 over its
// leading 32 bits, below the true value by less than 2^-28 of it.
RCS_HD uint32_t recip32(double b) {
  const uint32_t bh = hi32(b), bl = lo32(b);
  const uint32_t bn = (((bh & 0xfffffu) | 0x100000u) << 11) | (bl >> 21);  // leading 32 bits
  const uint32_t rb = umin(rcp_bits(0x3f800000u | ((bn >> 8) & 0x7ffffeu)), 0x3f7fffffu);
  const uint32_t V0 = (rb << 8) | SIGN_BIT;  // 2^63 / bn to 21 bits
  const int64_t dlt = (int64_t)(((uint64_t)SIGN_BIT << 32) - (uint64_t)V0 * bn);
  const int32_t dh = (int32_t)(dlt >> 12);
  return V0 + (uint32_t)(smulhi(dh, (int32_t)(V0 >> 1)) >> 18) - 6u;
}
// a / b with V = recip32(b)
RCS_HD double div_by(double a, double b, uint32_t V) {
  const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), bl = lo32(b);
  const uint32_t ea = (ah & EXP_MASK) - EXP_LO, eb = (bh & EXP_MASK) - EXP_LO;
  if (umax(ea, eb) > EXP_SPAN) {
    if (((bh << 1) | bl) != 0u && zero_times_finite(ah, al, bh, bl)) return make((ah ^ bh) & SIGN_BIT, 0u);
    return a / b;
  }
  const uint32_t mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
  const uint32_t an = (mah << 11) | (al >> 21);
  const uint32_t q1 = umulhi(an, V);  // 2^31 a / b, not above it
  const uint64_t ma = ((uint64_t)mah << 32) | al, mb = ((uint64_t)mbh << 32) | bl;
  const uint64_t r1 = (ma << 31) - ((uint64_t)q1 * bl + ((uint64_t)(q1 * mbh) << 32));
  uint32_t q2 = umulhi((uint32_t)(r1 >> 25), V) >> 4;
  const uint64_t r2 = (r1 << 23) - ((uint64_t)q2 * bl + ((uint64_t)(q2 * mbh) << 32));
  if (r2 >= mb) ++q2;
  uint64_t Q = ((uint64_t)q1 << 23) + q2;  // floor(2^54 a / b) of the significands
  uint32_t e = ea - eb + ((1023u - 1u) << 20);
  if (!(Q >> 54)) { Q <<= 1; e -= 1u << 20; }
  Q = (Q + 2) >> 2;
  return make(((uint32_t)(Q >> 32) + e) | ((ah ^ bh) & SIGN_BIT), (uint32_t)Q);
}
RCS_HD double div(double a, double b) { return div_by(a, b, recip32(b)); }

RCS_HD double sqrt(double a) {
  const uint32_t ah = hi32(a), al = lo32(a);
  if (ah - EXP_LO > EXP_SPAN) {
#ifdef __CUDA_ARCH__
    return ::sqrt(a);
#else
    return std::sqrt(a);
#endif
  }
  const uint32_t odd = (~ah >> 20) & 1u;  // the unbiased exponent is odd
  const uint32_t mh = (ah & 0xfffffu) | 0x100000u;
  const uint64_t x = (((uint64_t)mh << 32) | al) << odd;  // [2^52, 2^54)
  const uint32_t xn = (uint32_t)(x >> 22);                // [2^30, 2^32)
  const uint32_t f = 0x3f800000u + (odd << 23) + (((mh << 3) | (al >> 29)) & 0x7ffff8u);
  const uint32_t rb = umin(rsqrt_bits(f), 0x3f7fffffu);   // in [0.5, 1)
  const uint32_t Y0 = (rb << 8) | SIGN_BIT;                   // 2^32 / sqrt(x 2^-52), 22 bits
  // one Newton step: Y = Y0 + Y0 (1 - f Y0^2) / 2
  const uint32_t y2 = umulhi(Y0, Y0);                     // 2^32 Y^2
  const uint64_t t = (uint64_t)xn * y2;                   // 2^62 (f Y^2)
  const int64_t d = (int64_t)(((uint64_t)1 << 62) - t);
  const int32_t dh = (int32_t)(d >> 12);
  const uint32_t Y = Y0 + (uint32_t)(smulhi(dh, (int32_t)(Y0 >> 1)) >> 18);
  const uint32_t s1 = umulhi(xn, Y) << 1;                 // about 2^31 sqrt(f)
  const int64_t r1 = (int64_t)((x << 10) - (uint64_t)s1 * s1);
  const int32_t s2 = (int32_t)(((int64_t)smulhi((int32_t)(r1 >> 8), (int32_t)(Y >> 1))) >> 1);
  uint64_t S = ((uint64_t)s1 << 22) + (int64_t)s2;        // about 2^53 sqrt(f), off by a few units
  const uint32_t Sh = (uint32_t)(S >> 32), Sl = (uint32_t)S;
  int64_t T = (int64_t)((x << 54) - ((uint64_t)Sl * Sl + ((uint64_t)(2u * Sh * Sl) << 32)));
  if (T < 0) { S -= 1; T += 2 * (int64_t)S + 1; }
  if (T > 2 * (int64_t)S) { S += 1; }
  S = (S + 1) >> 1;
  return make64(S + ((uint64_t)(((((ah >> 20) + 1023u) >> 1) - 1u)) << 52));
}

}  // namespace rcs

#ifdef __CUDACC__
#include "rc_math.h"

namespace rc {

struct SoftMul {
  static RCM_HD double mul(double a, double b) { return rcs::mul(a, b); }
};
// One copy of each in the code: a call costs about 18 cycles of the 104-850
// that these take, and straight-line copies (a face flux holds some 60
// divisions and 32 exponentials) would not fit the instruction cache.
static __device__ __noinline__ double soft_div(double a, double b) { return rcs::div(a, b); }
static __device__ __noinline__ double soft_div_by(double a, double b, unsigned V) { return rcs::div_by(a, b, V); }
static __device__ __noinline__ double soft_sqrt(double a) { return rcs::sqrt(a); }
static __device__ __noinline__ double soft_exp(double x) { return rcm::exp_with<SoftMul>(x); }
static __device__ __noinline__ double soft_log(double x) { return rcm::log_with<SoftMul>(x); }
static __device__ __noinline__ double soft_pow(double x, double y, double logx) {
  return rcm::pow_log<SoftMul>(x, y, logx);
}

// A double whose divisions and square roots (and, with MUL, multiplications
// and elementary functions) run on the integer pipes; additions stay on the
// FP64 unit, negation, halving, doubling and comparisons are bit operations.
// Every operation gives the IEEE result, so an expression has the same bits in
// double and in Num.
template <bool MUL>
struct Num {
  double v;
  __device__ __forceinline__ Num() {}
  __device__ __forceinline__ Num(double x) : v(x) {}
  friend __device__ __forceinline__ Num operator+(Num a, Num b) { return a.v + b.v; }
  friend __device__ __forceinline__ Num operator-(Num a, Num b) { return a.v - b.v; }
  friend __device__ __forceinline__ Num operator-(Num a) {
    return __hiloint2double(__double2hiint(a.v) ^ (int)0x80000000, __double2loint(a.v));
  }
  friend __device__ __forceinline__ Num operator*(Num a, Num b) { return MUL ? rcs::mul(a.v, b.v) : a.v * b.v; }
  friend __device__ __forceinline__ Num operator/(Num a, Num b) { return soft_div(a.v, b.v); }
};

}  // namespace rc
#endif
