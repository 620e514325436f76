// Thermochemistry point functions of RocketCombustor on the device (FP64).
//
// Each function keeps the operation order of the reference routine it cites,
// so that with FMA contraction disabled (--fmad=false) +,-,*,/ and sqrt give
// the reference's IEEE results; exp/log/pow come from include/rc_math.h, the
// same code the CPU oracle runs, so the results are bit-identical.  Constants
// that depend on species data only (pair terms of the Wilke and Chapman-Enskog
// sums) are evaluated once on the host with the reference's expressions and
// passed in ThermoDev, with 32-bit reciprocals of the fixed divisors; divisions
// by those, and the transport fits' divisions by T and T^2, take the integer
// division of rc_soft.cuh with its reciprocal at hand (the IEEE quotient bit for
// bit, no FP64 operation).
#pragma once
#include <cstdint>

#include "rc_num.cuh"

namespace rc {

enum : unsigned {
  ERR_THERMO_T = 1u, ERR_TRANSPORT_T = 2u, ERR_NEG_TIMESTEP = 4u, ERR_NEG_FACE = 8u,
  ERR_NAN = 16u, ERR_BCTYPE = 32u, ERR_SYNC = 64u, ERR_LINSOLVE = 128u
};

template <int NSP>
struct ThermoDev {
  double R[NSP];                 // R_species
  double mw[NSP];                // mole_weight
  double Rconstant;
  double tlo, tcrit, thi;        // thermo_{lowest,critical,highest}_tem
  double cl[7][NSP], ch[7][NSP]; // low/high_coef_Cp_species(j,i) -> [j][i]
  double b1l[NSP], b1h[NSP];     // low/high_enthalpy_b1
  double trlo, trcrit, trhi;     // transport_{lowest,critical,highest}_tem
  double mu[2][4][NSP];          // [low/high][A..D][species]
  double kk[2][4][NSP];
  double wc[NSP][NSP];           // (mole_weight(j)/mole_weight(i))**0.25
  double wd[NSP][NSP];           // sqrt(1. + mole_weight(i)/mole_weight(j))
  double dlj[NSP][NSP];          // sqrt(LJ_energy(i)*LJ_energy(j))
  double dmw[NSP][NSP];          // sqrt(2./(1./mw(i)+1./mw(j))*1000)
  double dcd[NSP][NSP];          // (0.5*(sigma(i)+sigma(j)))**2
  int model;                     // code_chemical_model
  double Af, E;                  // Af_react(1), E_react(1)
  double prodc[NSP];             // 1000*mole_weight(ks)*(coef_r-coef_f)
  double mw1000[2];              // mole_weight(1..2)*1000
  double cfl;
  // rcs::recip32 of fixed divisors
  unsigned mwv[NSP], wdv[NSP][NSP], dljv[NSP][NSP], mw1000v[2];
  int cols;                      // bit j: column j of cl or ch has a non-zero coefficient
};

// The functions below take double or Num (rc_soft.cuh); the bits are the same.
__device__ __forceinline__ double fmin2(double a, double b) { return less(b, a) ? b : a; }
__device__ __forceinline__ double fmax2(double a, double b) { return less(a, b) ? b : a; }
template <bool M>
__device__ __forceinline__ Num<M> fmin2(Num<M> a, Num<M> b) { return less(b, a) ? b : a; }
template <bool M>
__device__ __forceinline__ Num<M> fmax2(Num<M> a, Num<M> b) { return less(a, b) ? b : a; }
// lo <= x && x <= hi (false for a NaN x)
__device__ __forceinline__ bool in_range(double lo, double x, double hi) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL && !less(x, lo) && !less(hi, x);
}

// The polynomial columns to evaluate at temperature t: those that hold a
// non-zero coefficient.  A column of zeros adds c b = +-0 to sums that start at
// +0, which changes no bit as long as its basis value b is finite: every
// column for a temperature outside 2^-100..2^100, whose powers and reciprocals
// need not be.  What a column costs is its basis value (two divisions for 1/t
// and 1/t^2, log t / t and three divisions in the enthalpy) and two operations
// per species; property files of this solver fill one to three of the seven.
template <int NSP>
__device__ __forceinline__ int poly_cols(const ThermoDev<NSP>& th, double t) {
  const unsigned e = (unsigned)__double2hiint(t) >> 20;  // sign and exponent
  return e - 923u <= 200u ? th.cols : 127;
}
// s_i + c_ij b for every species, c the range's coefficients of column j; the
// first column of `cols` starts the sums (0 + c b)
template <int NSP, class N>
__device__ __forceinline__ void poly_add(const ThermoDev<NSP>& th, int cols, int j, bool low, N b, N* s) {
  if ((cols & ((1 << j) - 1)) == 0) {
#pragma unroll
    for (int i = 0; i < NSP; ++i) s[i] = plus_zero((low ? th.cl[j][i] : th.ch[j][i]) * b);
  } else {
#pragma unroll
    for (int i = 0; i < NSP; ++i) s[i] = s[i] + (low ? th.cl[j][i] : th.ch[j][i]) * b;
  }
}
// the same for the column of the constant term, whose basis value is 1
template <int NSP, class N>
__device__ __forceinline__ void poly_add1(const ThermoDev<NSP>& th, int cols, int j, bool low, N* s) {
  if ((cols & ((1 << j) - 1)) == 0) {
#pragma unroll
    for (int i = 0; i < NSP; ++i) s[i] = plus_zero(low ? th.cl[j][i] : th.ch[j][i]);
  } else {
#pragma unroll
    for (int i = 0; i < NSP; ++i) s[i] = s[i] + (low ? th.cl[j][i] : th.ch[j][i]);
  }
}
// sum_i a_i b_i from +0 in index order
template <int NSP, class A, class N>
__device__ __forceinline__ N dot(const A* a, const N* b) {
  N s = plus_zero(a[0] * b[0]);
#pragma unroll
  for (int i = 1; i < NSP; ++i) s = s + a[i] * b[i];
  return s;
}
// the last species' mass fraction, 1 - sum of the others (from +0, in order)
template <int NSP, class N>
__device__ __forceinline__ N last_y(const N* Y) {
  if (NSP == 1) return 1.0 - 0.0;
  N s = plus_zero(Y[0]);
#pragma unroll
  for (int k = 1; k < NSP - 1; ++k) s = s + Y[k];
  return 1.0 - s;
}

// ComputeGasParameter (thermo_property.f90:78-112)
template <int NSP, class N>
__device__ __forceinline__ void gas(const ThermoDev<NSP>& th, const N* Y, N tem, N& Cp, N& gama, N& Rcpcv,
                                    unsigned& err) {
  const N t2 = tem * tem;
  const double t = val(tem);
  const bool low = in_range(th.tlo, t, th.tcrit);
  if (!low && !(less(th.tcrit, t) && !less(th.thi, t))) err |= ERR_THERMO_T;
  const int cols = poly_cols(th, t);
  N cps[NSP];
#pragma unroll
  for (int i = 0; i < NSP; ++i) cps[i] = 0.0;
  if (cols & 1) poly_add(th, cols, 0, low, 1.0 / t2, cps);
  if (cols & 2) poly_add(th, cols, 1, low, 1.0 / tem, cps);
  if (cols & 4) poly_add1(th, cols, 2, low, cps);
  if (cols & 8) poly_add(th, cols, 3, low, tem, cps);
  if (cols & 16) poly_add(th, cols, 4, low, t2, cps);
  if (cols & 32) poly_add(th, cols, 5, low, tem * t2, cps);
  if (cols & 64) poly_add(th, cols, 6, low, t2 * t2, cps);
#pragma unroll
  for (int i = 0; i < NSP; ++i) cps[i] = cps[i] * th.R[i];
  const N c = dot<NSP>(cps, Y), r = dot<NSP>(th.R, Y);
  Cp = c;
  Rcpcv = r;
  gama = c / (c - r);
}

// rcs::recip32 of 3 and 5: 2^63 over their leading 32 bits, less a little
constexpr unsigned THIRD_V = 0xaaaaaaa6u, FIFTH_V = 0xccccccc8u;
constexpr bool below_reciprocal(unsigned v, unsigned long long b) {
  return (1ull << 63) > v * b && (1ull << 63) - v * b < 1ull << 35;
}
static_assert(below_reciprocal(THIRD_V, 0xc0000000u) && below_reciprocal(FIFTH_V, 0xa0000000u), "as div_by needs");

// compute_enthalpy (thermo_property.f90:114-144)
template <int NSP, class N>
__device__ __forceinline__ void enthalpy(const ThermoDev<NSP>& th, N tem, N* entha, unsigned& err) {
  const N t2 = tem * tem;
  const double t = val(tem);
  const bool low = in_range(th.tlo, t, th.tcrit);
  if (!low && !(less(th.tcrit, t) && !less(th.thi, t))) err |= ERR_THERMO_T;
  const int cols = poly_cols(th, t);
  N s[NSP];
#pragma unroll
  for (int i = 0; i < NSP; ++i) s[i] = 0.0;
  if (cols & 1) poly_add(th, cols, 0, low, -(1.0 / t2), s);
  if (cols & 2) poly_add(th, cols, 1, low, n_log(tem) / tem, s);
  if (cols & 4) poly_add1(th, cols, 2, low, s);
  if (cols & 8) poly_add(th, cols, 3, low, half_of(tem), s);
  if (cols & 16) poly_add(th, cols, 4, low, div_fixed(t2, N(3.0), THIRD_V), s);
  if (cols & 32) poly_add(th, cols, 5, low, 0.25 * (tem * t2), s);
  if (cols & 64) poly_add(th, cols, 6, low, div_fixed(t2 * t2, N(5.0), FIFTH_V), s);
#pragma unroll
  for (int i = 0; i < NSP; ++i) entha[i] = th.R[i] * (tem * s[i] + (low ? th.b1l[i] : th.b1h[i]));
}

// Newton_temperature (thermo_property.f90:146-180); returns T, sets Rcpcv.
template <int NSP, class N>
__device__ __forceinline__ N newton_T(const ThermoDev<NSP>& th, N et, const N* Y, N t0, N& Rcpcv, unsigned& err) {
  N t = t0, Cp, gama;
  N entha[NSP];
  for (int it = 0; it < 200; ++it) {
    enthalpy<NSP>(th, t, entha, err);
    gas<NSP>(th, Y, t, Cp, gama, Rcpcv, err);
    const N h = dot<NSP>(Y, entha);
    const N ft = h - Rcpcv * t - et;
    const N dft = Cp - Rcpcv;
    const N dtt = -ft / dft;
    t = t + dtt;
    t = fmax2(t, N(th.tlo));
    t = fmin2(t, N(th.thi));
    if (less(n_abs(dtt), N(1.0e-5))) break;
  }
  return t;
}

// X_k = (Y_k / M_k) / sum_i Y_i / M_i as transport_property.f90 and
// diffusion_velocity.f90 form it
template <int NSP, class N>
__device__ __forceinline__ void mole_fractions(const ThermoDev<NSP>& th, const N* Y, N* X) {
  N s = plus_zero(div_fixed(Y[0], N(th.mw[0]), th.mwv[0]));
#pragma unroll
  for (int i = 1; i < NSP; ++i) s = s + div_fixed(Y[i], N(th.mw[i]), th.mwv[i]);
  const N ww = 1.0 / s;
#pragma unroll
  for (int i = 0; i < NSP; ++i) X[i] = div_fixed(ww * Y[i], N(th.mw[i]), th.mwv[i]);
}

// compute_transport_property (transport_property.f90:78-125); xx: mole_fractions
template <int NSP, class N>
__device__ __forceinline__ void transport(const ThermoDev<NSP>& th, N tem2, const N* xx, N& vmul, N& akmu,
                                          unsigned& err) {
  const N tem = fmax2(N(th.trlo), tem2);
  const double t = val(tem);
  N mul[NSP], Kl[NSP];
  const bool low = in_range(th.trlo, t, th.trcrit);
  if (!low && !(less(th.trcrit, t) && !less(th.trhi, t))) err |= ERR_TRANSPORT_T;
  const int rg = low ? 0 : 1;
  const N lt = n_log(tem);
  const N t2 = tem * tem;
  const unsigned rt = rcs::recip32(t), rt2 = rcs::recip32(val(t2));
#pragma unroll
  for (int i = 0; i < NSP; ++i) {
    mul[i] = n_exp(th.mu[rg][0][i] * lt + div_fixed(N(th.mu[rg][1][i]), tem, rt) +
                   div_fixed(N(th.mu[rg][2][i]), t2, rt2) + th.mu[rg][3][i]);
    Kl[i] = n_exp(th.kk[rg][0][i] * lt + div_fixed(N(th.kk[rg][1][i]), tem, rt) +
                  div_fixed(N(th.kk[rg][2][i]), t2, rt2) + th.kk[rg][3][i]);
  }
#pragma unroll
  for (int i = 0; i < NSP; ++i) { mul[i] = mul[i] * 1.0e-7; Kl[i] = Kl[i] * 1.0e-4; }
  N v = 0.0;
#pragma unroll
  for (int i = 0; i < NSP; ++i) {
    N phil = 0.0;
#pragma unroll
    for (int j = 0; j < NSP; ++j) {
      // sqrt(mul(i)/mul(i)) is exactly 1
      const N sq = (i == j) ? N(1.0) : n_sqrt(mul[i] / mul[j]);
      const N q = 1.0 + sq * th.wc[i][j];
      const N w = div_fixed(xx[j] * (q * q), N(th.wd[i][j]), th.wdv[i][j]);
      phil = j ? phil + w : plus_zero(w);
    }
    phil = (0.25 * sqrt(2.0)) * phil;
    const N w = xx[i] * mul[i] / phil;
    v = i ? v + w : plus_zero(w);
  }
  const N s1 = dot<NSP>(xx, Kl);
  N s2 = plus_zero(xx[0] / Kl[0]);
#pragma unroll
  for (int i = 1; i < NSP; ++i) s2 = s2 + xx[i] / Kl[i];
  vmul = v;
  akmu = half_of(s1 + 1.0 / s2);
}

// compute_diffusion_velocity (diffusion_velocity.f90:55-118); XX: mole_fractions.  D_ij is
// symmetric bit for bit (every pair term is), so each pair is evaluated once;
// the diagonal D_ii is never used.
template <int NSP, class N>
__device__ __forceinline__ void diffusion(const ThermoDev<NSP>& th, N pp, N tem, const N* XX, N* Dk) {
  const N num = 0.0266 * n_sqrt(tem * (tem * tem));
  N D[NSP][NSP];
#pragma unroll
  for (int i = 0; i < NSP; ++i)
#pragma unroll
    for (int j = i + 1; j < NSP; ++j) {
      const N tstar = div_fixed(tem, N(th.dlj[i][j]), th.dljv[i][j]);
      const N om = 1.06036 * n_pow(tstar, -0.15610) + 0.19300 * n_exp(-0.47635 * tstar) +
                   1.03587 * n_exp(-1.52996 * tstar) + 1.76474 * n_exp(-3.89411 * tstar);
      const N d = num / (pp * th.dmw[i][j] * th.dcd[i][j] * om);
      D[i][j] = d;
      D[j][i] = d;
    }
#pragma unroll
  for (int i = 0; i < NSP; ++i) {
    N xd = 0.0;
#pragma unroll
    for (int j = 0; j < NSP; ++j)
      if (j != i) {
        const N w = XX[j] / D[i][j];
        xd = j == (i == 0 ? 1 : 0) ? plus_zero(w) : xd + w;
      }
    Dk[i] = (1.0 - XX[i]) / (xd + 1.0e-16);
  }
}

// compute_production_rate (chemical_kinetics.f90:109-165)
template <int NSP, class N>
__device__ __forceinline__ void production(const ThermoDev<NSP>& th, N T, N rho, const N* Y2, N* prod) {
  N kf;
  const N y0 = fmin2(N(1.0), fmax2(N(0.0), Y2[0]));
  if (th.model == 0) {
    const N y1 = fmin2(N(1.0), fmax2(N(0.0), Y2[NSP > 1 ? 1 : 0]));
    kf = th.Af * n_exp(-th.E / (th.Rconstant * T));
    kf = kf * n_pow(div_fixed(y0 * rho, N(th.mw1000[0]), th.mw1000v[0]), 0.2);
    kf = kf * n_pow(div_fixed(y1 * rho, N(th.mw1000[1]), th.mw1000v[1]), 1.3);
  } else {
    kf = less(N(710.0), T) ? 1e4 : 0.0;
    kf = kf * div_fixed(y0 * rho, N(th.mw1000[0]), th.mw1000v[0]);
  }
#pragma unroll
  for (int k = 0; k < NSP; ++k) prod[k] = th.prodc[k] * kf;
}

}  // namespace rc
