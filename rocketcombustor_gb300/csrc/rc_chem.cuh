// Per-cell chemistry integrator on the device (FP64, built with --fmad=false).
//
// The reference has no chemistry ODE integrator; its explicit source adds
// vol*omega to the residual (sourceterm.f90:43-51).  This integrator is new.
// It is built on the reference's own Jacobians:
//   con_to_pri_jaco   Compute_Con_to_Pri_Jaco (Con_to_Pri_Jacobian.f90:1-87)
//   dwdp              compute_derivative_production_rate (chemical_kinetics.f90:167-265)
// and it keeps the operation order of the CPU oracle's restatement, so that
// the device result is bit-identical to the oracle's.
//
// chem_integrate: the isolated constant-volume adiabatic reactor of one cell
// over dt.  rho, u, v and e = h - R_mix T stay fixed and
// dY_k/dt = omega_k(T, rho, Y)/rho.  A substep of length hs is one linearly
// implicit (Rosenbrock-Euler) step in primitive variables:
//   (dU/dP - hs d omega/dP) dP = hs (0, 0, 0, 0, omega_1 .. omega_{Nsp-1}),
// solved by Gaussian elimination with partial pivoting.  Its flow rows keep
// rho, rho u, rho v and rho E.  Then Y += dP_Y, T comes from Newton_temperature
// at the fixed e (guess T + dP_T clamped to the thermo range), and
// p = rho R_mix T.
//
// Step control: d = max(max_k |dY_k| / (tol (|Y_k| + 1e-3)), |dT| / (0.1 tol T)).
// A substep with d > 1 is rejected and shortened to hs max(0.2, 0.9/d).  An
// accepted substep lets the next one grow to hs min(2, 0.9/d).  Substep
// number maxsub, and any attempt after 2 maxsub attempts, takes the remaining
// time unconditionally (implicit Euler is L-stable).
#pragma once
#include "rc_thermo.cuh"

namespace rc {

// dU/dP, row-major [V][V]; U = (rho, rho u, rho v, rho E, rho Y_1..), P = (p, u, v, T, Y_1..).
// r and Rcpcv return the density and the gas constant, for dwdp.
template <int NSP, class N>
__device__ __forceinline__ void con_to_pri_jaco(const ThermoDev<NSP>& th, const N* pri, N* J, N& r, N& Rcpcv,
                                                unsigned& err) {
  constexpr int V = 3 + NSP, NS1 = NSP - 1;
  const N p = pri[0], u = pri[1], v = pri[2], t = pri[3];
  N y2[NSP], entha[NSP], dhdy[NSP], drdy[NSP], Cp, gama;
#pragma unroll
  for (int i = 0; i < NS1; ++i) y2[i] = pri[4 + i];
  y2[NSP - 1] = last_y<NSP>(y2);
  gas<NSP>(th, y2, t, Cp, gama, Rcpcv, err);
  const N rt = Rcpcv * t;
  const unsigned rtv = rcs::recip32(val(rt));
  r = div_fixed(p, rt, rtv);
  enthalpy<NSP>(th, t, entha, err);
  N h = entha[NSP - 1];
#pragma unroll
  for (int i = 0; i < NS1; ++i) {
    h = h + pri[4 + i] * (entha[i] - entha[NSP - 1]);
    dhdy[i] = entha[i] - entha[NSP - 1];
  }
  const N drdp = div_fixed(N(1.), rt, rtv), drdt = -p / (rt * t);
  const N trr = t * Rcpcv * Rcpcv;
  const unsigned trrv = rcs::recip32(val(trr));
#pragma unroll
  for (int i = 0; i < NS1; ++i) drdy[i] = div_fixed(-N(th.R[i] - th.R[NSP - 1]) * p, trr, trrv);
  const N ke = h + half_of(u * u + v * v);
#pragma unroll
  for (int k = 0; k < V * V; ++k) J[k] = 0.0;
  J[0] = drdp; J[3] = drdt;
  J[V + 0] = u * drdp; J[V + 1] = r; J[V + 3] = u * drdt;
  J[2 * V + 0] = v * drdp; J[2 * V + 2] = r; J[2 * V + 3] = v * drdt;
  J[3 * V + 0] = ke * drdp - 1.; J[3 * V + 1] = r * u; J[3 * V + 2] = r * v; J[3 * V + 3] = r * Cp + ke * drdt;
#pragma unroll
  for (int i = 0; i < NS1; ++i) {
    const N yi = pri[4 + i];
    J[4 + i] = drdy[i];
    J[V + 4 + i] = u * drdy[i];
    J[2 * V + 4 + i] = v * drdy[i];
    J[3 * V + 4 + i] = ke * drdy[i] + r * dhdy[i];
    J[(4 + i) * V + 0] = drdp * yi;
    J[(4 + i) * V + 3] = drdt * yi;
#pragma unroll
    for (int j = 0; j < NS1; ++j) J[(4 + i) * V + 4 + j] = (j == i) ? r + yi * drdy[i] : yi * drdy[j];
  }
}

// d omega_i / dP, row-major [NSP-1][V].  Model 1 leaves dkfdy(3:) unset in
// the reference (chemical_kinetics.f90:228-243); it is taken as dkfdr*drdy(3:).
template <int NSP, class N>
__device__ __forceinline__ void dwdp(const ThermoDev<NSP>& th, const N* pri, N rho, N Rcpcv, N* D) {
  constexpr int V = 3 + NSP, NS1 = NSP - 1;
  const N p = pri[0], T = pri[3];
  N y[NSP], drdy[NSP], dkf[V];
#pragma unroll
  for (int i = 0; i < NS1; ++i) y[i] = fmin2(N(1.), fmax2(N(0.), pri[4 + i]));
  if (less(y[0], N(1.0e-12))) {
#pragma unroll
    for (int c = 0; c < V; ++c) dkf[c] = 0.;
  } else {
    N af = th.Af * n_exp(-th.E / (th.Rconstant * T));
    const N r1 = div_fixed(y[0] * rho, N(th.mw1000[0]), th.mw1000v[0]);
    const N dr1dr = div_fixed(y[0], N(th.mw1000[0]), th.mw1000v[0]);
    const N dr1dy1 = div_fixed(rho, N(th.mw1000[0]), th.mw1000v[0]);
    const N y1 = NS1 > 1 ? y[NS1 > 1 ? 1 : 0] : 0.0;
    const N r2 = div_fixed(y1 * rho, N(th.mw1000[1]), th.mw1000v[1]);
    const N dr2dr = div_fixed(y1, N(th.mw1000[1]), th.mw1000v[1]);
    const N dr2dy2 = div_fixed(rho, N(th.mw1000[1]), th.mw1000v[1]);
    const N drdp = rho / p, drdT = -rho / T;
    const unsigned Rv = rcs::recip32(val(Rcpcv));
#pragma unroll
    for (int i = 0; i < NS1; ++i) drdy[i] = div_fixed(-N(th.R[i] - th.R[NSP - 1]) * rho, Rcpcv, Rv);
    N dkfdr, dkfdT, dkfdy[NSP];
    if (th.model == 0) {
      const N l1 = n_log(r1), l2 = n_log(r2);
      const N p1 = n_pow(r1, 0.2, l1), p2 = n_pow(r2, 1.3, l2), p23 = n_pow(r2, 0.3, l2);
      const N dter1_dr = 0.2 * n_pow(rho, -0.8) * n_pow(dr1dr, 0.2);
      dkfdr = af * (p1 * 1.3 * p23 * dr2dr + dter1_dr * p2);
      dkfdT = af * p1 * p2 * th.E / (th.Rconstant * T * T) + dkfdr * drdT;
      dkfdy[0] = af * 0.2 * n_pow(r1, -0.8, l1) * dr1dy1 * p2 + dkfdr * drdy[0];
      if (NS1 > 1) dkfdy[1] = af * p1 * 1.3 * p23 * dr2dy2 + dkfdr * drdy[1];
    } else {
      af = 0.0;
      if (less(N(710.0), T)) af = 1e4;
      const N dter1_dr = dr1dr;
      dkfdr = af * (r1 * 0 * dr2dr + dter1_dr);
      dkfdT = 0.;
      dkfdy[0] = af * dr1dy1 + dkfdr * drdy[0];
      if (NS1 > 1) dkfdy[1] = af * r1 * 0 * dr2dy2 + dkfdr * drdy[1];
    }
#pragma unroll
    for (int i = 2; i < NS1; ++i) dkfdy[i] = dkfdr * drdy[i];
    dkf[0] = dkfdr * drdp; dkf[1] = 0.; dkf[2] = 0.; dkf[3] = dkfdT;
#pragma unroll
    for (int i = 0; i < NS1; ++i) dkf[4 + i] = dkfdy[i];
  }
#pragma unroll
  for (int i = 0; i < NS1; ++i)
#pragma unroll
    for (int k = 0; k < V; ++k) D[i * V + k] = th.prodc[i] * dkf[k];
}

// Gaussian elimination with partial pivoting, in place; b gets the solution.
// Returns false for a singular matrix.  Columns are a template recursion, so
// that every index is known and the system stays in registers (a loop over
// the columns was left rolled, with the matrix in local memory).
template <int NV, int K, class N>
__device__ __forceinline__ bool gepp_column(N* A, N* b, unsigned* V) {
  int piv = K;
  N best = n_abs(A[K * NV + K]);
#pragma unroll
  for (int r = K + 1; r < NV; ++r) {
    const N a = n_abs(A[r * NV + K]);
    if (less(best, a)) { best = a; piv = r; }
  }
  if (!less(N(0.0), best)) return false;
  if (piv != K) {
#pragma unroll
    for (int r = K + 1; r < NV; ++r)
      if (r == piv) {
#pragma unroll
        for (int c = K; c < NV; ++c) { const N t = A[K * NV + c]; A[K * NV + c] = A[r * NV + c]; A[r * NV + c] = t; }
        const N t = b[K]; b[K] = b[r]; b[r] = t;
      }
  }
  const N dk = A[K * NV + K];
  V[K] = rcs::recip32(val(dk));
#pragma unroll
  for (int r = K + 1; r < NV; ++r) {
    const N f = div_fixed(A[r * NV + K], dk, V[K]);
#pragma unroll
    for (int c = K + 1; c < NV; ++c) A[r * NV + c] = A[r * NV + c] - f * A[K * NV + c];
    b[r] = b[r] - f * b[K];
  }
  if constexpr (K + 1 < NV) return gepp_column<NV, K + 1>(A, b, V);
  return true;
}
template <int NV, class N>
__device__ __forceinline__ bool gepp_solve(N* A, N* b) {
  unsigned V[NV];  // recip32 of the pivots
  if (!gepp_column<NV, 0>(A, b, V)) return false;
#pragma unroll
  for (int k = NV - 1; k >= 0; --k) {
    N s = b[k];
#pragma unroll
    for (int c = k + 1; c < NV; ++c) s = s - A[k * NV + c] * b[c];
    b[k] = div_fixed(s, A[k * NV + k], V[k]);
  }
  return true;
}

// One reactor on its way: primitive state P, its fixed rho and e, the time
// left and the next substep.
template <int NSP, class N>
struct Reactor {
  N P[3 + NSP], rho, e, rem, hs;
  int nacc, natt;

  // starts at P over dt; false when there is nothing to integrate
  __device__ __forceinline__ bool begin(const ThermoDev<NSP>& th, N dt, unsigned& err) {
    N Y[NSP], entha[NSP], Cp, gama, Rcpcv;
#pragma unroll
    for (int i = 0; i < NSP - 1; ++i) Y[i] = P[4 + i];
    Y[NSP - 1] = last_y<NSP>(Y);
    gas<NSP>(th, Y, P[3], Cp, gama, Rcpcv, err);
    rho = P[0] / (Rcpcv * P[3]);
    enthalpy<NSP>(th, P[3], entha, err);
    e = dot<NSP>(Y, entha) - Rcpcv * P[3];
    rem = dt;
    hs = dt;
    nacc = 0;
    natt = 0;
    return less(N(0.0), rem);
  }

  // one attempted substep; false when the reactor has reached its end
  __device__ __forceinline__ bool attempt(const ThermoDev<NSP>& th, double tol, int maxsub, unsigned& err) {
    constexpr int V = 3 + NSP, NS1 = NSP - 1;
    N A[V * V], D[(NS1 > 0 ? NS1 : 1) * V], b[V], prod[NSP], Y[NSP], Rcpcv;
    const bool last = nacc + 1 >= maxsub || natt >= 2 * maxsub;
    if (last || less(rem, hs)) hs = rem;
    N r;
    con_to_pri_jaco<NSP>(th, P, A, r, Rcpcv, err);
    dwdp<NSP>(th, P, r, Rcpcv, D);
#pragma unroll
    for (int i = 0; i < NS1; ++i) Y[i] = P[4 + i];
    Y[NSP - 1] = last_y<NSP>(Y);
    production<NSP>(th, P[3], rho, Y, prod);
#pragma unroll
    for (int i = 0; i < NS1; ++i)
#pragma unroll
      for (int c = 0; c < V; ++c) A[(4 + i) * V + c] = A[(4 + i) * V + c] - hs * D[i * V + c];
#pragma unroll
    for (int k = 0; k < 4; ++k) b[k] = 0.0;
#pragma unroll
    for (int i = 0; i < NS1; ++i) b[4 + i] = hs * prod[i];
    if (!gepp_solve<V>(A, b)) { err |= ERR_NAN; return false; }
    ++natt;
    N d = n_abs(b[3]) / (N(0.1) * tol * P[3]);
#pragma unroll
    for (int i = 0; i < NS1; ++i) d = fmax2(d, n_abs(b[4 + i]) / (N(tol) * (n_abs(P[4 + i]) + 1.0e-3)));
    if (less(N(1.0), d) && !last) {
      hs = hs * fmax2(N(0.2), 0.9 / d);
      return true;
    }
#pragma unroll
    for (int i = 0; i < NS1; ++i) { P[4 + i] = P[4 + i] + b[4 + i]; Y[i] = P[4 + i]; }
    Y[NSP - 1] = last_y<NSP>(Y);
    const N tg = fmin2(fmax2(P[3] + b[3], N(th.tlo)), N(th.thi));
    const N t = newton_T<NSP>(th, e, Y, tg, Rcpcv, err);
    P[3] = t;
    P[0] = rho * Rcpcv * t;
    rem = rem - hs;
    ++nacc;
    if (less(N(0.0), d)) hs = hs * fmin2(N(2.0), 0.9 / d);
    else hs = twice_of(hs);
    if (less(rem - hs, 0.01 * hs)) hs = rem;
    return less(N(0.0), rem);
  }
};

}  // namespace rc
