// Unsteady dual-time BDF2 stage of RocketCombustor on the device (FP64, built
// with --fmad=false): the implicit_time_method 5 branch of the main loop,
// BDF2_stage / BDF2_LU_SGS (Time_BDF2.f90:4-337).  The backward Euler stage
// (implicit_time_method 3, Time_BackwardEuler.f90:4-324) runs the same
// kernels: its source term is vol/dt WA, its diagonal and right-hand side
// those of phi = 0.
//
// Per inner iteration, after the residual assembly that the steady path
// shares (timestep, reconstruction, flux_sourceterm):
//   k_bdf2_prep    every cell at once: the diagonal dd, the BDF2 right-hand
//                  side hWA - (1+phi) vol/dt WA + fixed, the cell's system
//                  matrix dU/dP dd - vol d omega/dP (Time_BDF2.f90:121-129),
//                  its equilibration, LU factors and condition estimate (the
//                  LAPACK dgesvx steps below), and the gas state the
//                  neighbours' sweeps read;
//   k_bdf2_sweep   one level of the forward or backward sweep: eight lanes
//                  per cell, each face slot's flux difference of the
//                  neighbour's increment split over two lanes, the terms added
//                  in NeighF order, then the cell's 7x7 solve with one lane per
//                  row (interchanges, triangular solves and the iterative
//                  refinement of dgerfs through warp shuffles);
//   k_bdf2_update  PA += dP, then primitve_to_conserved_variables.
// The system matrix depends on PA, dd and vol only, so both sweeps share one
// factorisation; the reference recomputes the same matrix in each sweep and
// factors it the same way, so the results are the same bits.
//
// The per-cell solve restates reference LAPACK 3.12's dgesvx('E', 'N') as
// called by advanced_linear_solve_lapack (la_math.f90:120-213): dgeequ +
// dlaqge, dgetrf with partial pivoting, dgecon (dlacn2 over triangular
// solves; only its comparison with eps matters: the reference stops there),
// dgetrs and the refinement loop of dgerfs, in the operation order of the
// netlib routines, which the CPU oracle restates too.
#include "rc_chem.cuh"
#include "rc_dev.cuh"
#include "rc_div.cuh"

namespace rc {

namespace bdf2 {
constexpr double EPS = 1.1102230246251565e-16;     // dlamch('E') = 2^-53
constexpr double SFMIN = 2.2250738585072014e-308;  // dlamch('S') = 2^-1022
constexpr double PREC = 2.220446049250313e-16;     // dlamch('P') = 2^-52
constexpr unsigned FULL = 0xffffffffu;

// gas state of a cell as a neighbour (bnb planes)
enum : int { NB_RR = 0, NB_RRC, NB_RT, NB_RCT, NB_RCP, NB_HH, NB_EK, NB_ROU, NB_ROV, NB_ROEPP, NB_H };
template <int NSP>
__host__ __device__ constexpr int nb_ry() { return NB_H + NSP; }
template <int NSP>
__host__ __device__ constexpr int nb_rct() { return NB_H + NSP + (NSP - 1); }  // recip32(Rcpcv T), as a bit pattern
template <int NSP>
__host__ __device__ constexpr int nbq() { return nb_rct<NSP>() + 1; }

// a recip32 in a slot of a double array
__device__ __forceinline__ double v_slot(unsigned v) { return __hiloint2double(0, (int)v); }
__device__ __forceinline__ unsigned slot_v(double x) { return (unsigned)__double2loint(x); }

// ---- dgesvx steps (T: T or Num, rc_num.cuh) on one row-major N x N matrix, a[r*N + c] = A(r, c)
template <int N, class T>
__device__ __forceinline__ int dgeequ(const T* a, T* r, T* c, T& rowcnd, T& colcnd,
                                      T& amax) {
  const T smlnum = SFMIN, bignum = 1.0 / SFMIN;
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = 0.0;
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = fmax2(r[i], n_abs(a[i * N + j]));
  T rcmin = bignum, rcmax = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) { rcmax = fmax2(rcmax, r[i]); rcmin = fmin2(rcmin, r[i]); }
  amax = rcmax;
  if (!nonzero(val(rcmin))) return 1;
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = 1.0 / fmin2(fmax2(r[i], smlnum), bignum);
  rowcnd = fmax2(rcmin, smlnum) / fmin2(rcmax, bignum);
#pragma unroll
  for (int j = 0; j < N; ++j) c[j] = 0.0;
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) c[j] = fmax2(c[j], n_abs(a[i * N + j]) * r[i]);
  rcmin = bignum; rcmax = 0.0;
#pragma unroll
  for (int j = 0; j < N; ++j) { rcmin = fmin2(rcmin, c[j]); rcmax = fmax2(rcmax, c[j]); }
  if (!nonzero(val(rcmin))) return 2;
#pragma unroll
  for (int j = 0; j < N; ++j) c[j] = 1.0 / fmin2(fmax2(c[j], smlnum), bignum);
  colcnd = fmax2(rcmin, smlnum) / fmin2(rcmax, bignum);
  return 0;
}
// dlaqge; returns bit 0 = rows scaled, bit 1 = columns scaled
template <int N, class T>
__device__ __forceinline__ int dlaqge(T* a, const T* r, const T* c, T rowcnd, T colcnd,
                                      T amax) {
  const double thresh = 0.1, small = SFMIN / PREC, large = 1.0 / small;
  if (val(rowcnd) >= thresh && val(amax) >= small && val(amax) <= large) {
    if (val(colcnd) >= thresh) return 0;
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < N; ++i) a[i * N + j] = c[j] * a[i * N + j];
    return 2;
  }
  if (val(colcnd) >= thresh) {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < N; ++i) a[i * N + j] = r[i] * a[i * N + j];
    return 1;
  }
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) a[i * N + j] = c[j] * r[i] * a[i * N + j];
  return 3;
}
// dgetrf (partial pivoting, unit L below the diagonal); returns 0 or the
// 1-based column of the first zero pivot
template <int N, class T>
__device__ __forceinline__ int dgetrf(T* a, int* ipiv) {
  int info = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    int jp = j;
    T m = n_abs(a[j * N + j]);
#pragma unroll
    for (int i = j + 1; i < N; ++i)
      if (less(m, n_abs(a[i * N + j]))) { jp = i; m = n_abs(a[i * N + j]); }
    ipiv[j] = jp;
    if (nonzero(val(a[jp * N + j]))) {
      if (jp != j) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
          const T t = a[j * N + k];
          a[j * N + k] = a[jp * N + k];
          a[jp * N + k] = t;
        }
      }
      if (j < N - 1) {
        if (!less(n_abs(a[j * N + j]), T(SFMIN))) {
          const T rp = 1.0 / a[j * N + j];
#pragma unroll
          for (int i = j + 1; i < N; ++i) a[i * N + j] = rp * a[i * N + j];
        } else {
#pragma unroll
          for (int i = j + 1; i < N; ++i) a[i * N + j] = a[i * N + j] / a[j * N + j];
        }
      }
    } else if (info == 0) {
      info = j + 1;
    }
#pragma unroll
    for (int jj = j + 1; jj < N; ++jj) {
      if (nonzero(val(a[j * N + jj]))) {
        const T temp = -a[j * N + jj];
#pragma unroll
        for (int i = j + 1; i < N; ++i) a[i * N + jj] = a[i * N + jj] + a[i * N + j] * temp;
      }
    }
  }
  return info;
}
// x >= 0.0
template <class T>
__device__ __forceinline__ bool nonneg(T x) {
  const long long b = dbits(val(x));
  return b >= 0 ? b <= 0x7ff0000000000000LL : (b << 1) == 0;
}
// the triangular solves of dgecon (uv: recip32 of U's diagonal): kase 1 inv(L) then inv(U), kase 2 inv(U^T) then inv(L^T)
template <int N, class T>
__device__ __forceinline__ void trs_kase(const T* af, const unsigned* uv, int kase, T* x) {
  if (kase == 1) {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (nonzero(val(x[j]))) {
        const T temp = x[j];
#pragma unroll
        for (int i = j + 1; i < N; ++i) x[i] = x[i] - temp * af[i * N + j];
      }
#pragma unroll
    for (int j = N - 1; j >= 0; --j)
      if (nonzero(val(x[j]))) {
        x[j] = rcs::div_by(val(x[j]), val(af[j * N + j]), uv[j]);
        const T temp = x[j];
#pragma unroll
        for (int i = j - 1; i >= 0; --i) x[i] = x[i] - temp * af[i * N + j];
      }
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      T temp = x[j];
#pragma unroll
      for (int i = 0; i < j; ++i) temp = temp - af[i * N + j] * x[i];
      x[j] = rcs::div_by(val(temp), val(af[j * N + j]), uv[j]);
    }
#pragma unroll
    for (int j = N - 1; j >= 0; --j) {
      T temp = x[j];
#pragma unroll
      for (int i = N - 1; i > j; --i) temp = temp - af[i * N + j] * x[i];
      x[j] = temp;
    }
  }
}
template <int N, class T>
__device__ __forceinline__ T dasum(const T* x) {
  T t = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) t = t + n_abs(x[i]);
  return t;
}
template <int N, class T>
__device__ __forceinline__ int idamax(const T* x) {
  int k = 0;
  T m = n_abs(x[0]);
#pragma unroll
  for (int i = 1; i < N; ++i)
    if (less(m, n_abs(x[i]))) { k = i; m = n_abs(x[i]); }
  return k;
}
// dgecon('1') with dlacn2 (at most 5 iterations) unrolled
template <int N, class T>
__device__ T dgecon(const T* af, const unsigned* uv, T anorm) {
  if (!nonzero(val(anorm))) return 0.0;
  if (isnan(val(anorm))) return anorm;
  T x[N], est, estold;
  int isgn[N];
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = 1.0 / (double)N;
  trs_kase<N>(af, uv, 1, x);
  if (N == 1) {
    est = n_abs(x[0]);
  } else {
    est = dasum<N>(x);
#pragma unroll
    for (int i = 0; i < N; ++i) { isgn[i] = nonneg(x[i]) ? 1 : -1; x[i] = nonneg(x[i]) ? 1.0 : -1.0; }
    trs_kase<N>(af, uv, 2, x);
    int j = idamax<N>(x), iter = 2;
    for (int guard = 0; guard < 8; ++guard) {
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = (i == j) ? 1.0 : 0.0;
      trs_kase<N>(af, uv, 1, x);
      estold = est;
      est = dasum<N>(x);
      bool same = true;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if ((nonneg(x[i]) ? 1 : -1) != isgn[i]) same = false;
      if (same || val(est) <= val(estold)) break;
#pragma unroll
      for (int i = 0; i < N; ++i) { isgn[i] = nonneg(x[i]) ? 1 : -1; x[i] = nonneg(x[i]) ? 1.0 : -1.0; }
      trs_kase<N>(af, uv, 2, x);
      const int jlast = j;
      j = idamax<N>(x);
      T xl = 0.0;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i == jlast) xl = x[i];
      T xj = 0.0;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i == j) xj = x[i];
      if (val(xl) != val(n_abs(xj)) && iter < 5) { iter = iter + 1; continue; }
      break;
    }
    double altsgn = 1.0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = altsgn * (1.0 + (double)i / (double)(N - 1));
      altsgn = -altsgn;
    }
    trs_kase<N>(af, uv, 1, x);
    const T temp = twice_of(dasum<N>(x) / T((double)(3 * N)));
    if (less(est, temp)) est = temp;
  }
  if (nonzero(val(est))) return (1.0 / est) / anorm;
  return 0.0;
}

}  // namespace bdf2

// fixed = vol/dt ((1+2 phi) WP - phi WP2) (Time_BDF2.f90:88-92), or for
// backward Euler vol/dt WA (Time_BackwardEuler.f90:75-79)
template <int NSP>
__global__ void __launch_bounds__(128) k_bdf2_fixed(const Dev d, int euler) {
  constexpr int V = 3 + NSP;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.NE) return;
  const int NE = d.NE;
  const double dt = d.bpar[0], phi = d.bpar[1];
  const double vd = d.vol[i] / dt;
#pragma unroll
  for (int k = 0; k < V; ++k)
    d.bfix[k * NE + i] = euler ? vd * d.WA[k * NE + i]
                               : vd * ((1 + 2 * phi) * d.WP[k * NE + i] - phi * d.WP2[k * NE + i]);
}

// Everything of BDF2_LU_SGS that the sweeps do not change, one thread per cell.
// FP64 throughput bounds it: the divisions, comparisons and halvings run on the
// integer pipes (Num).
template <int NSP>
__global__ void __launch_bounds__(128) k_bdf2_prep(const Dev d, const ThermoDev<NSP> th) {
  using namespace bdf2;
  using N = Num<false>;
  constexpr int V = 3 + NSP, RW = 2 * V + 3;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.NE) return;
  const int NE = d.NE;
  const N dt = d.bpar[0], phi = d.bpar[1], vol = d.vol[i];
  unsigned err = 0;
  // diagonal (Time_BDF2.f90:94-102) and right-hand side (:104-111)
  N s = 0.0;
  const int nf = d.nface[i];
  for (int q = 0; q < nf; ++q) s = s + half_of(d.alpaF[d.cface[q * NE + i]]);
  const N ddi = s + vol * (1. / N(d.step[i]) + (1. + phi) / dt);
  const N wdt = (1. + phi) * vol / dt;
#pragma unroll
  for (int k = 0; k < V; ++k)
    d.hWA[k * NE + i] = val(d.hWA[k * NE + i] - wdt * d.WA[k * NE + i] + d.bfix[k * NE + i]);
  // system matrix (:121-129)
  N pri[V];
#pragma unroll
  for (int k = 0; k < V; ++k) pri[k] = d.PA[k * NE + i];
  N a[V * V];
  N rj, Rj;
  con_to_pri_jaco<NSP>(th, pri, a, rj, Rj, err);
#pragma unroll
  for (int k = 0; k < V * V; ++k) a[k] = a[k] * ddi;
  if (NSP > 1) {
    N dw[(NSP > 1 ? NSP - 1 : 1) * V];
    dwdp<NSP>(th, pri, rj, Rj, dw);
#pragma unroll
    for (int j = 0; j < NSP - 1; ++j)
#pragma unroll
      for (int c = 0; c < V; ++c) a[(4 + j) * V + c] = a[(4 + j) * V + c] - vol * dw[j * V + c];
  }
  // dgesvx('E'): equilibrate, factor, condition estimate.  The equilibrated
  // matrix goes to the cell's record and gives its 1-norm (dlange('1')) before
  // the factorisation overwrites it in registers, so one V x V array is live
  // instead of two (the same operations as factoring a copy).
  N rs[V], cs[V], rowcnd = 0.0, colcnd = 0.0, amax = 0.0;
  int equ = 0;
  if (dgeequ<V>(a, rs, cs, rowcnd, colcnd, amax) == 0) equ = dlaqge<V>(a, rs, cs, rowcnd, colcnd, amax);
  double* m = d.bmat + (size_t)i * V * RW;
  N anorm = 0.0;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    N sum = 0.0;
#pragma unroll
    for (int r = 0; r < V; ++r) sum = sum + n_abs(a[r * V + j]);
    if (less(anorm, sum) || isnan(val(sum))) anorm = sum;
  }
#pragma unroll
  for (int r = 0; r < V; ++r)
#pragma unroll
    for (int c = 0; c < V; ++c) m[r * RW + c] = val(a[r * V + c]);
  N* af = a;
  int ipiv[V];
  const int info = dgetrf<V>(af, ipiv);
  unsigned uv[V];
#pragma unroll
  for (int r = 0; r < V; ++r) uv[r] = rcs::recip32(val(af[r * V + r]));
  if (info > 0) {
    err |= ERR_LINSOLVE;
  } else {
    if (val(dgecon<V>(af, uv, anorm)) < EPS) err |= ERR_LINSOLVE;
  }
  int src[V];
#pragma unroll
  for (int k = 0; k < V; ++k) src[k] = k;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int p = ipiv[k], t = src[k];
    src[k] = src[p];
    src[p] = t;
  }
#pragma unroll
  for (int r = 0; r < V; ++r) {
#pragma unroll
    for (int c = 0; c < V; ++c) m[r * RW + V + c] = val(af[r * V + c]);
    m[r * RW + 2 * V] = val(rs[r]);
    m[r * RW + 2 * V + 1] = val(cs[r]);
    m[r * RW + 2 * V + 2] = v_slot(uv[r]);
    d.bperm[i * 8 + r] = src[r];
  }
  d.bperm[i * 8 + 7] = equ;
  // this cell's gas state for its neighbours' sweeps (Time_BDF2.f90:145-166)
  N yy[NSP], entha[NSP], Cp, gama, Rcpcv;
#pragma unroll
  for (int k = 0; k < NSP - 1; ++k) yy[k] = pri[4 + k];
  yy[NSP - 1] = last_y<NSP>(yy);
  const N pp = pri[0], uu = pri[1], vv = pri[2], tt = pri[3];
  gas<NSP>(th, yy, tt, Cp, gama, Rcpcv, err);
  enthalpy<NSP>(th, tt, entha, err);
  const N hh = dot<NSP>(yy, entha);
  const N rct = Rcpcv * tt, rr = pp / rct, ek = half_of(uu * uu + vv * vv);
  double* nb = d.bnb;
  nb[NB_RR * NE + i] = val(rr);
  nb[NB_RRC * NE + i] = val(rr * Rcpcv);
  nb[NB_RT * NE + i] = val(rr * tt);
  nb[NB_RCT * NE + i] = val(rct);
  nb[NB_RCP * NE + i] = val(rr * Cp);
  nb[NB_HH * NE + i] = val(hh);
  nb[NB_EK * NE + i] = val(ek);
  nb[NB_ROU * NE + i] = val(rr * uu);
  nb[NB_ROV * NE + i] = val(rr * vv);
  nb[NB_ROEPP * NE + i] = val((rr * (hh + ek) - pp) + pp);
#pragma unroll
  for (int k = 0; k < NSP; ++k) nb[(NB_H + k) * NE + i] = val(entha[k]);
#pragma unroll
  for (int k = 0; k < NSP - 1; ++k) nb[(nb_ry<NSP>() + k) * NE + i] = val(rr * yy[k]);
  nb[nb_rct<NSP>() * NE + i] = v_slot(rcs::recip32(val(rct)));
  flag(d, err);
}

// What a sweep does not change, loaded before the wait for the previous level:
// the face of slot q of the cell at level position t and its neighbour's gas
// state (BSlot), and row r of the cell's factorised system (BRow).
template <int NSP>
struct BSlot {
  int j;
  bool act;
  double dx, dy, aF, uu, vv, rr, rrc, rt, rct, unormal, rou, rov, rcp, hh, ek, roepp;
  double ent[NSP], yy[NSP], ry[NSP];
  unsigned rctv;  // recip32(rct)
};
template <int NSP, bool FWD>
__device__ __forceinline__ BSlot<NSP> bslot_load(const Dev& d, int t, bool valid, int q) {
  using namespace bdf2;
  constexpr int DIR = FWD ? 0 : 1;
  const int NE = d.NE, NF = d.NF;
  BSlot<NSP> b;
  b.j = valid ? d.swj[DIR][q * NE + t] : -1;
  b.act = b.j >= 0;
  b.dx = b.dy = b.aF = b.uu = b.vv = b.rr = b.rrc = b.rt = b.rct = b.unormal = 0.0;
  b.rou = b.rov = b.rcp = b.hh = b.ek = b.roepp = 0.0;
  b.rctv = 0;
#pragma unroll
  for (int k = 0; k < NSP; ++k) { b.ent[k] = 0.0; b.yy[k] = 0.0; b.ry[k] = 0.0; }
  if (b.act) {
    const int j = b.j, fs = d.swf[DIR][q * NE + t], f = fs >= 0 ? fs : ~fs;
    b.dx = d.fvec[f];
    b.dy = d.fvec[NF + f];
    if (fs < 0) { b.dx = -b.dx; b.dy = -b.dy; }
    b.aF = d.alpaF[f];
    b.uu = d.PA[1 * NE + j];
    b.vv = d.PA[2 * NE + j];
    const double* nb = d.bnb;
    b.rr = nb[NB_RR * NE + j]; b.rrc = nb[NB_RRC * NE + j]; b.rt = nb[NB_RT * NE + j]; b.rct = nb[NB_RCT * NE + j];
    b.rctv = slot_v(nb[nb_rct<NSP>() * NE + j]);
    b.unormal = b.uu * b.dx + b.vv * b.dy;
    b.rou = nb[NB_ROU * NE + j];
    b.rov = nb[NB_ROV * NE + j];
    b.rcp = nb[NB_RCP * NE + j]; b.hh = nb[NB_HH * NE + j]; b.ek = nb[NB_EK * NE + j];
    b.roepp = nb[NB_ROEPP * NE + j];
#pragma unroll
    for (int k = 0; k < NSP; ++k) b.ent[k] = nb[(NB_H + k) * NE + j];
#pragma unroll
    for (int k = 0; k < NSP - 1; ++k) {
      b.yy[k] = d.PA[(4 + k) * NE + j];
      b.ry[k] = nb[(nb_ry<NSP>() + k) * NE + j];
    }
  }
  return b;
}
template <int NSP>
struct BRow {
  double arow[3 + NSP], lrow[3 + NSP], ukk[3 + NSP], rsc, csc;
  unsigned urv[3 + NSP];  // recip32(ukk)
  int src, equ;
};
template <int NSP>
__device__ __forceinline__ BRow<NSP> brow_load(const Dev& d, int i, bool valid, int r) {
  constexpr int V = 3 + NSP, RW = 2 * V + 3;
  BRow<NSP> w;
  w.rsc = 1.0; w.csc = 1.0; w.src = 0; w.equ = 0;
#pragma unroll
  for (int k = 0; k < V; ++k) { w.arow[k] = 0.0; w.lrow[k] = 0.0; w.ukk[k] = 1.0; w.urv[k] = 0; }
  if (valid) {
    const double* m = d.bmat + (size_t)i * V * RW;
    if (r < V) {
#pragma unroll
      for (int k = 0; k < V; ++k) { w.arow[k] = m[r * RW + k]; w.lrow[k] = m[r * RW + V + k]; }
      w.rsc = m[r * RW + 2 * V];
      w.csc = m[r * RW + 2 * V + 1];
      w.src = d.bperm[i * 8 + r];
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      w.ukk[k] = m[k * RW + V + k];
      w.urv[k] = bdf2::slot_v(m[k * RW + 2 * V + 2]);
    }
    w.equ = d.bperm[i * 8 + 7];
  }
  return w;
}
// A lane's record in shared memory, word w of lane l at [32 w + l]: a warp
// moves a word without bank conflicts, and reads only the words it uses (as
// an array of records of about 560 bytes the words met in two banks of the 32).
template <class S>
__device__ __forceinline__ void stage_put(double* sm, const S& s) {
  static_assert(sizeof(S) % 8 == 0, "whole words");
  double w[sizeof(S) / 8];
  memcpy(w, &s, sizeof(S));
#pragma unroll
  for (int k = 0; k < (int)(sizeof(S) / 8); ++k) sm[32 * k + (threadIdx.x & 31)] = w[k];
}
template <class S>
__device__ __forceinline__ S stage_get(const double* sm) {
  double w[sizeof(S) / 8];
#pragma unroll
  for (int k = 0; k < (int)(sizeof(S) / 8); ++k) w[k] = sm[32 * k + (threadIdx.x & 31)];
  S s;
  memcpy(&s, w, sizeof(S));
  return s;
}
// This lane's row in such a record (w: its first word of this lane).
template <int NSP>
struct BRowRef {
  static constexpr int V = 3 + NSP;
  static_assert(offsetof(BRow<NSP>, lrow) == 8 * V && offsetof(BRow<NSP>, ukk) == 16 * V &&
                    offsetof(BRow<NSP>, rsc) == 24 * V && offsetof(BRow<NSP>, urv) == 24 * V + 16 &&
                    offsetof(BRow<NSP>, src) == 24 * V + 16 + 4 * V,
                "words");
  const double* w;
  __device__ __forceinline__ double arow(int k) const { return w[32 * k]; }
  __device__ __forceinline__ double lrow(int k) const { return w[32 * (V + k)]; }
  __device__ __forceinline__ double ukk(int k) const { return w[32 * (2 * V + k)]; }
  __device__ __forceinline__ double rsc() const { return w[32 * 3 * V]; }
  __device__ __forceinline__ double csc() const { return w[32 * (3 * V + 1)]; }
  __device__ __forceinline__ unsigned half(int h) const {  // 32-bit word h after csc
    return reinterpret_cast<const unsigned*>(w + 32 * (3 * V + 2 + (h >> 1)))[h & 1];
  }
  __device__ __forceinline__ unsigned urv(int k) const { return half(k); }
  __device__ __forceinline__ int src() const { return (int)half(V); }
  __device__ __forceinline__ int equ() const { return (int)half(V + 1); }
};
// x: this row's right-hand side (already row-scaled); returns A^-1 x for this
// row (dgetrs('N')): the composed interchanges, then the column-oriented unit
// lower and upper solves of dtrsm, skipping zero entries as dtrsm does.  The
// divisions by the diagonal of U use its reciprocals (rcs::div_by: the same
// bits as the IEEE division).
template <int NSP>
__device__ __forceinline__ double getrs_rows(double x, const BRowRef<NSP>& rw, int r, int base) {
  constexpr int N = 3 + NSP;
  x = __shfl_sync(bdf2::FULL, x, base + rw.src());
#pragma unroll
  for (int k = 0; k < N - 1; ++k) {
    const double lu = rw.lrow(k);
    const double xk = __shfl_sync(bdf2::FULL, x, base + k);
    if (r > k && r < N && nonzero(xk)) x = x - xk * lu;
  }
#pragma unroll
  for (int k = N - 1; k >= 0; --k) {
    const double lu = rw.lrow(k), u = rw.ukk(k);
    const unsigned v = rw.urv(k);
    double xk = __shfl_sync(bdf2::FULL, x, base + k);
    if (nonzero(xk)) {
      xk = rcs::div_by(xk, u, v);
      if (r == k) x = xk;
      else if (r < k) x = x - xk * lu;
    }
  }
  return x;
}
// The flux difference of slot b's neighbour increment dP (Time_BDF2.f90:168-197),
// rows 1-3 (lo) or rows 4.. (energy and species) of the slot's terms.
// L2: the neighbour's increment read through L2 (ld.global.cg), as the
// dataflow launch needs (other SMs write it during the launch).
template <int NSP, bool L2 = false>
__device__ __forceinline__ void bslot_terms(const Dev& d, const ThermoDev<NSP>& th, const BSlot<NSP>& b, bool lo,
                                            double* c) {
  constexpr int V = 3 + NSP;
  const int NE = d.NE;
  auto ld = [](const double* p) { return L2 ? __ldcg(p) : *p; };
#pragma unroll
  for (int k = 0; k < V; ++k) c[k] = 0.0;
  if (!b.act) return;
  const int j = b.j;
  const double dpp = ld(d.hWA + 0 * NE + j), duu = ld(d.hWA + 1 * NE + j), dvv = ld(d.hWA + 2 * NE + j),
               dtt = ld(d.hWA + 3 * NE + j);
  double dyy[NSP], s = 0.0;
#pragma unroll
  for (int k = 0; k < NSP - 1; ++k) { dyy[k] = ld(d.hWA + (4 + k) * NE + j); s = s + dyy[k]; }
  dyy[NSP - 1] = -s;
  double s1 = 0.0;
#pragma unroll
  for (int k = 0; k < NSP; ++k) s1 = s1 + th.R[k] * dyy[k];
  const double drr = rcs::div_by(dpp - b.rrc * dtt - b.rt * s1, b.rct, b.rctv);
  const double dunormal = duu * b.dx + dvv * b.dy;
  const double aF = b.aF, unormal = b.unormal, rr = b.rr;
  if (lo) {
    const double dru = rr * duu + b.uu * drr;
    const double drv = rr * dvv + b.vv * drr;
    c[0] = half_of(-aF * drr + dru * b.dx + drv * b.dy);
    c[1] = half_of(-aF * dru + dru * unormal + b.rou * dunormal + dpp * b.dx);
    c[2] = half_of(-aF * drv + drv * unormal + b.rov * dunormal + dpp * b.dy);
  } else {
    double s2 = 0.0;
#pragma unroll
    for (int k = 0; k < NSP; ++k) s2 = s2 + b.ent[k] * dyy[k];
    const double dre = b.rcp * dtt + rr * s2 + b.hh * drr + rr * (b.uu * duu + b.vv * dvv) + b.ek * drr - dpp;
    c[3] = half_of(-aF * dre + dunormal * b.roepp + unormal * (dre + dpp));
#pragma unroll
    for (int k = 0; k < NSP - 1; ++k) {
      const double dry = rr * dyy[k] + b.yy[k] * drr;
      c[4 + k] = half_of(-aF * dry + dry * unormal + b.ry[k] * dunormal);
    }
  }
}
template <int NSP>
__device__ __forceinline__ void bslot_put(double* w, bool lo, int q, const double* c) {
  constexpr int V = 3 + NSP;
  if (lo) {
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k * 4 + q] = c[k];
  } else {
#pragma unroll
    for (int k = 3; k < V; ++k) w[k * 4 + q] = c[k];
  }
}
// the backward error of one refinement pass over a cell's rows (8 lanes):
// max over the rows of |y| / w (or the guarded form), as a bit pattern.  A cell
// that is done (go false; its result is not used) and a row whose residual is
// zero divide nothing: rcs::div leaves a zero to the hardware's division,
// and one lane that takes it holds up the warp.
template <int V>
__device__ __forceinline__ long long berr_bits(double y, double wk, int r, bool go) {
  using namespace bdf2;
  const double safe1 = (V + 1) * SFMIN, safe2 = safe1 / EPS;
  long long vb = 0;
  const bool plain = dbits(wk) > dbits(safe2);
  if (r < V && go && (nonzero(y) || !plain || isnan(wk)))
    vb = dbits(plain ? rcs::div(fabs(y), wk) : (fabs(y) + safe1) / (wk + safe1));
  vb = max(vb, (long long)__shfl_xor_sync(FULL, (unsigned long long)vb, 1));
  vb = max(vb, (long long)__shfl_xor_sync(FULL, (unsigned long long)vb, 2));
  vb = max(vb, (long long)__shfl_xor_sync(FULL, (unsigned long long)vb, 4));
  return vb;
}

// The sweep step of up to four cells on one warp, eight lanes per cell (lane
// = 8 cell + r; lanes of cell slots >= CPW only join the shuffles): the flux
// differences of the neighbours' increments (sp: this lane's slot, q = r % 4,
// rows 1-3 on lanes r < 4, rows 4.. on the others), added in NeighF order
// through w (this warp's [cell][row][slot] scratch), then the cell's system
// (rw: row r of its factorisation) solved with one lane per row and refined
// as dgerfs does; hown is the cell's own increment (row r), i its index.
// part 0: the whole step on this warp.  part 1 and 2: two warps (warp 0 and
// warp 1 of the block) on the same cells, part 1 forming rows 1-3 of every
// slot's terms, part 2 rows 4..; they meet at named barrier 6 (64 threads),
// after which part 1 solves and part 2 returns.  The terms, their places in w
// and the sums are the same in every part.
// part and fwd are arguments, and the first solve and the corrections one
// loop, so that every pass runs the same instructions: they have to come
// from the instruction cache, and a pass runs each of them only a few times.
template <int NSP, int CPW, bool L2>
__device__ __forceinline__ void bdf2_cell_step(const Dev& d, const ThermoDev<NSP>& th, const BSlot<NSP>& sp,
                                               const BRowRef<NSP>& rw, bool fwd, int part, double hown, int i,
                                               bool valid, double* wsm) {
  using namespace bdf2;
  constexpr int V = 3 + NSP;
  const int lane = threadIdx.x & 31, cell = lane >> 3, r = lane & 7, base = cell * 8;
  const int q = r & 3;
  // part 0: lanes 0-3 keep flux rows 1-3 of their slot, lanes 4-7 rows 4..
  // (energy, species); part 1 / 2: all lanes the one half, lanes 0-3 store it
  const bool lo = part == 0 ? r < 4 : part == 1;
  const int NE = d.NE;
  double c[V];
  bslot_terms<NSP, L2>(d, th, sp, lo, c);
  double* w = wsm + (cell < CPW ? cell : 0) * V * 4;  // [row][slot]
  if (cell < CPW && (part == 0 || r < 4)) bslot_put<NSP>(w, lo, q, c);
  __syncwarp();
  if (part == 2) {
    bar_arrive(6, 64);
    return;
  }
  if (part == 1) bar_named(6, 64);
  double dflux = 0.0;
  if (r < V) {
#pragma unroll
    for (int sl = 0; sl < 4; ++sl) dflux = dflux + w[r * 4 + sl];
  }
  // --- the cell's system, one row per lane (dgesvx after the factorisation)
  const int equ = rw.equ();
  const bool rowequ = equ & 1, colequ = equ & 2;
  double b = fwd ? hown - dflux : dflux;
  if (rowequ) b = rw.rsc() * b;
  if (!(valid && r < V)) b = 0.0;
  // the solve, then dgerfs refinement: residual, componentwise backward error,
  // correction.  The backward error is non-negative: its maximum and the loop
  // tests compare bit patterns; 2 berr <= lstres is berr <= lstres/2 (both exact).
  double x = 0.0, y = b;
  long long lstres_half = dbits(1.5);  // lstres = 3
  bool go = valid;
#pragma unroll 1
  for (int it = 0;; ++it) {
    const double xi = getrs_rows<NSP>(y, rw, r, base);
    if (it == 0) x = xi;
    else if (go) x = x + xi;
    // y = b - A x and w = |b| + |A| |x| on the same products (rounding is
    // symmetric: (-x) a = -(x a) and |a| |x| = |x a|)
    double wk = fabs(b);
    y = b;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const double p = __shfl_sync(FULL, x, base + k) * rw.arow(k);
      y = y - p;
      wk = wk + fabs(p);
    }
    const long long vb = berr_bits<V>(y, wk, r, go);
    // a cell that goes on has made `it` corrections
    go = go && vb > dbits(EPS) && vb <= lstres_half && it < 5;
    if (!__any_sync(FULL, go)) break;
    lstres_half = vb - (1LL << 52);  // berr / 2: berr > eps is a normal number (unused once go is false)
  }
  if (colequ) x = rw.csc() * x;
  if (valid && r < V) d.hWA[r * NE + i] = fwd ? x : hown - x;
}

// One level of the forward (FWD) or backward sweep, cells t0..t1-1 of the
// level order; eight lanes per cell, CPW cells per warp (one warp per block;
// lanes of cell slots >= CPW only join the shuffles).
template <int NSP, bool FWD, int CPW>
__global__ void __launch_bounds__(32) k_bdf2_sweep(const Dev d, const ThermoDev<NSP> th, int t0, int t1) {
  using namespace bdf2;
  constexpr int V = 3 + NSP, DIR = FWD ? 0 : 1;
  static_assert(V <= 7, "one lane per row and the flags in slot 7");
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, cell = lane >> 3, r = lane & 7;
  const int q = r & 3;
  const int NE = d.NE;
  const int t = t0 + blockIdx.x * CPW + cell;
  const bool valid = cell < CPW && t < t1;
  const int i = valid ? d.swi[DIR][t] : 0;
  const BSlot<NSP> sp = bslot_load<NSP, FWD>(d, t, valid, q);
  const BRow<NSP> rw = brow_load<NSP>(d, i, valid, r);
  double hown = 0.0;
  if (FWD && valid && r < V) hown = d.hWA[r * NE + i];  // written by k_bdf2_prep, complete before this grid
  pdl_wait();
  if (!FWD && valid && r < V) hown = d.hWA[r * NE + i];
  __shared__ double wsm[CPW * V * 4];
  __shared__ double s_row[32 * sizeof(BRow<NSP>) / 8];
  stage_put(s_row, rw);  // each lane reads its own
  bdf2_cell_step<NSP, CPW, false>(d, th, sp, BRowRef<NSP>{s_row + lane}, FWD, 0, hown, i, valid, wsm);
}

// Both BDF2 sweeps as one cooperative dataflow launch on the pass tables of
// k_lusgs_flow (FlowDev with passes of up to 8 consecutive positions of one
// level owned by one block; one block per SM).  A cell's step is long (two
// 7 x 7 solves and up to five refinement passes, about 12 us of dependent
// FP64) and uneven: with one launch per level every level lasts as long as
// its slowest cell, here a slow cell holds up only the passes that read it.
// Warps 0 and 1 take four cells of each pass each.  Warps 3 and 4 stage one
// pass ahead what the sweep does not change (the slot data, the cell's
// factorised rows, its index and, forward, its right-hand side) in a double
// buffer of shared memory, for warp 0 and warp 1 respectively, and arrive on
// barrier 5.  Warp 2 looks at the flags of the next pass; once the current
// pass is done (barrier 4) and the next one is staged (barrier 5) it hands
// the next one over (barrier 3, which the staging warps also wait on before
// they refill the other buffer), and it publishes the finished pass (flag =
// this launch's epoch) before any blocking wait.  s_go[k % 2] = 0 after a
// bounded wait gave up (ERR_SYNC): the compute warps then skip the pass.  The
// last block to finish advances the epoch counter; the primitive update
// follows as its own launch.
struct BTail {
  double hown;
  int i, valid;
};
template <int NSP>
struct BStage {
  BSlot<NSP> sp;
  BRow<NSP> rw;
  BTail t;
};
// A pass is one chain: per cell, of about 22,000 cycles, the record 2,500, the
// terms with the neighbours' increments from L2 4,200, the solve 6,600, a check of
// the backward error 2,700 (3,300 with the hardware's division for zero residuals
// and finished cells, see berr_bits), the correction's solve 4,500.  An inner
// iteration on 120,000 cells: 10.2 -> 8.6 ms with that, the divisions by shared
// reciprocals and the records by word.
// A pass of at most four cells runs on both compute warps split by rows
// (bdf2_cell_step, part 1 and 2), otherwise four cells on each (part 0).
constexpr int BFLOW_THREADS = 160, BFLOW_NB = 96;  // all five warps; a role pair and the coordinator
template <int NSP>
constexpr int bflow_smem() { return (int)(2 * 2 * 32 * sizeof(BStage<NSP>)); }
template <int NSP>
__global__ void __launch_bounds__(BFLOW_THREADS, 1) k_bdf2_flow(const Dev d, const ThermoDev<NSP> th, const FlowDev f) {
  using namespace bdf2;
  constexpr int V = 3 + NSP;
  static_assert(V <= 7, "one lane per row and the flags in slot 7");
  extern __shared__ __align__(16) uint8_t bflow_smem_raw[];
  auto buffer = [&](int k, int w) {  // the record of pass k for compute warp w
    return reinterpret_cast<double*>(bflow_smem_raw) + ((k & 1) * 2 + w) * (int)(4 * sizeof(BStage<NSP>));
  };
  __shared__ double wsm[2][4 * V * 4];
  __shared__ unsigned s_epoch;
  __shared__ volatile int s_bad, s_go[2], s_split[2];
  if (threadIdx.x == 0) {
    s_epoch = ld_acquire(f.ctr) + 1u;
    s_bad = 0;
    s_go[0] = 0;
    s_go[1] = 0;
  }
  __syncthreads();
  const unsigned epoch = s_epoch;
  const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int f0 = f.boff[0][b], b0 = f.boff[1][b];
  const int nf = f.boff[0][b + 1] - f0, n = nf + (f.boff[1][b + 1] - b0);
  auto pass_of = [&](int k) { return k < nf ? f.blist[0][f0 + k] : f.blist[1][b0 + k - nf]; };
  const int cell = lane >> 3, r = lane & 7, q = r & 3;
  if (warp == 2) {
    auto poll = [&](int k) {
      if (s_bad) return;
      const int pz = pass_of(k), d0 = f.doff[pz], nd = f.doff[pz + 1] - d0;
      bool ok = true;
      for (int u = lane; u < nd; u += 32) ok = ok && wait_flag(f.pflag + f.deps[d0 + u], epoch, d.err, d.spin_limit);
      if (__any_sync(FULL, !ok) && lane == 0) s_bad = 1;
      __syncwarp();
    };
    auto ready = [&](int k) -> bool {
      if (s_bad) return true;
      const int pz = pass_of(k), d0 = f.doff[pz], nd = f.doff[pz + 1] - d0;
      bool ok = true;
      for (int u = lane; u < nd; u += 32) ok = ok && ld_acquire(f.pflag + f.deps[d0 + u]) >= epoch;
      return __all_sync(FULL, ok) != 0;
    };
    // pass k is staged (barrier 5), then handed over (barrier 3)
    auto hand_over = [&](int k) {
      bar_named(5, BFLOW_NB);
      if (lane == 0) s_go[k & 1] = s_bad ? 0 : 1;
      __syncwarp();
      __threadfence_block();
      bar_arrive(3, BFLOW_THREADS);
    };
    if (n > 0) {
      poll(0);
      hand_over(0);
    }
    for (int k = 0; k < n; ++k) {
      const bool more = k + 1 < n;
      const bool go = more && ready(k + 1);
      bar_named(4, BFLOW_NB);
      if (go) hand_over(k + 1);
      if (lane == 0 && !s_bad) st_release(f.pflag + pass_of(k), epoch);
      if (more && !go) {
        poll(k + 1);
        hand_over(k + 1);
      }
    }
  } else if (warp >= 3) {
    const int w = warp - 3;  // stages for compute warp w
    auto stage = [&](int k) {
      const bool fwd = k < nf;
      const int pz = pass_of(k), t0 = f.pstart[pz], t1 = t0 + f.pcount[pz];
      const bool split = t1 - t0 <= 4;  // both compute warps on cells t0 .. t0 + 3
      const int t = t0 + (split ? 0 : 4 * w) + cell;
      const bool valid = t < t1;
      if (w == 0 && lane == 0) s_split[k & 1] = split ? 1 : 0;
      const int i = valid ? d.swi[fwd ? 0 : 1][t] : 0;
      BStage<NSP> e;
      e.sp = fwd ? bslot_load<NSP, true>(d, t, valid, q) : bslot_load<NSP, false>(d, t, valid, q);
      e.rw = brow_load<NSP>(d, i, valid, r);
      // forward: the set-up's right-hand side, which only this cell's own
      // forward step changes
      e.t.hown = fwd && valid && r < V ? __ldcg(d.hWA + r * d.NE + i) : 0.0;
      e.t.i = i;
      e.t.valid = valid ? 1 : 0;
      stage_put(buffer(k, w), e);
      __syncwarp();
      __threadfence_block();
      bar_arrive(5, BFLOW_NB);
    };
    if (n > 0) stage(0);
    for (int k = 0; k < n; ++k) {
      bar_named(3, BFLOW_THREADS);  // pass k handed over: the other buffer is free
      if (k + 1 < n) stage(k + 1);
    }
  } else {
    for (int k = 0; k < n; ++k) {
      const bool fwd = k < nf;
      bar_named(3, BFLOW_THREADS);
      const double* rec = buffer(k, warp);
      const BRowRef<NSP> rw = {rec + 4 * offsetof(BStage<NSP>, rw) + lane};
      const BTail t = stage_get<BTail>(rec + 4 * offsetof(BStage<NSP>, t));
      const int i = t.i;
      const bool valid = t.valid != 0;
      // backward: the cell's own increment, as this block's forward pass of
      // the cell wrote it (read after the hand-over: the other warp may have
      // been finishing the forward pass that holds the same cell)
      const double hown = fwd ? t.hown : valid && r < V ? __ldcg(d.hWA + r * d.NE + i) : 0.0;
      if (s_go[k & 1]) {
        // both warps on the same cells, or four cells each
        const bool split = s_split[k & 1] != 0;
        bdf2_cell_step<NSP, 4, true>(d, th, stage_get<BSlot<NSP>>(rec + 4 * offsetof(BStage<NSP>, sp)), rw, fwd,
                                     split ? 1 + warp : 0, hown, i, valid, split ? wsm[0] : wsm[warp]);
      }
      __syncwarp();
      bar_arrive(4, BFLOW_NB);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(f.ctr + 1, 1u) == gridDim.x - 1) {
      f.ctr[1] = 0u;
      __threadfence();
      st_release(f.ctr, epoch);
    }
  }
}

// PA += dP, then primitve_to_conserved_variables (update_flow_variables.f90:50-84)
template <int NSP>
__global__ void __launch_bounds__(128) k_bdf2_update(const Dev d, const ThermoDev<NSP> th) {
  constexpr int V = 3 + NSP;
  using N = Num<false>;
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.NE) return;
  const int NE = d.NE;
  unsigned err = 0;
  N P[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    P[k] = d.PA[k * NE + i] + d.hWA[k * NE + i];
    d.PA[k * NE + i] = val(P[k]);
  }
  N yy[NSP], entha[NSP], Cp, gama, Rcpcv;
#pragma unroll
  for (int k = 0; k < NSP - 1; ++k) yy[k] = P[4 + k];
  yy[NSP - 1] = last_y<NSP>(yy);
  const N pp = P[0], uu = P[1], vv = P[2], tt = P[3];
  gas<NSP>(th, yy, tt, Cp, gama, Rcpcv, err);
  const N rr = pp / (Rcpcv * tt);
  enthalpy<NSP>(th, tt, entha, err);
  const N hh = dot<NSP>(yy, entha);
  d.WA[0 * NE + i] = val(rr);
  d.WA[1 * NE + i] = val(rr * uu);
  d.WA[2 * NE + i] = val(rr * vv);
  d.WA[3 * NE + i] = val(rr * (hh + half_of(uu * uu + vv * vv)) - pp);
#pragma unroll
  for (int k = 0; k < NSP - 1; ++k) d.WA[(4 + k) * NE + i] = val(rr * yy[k]);
  if (i == 0 && isnan(val(rr))) err |= ERR_NAN;
  flag(d, err);
}

inline unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

template <int NSP>
void bdf2_fixed(const Dev& d, int bs, int euler, cudaStream_t s) {
  k_bdf2_fixed<NSP><<<nblk(d.NE, bs), bs, 0, s>>>(d, euler);
}
template <int NSP>
void bdf2_prep(const Dev& d, const void* th, int bs, cudaStream_t s) {
  k_bdf2_prep<NSP><<<nblk(d.NE, bs), bs, 0, s>>>(d, *static_cast<const ThermoDev<NSP>*>(th));
}
template <int NSP, int CPW>
void bdf2_sweep_cpw(const Dev& d, const ThermoDev<NSP>& T, bool fwd, int t0, int t1, cudaStream_t s) {
  if (fwd) launch_pdl(k_bdf2_sweep<NSP, true, CPW>, nblk(t1 - t0, CPW), 32, s, d, T, t0, t1);
  else launch_pdl(k_bdf2_sweep<NSP, false, CPW>, nblk(t1 - t0, CPW), 32, s, d, T, t0, t1);
}
template <int NSP>
void bdf2_sweep(const Dev& d, const void* th, bool fwd, int t0, int t1, int cpw, cudaStream_t s) {
  const auto& T = *static_cast<const ThermoDev<NSP>*>(th);
  if (cpw >= 4) bdf2_sweep_cpw<NSP, 4>(d, T, fwd, t0, t1, s);
  else if (cpw == 2) bdf2_sweep_cpw<NSP, 2>(d, T, fwd, t0, t1, s);
  else bdf2_sweep_cpw<NSP, 1>(d, T, fwd, t0, t1, s);
}
// the cooperative dataflow launch of both sweeps (grid: one block per SM)
template <int NSP>
cudaError_t bdf2_flow(const Dev& d, const void* th, const FlowDev& f, int grid, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(BFLOW_THREADS);
  cfg.dynamicSmemBytes = (size_t)bflow_smem<NSP>();
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_bdf2_flow<NSP>, d, *static_cast<const ThermoDev<NSP>*>(th), f);
}
template <int NSP>
int bdf2_flow_occupancy() {
  int nb = 0;
  if (cudaFuncSetAttribute(k_bdf2_flow<NSP>, cudaFuncAttributeMaxDynamicSharedMemorySize, bflow_smem<NSP>()) !=
      cudaSuccess)
    return 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_bdf2_flow<NSP>, BFLOW_THREADS, bflow_smem<NSP>());
  return nb;
}
template <int NSP>
void bdf2_update(const Dev& d, const void* th, int bs, cudaStream_t s) {
  launch_pdl(k_bdf2_update<NSP>, nblk(d.NE, bs), bs, s, d, *static_cast<const ThermoDev<NSP>*>(th));
}
template <int NSP>
int bdf2_nbq() { return bdf2::nbq<NSP>(); }

#define RC_BDF2_INST(N)                                                             \
  template void bdf2_fixed<N>(const Dev&, int, int, cudaStream_t);                  \
  template void bdf2_prep<N>(const Dev&, const void*, int, cudaStream_t);           \
  template void bdf2_sweep<N>(const Dev&, const void*, bool, int, int, int, cudaStream_t); \
  template void bdf2_update<N>(const Dev&, const void*, int, cudaStream_t);         \
  template cudaError_t bdf2_flow<N>(const Dev&, const void*, const FlowDev&, int, cudaStream_t); \
  template int bdf2_flow_occupancy<N>();                                           \
  template int bdf2_nbq<N>();
RC_BDF2_INST(1)
RC_BDF2_INST(4)

}  // namespace rc
