// Finite-rate chemistry: operator-split point-implicit reaction advance, four lanes per solution node, and the
// rates alone, one thread per sample; float64 throughout.
//
// Follows the reference's hybrid/chemistry package:
//   nasa.py:47-118          NASA-7 cp/R, h/RT, s/R with T clamped to each species' range
//   mechanism.py:125-220    forward rates, Gibbs equilibrium constants, mass-action net
//                           rates with third bodies, mass-conserving correction
//   mechanism.py:262-287    T(e) damped Newton inversion
//   integrator.py:31-104    Newton on R(rho) = rho - rho0 - dt w(rho, T) with the exact
//                           Jacobian, max(., 0) clipping, T re-derived from the initial
//                           internal energy after every update, final mass rescale
//   coupling.py:116-197     per-node coupling (species renormalisation, thermal energy,
//                           dimensionless scaling)
// The reference differentiates the residual with JAX; here d w/d rho is assembled
// analytically from the reaction structure, with JAX's convention at ties of max/clip
// (the derivative is split evenly between the two arguments).
//
// Layout of the advance (k_react): four lanes per node, eight nodes per warp.  The Newton matrix and
// its right-hand side stay in registers, up to three rows a lane; a twelfth row of the same kind
// holds the mass-weighted sum over the species, which the mass-conserving correction needs.  Each
// lane evaluates every fourth reaction and writes that reaction's row [dq/drho_j | q] to shared
// memory, kPass reactions at a time; a lane then adds to its rows the reactions that they take part
// in (host-built lists, the longest rows of the four lanes side by side).  Elimination is by lanes,
// the pivot row going round by shuffles.  With a thread per node, the matrix in shared memory let five
// warps share an SM and every addition to it waited out a shared-memory round trip; now twelve warps do
// and the chains are register arithmetic: 54,000 nodes of 12 iterations took 4.7 ms before and
// take 1.6 ms.
//
// The rates alone (k_rates) take one thread per sample: the mechanism is one __grid_constant__ kernel
// parameter, and the matrix and the species vectors that the reaction loops index live in shared memory
// with a stride of one thread.
//
// Work saved against a literal evaluation, each with the same result up to rounding:
//  - a reaction whose stoichiometric coefficients are all whole numbers up to 3 forms
//    prod C^nu by multiplication instead of exp(sum nu log C) (the clip at |.| = 700 is
//    applied to the product);
//  - the temperature inversion stops once an update moves T by at most 1e-13 T: Newton on
//    e(T) converges quadratically, so the remaining iterations of the fixed count change T
//    only in its last bits;
//  - in the same way a node keeps its state once a Newton iteration has moved each density by at most
//    1e-13 of it and T by at most 1e-13 T.  T is inverted after the densities, outside the Jacobian, so the iterations
//    converge linearly: an iteration shrinks the change by 1e-3 in the median and by 0.13 in the slowest hot nodes, so
//    that the remaining ones would still move a density by at most 1e-13 0.13 / 0.87 = 1.5e-14 of it, within the
//    round-off that every further iteration leaves anew.  Root mean square of a node's largest error in any density, against
//    the converged iterations in extended precision, after the stop and after all 12 (after 11 and 13): hot mixtures 1.087e-14 and
//    1.085e-14 (1.079, 1.083), at a tenth of the step 4.37e-15 and 4.40e-15, free stream 3.071e-14 and 3.073e-14,
//    behind a Mach 8 shock 1.394e-14 and 1.399e-14 (1.411, 1.406).
//    A warp stops when its eight nodes have.  Nodes whose iterations do not settle that far (I - dt J
//    ill-conditioned) run the whole count;
//  - with one temperature (T_v = T) the three controlling temperatures of a reaction, floored at 10 K,
//    are the same number (sqrt(T T) is T in binary floating point).
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "dgb200.h"

namespace dgb {
int set_error(int code, const std::string& msg);
}

namespace {

constexpr int kThreads = 32;
constexpr int kMaxList = 6;
constexpr double kClipExp = 700.0, kMinKc = 1.0e-300, kMinC = 1.0e-100;
// exp(-700) and exp(700): the clip of the mass-action exponent applied to a product
constexpr double kExpLo = 9.8597628436862264e-305, kExpHi = 1.0142320547350045e304;
// the temperature inversion's convergence test (relative step)
constexpr double kTStop = 1.0e-13;
constexpr double kRUniv = 8.31446261815324, kPStd = 101325.0;
// k_react: lanes per node, CTA size, reactions per pass, rows
constexpr int kLanes = 4, kReactThreads = 128, kPass = 8, kRows = 12;
constexpr int kPasses = (DGB_CHEM_MAX_REACTIONS + kPass - 1) / kPass;
// a node has settled once an update moves no density by more than this share of it
constexpr double kSettled = 1.0e-13;

struct Reaction {
  double A, b, theta, dn;                 // Arrhenius; sum of net stoichiometry
  int fmode, rmode, third, nf, nr, nd;    // temperature modes, third-body flag, list sizes
  int whole;                              // every nu' and nu'' a whole number in 1..3
  int f_pw[3], r_pw[3];                   // those whole numbers
  int f_sp[3], r_sp[3], d_sp[kMaxList];   // species of nu', nu'', nu''-nu' (ascending)
  double f_nu[3], r_nu[3], d_nu[kMaxList];
};

struct Tables {
  int ns, nr;
  double W[DGB_CHEM_MAX_SPECIES];             // molar mass
  double RW[DGB_CHEM_MAX_SPECIES];            // R_univ / W
  double iW[DGB_CHEM_MAX_SPECIES];            // 1 / W
  double trange[DGB_CHEM_MAX_SPECIES][3];
  double clamp_log[DGB_CHEM_MAX_SPECIES][2];  // ln t_low, ln t_high
  double clamp_inv[DGB_CHEM_MAX_SPECIES][2];  // 1 / t_low, 1 / t_high
  double cp[DGB_CHEM_MAX_SPECIES][2][5];      // a0..a4
  double h[DGB_CHEM_MAX_SPECIES][2][6];       // a0, a1/2, a2/3, a3/4, a4/5, a5
  double s[DGB_CHEM_MAX_SPECIES][2][6];       // a0, a1, a2/2, a3/3, a4/4, a6
  double alpha[DGB_CHEM_MAX_REACTIONS][DGB_CHEM_MAX_SPECIES];
  Reaction rx[DGB_CHEM_MAX_REACTIONS];
  // k_react: species of row slot * 4 + lane (-1: none, ns: the mass-weighted sum), and per pass of
  // kPass reactions the row's entries [ptr, ptr of the next row): reaction in the pass, weight
  int row_of[kRows];
  int list_ptr[kPasses * kRows + 1];
  short list_rx[DGB_CHEM_MAX_REACTIONS * (kMaxList + 1)];
  double list_w[DGB_CHEM_MAX_REACTIONS * (kMaxList + 1)];
  // coupler (coupling.py:26-71)
  int iters, dimensionless;
  double T_ref, rho_ref, e_ref, t_ref, gamma;
};

// max/min that propagate NaN like jnp.maximum/jnp.minimum
__device__ __forceinline__ double jmax(double a, double b) { return (a > b || a != a) ? a : b; }
__device__ __forceinline__ double jmin(double a, double b) { return (a < b || a != a) ? a : b; }
__device__ __forceinline__ double jclip(double x, double lo, double hi) { return jmin(jmax(x, lo), hi); }
// d max(x, c)/dx under JAX's tie rule
__device__ __forceinline__ double dmax_tie(double x, double c) { return x > c ? 1.0 : (x == c ? 0.5 : 0.0); }

template <int NS>
struct Slots {
  double* base;
  int stride;
  __device__ double& A(int i, int j) const { return base[(i * (NS + 1) + j) * stride]; }
  __device__ double& om(int q) const { return A(q, NS); }                              // net rates
  __device__ double& C(int q) const { return base[(NS * (NS + 1) + q) * stride]; }     // max(C, 1e-100)
  __device__ double& dlog(int q) const { return base[(NS * (NS + 2) + q) * stride]; }
  __device__ double& g(int q) const { return base[(NS * (NS + 3) + q) * stride]; }
  static constexpr int kDoubles = NS * (NS + 4);
};

// Temperature powers shared by every species at one temperature T: ln T and 1/T.  A species
// whose fit range clamps T uses the host-computed ln and reciprocal of its range end.
struct TPow {
  double T, lnT, invT;
};

__device__ __forceinline__ TPow tpow(double T) { return TPow{T, log(T), 1.0 / T}; }

// species q at T: T clamped to [t_low, t_high], coefficient set by T_c < t_mid
__device__ __forceinline__ int nasa_range(const Tables& M, int q, const TPow& t, double& Tc, double& lnTc,
                                          double& invTc) {
  Tc = jclip(t.T, M.trange[q][0], M.trange[q][2]);
  const bool lo = Tc == M.trange[q][0] && Tc != t.T;
  const bool hi = Tc == M.trange[q][2] && Tc != t.T;
  lnTc = lo ? M.clamp_log[q][0] : (hi ? M.clamp_log[q][1] : t.lnT);
  invTc = lo ? M.clamp_inv[q][0] : (hi ? M.clamp_inv[q][1] : t.invT);
  return Tc < M.trange[q][1] ? 0 : 1;
}

__device__ __forceinline__ double g_RT(const Tables& M, int q, const TPow& t) {
  double Tc, lnTc, invTc;
  const int r = nasa_range(M, q, t, Tc, lnTc, invTc);
  const double* a = M.h[q][r];
  const double* c = M.s[q][r];
  const double T2 = Tc * Tc;
  const double h = a[0] + a[1] * Tc + a[2] * T2 + a[3] * (T2 * Tc) + a[4] * (T2 * T2) + a[5] * invTc;
  const double s = c[0] * lnTc + c[1] * Tc + c[2] * T2 + c[3] * (T2 * Tc) + c[4] * (T2 * T2) + c[5];
  return h - s;
}

// mechanism.py:125-128 with Tv = T (single temperature)
__device__ __forceinline__ double select_T(int mode, double T, double Tv) {
  if (mode == 1) return sqrt(jmax(T * Tv, 1.0));
  return mode == 2 ? Tv : T;
}

// prod_k C[sp[k]]^pw[k] for whole exponents, clipped to [exp(-700), exp(700)] as the
// exponential of the summed logarithms is; ok receives d(clip)/d(arg) under JAX's tie rule.
template <int NS>
__device__ __forceinline__ double mass_action(const Slots<NS>& sl, int n, const int* sp, const int* pw, double& ok) {
  double v = 1.0;
  for (int k = 0; k < n; ++k) {
    const double c = sl.C(sp[k]);
    v *= pw[k] == 1 ? c : (pw[k] == 2 ? c * c : c * c * c);
  }
  ok = (v > kExpLo && v < kExpHi) ? 1.0 : ((v == kExpLo || v == kExpHi) ? 0.5 : 0.0);
  return jclip(v, kExpLo, kExpHi);
}

// Net rates at (rho, T): omega -> sl.om, and, when jac, sum_r dnu[r][s] dq_r/drho_j
// into sl.A(s, j) (d w/d rho before the molar-mass scaling and the mass correction).
template <int NS>
__device__ void rates(const Tables& M, const Slots<NS>& sl, const double (&rho)[NS], double T, bool jac) {
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const double craw = rho[q] * M.iW[q];
    const double c = jmax(craw, 0.0);
    const double dc = dmax_tie(craw, 0.0) * M.iW[q];
    const double cc = jmax(c, kMinC);
    sl.C(q) = cc;
    sl.dlog(q) = dmax_tie(c, kMinC) * dc / cc;
    sl.om(q) = 0.0;
  }
  const double Tg = jmax(T, 10.0);
  const TPow tg = tpow(Tg);
  const double base_g = kPStd / (kRUniv * Tg);
#pragma unroll
  for (int q = 0; q < NS; ++q) sl.g(q) = g_RT(M, q, tg);
  if (jac) {
#pragma unroll
    for (int i = 0; i < NS; ++i)
#pragma unroll
      for (int j = 0; j < NS; ++j) sl.A(i, j) = 0.0;
  }
  for (int r = 0; r < M.nr; ++r) {
    const Reaction& R = M.rx[r];
    // kf = A T^b exp(-theta/T) as A exp(b ln T - theta/T); ln T and 1/T are shared
    const double Tf = jmax(select_T(R.fmode, T, T), 10.0);
    const TPow tf = Tf == Tg ? tg : tpow(Tf);
    const double kf = R.A * exp(R.b * tf.lnT - R.theta * tf.invT);
    const double Tr = jmax(select_T(R.rmode, T, T), 10.0);
    double dG = 0.0;
    if (Tr == Tg) {
#pragma unroll 1
      for (int k = 0; k < R.nd; ++k) dG += R.d_nu[k] * sl.g(R.d_sp[k]);
    } else {
      const TPow tr = tpow(Tr);
#pragma unroll 1
      for (int k = 0; k < R.nd; ++k) dG += R.d_nu[k] * g_RT(M, R.d_sp[k], tr);
    }
    const double base = Tr == Tg ? base_g : kPStd / (kRUniv * Tr);
    const double conv = R.dn == 0.0 ? 1.0 : (R.dn == 1.0 ? base : (R.dn == -1.0 ? 1.0 / base : pow(base, R.dn)));
    const double Kc = exp(-jclip(dG, -kClipExp, kClipExp)) * conv;
    const double kr = kf / jmax(Kc, kMinKc);
    double fwd, rev, okf, okr;
    if (R.whole) {
      fwd = mass_action(sl, R.nf, R.f_sp, R.f_pw, okf);
      rev = mass_action(sl, R.nr, R.r_sp, R.r_pw, okr);
    } else {
      double lf = 0.0, lr = 0.0;
      for (int k = 0; k < R.nf; ++k) lf += R.f_nu[k] * log(sl.C(R.f_sp[k]));
      for (int k = 0; k < R.nr; ++k) lr += R.r_nu[k] * log(sl.C(R.r_sp[k]));
      fwd = exp(jclip(lf, -kClipExp, kClipExp));
      rev = exp(jclip(lr, -kClipExp, kClipExp));
      // d q / d log C_j through the clipped exponentials; the tie rule at |l| == 700
      okf = fabs(lf) < kClipExp ? 1.0 : (fabs(lf) == kClipExp ? 0.5 : 0.0);
      okr = fabs(lr) < kClipExp ? 1.0 : (fabs(lr) == kClipExp ? 0.5 : 0.0);
    }
    double coll = 1.0;
    if (R.third) {
      coll = 0.0;
#pragma unroll
      for (int q = 0; q < NS; ++q) coll += M.alpha[r][q] * jmax(rho[q] * M.iW[q], 0.0);
    }
    const double qf = kf * fwd * coll, qr = kr * rev * coll;
    const double qn = qf - qr;
    for (int k = 0; k < R.nd; ++k) sl.om(R.d_sp[k]) += R.d_nu[k] * qn;
    if (!jac) continue;
    const double a = kf * fwd * okf * coll, b = kr * rev * okr * coll;
    const double qc = kf * fwd - kr * rev;
    for (int kd = 0; kd < R.nd; ++kd) {
      const int s = R.d_sp[kd];
      const double dn = R.d_nu[kd];
      for (int m = 0; m < R.nf; ++m) {
        const int j = R.f_sp[m];
        sl.A(s, j) += dn * (a * R.f_nu[m] * sl.dlog(j));
      }
      for (int m = 0; m < R.nr; ++m) {
        const int j = R.r_sp[m];
        sl.A(s, j) -= dn * (b * R.r_nu[m] * sl.dlog(j));
      }
      if (R.third) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          const double dC = dmax_tie(rho[j] * M.iW[j], 0.0) * M.iW[j];
          sl.A(s, j) += dn * (qc * M.alpha[r][j] * dC);
        }
      }
    }
  }
}

// Mass-conserving correction (mechanism.py:214-218): w = W omega - Y sum(W omega) replaces
// omega in sl.om, and its Jacobian J = dwd - dY sum(wd) - Y colsum(dwd) replaces sl.A.
template <int NS>
__device__ void finish(const Tables& M, const Slots<NS>& sl, const double (&rho)[NS], bool jac) {
  double Sraw = 0.0;
#pragma unroll
  for (int q = 0; q < NS; ++q) Sraw += rho[q];
  const double S = jmax(Sraw, 1.0e-14);
  const double dS = dmax_tie(Sraw, 1.0e-14);
  double sw = 0.0;
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const double wd = sl.om(q) * M.W[q];
    sl.om(q) = wd;
    sw += wd;
  }
#pragma unroll
  for (int q = 0; q < NS; ++q) sl.om(q) = sl.om(q) - (jmax(rho[q], 0.0) / S) * sw;
  if (!jac) return;
  // per row: Y_i, and dY_i/drho_j off the diagonal (the diagonal adds dmax(rho_i, 0)/S)
  double Yr[NS], dYo[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    Yr[i] = jmax(rho[i], 0.0) / S;
    dYo[i] = -(jmax(rho[i], 0.0) / (S * S)) * dS;
  }
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    double col = 0.0;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      const double v = M.W[i] * sl.A(i, j);
      sl.A(i, j) = v;
      col += v;
    }
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      const double dY = i == j ? dmax_tie(rho[i], 0.0) / S + dYo[i] : dYo[i];
      sl.A(i, j) = sl.A(i, j) - dY * sw - Yr[i] * col;
    }
  }
}

// ------------------------------------------------------------------------------------ point-implicit step
// Node arrays in shared memory (doubles): the species vectors [C | dlog | c | dC | g], kRows each, then
// kPass reaction rows.  The reaction rows and the nodes are an odd number of 16-byte units apart, so that
// the lanes of a warp, which read rows of their own, spread over the banks.
constexpr int kVec = 5 * kRows, kRxRow = kRows + 2;
constexpr int kNodeDoubles = kVec + kPass * kRxRow + 2;
static_assert((kNodeDoubles / 2) % 2 == 1 && (kRxRow / 2) % 2 == 1, "odd strides");

__device__ __forceinline__ double quad_sum(double x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x;
}

// NASA-7 fits of species q at T (lnT and 1/T given): the temperature clamped to the fit's range.
__device__ __forceinline__ double species_energy(const Tables& M, int q, double T, double invT, double& cv) {
  const TPow t{T, 0.0, invT};
  double Tc, lnTc, invTc;
  const int r = nasa_range(M, q, t, Tc, lnTc, invTc);
  const double* a = M.h[q][r];
  const double* c = M.cp[q][r];
  const double T2 = Tc * Tc, T3 = T2 * Tc, T4 = T2 * T2;
  const double h = a[0] + a[1] * Tc + a[2] * T2 + a[3] * T3 + a[4] * T4 + a[5] * invTc;
  const double cp = c[0] + c[1] * Tc + c[2] * T2 + c[3] * T3 + c[4] * T4;
  cv = (cp - 1.0) * M.RW[q];
  return (h - 1.0) * (T * M.RW[q]);
}

// The species of each of a lane's rows (NS and above: none), as kept in registers.
template <int SLOTS>
struct RowSpecies {
  int q[SLOTS];
};

// recover_temperature_from_energy, mechanism.py:262-287, the species spread over the node's lanes
template <int NS, int SLOTS>
__device__ __noinline__ double recover_T(const Tables& M, const RowSpecies<SLOTS>& row, const double (&rho)[SLOTS], double target,
                            double T, int iters) {
  double S = 0.0;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) S += row.q[s] < NS ? rho[s] : 0.0;
  S = jmax(quad_sum(S), 1.0e-14);
  double Y[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) Y[s] = row.q[s] < NS ? jmax(rho[s], 0.0) / S : 0.0;
  bool done = false;
#pragma unroll 1
  for (int it = 0; it < iters; ++it) {
    const double Ts = jclip(T, 50.0, 50000.0);
    const double invT = 1.0 / Ts;
    double e = 0.0, cv = 0.0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      double c;
      const double es = species_energy(M, row.q[s] < NS ? row.q[s] : 0, Ts, invT, c);
      e += Y[s] * es;
      cv += Y[s] * c;
    }
    e = quad_sum(e);
    cv = quad_sum(cv);
    const double dT = -(e - target) / jmax(cv, 1.0e-5);
    const double Tn = jclip(T + jclip(dT, -0.5 * T, 0.5 * T), 100.0, 50000.0);
    const bool now = fabs(Tn - T) <= kTStop * T;
    if (!done) T = Tn;
    done = done || now;
    if (__all_sync(0xffffffffu, done)) break;
  }
  return T;
}

// prod_k C[sp[k]]^pw[k] from the node's concentrations, clipped as mass_action above
__device__ __forceinline__ double node_mass_action(const double* C, int n, const int* sp, const int* pw, double& ok) {
  double v = 1.0;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const double c = C[sp[k]];
    v *= pw[k] == 1 ? c : (pw[k] == 2 ? c * c : c * c * c);
  }
  ok = (v > kExpLo && v < kExpHi) ? 1.0 : ((v == kExpLo || v == kExpHi) ? 0.5 : 0.0);
  return jclip(v, kExpLo, kExpHi);
}

// The paths that whole-number mechanisms such as Air-11 do not take stay out of the kernel's code, which
// the warps stream through the instruction cache once per iteration.
__device__ __noinline__ double rare_pow(double x, double y) { return pow(x, y); }
__device__ __noinline__ double fractional_mass_action(const double* C, int n, const int* sp, const double* nu, double* ok) {
  double l = 0.0;
  for (int k = 0; k < n; ++k) l += nu[k] * log(C[sp[k]]);
  // d q / d log C_j through the clipped exponential; the tie rule at |l| == 700
  *ok = fabs(l) < kClipExp ? 1.0 : (fabs(l) == kClipExp ? 0.5 : 0.0);
  return exp(jclip(l, -kClipExp, kClipExp));
}

// Reaction r's row [dq/drho_j | q] at the node's concentrations (the vectors of node) and temperature.
template <int NS>
__device__ __forceinline__ void reaction_row(const Tables& M, int r, const double* node, const TPow& tg, double base,
                                             double* out) {
  const double *C = node, *dlog = node + kRows, *cpos = node + 2 * kRows, *dC = node + 3 * kRows, *g = node + 4 * kRows;
  const Reaction& R = M.rx[r];
  const double kf = R.A * exp(R.b * tg.lnT - R.theta * tg.invT);
  double dG = 0.0;
#pragma unroll 1
  for (int k = 0; k < R.nd; ++k) dG += R.d_nu[k] * g[R.d_sp[k]];
  const double conv = R.dn == 0.0 ? 1.0 : (R.dn == 1.0 ? base : (R.dn == -1.0 ? 1.0 / base : rare_pow(base, R.dn)));
  const double Kc = exp(-jclip(dG, -kClipExp, kClipExp)) * conv;
  const double kr = kf / jmax(Kc, kMinKc);
  double fwd, rev, okf, okr;
  if (R.whole) {
    fwd = node_mass_action(C, R.nf, R.f_sp, R.f_pw, okf);
    rev = node_mass_action(C, R.nr, R.r_sp, R.r_pw, okr);
  } else {
    fwd = fractional_mass_action(C, R.nf, R.f_sp, R.f_nu, &okf);
    rev = fractional_mass_action(C, R.nr, R.r_sp, R.r_nu, &okr);
  }
  const double F = kf * fwd, B = kr * rev;
  double coll = 1.0;
  if (R.third) {
    coll = 0.0;
#pragma unroll
    for (int q = 0; q < NS; ++q) coll += M.alpha[r][q] * cpos[q];
    const double qc = F - B;
#pragma unroll
    for (int q = 0; q < NS; ++q) out[q] = qc * M.alpha[r][q] * dC[q];
  } else {
#pragma unroll
    for (int q = 0; q < NS; ++q) out[q] = 0.0;
  }
  const double a = F * okf * coll, b = B * okr * coll;
#pragma unroll 1
  for (int m = 0; m < R.nf; ++m) out[R.f_sp[m]] += a * R.f_nu[m] * dlog[R.f_sp[m]];
#pragma unroll 1
  for (int m = 0; m < R.nr; ++m) out[R.r_sp[m]] -= b * R.r_nu[m] * dlog[R.r_sp[m]];
  out[NS] = F * coll - B * coll;
}

// ReactingFlowCoupler._react_single_cell for every node of a block.
template <int NS>
__global__ void __launch_bounds__(kReactThreads, 3)
    k_react(const __grid_constant__ Tables params, const double* U, double* out, long long nodes, int num_nodes, int nvars,
            double dt, const double* __restrict__ dt_elem) {
  constexpr int SLOTS = (NS + 1 + kLanes - 1) / kLanes, NC = NS + 1;   // rows a lane; columns with the right side
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) double smem[];
  // the mechanism in shared memory: the lanes of a node read different reactions and species
  constexpr int kTableDoubles = (int)((sizeof(Tables) + 15) / 16 * 2);
  {
    const int* src = reinterpret_cast<const int*>(&params);
    int* dst = reinterpret_cast<int*>(smem);
    for (int i = threadIdx.x; i < (int)(sizeof(Tables) / sizeof(int)); i += kReactThreads) dst[i] = src[i];
  }
  __syncthreads();
  const Tables& M = *reinterpret_cast<const Tables*>(smem);
  const int lane = threadIdx.x % kLanes;
  const long long want = ((long long)blockIdx.x * kReactThreads + threadIdx.x) / kLanes;
  const bool live = want < nodes;
  const long long n = live ? want : nodes - 1;          // spare lanes repeat the last node and store nothing
  double* node = smem + kTableDoubles + (threadIdx.x / kLanes) * kNodeDoubles;
  const double* u = U + n * nvars;
  const double step = dt_elem ? dt_elem[n / num_nodes] : dt;
  RowSpecies<SLOTS> row;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    const int q = M.row_of[s * kLanes + lane];
    row.q[s] = q < 0 ? NS + 1 : q;                       // NS: the mass-weighted sum, NS + 1: no row
  }

  const double rho_t = jmax(u[0], 1.0e-14);
  double rs[SLOTS], ssum = 0.0;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    rs[s] = row.q[s] < NS ? jmax(u[5 + row.q[s]], 0.0) : 0.0;
    ssum += rs[s];
  }
  ssum = quad_sum(ssum);
  const double scale = rho_t / jmax(ssum, 1.0e-20);
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) rs[s] *= scale;
  const double ek = 0.5 * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / (rho_t * rho_t);

  double T0, dtp, target;
  if (M.dimensionless) {
    const double es = jmax(u[4] / rho_t - ek, 1.0e-4);
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) rs[s] *= M.rho_ref;
    T0 = jmax((M.gamma - 1.0) * es * M.T_ref, 200.0);
    target = es * M.e_ref;
    dtp = step * M.t_ref;
  } else {
    target = jmax(u[4] / rho_t - ek, 1.0e3);
    T0 = 1000.0;
    dtp = step;
  }
  T0 = recover_T<NS, SLOTS>(M, row, rs, target, T0, 8);

  // PointImplicitIntegrator.step, constant_temperature=False
  double rho[SLOTS], r0[SLOTS], total = 0.0;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    rho[s] = r0[s] = row.q[s] < NS ? jmax(rs[s], 1.0e-20) : 0.0;
    total += rho[s];
  }
  total = quad_sum(total);
  double e_init = 0.0;
  {
    const double S = jmax(total, 1.0e-14), invT = 1.0 / T0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      double c;
      const double es = species_energy(M, row.q[s] < NS ? row.q[s] : 0, T0, invT, c);
      e_init += row.q[s] < NS ? (jmax(rho[s], 0.0) / S) * es : 0.0;
    }
    e_init = quad_sum(e_init);
  }
  double Tk = T0;
  bool settled = false;
#pragma unroll 1
  for (int it = 0; it < M.iters; ++it) {
    // ---- the node's species vectors
    const double Tg = jmax(Tk, 10.0);
    const TPow tg = tpow(Tg);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int q = row.q[s];
      if (q >= NS) continue;
      const double craw = rho[s] * M.iW[q];
      const double c = jmax(craw, 0.0);
      const double dC = dmax_tie(craw, 0.0) * M.iW[q];
      const double cc = jmax(c, kMinC);
      node[q] = cc;
      node[kRows + q] = dmax_tie(c, kMinC) * dC / cc;
      node[2 * kRows + q] = c;
      node[3 * kRows + q] = dC;
      node[4 * kRows + q] = g_RT(M, q, tg);
    }
    __syncwarp();
    // ---- rows of d omega/d rho and omega (last column), and their mass-weighted sum
    const double base = kPStd / (kRUniv * Tg);
    double a[SLOTS][NC];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)
#pragma unroll
      for (int j = 0; j < NC; ++j) a[s][j] = 0.0;
#pragma unroll 1
    for (int pass = 0; pass * kPass < M.nr; ++pass) {
#pragma unroll 1
      for (int r = lane; r < kPass; r += kLanes)
        if (pass * kPass + r < M.nr)
          reaction_row<NS>(M, pass * kPass + r, node, tg, base, node + kVec + r * kRxRow);
      __syncwarp();
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        const int* ptr = M.list_ptr + pass * kRows + s * kLanes + lane;
        const int end = ptr[1];
#pragma unroll 1
        for (int k = ptr[0]; k < end; ++k) {
          const double w = M.list_w[k];
          const double* x = node + kVec + M.list_rx[k] * kRxRow;
#pragma unroll
          for (int j = 0; j + 1 < NC; j += 2) {
            const double2 v = *reinterpret_cast<const double2*>(x + j);
            a[s][j] += w * v.x;
            a[s][j + 1] += w * v.y;
          }
          if (NC % 2) a[s][NC - 1] += w * x[NC - 1];
        }
      }
      __syncwarp();
    }
    // ---- mass-conserving correction and the Newton system [I - dt J | -res]
    double S = 0.0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) S += row.q[s] < NS ? rho[s] : 0.0;
    const double Sraw = quad_sum(S);
    S = jmax(Sraw, 1.0e-14);
    const double dS = dmax_tie(Sraw, 1.0e-14);
    // the mass-weighted sum is the last slot of the last lane
    double col[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) col[j] = __shfl_sync(kAll, a[SLOTS - 1][j], (threadIdx.x & 28) | (kLanes - 1));
    const double sw = col[NS];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int q = row.q[s];
      const double W = q < NS ? M.W[q] : 0.0;
      const double Y = jmax(rho[s], 0.0) / S;
      const double dYo = -(jmax(rho[s], 0.0) / (S * S)) * dS, dYd = dmax_tie(rho[s], 0.0) / S;
      const double w = W * a[s][NS] - Y * sw;
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const double dY = j == q ? dYd + dYo : dYo;
        const double J = W * a[s][j] - dY * sw - Y * col[j];
        a[s][j] = (j == q ? 1.0 : 0.0) - dtp * J;
      }
      a[s][NS] = -(rho[s] - r0[s] - dtp * w);
    }
    // ---- LU with partial pivoting: the pivot is the largest entry of the column to 16 bits of the mantissa, so that
    // one integer maximum finds value and row.  Which of two entries that agree to 1.5e-5 is the pivot enters no value:
    // the factors stay below 1 + 1.5e-5 instead of 1.  The largest by all bits took 6 % longer (54,000 nodes: 1628 ->
    // 1731 us) and left the same states bit for bit.
    unsigned used = 0;                                   // slots of this lane that have been pivot rows
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) used |= row.q[s] < NS ? 0u : 1u << s;
    unsigned long long order = 0;                        // 4 bits a column: its pivot row
#pragma unroll
    for (int k = 0; k < NS; ++k) {
      unsigned key = 0;
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        const unsigned hi = (unsigned)__double2hiint(a[s][k]) & 0x7ffffff0u;
        const unsigned mine = (used >> s) & 1 ? 0u : hi | (15u - (unsigned)(s * kLanes + lane));
        key = mine > key ? mine : key;
      }
      key = max(key, __shfl_xor_sync(kAll, key, 1));
      key = max(key, __shfl_xor_sync(kAll, key, 2));
      const int p = 15 - (int)(key & 15u), ps = p / kLanes, pl = p % kLanes;
      order |= (unsigned long long)p << (4 * k);
      double pv[NC];
#pragma unroll
      for (int j = k; j < NC; ++j) {
        double v = a[0][j];
#pragma unroll
        for (int s = 1; s < SLOTS; ++s) v = ps == s ? a[s][j] : v;
        pv[j] = __shfl_sync(kAll, v, (threadIdx.x & 28) | pl);
      }
      if (lane == pl) used |= 1u << ps;
      const double rp = 1.0 / pv[k];
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        const double f = (used >> s) & 1 ? 0.0 : a[s][k] * rp;
#pragma unroll
        for (int j = k + 1; j < NC; ++j) a[s][j] -= f * pv[j];
      }
    }
    double d[SLOTS];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) d[s] = 0.0;
#pragma unroll
    for (int k = NS - 1; k >= 0; --k) {
      const int p = (int)((order >> (4 * k)) & 15u), ps = p / kLanes, pl = p % kLanes;
      double num = a[0][NS], den = a[0][k];
#pragma unroll
      for (int s = 1; s < SLOTS; ++s) {
        num = ps == s ? a[s][NS] : num;
        den = ps == s ? a[s][k] : den;
      }
      const double x = __shfl_sync(kAll, num / den, (threadIdx.x & 28) | pl);
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        a[s][NS] -= a[s][k] * x;
        d[s] = row.q[s] == k ? x : d[s];
      }
    }
    // ---- update; a node that has settled keeps its state
    bool still = true;
    double next[SLOTS];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      next[s] = jmax(rho[s] + d[s], 0.0);
      if (row.q[s] >= NS) next[s] = 0.0;
      still = still && fabs(next[s] - rho[s]) <= kSettled * rho[s];
      if (!settled) rho[s] = next[s];
    }
    const double Tn = recover_T<NS, SLOTS>(M, row, rho, e_init, Tk, 10);
    still = still && fabs(Tn - Tk) <= kTStop * Tk;
    if (!settled) Tk = Tn;
    const unsigned votes = __ballot_sync(kAll, still) >> (threadIdx.x & 28) & 15u;
    settled = settled || votes == 15u;
    if (__all_sync(kAll, settled)) break;
  }
  double fsum = 0.0;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) fsum += row.q[s] < NS ? rho[s] : 0.0;
  const double fs = total / quad_sum(fsum);
  double nsum = 0.0;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    double v = rho[s] * fs;
    if (M.dimensionless) v = v / M.rho_ref;
    rho[s] = row.q[s] < NS ? jmax(v, 0.0) : 0.0;
    nsum += rho[s];
  }
  const double back = rho_t / jmax(quad_sum(nsum), 1.0e-20);
  if (!live) return;
  double* o = out + n * nvars;
  if (o != u) {
    for (int v = lane; v < 5; v += kLanes) o[v] = u[v];
    for (int v = 5 + NS + lane; v < nvars; v += kLanes) o[v] = u[v];
  }
#pragma unroll
  for (int s = 0; s < SLOTS; ++s)
    if (row.q[s] < NS) o[5 + row.q[s]] = rho[s] * back;
}

// ReactionMechanism.net_production_rates (and its Jacobian) for independent samples.
template <int NS>
__global__ void __launch_bounds__(kThreads) k_rates(const __grid_constant__ Tables M, const double* __restrict__ rho_in,
                                                    const double* __restrict__ T_in, long long count,
                                                    double* __restrict__ omega, double* __restrict__ wdot,
                                                    double* __restrict__ jac) {
  extern __shared__ double smem[];
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= count) return;
  const Slots<NS> sl{smem + threadIdx.x, (int)blockDim.x};
  double rho[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) rho[q] = rho_in[n * NS + q];
  const bool want = jac != nullptr;
  rates<NS>(M, sl, rho, T_in[n], want);
#pragma unroll
  for (int q = 0; q < NS; ++q)
    if (omega) omega[n * NS + q] = sl.om(q);
  finish<NS>(M, sl, rho, want);
#pragma unroll
  for (int q = 0; q < NS; ++q)
    if (wdot) wdot[n * NS + q] = sl.om(q);
  if (want) {
#pragma unroll
    for (int i = 0; i < NS; ++i)
#pragma unroll
      for (int j = 0; j < NS; ++j) jac[(n * NS + i) * NS + j] = sl.A(i, j);
  }
}

int fail(int code, const std::string& msg) { return dgb::set_error(code, msg); }

template <int NS>
size_t smem_bytes() {
  return sizeof(double) * (size_t)Slots<NS>::kDoubles * kThreads;
}

template <int NS>
int launch_react(const Tables& M, const double* U, double* out, long long nodes, int num_nodes, int nvars, double dt,
                 const double* dt_elem, cudaStream_t st) {
  constexpr int per = kReactThreads / kLanes;
  const size_t sm = (sizeof(Tables) + 15) / 16 * 16 + sizeof(double) * (size_t)per * kNodeDoubles;
  cudaError_t err = cudaFuncSetAttribute(k_react<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  // the largest shared-memory carve-out, so that three CTAs share an SM
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(k_react<NS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
  if (err != cudaSuccess) return fail(DGB_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(err));
  const unsigned grid = (unsigned)((nodes + per - 1) / per);
  k_react<NS><<<grid, kReactThreads, sm, st>>>(M, U, out, nodes, num_nodes, nvars, dt, dt_elem);
  err = cudaGetLastError();
  if (err != cudaSuccess) return fail(DGB_ERR_CUDA, std::string("k_react: ") + cudaGetErrorString(err));
  return DGB_OK;
}

template <int NS>
int launch_rates(const Tables& M, const double* rho, const double* T, long long count, double* omega, double* wdot,
                 double* jac, cudaStream_t st) {
  const size_t sm = smem_bytes<NS>();
  cudaError_t err = cudaFuncSetAttribute(k_rates<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (err != cudaSuccess) return fail(DGB_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(err));
  const unsigned grid = (unsigned)((count + kThreads - 1) / kThreads);
  k_rates<NS><<<grid, kThreads, sm, st>>>(M, rho, T, count, omega, wdot, jac);
  err = cudaGetLastError();
  if (err != cudaSuccess) return fail(DGB_ERR_CUDA, std::string("k_rates: ") + cudaGetErrorString(err));
  return DGB_OK;
}

}  // namespace

struct dgb_chem {
  Tables tables;
};

extern "C" {

int dgb_chem_create(const dgb_chem_mechanism* m, const dgb_chem_params* prm, dgb_chem** out) {
  if (!m || !prm || !out) return fail(DGB_ERR_ARGUMENT, "null argument");
  *out = nullptr;
  const int ns = m->num_species, nr = m->num_reactions;
  if (ns != 3 && ns != 11) return fail(DGB_ERR_UNSUPPORTED, "chemistry kernels are compiled for 3 or 11 species");
  if (nr < 1 || nr > DGB_CHEM_MAX_REACTIONS) return fail(DGB_ERR_UNSUPPORTED, "too many reactions");
  if (!m->molar_mass || !m->nu_forward || !m->nu_reverse || !m->efficiency || !m->arrhenius || !m->third_body ||
      !m->forward_mode || !m->reverse_mode || !m->nasa_range || !m->nasa_coeffs)
    return fail(DGB_ERR_ARGUMENT, "null mechanism table");
  if (prm->max_newton_iters < 0) return fail(DGB_ERR_ARGUMENT, "max_newton_iters must be >= 0");
  dgb_chem* c = new dgb_chem;
  Tables& M = c->tables;
  memset(&M, 0, sizeof(M));
  M.ns = ns;
  M.nr = nr;
  for (int q = 0; q < ns; ++q) {
    M.W[q] = m->molar_mass[q];
    M.RW[q] = kRUniv / m->molar_mass[q];
    M.iW[q] = 1.0 / m->molar_mass[q];
    for (int k = 0; k < 3; ++k) M.trange[q][k] = m->nasa_range[q * 3 + k];
    if (!(M.trange[q][0] > 0.0) || !(M.trange[q][2] > M.trange[q][0])) {
      delete c;
      return fail(DGB_ERR_ARGUMENT, "NASA-7 ranges must satisfy 0 < t_low < t_high");
    }
    M.clamp_log[q][0] = log(M.trange[q][0]);
    M.clamp_log[q][1] = log(M.trange[q][2]);
    M.clamp_inv[q][0] = 1.0 / M.trange[q][0];
    M.clamp_inv[q][1] = 1.0 / M.trange[q][2];
    for (int r = 0; r < 2; ++r) {
      const double* a = m->nasa_coeffs + (q * 2 + r) * 7;
      for (int k = 0; k < 5; ++k) M.cp[q][r][k] = a[k];
      M.h[q][r][0] = a[0];
      M.h[q][r][1] = a[1] / 2.0;
      M.h[q][r][2] = a[2] / 3.0;
      M.h[q][r][3] = a[3] / 4.0;
      M.h[q][r][4] = a[4] / 5.0;
      M.h[q][r][5] = a[5];
      M.s[q][r][0] = a[0];
      M.s[q][r][1] = a[1];
      M.s[q][r][2] = a[2] / 2.0;
      M.s[q][r][3] = a[3] / 3.0;
      M.s[q][r][4] = a[4] / 4.0;
      M.s[q][r][5] = a[6];
    }
  }
  for (int r = 0; r < nr; ++r) {
    Reaction& R = M.rx[r];
    R.A = m->arrhenius[r * 3 + 0];
    R.b = m->arrhenius[r * 3 + 1];
    R.theta = m->arrhenius[r * 3 + 2];
    R.third = m->third_body[r] ? 1 : 0;
    R.fmode = m->forward_mode[r];
    R.rmode = m->reverse_mode[r];
    if (R.fmode < 0 || R.fmode > 2 || R.rmode < 0 || R.rmode > 2) {
      delete c;
      return fail(DGB_ERR_ARGUMENT, "temperature mode must be 0, 1 or 2");
    }
    double dn = 0.0;
    for (int q = 0; q < ns; ++q) {
      const double f = m->nu_forward[r * ns + q], p = m->nu_reverse[r * ns + q], d = p - f;
      M.alpha[r][q] = m->efficiency[r * ns + q];
      dn += d;
      if (f != 0.0) {
        if (R.nf == 3) { delete c; return fail(DGB_ERR_UNSUPPORTED, "more than 3 reactant species"); }
        R.f_sp[R.nf] = q;
        R.f_nu[R.nf++] = f;
      }
      if (p != 0.0) {
        if (R.nr == 3) { delete c; return fail(DGB_ERR_UNSUPPORTED, "more than 3 product species"); }
        R.r_sp[R.nr] = q;
        R.r_nu[R.nr++] = p;
      }
      if (d != 0.0) {
        if (R.nd == kMaxList) { delete c; return fail(DGB_ERR_UNSUPPORTED, "more than 6 net species"); }
        R.d_sp[R.nd] = q;
        R.d_nu[R.nd++] = d;
      }
    }
    R.dn = dn;
    R.whole = 1;
    for (int k = 0; k < R.nf; ++k) {
      const double v = R.f_nu[k];
      R.whole &= (v == 1.0 || v == 2.0 || v == 3.0) ? 1 : 0;
      R.f_pw[k] = (int)v;
    }
    for (int k = 0; k < R.nr; ++k) {
      const double v = R.r_nu[k];
      R.whole &= (v == 1.0 || v == 2.0 || v == 3.0) ? 1 : 0;
      R.r_pw[k] = (int)v;
    }
  }
  // k_react's rows: the species by falling number of reactions, four side by side, so that the lanes
  // of a node walk lists of similar length; the mass-weighted sum is the last row of NS + 1
  {
    const int rows = (ns + 1 + kLanes - 1) / kLanes * kLanes;
    std::vector<int> sp(ns), count(ns, 0);
    for (int q = 0; q < ns; ++q) sp[q] = q;
    for (int r = 0; r < nr; ++r)
      for (int k = 0; k < M.rx[r].nd; ++k) ++count[M.rx[r].d_sp[k]];
    std::stable_sort(sp.begin(), sp.end(), [&](int a, int b) { return count[a] > count[b]; });
    for (int i = 0; i < kRows; ++i) M.row_of[i] = i < ns ? sp[i] : -1;
    M.row_of[rows - 1] = ns;
    int n = 0;
    for (int pass = 0; pass < kPasses; ++pass)
      for (int i = 0; i < kRows; ++i) {
        M.list_ptr[pass * kRows + i] = n;
        const int q = M.row_of[i];
        if (q < 0) continue;
        for (int r = pass * kPass; r < nr && r < (pass + 1) * kPass; ++r) {
          const Reaction& R = M.rx[r];
          double w = 0.0;
          for (int k = 0; k < R.nd; ++k)
            if (q == ns) w += M.W[R.d_sp[k]] * R.d_nu[k];
            else if (R.d_sp[k] == q) w = R.d_nu[k];
          if (w == 0.0) continue;
          M.list_rx[n] = (short)(r - pass * kPass);
          M.list_w[n++] = w;
        }
      }
    M.list_ptr[kPasses * kRows] = n;
  }
  // coupling.py:55-67
  M.iters = prm->max_newton_iters;
  M.dimensionless = prm->dimensionless ? 1 : 0;
  M.gamma = prm->gamma;
  M.T_ref = prm->reference_temperature;
  const double mw_n2 = 2.0 * 0.0140067, mw_o2 = 2.0 * 0.015999;
  const double mean_mw = 1.0 / (0.767 / mw_n2 + 0.233 / mw_o2);
  const double R_ref = kRUniv / mean_mw;
  M.rho_ref = prm->reference_pressure / (R_ref * prm->reference_temperature);
  const double u_ref = sqrt(R_ref * prm->reference_temperature);
  M.e_ref = u_ref * u_ref;
  M.t_ref = prm->reference_length / u_ref;
  *out = c;
  return DGB_OK;
}

int dgb_chem_destroy(dgb_chem* chem) {
  delete chem;
  return DGB_OK;
}

int dgb_react_block(dgb_chem* chem, const double* U, double* out, int64_t num_elements, int num_nodes, int nvars,
                    double dt, const double* dt_per_element, void* stream) {
  if (!chem) return fail(DGB_ERR_ARGUMENT, "null argument");
  const Tables& M = chem->tables;
  if (nvars < 5 + M.ns)
    return fail(DGB_ERR_ARGUMENT, "State has " + std::to_string(nvars) + " variables; expected at least " +
                                      std::to_string(5 + M.ns) + " for reacting mixture.");
  if (num_elements < 0 || num_nodes < 0) return fail(DGB_ERR_ARGUMENT, "negative block size");
  const long long nodes = (long long)num_elements * num_nodes;
  if (nodes == 0) return DGB_OK;                    // an empty block needs no buffers
  if (!U || !out) return fail(DGB_ERR_ARGUMENT, "null argument");
  if (nodes / (kReactThreads / kLanes) >= 0x7fffffffLL) return fail(DGB_ERR_ARGUMENT, "block too large");
  cudaStream_t st = (cudaStream_t)stream;
  return M.ns == 11 ? launch_react<11>(M, U, out, nodes, num_nodes, nvars, dt, dt_per_element, st)
                    : launch_react<3>(M, U, out, nodes, num_nodes, nvars, dt, dt_per_element, st);
}

int dgb_chem_rates(dgb_chem* chem, const double* rho, const double* T, int64_t count, double* omega, double* wdot,
                   double* jacobian, void* stream) {
  if (!chem || !rho || !T) return fail(DGB_ERR_ARGUMENT, "null argument");
  if (count < 0) return fail(DGB_ERR_ARGUMENT, "negative count");
  if (count == 0) return DGB_OK;
  const Tables& M = chem->tables;
  cudaStream_t st = (cudaStream_t)stream;
  return M.ns == 11 ? launch_rates<11>(M, rho, T, count, omega, wdot, jacobian, st)
                    : launch_rates<3>(M, rho, T, count, omega, wdot, jacobian, st);
}

}  // extern "C"
