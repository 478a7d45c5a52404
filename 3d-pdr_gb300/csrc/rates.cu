// rates.cu -- batched reaction-rate evaluation with self-shielding
// (GPU form of CALCULATE_REACTION_RATES, calc_reac_rates.F90:16-401).
//
// rates_kernel takes a batch of cells per block and gives every lane of every
// phase an item of its own: the cells (per-cell logarithms and reciprocals),
// the (cell, ray) pairs (shielding, scattering), the (cell, photo-reaction)
// pairs (a sum over the rays in ray order), and the (cell, reaction) pairs of
// the other reactions, class by class.  Powers of T and exponentials of 1/T
// are one exponential 2^(b L - g G) of per-cell L = 1024 log2(T/300) and
// G = 1024/(T ln 2).  Each reaction's branch, duplicate-group selection (the
// first member whose RTMAX >= T, else the last member,
// calc_reac_rates.F90:117-145) and the clamps of :387-396 are the reference's.
// Shielding follows shield.F90: Federman H2SHIELD1 (:231), the van Dishoeck &
// Black 2-D spline COSHIELD (:375, natural splines of spline.F90), SCATTER
// (:449) with XLAMBDA (:525) and LBAR (:570); H2 formation on grains follows
// h2_form.F90:8-113.
//
// Cells outside the fast path's ranges (rates_cell_ok) are evaluated by
// rates_cell_general, one warp per cell, expression by expression.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

#include <mutex>

#include "fp64_fast.cuh"
#include "pdr_internal.h"

namespace pdr {

// Savage & Mathis (1979) tau(lambda)/tau(V) (the extinction table of the
// reference, modules.F90:354-366) and the van Dishoeck & Black (1988) log10
// 12CO shielding grid (modules.F90:346-351, values 3DPDR.F90:1532-1537).
static const double kLGrid[30] = {910.0, 950.0, 1000.0, 1050.0, 1110.0, 1180.0, 1250.0, 1390.0,
                                  1490.0, 1600.0, 1700.0, 1800.0, 1900.0, 2000.0, 2100.0, 2190.0,
                                  2300.0, 2400.0, 2500.0, 2740.0, 3440.0, 4000.0, 4400.0, 5500.0,
                                  7000.0, 9000.0, 12500.0, 22000.0, 34000.0, 1.0e9};
static const double kXGrid[30] = {5.76, 5.18, 4.65, 4.16, 3.73, 3.40, 3.11, 2.74, 2.63, 2.62,
                                  2.54, 2.50, 2.58, 2.78, 3.01, 3.12, 2.86, 2.58, 2.35, 2.00,
                                  1.58, 1.42, 1.32, 1.00, 0.75, 0.48, 0.28, 0.12, 0.05, 0.00};
static const double kNCOGrid[8] = {12.0, 13.0, 14.0, 15.0, 16.0, 17.0, 18.0, 19.0};
static const double kNH2Grid[6] = {18.0, 19.0, 20.0, 21.0, 22.0, 23.0};
// [iNH2][iNCO]
static const double kSCO[6][8] = {
    {0.000e+00, -1.408e-02, -1.099e-01, -4.400e-01, -1.154e+00, -1.888e+00, -2.760e+00, -4.001e+00},
    {-8.539e-02, -1.015e-01, -2.104e-01, -5.608e-01, -1.272e+00, -1.973e+00, -2.818e+00, -4.055e+00},
    {-1.451e-01, -1.612e-01, -2.708e-01, -6.273e-01, -1.355e+00, -2.057e+00, -2.902e+00, -4.122e+00},
    {-4.559e-01, -4.666e-01, -5.432e-01, -8.665e-01, -1.602e+00, -2.303e+00, -3.146e+00, -4.421e+00},
    {-1.303e+00, -1.312e+00, -1.367e+00, -1.676e+00, -2.305e+00, -3.034e+00, -3.758e+00, -5.077e+00},
    {-3.883e+00, -3.888e+00, -3.936e+00, -4.197e+00, -4.739e+00, -5.165e+00, -5.441e+00, -6.446e+00}};

struct ShieldTables {
  double lgrid[30], xgrid[30], xderiv[30];
  double nco[8], nh2[6], sco[8][6], scoderiv[8][6];
};
__constant__ ShieldTables c_shield;

// natural cubic spline second derivatives (the tridiagonal sweep of the
// Numerical-Recipes routine the reference uses, spline.F90:65-125)
template <class R>
__host__ __device__ void spline_natural(const R *x, const R *y, int n, R *y2, R *u) {
  y2[0] = 0.0;
  u[0] = 0.0;
  for (int i = 1; i < n - 1; i++) {
    const R sig = (x[i] - x[i - 1]) / (x[i + 1] - x[i - 1]);
    const R p = sig * y2[i - 1] + 2.0;
    y2[i] = (sig - 1.0) / p;
    u[i] = (6.0 * ((y[i + 1] - y[i]) / (x[i + 1] - x[i]) - (y[i] - y[i - 1]) / (x[i] - x[i - 1])) /
                (x[i + 1] - x[i - 1]) - sig * u[i - 1]) / p;
  }
  y2[n - 1] = 0.0;
  for (int i = n - 2; i >= 0; i--) y2[i] = y2[i] * y2[i + 1] + u[i];
}

// cubic spline value with the bisection bracket of spline.F90:182-277
template <class R>
__host__ __device__ R splint(const R *xa, const R *ya, const R *y2a, int n, R x) {
  const bool asc = xa[n - 1] > xa[0];
  int lo = 0, hi = n + 1;
  while (hi - lo != 1) {
    const int mid = (hi + lo) / 2;
    if ((x > xa[mid - 1]) == asc) lo = mid;
    else hi = mid;
  }
  if (lo == 0) { lo = 1; hi = 2; }
  if (lo == n) { lo = n - 1; hi = n; }
  const R h = xa[hi - 1] - xa[lo - 1];
  const R A = (xa[hi - 1] - x) / h, B = (x - xa[lo - 1]) / h;
  return A * ya[lo - 1] + B * ya[hi - 1] +
         ((A * A * A - A) * y2a[lo - 1] + (B * B * B - B) * y2a[hi - 1]) * (h * h) / 6.0;
}

// The same functions as the fast path evaluates them: COSHIELD's two natural
// splines as bicubic patches (coefficient of x^n y^m at [n][m], x and y from
// the patch's lower corner in log10 N(CO), log10 N(H2)), and XLAMBDA's cubic
// pieces over LBAR's range (c0..c3, the piece's start, 1/its width) for the
// natural spline [0] and the linear variant [1].  (A patch is read with 16-byte
// loads.)
struct alignas(16) ShieldFast {
  double patch[7][5][4][4];
  double lam[2][4][6];
};
__device__ ShieldFast d_shield;

// cubic c0..c3 in B = (x - x0)/h of the spline piece with values ya, yb and second derivatives a2, b2
template <class R>
static void piece(R ya, R yb, R a2, R b2, R h, R *c) {
  const R q = h * h / 6;
  c[0] = ya;
  c[1] = yb - ya - q * (2 * a2 + b2);
  c[2] = 3 * q * a2;
  c[3] = q * (b2 - a2);
}

#pragma nv_diag_suppress 20208   // the host evaluates these in long double; no device code is made of it
static void shield_fast_tables(const ShieldTables &t, ShieldFast &f) {
  using R = long double;
  R nco[8], nh2[6], u[8];
  for (int i = 0; i < 8; i++) nco[i] = t.nco[i];
  for (int j = 0; j < 6; j++) nh2[j] = t.nh2[j];
  R rows[8][5][4];
  for (int i = 0; i < 8; i++) {
    R row[6], y2[6];
    for (int j = 0; j < 6; j++) row[j] = t.sco[i][j];
    spline_natural<R>(nh2, row, 6, y2, u);
    for (int q = 0; q < 5; q++) piece<R>(row[q], row[q + 1], y2[q], y2[q + 1], R(1), rows[i][q]);
  }
  R acc[7][5][4][4];
  for (auto &a : acc) for (auto &b : a) for (auto &c : b) for (R &d : c) d = 0;
  for (int i = 0; i < 8; i++) {
    R e[8], y2[8];
    for (int j = 0; j < 8; j++) e[j] = (i == j);
    spline_natural<R>(nco, e, 8, y2, u);
    for (int p = 0; p < 7; p++) {
      R w[4];
      piece<R>(e[p], e[p + 1], y2[p], y2[p + 1], R(1), w);
      for (int q = 0; q < 5; q++)
        for (int n = 0; n < 4; n++)
          for (int m = 0; m < 4; m++) acc[p][q][n][m] += w[n] * rows[i][q][m];
    }
  }
  for (int p = 0; p < 7; p++)
    for (int q = 0; q < 5; q++)
      for (int n = 0; n < 4; n++)
        for (int m = 0; m < 4; m++) f.patch[p][q][n][m] = (double)acc[p][q][n][m];
  for (int v = 0; v < 2; v++)
    for (int i = 0; i < 4; i++) {
      const double h = t.lgrid[i + 1] - t.lgrid[i];
      R c[4];
      piece<R>(t.xgrid[i], t.xgrid[i + 1], v ? 0.0 : t.xderiv[i], v ? 0.0 : t.xderiv[i + 1], h, c);
      for (int k = 0; k < 4; k++) f.lam[v][i][k] = (double)c[k];
      f.lam[v][i][4] = t.lgrid[i];
      f.lam[v][i][5] = 1.0 / h;
    }
}

// the tables of every device, made once per process
struct ShieldHost {
  ShieldTables t;
  ShieldFast f;
  ShieldHost() {
    double u[30];
    for (int i = 0; i < 30; i++) { t.lgrid[i] = kLGrid[i]; t.xgrid[i] = kXGrid[i]; }
    spline_natural<double>(t.lgrid, t.xgrid, 30, t.xderiv, u);
    for (int i = 0; i < 8; i++) t.nco[i] = kNCOGrid[i];
    for (int j = 0; j < 6; j++) t.nh2[j] = kNH2Grid[j];
    for (int i = 0; i < 8; i++) {
      double row[6], y2[6];
      for (int j = 0; j < 6; j++) { row[j] = kSCO[j][i]; t.sco[i][j] = kSCO[j][i]; }
      spline_natural<double>(t.nh2, row, 6, y2, u);
      for (int j = 0; j < 6; j++) t.scoderiv[i][j] = y2[j];
    }
    shield_fast_tables(t, f);
  }
};

// Uploads the tables to `dev`, the calling thread's device, at its first call.
// Any number of threads may make that call: one copies, the others return when
// the device has the tables, and none copies over tables that are in use.
int upload_shield_tables(int dev) {
  static std::mutex mu;
  static bool ready[64];
  static const ShieldHost host;
  std::lock_guard<std::mutex> lk(mu);
  const bool known = dev >= 0 && dev < 64;
  if (known && ready[dev]) return 0;
  cudaError_t e = cudaMemcpyToSymbol(c_shield, &host.t, sizeof host.t);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyToSymbol(shield tables)");
  e = cudaMemcpyToSymbol(d_shield, &host.f, sizeof host.f);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyToSymbol(shield pieces)");
  if (known) ready[dev] = true;
  return 0;
}

// host copies for the test/diagnostic export
void shield_tables_host(double *xderiv30, double *scoderiv48) {
  double lg[30], xg[30], u[64];
  for (int i = 0; i < 30; i++) { lg[i] = kLGrid[i]; xg[i] = kXGrid[i]; }
  spline_natural<double>(lg, xg, 30, xderiv30, u);
  double nh2[6];
  for (int j = 0; j < 6; j++) nh2[j] = kNH2Grid[j];
  for (int i = 0; i < 8; i++) {
    double row[6], y2[6];
    for (int j = 0; j < 6; j++) row[j] = kSCO[j][i];
    spline_natural<double>(nh2, row, 6, y2, u);
    for (int j = 0; j < 6; j++) scoderiv48[i * 6 + j] = y2[j];
  }
}

// tau(1000 A)/tau(V)/1.086, spline and linear
static void shield_x1000(double *x) {
  static double v[2];
  static std::once_flag once;
  std::call_once(once, [] {
    double xd[30], zero[30] = {}, u[64];
    spline_natural<double>(kLGrid, kXGrid, 30, xd, u);
    v[0] = splint<double>(kLGrid, kXGrid, xd, 30, 1000.0) / 1.086;
    v[1] = splint<double>(kLGrid, kXGrid, zero, 30, 1000.0) / 1.086;
  });
  x[0] = v[0];
  x[1] = v[1];
}

namespace {

constexpr double KB = 1.38065040e-16, AU = 1.66053878e-24;
constexpr double PI = 3.141592653589793238462643383279502884197;

__device__ double xlambda(double lambda, int linear) {
  const ShieldTables &t = c_shield;
  if (lambda < t.lgrid[0]) lambda = t.lgrid[0];
  if (lambda > t.lgrid[29]) lambda = t.lgrid[29];
  double zero[30];
  if (linear)
    for (int i = 0; i < 30; i++) zero[i] = 0.0;
  return splint<double>(t.lgrid, t.xgrid, linear ? zero : t.xderiv, 30, lambda);
}

__device__ double scatter(double av, double lambda, int linear) {
  const double A[6] = {1.000, 2.006, -1.438, 0.7364, -0.5076, -0.0592};
  const double K[6] = {0.7514, 0.8490, 1.013, 1.282, 2.005, 5.832};
  const double taul = (av / 1.086) * xlambda(lambda, linear);
  double s = 0.0;
  if (taul < 1.0) {
    const double e = K[0] * taul;
    if (e < 100.0) s = A[0] * exp(-e);
  } else {
    for (int i = 1; i <= 5; i++) {
      const double e = K[i] * taul;
      if (e < 100.0) s = s + A[i] * exp(-e);
    }
  }
  return s;
}

__device__ double h2shield1(double nh2, double dopw, double radw) {
  const double taud = nh2 * 0.5 * (1.497358985e-2) * 1.0e-2 / dopw;
  double jd, jr;
  if (taud == 0.0) jd = 1.0;
  else if (taud < 2.0) jd = exp(-(0.666666667 * taud));
  else if (taud < 10.0) jd = 0.638 * pow(taud, -1.25);
  else if (taud < 100.0) jd = 0.505 * pow(taud, -1.15);
  else jd = 0.344 * pow(taud, -1.0667);
  if (radw == 0.0) jr = 0.0;
  else {
    const double r = radw / (1.772453851 * dopw);
    const double t = 3.02 * pow(r * 1.0e3, -0.064);
    const double u = sqrt(taud * r) / t;
    jr = r / (t * sqrt(0.785398163 + u * u));
  }
  return jd + jr;
}

__device__ double coshield(double nco, double nh2) {
  const ShieldTables &t = c_shield;
  double lnco = log10(nco + 1.0), lnh2 = log10(nh2 + 1.0);
  if (lnco < t.nco[0]) lnco = t.nco[0];
  if (lnh2 < t.nh2[0]) lnh2 = t.nh2[0];
  if (lnco > t.nco[7]) lnco = t.nco[7];
  if (lnh2 > t.nh2[5]) lnh2 = t.nh2[5];
  double yy[8], yy2[8], u[8];
  for (int i = 0; i < 8; i++) yy[i] = splint<double>(t.nh2, t.sco[i], t.scoderiv[i], 6, lnh2);
  spline_natural<double>(t.nco, yy, 8, yy2, u);
  return pow(10.0, splint<double>(t.nco, yy, yy2, 8, lnco));
}

__device__ double lbar(double nco, double nh2) {
  const double u = log10(nco + 1.0), w = log10(nh2 + 1.0);
  double l = (5675.0 - 200.6 * w) - (571.6 - 24.09 * w) * u + (18.22 - 0.7664 * w) * (u * u);
  if (l < 913.6) l = 913.6;
  if (l > 1076.1) l = 1076.1;
  return l;
}

__device__ double h2_formation(double Tg, double Td, double Z, double g2d) {
  const double vth = 1.45e5 * sqrt(Tg / 1.0e2);
  const double tt = Tg / 1.0e2;
  const double stick = 1.0 / (1.0 + 0.04 * sqrt(Tg + Td) + 0.2 * tt + 0.08 * (tt * tt));
  const double flux = 1.0e-10, mu = 0.005, nu_h2 = 3.0e12, nu_hc = 1.3e13, ehc = 3.0e4;
  const double es[2] = {110.0, 260.0}, eh2[2] = {320.0, 520.0}, ehp[2] = {450.0, 800.0};
  double eff[2];
  for (int g = 0; g < 2; g++) {
    const double f1 = mu * flux / (2 * nu_h2 * exp(-eh2[g] / Td));
    const double sq = 1.0 + sqrt((ehc - es[g]) / (ehp[g] - es[g]));
    const double f2 = 1.0 * (sq * sq) / 4.0 * exp(-es[g] / Td);
    const double eps = 1.0 / (1.0 + nu_hc / (2 * flux) * exp(-1.5 * ehc / Td) * (sq * sq));
    eff[g] = 1.0 / (1.0 + f1 + f2) * eps;
  }
  return 0.5 * vth * (8.473e-22 * eff[0] + 7.908e-22 * eff[1]) * stick * Z * 100. / g2d;
}

struct RateRow {
  double alpha, beta, gamma, rtmin;
  int kind, flags;
};
__device__ __forceinline__ RateRow rate_row(const RateTables &T, int r) {
  RateRow w;
  w.alpha = __ldg(&T.alpha[r]); w.beta = __ldg(&T.beta[r]); w.gamma = __ldg(&T.gamma[r]);
  w.rtmin = __ldg(&T.rtmin[r]);
  w.kind = __ldg(&T.kind[r]);
  w.flags = __ldg(&T.flags[r]);
  return w;
}

// only the selected member of a duplicate group gets a rate (the member whose
// temperature range holds T, else the group's last)
__device__ __forceinline__ bool dup_selected(const RateTables &T, int r, double t) {
  const int d = __ldg(&T.dup[r]), kind = __ldg(&T.kind[r]);
  if (d > 0 && (kind == RK_THERMAL || kind == RK_PHOTO || kind == RK_CRP || kind == RK_CRPHOT)) {
    int head = r;
    while (head > 0 && __ldg(&T.dup[head]) > 1) head--;
    int sel = head;
    // the group ends where the next reaction's DUPLICATE does not go on
    while (!(t <= __ldg(&T.rtmax[sel]) || __ldg(&T.dup_next[sel]) < __ldg(&T.dup[sel]) || __ldg(&T.dup_next[sel]) < 0)) sel++;
    return sel == r;
  }
  return true;
}

// one ray's term of a ray-summed rate (the summand of calc_reac_rates.F90's
// loop over the rays, the same expression in the same order)
__device__ __forceinline__ double ray_term(const RateRow &w, double t, const double *rs, const double *av,
                                           const double *cc, int ray, double dopw, double radw, int linear) {
  const double a = w.alpha, g = w.gamma;
  switch (w.kind) {
    case RK_PHOTO_H2:
    case RK_PHOTO_HD: {
      const int c = (w.kind == RK_PHOTO_H2) ? 0 : 1;
      return a * rs[ray] * h2shield1(cc[ray * 5 + c], dopw, radw) * scatter(av[ray], 1000.0, linear) / 2.0;
    }
    case RK_PHOTO_CO: {
      const double nco = cc[ray * 5 + 2], nh2 = cc[ray * 5 + 0];
      return a * rs[ray] * coshield(nco, nh2) * scatter(av[ray], lbar(nco, nh2), linear) / 2.0;
    }
    case RK_PHOTO_CI: {
      const double tauc = g * av[ray] + 1.1e-17 * cc[ray * 5 + 3] +
                          (0.9 * pow(t, 0.27) * pow(cc[ray * 5 + 0] / 1.59e21, 0.45));
      return a * rs[ray] * exp(-tauc) / 2.0;
    }
    case RK_PHOTD: {
      const double y = (t < 50.0) ? 3.5e-3 : (t < 85.0 ? 4.0e-3 : (t < 100.0 ? 5.5e-3 : 7.5e-3));
      return 1.7e8 * rs[ray] * exp(-(1.8 * av[ray])) * 2.4e-22 * y;
    }
    default:   // RK_PHOTO, RK_PHOTO_SI
      return a * rs[ray] * exp(-(g * av[ray])) / 2.0;
  }
}

// calc_reac_rates.F90's clamps: a negative rate is reported, rates above 1
// are capped unless the first reactant is a grain, rates below 1e-99 are zero
__device__ __forceinline__ void store_rate(double k, const RateRow &w, int r, double *out, bool &neg, int &negr) {
  if (k < 0.0) { negr = neg ? min(negr, r + 1) : r + 1; neg = true; }
  if (k > 1.0 && !(w.flags & 1)) k = 1.0;
  if (k < 1.0e-99) k = 0.0;
  out[r] = k;
}

// One reaction that is not a sum over the rays, as the reference writes it.
__device__ __noinline__ double other_rate(RateRow w, double t, double td, double zeta, const pdr_phys &ph) {
  const double a = w.alpha, b = w.beta, g = w.gamma;
  switch (w.kind) {
    case RK_H2FORM: return ph.h2form ? h2_formation(t, td, ph.metallicity, ph.g2d) : 3.0e-18 * sqrt(t);
    case RK_PAH: return a * pow(t / 100.0, b) * 0.4;
    case RK_THERMAL: return (g < -200.0 && t < w.rtmin) ? 0.0 : a * pow(t / 300.0, b) * exp(-(g / t));
    case RK_CRP: return a * zeta;
    case RK_CRPHOT: return a * zeta * pow(t / 300.0, b) * g / (1.0 - ph.omega);
    case RK_FREEZE:
    case RK_ELFRZE: {
      const double cion = (b == 0.0) ? 1.0 : (b == 1.0 ? 1.0 + 16.71e-4 / (ph.grain_radius * t) : 0.0);
      return a * 4.57e4 * 2.4e-22 * sqrt(t / g) * cion * 0.3;
    }
    case RK_CRH: return 2.06e-3 * zeta * 2.4e-22 * ((g <= 1210.0) ? 1.0e5 : 0.0);
    case RK_THERM: return sqrt(2.0 * 1.5e15 * KB / (PI * PI * AU) * a / g) * exp(-(a / td));
    case RK_GRAIN: return a;
    default: return 0.0;
  }
}

// Constants of one call: which shielded reactions the network has, the H2
// shielding's per-column optical depth and radiative-wing factors, and
// tau(1000 A)/tau(V)/1.086; fast = 0 sends every cell to the general path.
struct RateShield {
  int fast, has_h2, has_hd, has_co, has_ci;
  double ci_gamma, taud, jr_a, jr_b, x1000[2];
};

struct RatesArgs {
  RateTables T;
  RateShield S;
  pdr_phys ph;
  int ncell, nrays, batch;   // batch: cells per block and round
  const double *Tg, *Td, *rad, *AV, *col5, *zeta;
  double *rate;
  int *status;
};

// Every reaction of one cell by one warp, the reference's expressions: for the
// cells whose values the fast path does not take.
__device__ __noinline__ void rates_cell_general(const RatesArgs &A, int cell) {
  const RateTables &T = A.T;
  const pdr_phys &ph = A.ph;
  const int lane = threadIdx.x & 31, nrays = A.nrays;
  const double dopw = ph.v_turb / (1000.0 * 1.0e-8), radw = 8.0e7;
  const int linear = ph.xlambda_linear;
  const double t = A.Tg[cell], td = A.Td[cell];
  // ZETA, or the cell's own rate in the cosmic-ray variant (zetacrlocal)
  const double zeta = A.zeta ? A.zeta[cell] : ph.zeta;
  const double *rs = A.rad + (size_t)cell * nrays;
  const double *av = A.AV + (size_t)cell * nrays;
  const double *cc = A.col5 + (size_t)cell * nrays * 5;
  double *out = A.rate + (size_t)cell * T.nreac;
  bool neg = false;
  int negr = 0;
  for (int j = lane; j < T.nray + T.nother; j += 32) {
    const int r = j < T.nray ? __ldg(&T.ray_reac[j]) : __ldg(&T.other_reac[j - T.nray]);
    const RateRow w = rate_row(T, r);
    double k = 0.0;
    if (dup_selected(T, r, t)) {
      if (j < T.nray)
        for (int ray = 0; ray < nrays; ray++) k = k + ray_term(w, t, rs, av, cc, ray, dopw, radw, linear);
      else
        k = other_rate(w, t, td, zeta, ph);
    }
    store_rate(k, w, r, out, neg, negr);
  }
  // the lowest-numbered negative rate of the cell, as a negative status
  const unsigned anyneg = __ballot_sync(0xffffffffu, neg);
  if (A.status) {
    int rr = neg ? negr : 0x7fffffff;
    for (int o = 16; o > 0; o >>= 1) rr = min(rr, __shfl_xor_sync(0xffffffffu, rr, o));
    if (lane == 0) A.status[cell] = anyneg ? -rr : 0;
  }
}

__device__ __forceinline__ bool in_range(double x, double lo, double hi) { return x >= lo && x <= hi; }   // false for NaN

// per-cell values of the fast path
struct CellRates {
  double t, td, zeta;
  double Lh, Ll;      // 1024 log2(T/300)
  double Gh, Gl;      // 1024/(T ln 2)
  double t27;         // 0.9 T^0.27 (the C photo-rate's H2 line opacity)
  float Lf, Gf;
  int ok;             // 0: general path
  int neg;            // lowest negative reaction number
};
// per-(cell, ray) values: A_V 1024/ln 2 = av2 + av2_lo, the field, and the field
// times the shielding functions of H2, HD, CO and C
struct RayRates {
  double av2, rs, h2, hd, co, ci;
  float av2_lo;
};

// The reference's expressions jump where they change (SCATTER by 3.8e-4 at tau =
// 1), and the fast path's arguments may be an ulp or so from the reference's.  So
// each choice is made on all the bits of the argument, by integer compares, and
// within 4,096 ulp (9e-13) of a jump the reference's own expression decides: a
// rare call.
__device__ __forceinline__ bool at_jump(double x, double jump) {
  return (unsigned long long)(__double_as_longlong(x) - __double_as_longlong(jump) + 4096) < 8192ull;
}
__device__ __noinline__ double scatter_at_jump(double av, double nco, double nh2, bool co, int linear) {
  return scatter(av, co ? lbar(nco, nh2) : 1000.0, linear);
}
__device__ __noinline__ double h2_taud(double nh2, double v_turb) {
  const double dopw = v_turb / (1000.0 * 1.0e-8);
  return nh2 * 0.5 * (1.497358985e-2) * 1.0e-2 / dopw;
}

// SCATTER(A_V, lambda) (shield.F90:449) from tl = tau(lambda) 1024/ln 2: one
// exponential below tau = 1, else five, those with an exponent of 100 or more
// left out (c_scat_end: where that is, and tau = 1 in the first place); jump: the
// caller has to take the reference's expression
__constant__ double c_scat_a[6] = {1.000, 2.006, -1.438, 0.7364, -0.5076, -0.0592};
__constant__ double c_scat_k[6] = {0.7514, 0.8490, 1.013, 1.282, 2.005, 5.832};
__constant__ float c_scat_kf[6] = {0.7514f, 0.8490f, 1.013f, 1.282f, 2.005f, 5.832f};
__constant__ double c_scat_end[6] = {fp64::K_LN2, 100.0 / 0.8490 * fp64::K_LN2, 100.0 / 1.013 * fp64::K_LN2,
                                     100.0 / 1.282 * fp64::K_LN2, 100.0 / 2.005 * fp64::K_LN2, 100.0 / 5.832 * fp64::K_LN2};
__device__ __forceinline__ double scatter_fast(double tl, bool &jump) {
  const float tf = fp64::d2f(tl);
  const bool thin = __double_as_longlong(tl) < __double_as_longlong(fp64::K_LN2);
  jump = at_jump(tl, fp64::K_LN2);
  double s = 0.0;
  for (int i = thin ? 0 : 1; i < (thin ? 1 : 6); i++) {
    jump |= at_jump(tl, c_scat_end[i]);
    if (__double_as_longlong(tl) >= __double_as_longlong(c_scat_end[i])) continue;
    float kf;
    const int k = fp64::rint_f(-c_scat_kf[i] * tf, kf);
    const double r = fma(-c_scat_k[i], tl, fp64::flip(fp64::f2d(kf)));
    const double t = c_scat_a[i] * fp64::exp2_int(k);
    s = fma(t, fma(r, fp64::exp2_slope(r), 1.0), s);
  }
  return s;
}

// H2SHIELD1 (shield.F90:231) for a positive Doppler width
__device__ __forceinline__ double h2shield_fast(double nh2, const RateShield &S, double v_turb) {
  double taud = nh2 * S.taud;
  if (at_jump(taud, 2.0) || at_jump(taud, 10.0) || at_jump(taud, 100.0)) taud = h2_taud(nh2, v_turb);
  double jd = 1.0;
  if (taud >= 2.0) {
    const double p = taud < 10.0 ? -1.25 : (taud < 100.0 ? -1.15 : -1.0667);
    const double c = taud < 10.0 ? 0.638 : (taud < 100.0 ? 0.505 : 0.344);
    jd = c * fp64::powk(fp64::log2k(taud), p);
  } else if (taud > 0.0) {
    jd = fp64::exp_fast(-0.666666667 * taud);
  }
  return fma(S.jr_a, fp64::rsqrt_fast(fma(taud, S.jr_b, 0.785398163)), jd);
}

// COSHIELD (shield.F90:375) from the clamped log10 columns: the bicubic patch
// of the two natural splines, then 10^x
__device__ __forceinline__ double coshield_fast(double u, double w) {
  u = fmin(fmax(u, 12.0), 19.0);
  w = fmin(fmax(w, 18.0), 23.0);
  const int p = min((int)fp64::d2f(u) - 12, 6), q = min((int)fp64::d2f(w) - 18, 4);
  const double x = u - fp64::f2d((float)(p + 12)), y = w - fp64::f2d((float)(q + 18));
  static_assert(alignof(ShieldFast) % alignof(double2) == 0 && sizeof(d_shield.patch[0][0]) % sizeof(double2) == 0 &&
                    offsetof(ShieldFast, patch) % alignof(double2) == 0,
                "a patch is read with 16-byte loads");
  const double2 *K = reinterpret_cast<const double2 *>(d_shield.patch[p][q]);
  double f = 0.0;
#pragma unroll 1
  for (int n = 3; n >= 0; n--) {
    const double2 a = __ldg(K + 2 * n), b = __ldg(K + 2 * n + 1);
    f = fma(f, x, fma(y, fma(y, fma(y, b.y, b.x), a.y), a.x));
  }
  // 10^f: 1024 log2(10) f = k + r
  constexpr double T10 = 3401.654369164659, T10L = 1.7014963373809582e-13;
  float kf;
  const int k = fp64::rint_f(fp64::d2f(f) * (float)T10, kf);
  return fp64::exp2k(k, fma(f, T10L, fma(f, T10, fp64::flip(fp64::f2d(kf)))));
}

// LBAR (shield.F90:570), then tau(LBAR)/tau(V) from its spline's cubic pieces
__device__ __forceinline__ double xlambda_lbar(double u, double w, int linear) {
  double l = fma(u * u, fma(-0.7664, w, 18.22), fma(-u, fma(-24.09, w, 571.6), fma(-200.6, w, 5675.0)));
  if (l < 913.6) l = 913.6;
  if (l > 1076.1) l = 1076.1;
  const float lf = fp64::d2f(l);
  const int i = lf > 1050.0f ? 3 : (lf > 1000.0f ? 2 : (lf > 950.0f ? 1 : 0));
  const double *c = d_shield.lam[linear][i];
  const double x = (l - __ldg(c + 4)) * __ldg(c + 5);
  return fma(x, fma(x, fma(x, __ldg(c + 3), __ldg(c + 2)), __ldg(c + 1)), __ldg(c));
}

__device__ __forceinline__ bool column_ok(double n) { return n == 0.0 || in_range(n, 1.0e-30, 1.0e30); }

// a 2^((k + r)/1024); exponents below the normal range give 0
__device__ __forceinline__ double scaled_exp2(double a, int k, double r) {
  return k < -1000 * 1024 ? 0.0 : fp64::exp2_times(a, min(k, 1000 * 1024), r);
}

// store_rate on the bit pattern of a finite rate (no FP64 compares)
__device__ __forceinline__ void store_rate_bits(double k, int r, int flags, double *out, int *neg) {
  const long long b = __double_as_longlong(k);
  if (b < 0) {
    if (b != (long long)0x8000000000000000ull) atomicMin(neg, r + 1);
    k = 0.0;
  } else if (b > 0x3ff0000000000000ll && !(flags & 1)) {
    k = 1.0;
  } else if (b < 0x2b617f7d4ed8c33ell) {   // 1e-99
    k = 0.0;
  }
  out[r] = k;
}

constexpr int RATES_THREADS = 256;

// What bounds it: the FP64 pipe (64 to 76 cycles per warp instruction).  So the
// lanes are kept full -- items of every phase are flattened over the batch's
// cells -- and the powers and exponentials take 3 to 9 FP64 instructions each
// (fp64_fast.cuh) instead of 19 (exp) and 95 (pow).  100,003 cells of the
// reduced network take 1.25 ms (one warp per cell with the library functions:
// 24.2 ms), 8,000 of the full one 0.46 ms (8.13 ms).  Against 113-bit values
// a (T/300)^b is 6.7e-17 off (rms, as with a correctly rounded pow) and
// a exp(-g/T) 6.7e-17 (1.3e-15 where g/T is rounded first).
// Over all thermal and photo-reactions of 400 full-network cells: thermal
// 5.8e-17 rms (library functions 6.8e-16), photo 1.44e-16 rms, 6.8e-16 at most.
// The reference rounds gamma A_V, and with the library's exp has 1.59e-16 and
// 1.6e-15 (host evaluation); rounding A_V 1024/ln 2 alone was 1.76e-16, so its
// low part goes along (no FP64 instruction more).  The table's tail in the
// photo sum would cost an addition and gains nothing (the sum then rounds twice
// a ray: 1.93e-16, 1.26 -> 1.32 ms).
__global__ void __launch_bounds__(RATES_THREADS, 3) rates_kernel(const __grid_constant__ RatesArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  CellRates *cells = reinterpret_cast<CellRates *>(smem);
  RayRates *rays = reinterpret_cast<RayRates *>(cells + A.batch);
  const RateTables &T = A.T;
  const RateShield &S = A.S;
  const int tid = threadIdx.x, nrays = A.nrays, nreac = T.nreac;
  const int linear = A.ph.xlambda_linear ? 1 : 0;
  for (long long base = (long long)blockIdx.x * A.batch; base < A.ncell; base += (long long)gridDim.x * A.batch) {
    const int nb = (int)min((long long)A.batch, A.ncell - base);
    for (int c = tid; c < nb; c += RATES_THREADS) {
      cells[c].ok = S.fast;
      cells[c].neg = 0x7fffffff;
    }
    __syncthreads();
    // the cells, and (from the second warp on, the first joining last) the rays
    for (int c = tid; c < nb; c += RATES_THREADS) {
      CellRates &C = cells[c];
      C.t = A.Tg[base + c];
      C.td = A.Td[base + c];
      // ZETA, or the cell's own rate in the cosmic-ray variant (zetacrlocal)
      C.zeta = A.zeta ? A.zeta[base + c] : A.ph.zeta;
      if (in_range(C.t, 1.0e-2, 1.0e8) && in_range(C.zeta, -1.0e30, 1.0e30)) {
        const fp64::Log2 L = fp64::log2k(C.t / 300.0);
        C.Lh = L.h;
        C.Ll = L.l;
        C.Lf = fp64::d2f(L.h);
        C.Gh = fp64::K_LN2 / C.t;
        C.Gl = (fma(-C.Gh, C.t, fp64::K_LN2) + (double)fp64::K_LN2_LO) / C.t;
        C.Gf = fp64::d2f(C.Gh);
        C.t27 = S.has_ci ? 0.9 * fp64::powk(fp64::log2k(C.t), 0.27) : 0.0;
      } else {
        C.ok = 0;
      }
    }
    if (S.fast)
      for (int i = (tid + RATES_THREADS - 32) % RATES_THREADS; i < nb * nrays; i += RATES_THREADS) {
        const size_t g = (size_t)base * nrays + i;
        RayRates &R = rays[i];
        const double av = A.AV[g];
        R.rs = A.rad[g];
        const double *col = A.col5 + g * 5;
        const double nh2 = (S.has_h2 | S.has_co | S.has_ci) ? col[0] : 0.0, nhd = S.has_hd ? col[1] : 0.0;
        const double nco = S.has_co ? col[2] : 0.0, nc = S.has_ci ? col[3] : 0.0;
        if (!(in_range(av, 0.0, 1.0e30) && in_range(R.rs, 0.0, 1.0e30) && column_ok(nh2) && column_ok(nhd) &&
              column_ok(nco) && column_ok(nc))) {
          cells[i / nrays].ok = 0;
          continue;
        }
        R.av2 = av * fp64::K_LN2;
        R.av2_lo = fp64::d2f(fma(av, fp64::K_LN2, -R.av2)) + fp64::d2f(av) * fp64::K_LN2_LO;
        if (S.has_h2 | S.has_hd) {
          bool jump;
          double s = scatter_fast(R.av2 * S.x1000[linear], jump);
          if (jump) s = scatter_at_jump(av, 0.0, 0.0, false, linear);
          s = R.rs * s;
          if (S.has_h2) R.h2 = s * h2shield_fast(nh2, S, A.ph.v_turb);
          if (S.has_hd) R.hd = s * h2shield_fast(nhd, S, A.ph.v_turb);
        }
        if (S.has_co) {
          const double u = fp64::log10_fast(nco + 1.0), w = fp64::log10_fast(nh2 + 1.0);
          const double tl = R.av2 * (xlambda_lbar(u, w, linear) * (1.0 / 1.086));
          bool jump;
          double s = scatter_fast(tl, jump);
          if (jump) s = scatter_at_jump(av, nco, nh2, true, linear);
          R.co = R.rs * s * coshield_fast(u, w);
        }
        // the C photo-rate's H2 line opacity without its T^0.27, which the cell's lane may still be computing
        if (S.has_ci) R.ci = nh2 > 0.0 ? fp64::powk(fp64::log2k(nh2 * (1.0 / 1.59e21)), 0.45) : 0.0;
      }
    __syncthreads();
    if (S.fast && S.has_ci) {
      for (int i = tid; i < nb * nrays; i += RATES_THREADS) {
        const CellRates &C = cells[i / nrays];
        if (!C.ok) continue;
        RayRates &R = rays[i];
        const double x = fma(C.t27, R.ci, 1.1e-17 * A.col5[((size_t)base * nrays + i) * 5 + 3]);
        const double arg = fma(S.ci_gamma, R.av2, x * fp64::K_LN2);
        float kf;
        const int k = fp64::rint_f(fmaxf(-fp64::d2f(arg), -2.0e6f), kf);
        R.ci = scaled_exp2(R.rs, k, k <= -1999999 ? 0.0 : -arg - fp64::f2d(kf));
      }
      __syncthreads();
    }
    // the photo-reactions: sum over the rays in ray order
    for (int i = tid; i < nb * T.nray; i += RATES_THREADS) {
      const int c = i / T.nray, j = i - c * T.nray;
      const CellRates &C = cells[c];
      if (!C.ok) continue;
      const RayRates *R = rays + c * nrays;
      const int r = __ldg(&T.ray_reac[j]), kind = __ldg(&T.kind[r]);
      double a = __ldg(&T.alpha[r]) * 0.5, k = 0.0;
      if (!__ldg(&T.dup[r]) || dup_selected(T, r, C.t)) {
        switch (kind) {
          case RK_PHOTO_H2: for (int q = 0; q < nrays; q++) k += R[q].h2; break;
          case RK_PHOTO_HD: for (int q = 0; q < nrays; q++) k += R[q].hd; break;
          case RK_PHOTO_CO: for (int q = 0; q < nrays; q++) k += R[q].co; break;
          case RK_PHOTO_CI: for (int q = 0; q < nrays; q++) k += R[q].ci; break;
          default: {
            double g = __ldg(&T.gamma[r]);
            float gf = __ldg(&T.gamma_f[r]);
            if (kind == RK_PHOTD) {
              g = 1.8;
              gf = 1.8f;
              a = 1.7e8 * 2.4e-22 * (C.t < 50.0 ? 3.5e-3 : (C.t < 85.0 ? 4.0e-3 : (C.t < 100.0 ? 5.5e-3 : 7.5e-3)));
            }
            // the exponent's low part, -g av2_lo ln 2/1024, is a few units of 2^-53:
            // it goes into the series' leading 1 by an integer addition
            const float glo = gf * (float)(-fp64::C1 * 9007199254740992.0);
#pragma unroll 2
            for (int q = 0; q < nrays; q++) {
              const double av2 = R[q].av2;
              float kf;
              const int m = fp64::rint_f(fmaxf(-gf * fp64::d2f(av2), -2.0e6f), kf);
              const double x = fma(-g, av2, fp64::flip(fp64::f2d(kf)));
              const double t = m < -1000 * 1024 ? 0.0 : R[q].rs * fp64::exp2_int(m);
              const int lo = __float2int_rn(glo * R[q].av2_lo);
              const double one = __longlong_as_double(0x3ff0000000000000ll + (lo > 0 ? (lo + 1) >> 1 : lo));
              k = fma(t, m < -1000 * 1024 ? 1.0 : fma(x, fp64::exp2_slope(x), one), k);
            }
          }
        }
        k = a * k;
      }
      store_rate_bits(k, r, __ldg(&T.flags[r]), A.rate + (base + c) * nreac, &cells[c].neg);
    }
    // the others, class by class: lanes over (cell, reaction)
    for (int cls = 0; cls < RC_GENERAL; cls++) {
      const int n = T.class_n[cls];
      const int *list = T.other_reac + T.class_off[cls];
      for (int i = tid; i < nb * n; i += RATES_THREADS) {
        const int c = i / n, r = __ldg(&list[i - c * n]);
        const CellRates &C = cells[c];
        if (!C.ok) continue;
        const int flags = __ldg(&T.flags[r]);
        double a = __ldg(&T.alpha[r]), k = 0.0;
        if (!__ldg(&T.dup[r]) || dup_selected(T, r, C.t)) {
          if (cls == RC_CONST) k = a;
          else if (cls == RC_CRP) k = a * C.zeta;
          else {
            // a 2^(b L - g G): the integer parts in FP32, the remainders by FMAs
            int m = 0;
            double x = 0.0;
            bool zero = false, far = false;
            if (cls == RC_BETA || cls == RC_BOTH || cls == RC_CRPHOT) {
              const double b = __ldg(&T.beta[r]);
              float kf;
              m = fp64::rint_f(__ldg(&T.beta_f[r]) * C.Lf, kf);
              x = fma(b, C.Ll, fma(b, C.Lh, fp64::flip(fp64::f2d(kf))));
            }
            if (cls == RC_GAMMA || cls == RC_BOTH) {
              const double g = __ldg(&T.gamma[r]);
              const float gf = __ldg(&T.gamma_f[r]), arg = gf * C.Gf;
              float kf;
              far = fabsf(arg) > 3.0e6f;
              m -= fp64::rint_f(fminf(fmaxf(arg, -3.0e6f), 3.0e6f), kf);
              const double y = fma(g, C.Gl, fma(g, C.Gh, fp64::flip(fp64::f2d(kf))));
              x = (cls == RC_BOTH) ? x - y : fp64::flip(y);
              if (flags & 2) zero = C.t < __ldg(&T.rtmin[r]);
            }
            if (cls == RC_CRPHOT) a = a * C.zeta;
            k = zero ? 0.0 : scaled_exp2(a, m, far ? 0.0 : x);
            if (cls == RC_CRPHOT) k = fp64::div_fast(k * __ldg(&T.gamma[r]), 1.0 - A.ph.omega);
          }
        }
        store_rate_bits(k, r, flags, A.rate + (base + c) * nreac, &cells[c].neg);
      }
    }
    // reactions of the rarer kinds, in the reference's expressions: lanes over cells
    for (int i = tid; i < nb * T.class_n[RC_GENERAL]; i += RATES_THREADS) {
      const int j = i / nb, c = i - j * nb, r = __ldg(&T.other_reac[T.class_off[RC_GENERAL] + j]);
      const CellRates &C = cells[c];
      if (!C.ok) continue;
      const RateRow w = rate_row(T, r);
      bool neg = false;
      int negr = 0;
      const double k = dup_selected(T, r, C.t) ? other_rate(w, C.t, C.td, C.zeta, A.ph) : 0.0;
      store_rate(k, w, r, A.rate + (base + c) * nreac, neg, negr);
      if (neg) atomicMin(&cells[c].neg, negr);
    }
    __syncthreads();
    for (int c = tid >> 5; c < nb; c += RATES_THREADS >> 5) {
      if (!cells[c].ok) rates_cell_general(A, (int)base + c);
      // the lowest-numbered negative rate of the cell, as a negative status
      else if (A.status && (tid & 31) == 0) A.status[base + c] = cells[c].neg == 0x7fffffff ? 0 : -cells[c].neg;
    }
    __syncthreads();
  }
}

}  // namespace

int launch_rates(const pdr_net *net, const pdr_phys &ph, int ncell, int nrays, const double *T,
                 const double *Td, const double *rad, const double *AV, const double *col5, const double *zeta,
                 double *rate, int *status, int sm_count, cudaStream_t st) {
  RatesArgs A;
  A.T = net->rates;
  A.ph = ph;
  A.ncell = ncell;
  A.nrays = nrays;
  A.Tg = T;
  A.Td = Td;
  A.rad = rad;
  A.AV = AV;
  A.col5 = col5;
  A.zeta = zeta;
  A.rate = rate;
  A.status = status;
  RateShield &S = A.S;
  const RateTables &rt = net->rates;
  S.has_h2 = rt.has_h2;
  S.has_hd = rt.has_hd;
  S.has_co = rt.has_co;
  S.has_ci = rt.has_ci;
  S.ci_gamma = rt.ci_gamma;
  const double dopw = ph.v_turb / (1000.0 * 1.0e-8);
  const double r = 8.0e7 / (1.772453851 * dopw), tw = 3.02 * std::pow(r * 1.0e3, -0.064);
  S.taud = 0.5 * 1.497358985e-2 * 1.0e-2 / dopw;
  S.jr_a = r / tw;
  S.jr_b = r / (tw * tw);
  shield_x1000(S.x1000);
  // the general path takes what the fast one's ranges leave out: networks with
  // parameters beyond them, a Doppler width or albedo that is not positive and
  // ordinary, and more rays than a block's shared memory holds
  S.fast = rt.fast_ok && dopw >= 1.0 && dopw <= 1.0e20 && std::fabs(1.0 - ph.omega) >= 1.0e-6 &&
           std::fabs(1.0 - ph.omega) <= 1.0e6 && nrays <= 512;
  // cells per block and round: up to 32, so that the per-cell phase fills a
  // warp, and fewer where that leaves SMs idle
  const size_t per_cell = sizeof(CellRates) + (S.fast ? sizeof(RayRates) * (size_t)nrays : 0);
  constexpr int PER_SM = 3;
  const long long blocks_max = (long long)sm_count * PER_SM;
  long long batch = (ncell + blocks_max - 1) / blocks_max;
  batch = std::min<long long>(std::min<long long>(batch, 32), (long long)(48 * 1024 / per_cell));
  A.batch = (int)std::max<long long>(batch, 1);
  const size_t smem = per_cell * A.batch;
  long long blocks = std::min(((long long)ncell + A.batch - 1) / A.batch, blocks_max);
  rates_kernel<<<(int)blocks, RATES_THREADS, smem, st>>>(A);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "rates_kernel launch");
}

}  // namespace pdr
