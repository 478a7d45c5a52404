// levpop.cu -- batched statistical-equilibrium solves for one coolant
// (the per-cell, per-coolant step of 3DPDR.F90:756-843: FIND_CCOEFF,
// escape_probability after the optical depths are known, solvlevpop).
//
// Coolants of more than 8 levels (CO) take one warp per cell; the lanes share
// its work:
//   field  per radiative pair: CMB + dust Planck background, source function,
//          ray-averaged escape probability beta(tau) with the masing and
//          small-tau guards (escape_probability.F90:51-167; PSEUDO_1D uses ray 6);
//   C_ij   linear-in-T interpolation of each partner's table, partners summed in
//          LAMDA-id order with the para/ortho split (find_Ccoeff.F90:35-147);
//   R_ij = A_ij + B_ij <J_ij> + C_ij (|R| < 1e-50 -> 0);
//   the solvlevpop matrix (transposed rates, diagonal = -row sum, last row
//   1e-8, rhs = density*1e-8, solvlevpop.F90:18-35) held in shared memory and
//   solved either in FP64 by Gaussian elimination with the full pivoting of the
//   reference's Gauss-Jordan (the same pivots), or (mixed) by the FP32 LU factors of the row-equilibrated matrix (partial
//   pivoting) and up to two refinement steps, the residual in FP64 and the
//   correction in FP32, each accepted by the size of the next
//   correction (cells that fail the check are re-solved in FP64, status 2);
//   negative populations are set to zero.
// The fine-structure coolants (at most 8 levels) take a batch of cells per
// block, a lane per (cell, pair), (cell, entry), and for the elimination per
// cell: see levpop_small_kernel.
#include <algorithm>
#include <mutex>
#include <vector>

#include "fp64_fast.cuh"
#include "pdr_internal.h"

namespace pdr {
namespace {

constexpr double KB = 1.38065040e-16, HP = 6.62606896e-27;
constexpr double PI = 3.141592653589793238462643383279502884197;
constexpr unsigned FULL = 0xffffffffu;

// per-warp shared memory: the nlev^2 FP64 rate matrix (before it, the rays'
// escape probabilities), the right-hand side, and one region that has, in turn,
// the radiative pairs' line values and rates up and down with the current
// populations, then what the solve needs: the multipliers, the active indices
// and the solution of the FP64 elimination, or the FP32 factors (beside the
// solution), whose place the elimination takes again for a cell that is
// re-solved.  Side by side they were 24.9 KB a warp for CO mixed and 16.3 KB
// FP64, 9 and 14 warps on an SM; 23.1 and 15.1 KB let 10 and 15: 64,000 cells
// mixed 5.80 -> 5.27 ms, 20,011 cells FP64 3.25 -> 3.10 ms.
struct LevLayout {
  size_t R, lines, b, sp, x, rs, act, Mf, upan, total;
};
__host__ __device__ inline LevLayout levpop_layout(int n, int nrad, bool mixed) {
  auto al = [](size_t v) { return (v + 15) & ~size_t(15); };
  auto most = [](size_t p, size_t q) { return p > q ? p : q; };
  LevLayout L;
  size_t o = 0;
  L.R = o; o += al(8 * (size_t)n * n);
  L.b = o; o += al(8 * (size_t)n);
  L.x = o;
  if (mixed) o += al(8 * (size_t)n);   // kept while the factors and, later, the elimination are in the region
  L.lines = L.Mf = o;
  L.sp = L.lines + al(24 * (size_t)(nrad > 0 ? nrad : 1));
  size_t end = L.sp + al(8 * (size_t)n);
  L.rs = mixed ? o : L.x + al(8 * (size_t)n);
  L.act = L.rs + al(8 * (size_t)n);
  end = most(end, L.act + al(4 * (size_t)n));
  L.upan = o;
  if (mixed) {
    const size_t n4 = ((size_t)n + 3) & ~size_t(3);
    L.upan = L.Mf + al(4 * n4 * (n4 | 1));
    end = most(end, L.upan + al(4 * 6 * n4));   // the panel, the reciprocal pivots, the pivot order
  }
  L.total = end;
  return L;
}

struct LevArgs {
  int ncell, nrays, pseudo1d;
  double metallicity, g2d;
  const double *density, *T, *Td, *partner5, *cdens, *spop, *tau;
  double *pop, *cooling, *line;
  int *status;
};

// magnitude bit pattern of a value: ordered like |x| for finite values
__device__ __forceinline__ long long mag_bits(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffll; }

// (1 - exp(-tau))/tau with the masing and small-tau guards
// (escape_probability.F90:110-125), the comparisons on the bit patterns
__device__ __forceinline__ double escape_ray(double t) {
  const long long bits = __double_as_longlong(t), mag = bits & 0x7fffffffffffffffll;
  constexpr long long SMALL = 0x3e45798ee2308c3all, FIVE = 0x4014000000000000ll, BIG = 0x4085e00000000000ll,
                      INF = 0x7ff0000000000000ll;   // 1e-8, 5, 700, infinity
  if (mag < SMALL) return 1.0;
  if (bits < 0 && mag > FIVE && mag <= INF) return (1.0 - exp(5.0)) / (-5.0);
  if (mag > 0x7e00000000000000ll) return (1.0 - exp(-t)) / t;
  double num = 1.0;   // from 700 on, exp(-t) is below half an ulp of 1
  if (mag < BIG) num = 1.0 - fp64::exp_fast(fp64::flip(t));
  return fp64::div_fast(num, t);   // one division: a warp's lanes have tau on both sides
}

// exp(x) - 1 > 0 as escape_probability.F90 writes it, for x = h nu / k T
__device__ __forceinline__ double planck_expm1(double x) {
  if (x < 690.0 && x > 0.0) return fp64::exp_fast(x) - 1.0;
  return exp(x) - 1.0;
}

// One radiative pair of a cell from its mean escape probability's ray sum:
// the line value and the radiative rates A + B J up and down the pair
__device__ __forceinline__ void radiative_pair(const CoolantTables &C, int pe, double Td, double ngrain, double spi,
                                               double spj, double bsum, int nrays, bool pseudo1d, double &line,
                                               double &down, double &up) {
  // per-pair constants (2 h nu^3 / c^2, the 2.7 K background, the dust
  // emissivity factor) come precomputed with the coolant
  const double tmp2 = C.pair_tmp2[pe];
  const double emis = (2.0 * ngrain) * C.pair_emis[pe];
  const double w = fp64::div_any(1.0, planck_expm1(fp64::div_any(C.pair_hk[pe], Td)));
  const double bb = C.pair_cmb[pe] + tmp2 * (w * emis);
  double S = 0.0, beta = 1.0;
  line = 0.0;
  if (spi != 0.0) {
    const double gi = C.pair_g[2 * pe], gj = C.pair_g[2 * pe + 1];
    const double tpop = fp64::div_any(spj * gi, spi * gj) - 1.0;
    if (fabs(tpop) < 1.0e-50) {
      S = HP * C.freq[C.rad_pairs[pe]] * spi * C.pair_ab[4 * pe] / 4. / PI;
    } else {
      S = fp64::div_any(tmp2, tpop);
      beta = pseudo1d ? bsum : fp64::div_any(bsum, (double)nrays);
    }
    line = fp64::div_any(C.pair_ahf[pe] * spi * beta * (S - bb), S);
  }
  const double field = (1.0 - beta) * S + beta * bb;
  down = C.pair_ab[4 * pe] + C.pair_ab[4 * pe + 1] * field;
  up = C.pair_ab[4 * pe + 2] + C.pair_ab[4 * pe + 3] * field;
}

// Collision partner q at temperature T: its table row, the interpolation step
// and the partner's density (find_Ccoeff.F90:35-147)
__device__ __forceinline__ void partner_at(const CoolantTables &C, int q, double T, const double *p5, int &row,
                                           double &step, double &dens) {
  const double nH = p5[0], nHp = p5[1], ne = p5[2], nHe = p5[3], nH2 = p5[4];
  const int p = C.part[q];
  const double *tp = C.temps + (size_t)q * C.ntemp;
  int klo = 0, khi = 0;
  for (int k = 1; k <= C.ntemp; k++) {
    const double t = __ldg(&tp[k - 1]);
    if (t > T) { klo = k - 1; khi = k; break; }
    else if (t == 0.0) { klo = k - 1; khi = k - 1; break; }
  }
  if (khi == 0) { klo = C.ntemp; khi = C.ntemp; }
  else if (khi == 1) { klo = 1; khi = 1; }
  row = klo - 1;
  step = (klo == khi) ? 0.0 : (T - tp[klo - 1]) / (tp[khi - 1] - tp[klo - 1]);
  if (p == 1 || p == 2) {
    // para and ortho H2
    double f = 0.0;
    if (nH2 > 0.0) {
      f = 1.0 / (1.0 + 9.0 * exp(-170.5 / T));
      if (p == 2) f = 1.0 - f;
    }
    dens = nH2 * f;
  } else {
    dens = (p == 0 ? nH2 : p == 3 ? ne : p == 4 ? nH : p == 5 ? nHe : nHp);
  }
}

// warp argmax of (value, index) with ties resolved to the larger index
__device__ __forceinline__ void argmax_last(long long &v, int &idx) {
  const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
  const bool have = idx >= 0;
  const unsigned mh = __reduce_max_sync(FULL, have ? hi : 0u);
  const unsigned ml = __reduce_max_sync(FULL, (have && hi == mh) ? lo : 0u);
  idx = __reduce_max_sync(FULL, (have && hi == mh && lo == ml) ? idx : -1);
}

// Gaussian elimination with the full pivoting of the reference's Gauss-Jordan
// (solvlevpop.F90:65-174) on a (n x n, row stride n, n <= 64) and one rhs b,
// warp-cooperative; x receives the solution.  The pivots and their order are
// the reference's:
//  * pivot search: the last maximum in row-major order over the unpivoted rows
//    and columns; each lane notes its largest new element as it stores it, so
//    no pass over the matrix is spent on the search;
//  * a row interchange brings the pivot to the diagonal, so one list (act) has
//    the rows and the columns that are still to be pivoted, and behind them the
//    pivots taken, last one first;
//  * elimination: every element of the active rows and columns, b as the last
//    column, updated by one lane with one fused operation.  The pivoted rows
//    keep their part of U and are solved at the end (a row a lane), in place of
//    the Gauss-Jordan's elimination of them at every step.
// What bounds it: the FP64 instructions of the updates, n^3/3 fused ones
// against the n^3/2 pairs of the Gauss-Jordan on the active columns (an FMA
// takes the pipe 64 cycles, a product and a difference 152).  20,011 CO cells:
// 5.41 -> 3.39 ms (errors against 64-bit-exact solutions unchanged, 4.7e-15).
// l: n values, act: n ints, x: n values.  False on a singular matrix: x is then
// the solution of the rows pivoted so far, and b of the others.
__device__ __forceinline__ bool gauss_full(double *a, double *b, int n, double *l, int *act, double *x) {
  const int lane = threadIdx.x & 31;
  long long best = -1;
  int bidx = -1;
  bool ok = true;
  for (int i = lane; i < n; i += 32) act[i] = i;
  for (int e = lane; e < n * n; e += 32) {
    // |a| compared through its bit pattern (the order of non-negative
    // IEEE values), on the integer pipe instead of the FP64 one
    const long long v = mag_bits(a[e]);
    if (v >= best) { best = v; bidx = e; }
  }
  __syncwarp();
  int np = 0;   // pivots taken
  for (; np < n; np++) {
    argmax_last(best, bidx);
    if (bidx < 0) { ok = false; break; }
    const int irow = bidx / n, icol = bidx - irow * n;
    const int nact = n - 1 - np;   // indices that stay active
    // the pivot leaves the list, the last one takes its place
    const int hit = (lane <= nact && act[lane] == icol) ? lane : ((lane + 32 <= nact && act[lane + 32] == icol) ? lane + 32 : -1);
    __syncwarp();
    if (hit >= 0) {
      act[hit] = act[nact];
      act[nact] = icol;
    }
    __syncwarp();
    if (irow != icol) {
      // row interchange of the columns that matter (the pivot column with them)
      for (int q = lane; q <= nact; q += 32) {
        const int c = act[q];
        const double d = a[irow * n + c];
        a[irow * n + c] = a[icol * n + c];
        a[icol * n + c] = d;
      }
      if (lane == 0) { const double d = b[irow]; b[irow] = b[icol]; b[icol] = d; }
      __syncwarp();
    }
    const double piv = a[icol * n + icol];
    if (piv == 0.0) { ok = false; break; }
    const double pivinv = fp64::rcp_near(piv);
    if (lane == 0) x[icol] = pivinv;
    for (int p = lane; p < nact; p += 32) l[p] = a[act[p] * n + icol] * pivinv;
    __syncwarp();
    const int w = nact + 1;   // active columns and b
    const float inv = 1.0f / (float)w;
    best = -1;
    bidx = -1;
    for (int e = lane; e < nact * w; e += 32) {
      const int p = __float2int_rz(__fmul_rn((float)e + 0.5f, inv));   // e / w, exact for e < 64^2
      const int q = e - p * w, r = act[p];
      // one path for the matrix and b: a branch would pay the FP64 instruction twice
      const bool mat = q < nact;
      const int c = mat ? act[q] : 0, at = r * n + c;
      double *dst = mat ? a + at : b + r;
      const double v = fma(-(mat ? a[icol * n + c] : b[icol]), l[p], *dst);
      *dst = v;
      if (mat) {
        const long long m = mag_bits(v);
        if (m > best || (m == best && at > bidx)) { best = m; bidx = at; }
      }
    }
    __syncwarp();
  }
  __syncwarp();
  // U x = b, pivot k = act[n - 1 - k]; lane j keeps the running values of pivots j and j + 32
  const int c0 = lane < np ? act[n - 1 - lane] : 0, c1 = lane + 32 < np ? act[n - 33 - lane] : 0;
  double b0 = b[c0], b1 = b[c1];
  const double p0 = x[c0], p1 = x[c1];
  for (int i = lane; i < n - np; i += 32) x[act[i]] = b[act[i]];   // (singular) the rows that have no pivot
  for (int k = np - 1; k >= 0; k--) {
    const int c = act[n - 1 - k];
    const double xk = __shfl_sync(FULL, (k < 32 ? b0 : b1) * (k < 32 ? p0 : p1), k & 31);
    if (lane == 0) x[c] = xk;
    b0 = fma(-a[c0 * n + c], xk, b0);
    if (k > 32) b1 = fma(-a[c1 * n + c], xk, b1);
  }
  __syncwarp();
  return ok;
}

// The mixed solve's acceptance test on the correction s that a further
// refinement step would make to population x: above 1e-6 of the coolant
// density it must be below 1e-7 of x, above 1e-12 of the density below 1e-4
// of x (ten times inside the 1e-6 and 1e-3 the results are held to), and it
// must contract (at most half the previous correction, or negligible).  A NaN
// among them is refused; as itself is a finite FP32 value.
__device__ __forceinline__ bool refine_ok(double ax, double as, double prev, double dens) {
  const bool contracts = as <= 0.5 * prev || as <= 1.0e-12 * ax;
  if (!(ax <= 1.0e-6 * dens)) return as <= 1.0e-7 * ax && contracts;
  if (!(ax <= 1.0e-12 * dens)) return as <= 1.0e-4 * ax && contracts;
  return true;
}

// ---- the mixed solve's FP32 factors ----
//
// LU with partial pivoting (largest magnitude among the rows not yet pivoted,
// lowest row on ties) of the row-equilibrated matrix, and solves with it.  They
// only precondition the FP64 refinement, so they need not follow the
// reference's full-pivot order.  n4 is the order rounded up to a multiple of
// four (identity rows and columns behind the matrix), ld its odd row stride.
// Lane i owns rows i and i + 32; rows stay in place.  Panels of four columns,
// the row's panel entries in registers, so that a trailing entry is loaded
// and stored once for four updates; the solves move four columns per round of
// shuffles.  (The Gauss-Jordan inverse this replaces updated all n^2 entries
// at each of n steps, one dependent load, FMA and store after the other.)
// 64,000 CO cells, mixed: 14.9 -> 5.3 ms (6.1 before the shared row sums,
// the separate pass over the radiative entries and the smaller layout).

// n4 x n4 factors at a; upan: 4 n4 floats, 16-byte aligned; perm[k] the pivot
// row of step k, dinv[k] its reciprocal pivot
__device__ __forceinline__ bool lu_pp(float *a, int n4, int ld, float *upan, int *perm, float *dinv) {
  const int lane = threadIdx.x & 31;
  const bool has1 = lane + 32 < n4;
  float *row0 = a + (lane < n4 ? lane : 0) * ld, *row1 = a + (has1 ? lane + 32 : 0) * ld;
  bool free0 = lane < n4, free1 = has1, ok = true;
#pragma unroll 1
  for (int k0 = 0; k0 < n4; k0 += 4) {
    float r0[4], r1[4];
    int pt[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      r0[t] = row0[k0 + t];
      r1[t] = has1 ? row1[k0 + t] : 0.0f;
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const unsigned m0 = free0 ? __float_as_uint(fabsf(r0[t])) : 0u, m1 = free1 ? __float_as_uint(fabsf(r1[t])) : 0u;
      const unsigned mx = __reduce_max_sync(FULL, max(m0, m1));
      const unsigned b0 = __ballot_sync(FULL, free0 && m0 == mx), b1 = __ballot_sync(FULL, free1 && m1 == mx);
      ok = ok && mx != 0u;   // a column of zeros: finish on any row, the caller discards the factors
      const bool hi = b0 == 0u;
      const int src = __ffs(hi ? b1 : b0) - 1;
      const int p = max(src, 0) + (hi ? 32 : 0);
      pt[t] = p;
      float u[4];
#pragma unroll
      for (int j = t; j < 4; j++) u[j] = __shfl_sync(FULL, hi ? r1[j] : r0[j], p & 31);
      const float rinv = __fdividef(1.0f, u[t]);
      if (lane == (p & 31)) {
        if (hi) free1 = false;
        else free0 = false;
        perm[k0 + t] = p;
        dinv[k0 + t] = rinv;
      }
      if (free0) {
        r0[t] *= rinv;
#pragma unroll
        for (int j = t + 1; j < 4; j++) r0[j] = fmaf(-r0[t], u[j], r0[j]);
      }
      if (free1) {
        r1[t] *= rinv;
#pragma unroll
        for (int j = t + 1; j < 4; j++) r1[j] = fmaf(-r1[t], u[j], r1[j]);
      }
    }
    if (lane < n4) {
#pragma unroll
      for (int t = 0; t < 4; t++) row0[k0 + t] = r0[t];
    }
    if (has1) {
#pragma unroll
      for (int t = 0; t < 4; t++) row1[k0 + t] = r1[t];
    }
    __syncwarp();
    // the pivot rows' entries right of the panel
    const float m10 = a[pt[1] * ld + k0], m20 = a[pt[2] * ld + k0], m21 = a[pt[2] * ld + k0 + 1];
    const float m30 = a[pt[3] * ld + k0], m31 = a[pt[3] * ld + k0 + 1], m32 = a[pt[3] * ld + k0 + 2];
    for (int j = k0 + 4 + lane; j < n4; j += 32) {
      const float u0 = a[pt[0] * ld + j];
      const float u1 = fmaf(-m10, u0, a[pt[1] * ld + j]);
      const float u2 = fmaf(-m21, u1, fmaf(-m20, u0, a[pt[2] * ld + j]));
      const float u3 = fmaf(-m32, u2, fmaf(-m31, u1, fmaf(-m30, u0, a[pt[3] * ld + j])));
      a[pt[1] * ld + j] = u1;
      a[pt[2] * ld + j] = u2;
      a[pt[3] * ld + j] = u3;
      reinterpret_cast<float4 *>(upan)[j] = make_float4(u0, u1, u2, u3);
    }
    __syncwarp();
    const bool any1 = __any_sync(FULL, free1);
#pragma unroll 1
    for (int j = k0 + 4; j < n4; j += 4) {
      float4 u[4];
      float s0[4], s1[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        u[c] = reinterpret_cast<const float4 *>(upan)[j + c];
        s0[c] = row0[j + c];
      }
      if (any1) {
#pragma unroll
        for (int c = 0; c < 4; c++) s1[c] = row1[j + c];
      }
      if (free0) {
#pragma unroll
        for (int c = 0; c < 4; c++)
          row0[j + c] = fmaf(-r0[3], u[c].w, fmaf(-r0[2], u[c].z, fmaf(-r0[1], u[c].y, fmaf(-r0[0], u[c].x, s0[c]))));
      }
      if (free1) {
#pragma unroll
        for (int c = 0; c < 4; c++)
          row1[j + c] = fmaf(-r1[3], u[c].w, fmaf(-r1[2], u[c].z, fmaf(-r1[1], u[c].y, fmaf(-r1[0], u[c].x, s1[c]))));
      }
    }
    __syncwarp();
  }
  return ok;
}

// x = (LU)^-1 b: (b0, b1) the right-hand side's entries lane and lane + 32, the
// solution's come back in them
__device__ __forceinline__ void lu_pp_solve(const float *a, int n4, int ld, const int *perm, const float *dinv, float &b0,
                                            float &b1) {
  const int lane = threadIdx.x & 31;
  const int p0 = lane < n4 ? perm[lane] : 0, p1 = lane + 32 < n4 ? perm[lane + 32] : 0;
  const float *row0 = a + p0 * ld, *row1 = a + p1 * ld;
  {
    // into pivot order
    const float x0 = __shfl_sync(FULL, b0, p0 & 31), x1 = __shfl_sync(FULL, b1, p0 & 31);
    const float y0 = __shfl_sync(FULL, b0, p1 & 31), y1 = __shfl_sync(FULL, b1, p1 & 31);
    b0 = p0 < 32 ? x0 : x1;
    b1 = p1 < 32 ? y0 : y1;
  }
#pragma unroll 1
  for (int k = 0; k < n4; k += 4) {
    const float *q1 = a + perm[k + 1] * ld + k, *q2 = a + perm[k + 2] * ld + k, *q3 = a + perm[k + 3] * ld + k;
    const bool hi = k >= 32;
    const float c = hi ? b1 : b0;
    const float y0 = __shfl_sync(FULL, c, k & 31), c1 = __shfl_sync(FULL, c, (k + 1) & 31);
    const float c2 = __shfl_sync(FULL, c, (k + 2) & 31), c3 = __shfl_sync(FULL, c, (k + 3) & 31);
    const float y1 = fmaf(-q1[0], y0, c1);
    const float y2 = fmaf(-q2[1], y1, fmaf(-q2[0], y0, c2));
    const float y3 = fmaf(-q3[2], y2, fmaf(-q3[1], y1, fmaf(-q3[0], y0, c3)));
    if (lane > k) b0 = fmaf(-row0[k], y0, b0);
    if (lane > k + 1) b0 = fmaf(-row0[k + 1], y1, b0);
    if (lane > k + 2) b0 = fmaf(-row0[k + 2], y2, b0);
    if (lane > k + 3) b0 = fmaf(-row0[k + 3], y3, b0);
    if (lane + 32 > k) b1 = fmaf(-row1[k], y0, b1);
    if (lane + 32 > k + 1) b1 = fmaf(-row1[k + 1], y1, b1);
    if (lane + 32 > k + 2) b1 = fmaf(-row1[k + 2], y2, b1);
    if (lane + 32 > k + 3) b1 = fmaf(-row1[k + 3], y3, b1);
  }
#pragma unroll 1
  for (int k = n4 - 4; k >= 0; k -= 4) {
    const float *q0 = a + perm[k] * ld + k, *q1 = a + perm[k + 1] * ld + k, *q2 = a + perm[k + 2] * ld + k;
    const bool hi = k >= 32;
    const float c = hi ? b1 : b0;
    const float c0 = __shfl_sync(FULL, c, k & 31), c1 = __shfl_sync(FULL, c, (k + 1) & 31);
    const float c2 = __shfl_sync(FULL, c, (k + 2) & 31), c3 = __shfl_sync(FULL, c, (k + 3) & 31);
    const float x3 = c3 * dinv[k + 3];
    const float x2 = fmaf(-q2[3], x3, c2) * dinv[k + 2];
    const float x1 = fmaf(-q1[2], x2, fmaf(-q1[3], x3, c1)) * dinv[k + 1];
    const float x0 = fmaf(-q0[1], x1, fmaf(-q0[2], x2, fmaf(-q0[3], x3, c0))) * dinv[k];
    const int at = lane - (k & 31);   // this lane's place in the block, 0..3
    const float x = at == 0 ? x0 : at == 1 ? x1 : at == 2 ? x2 : x3;
    if (lane < k) b0 = fmaf(-row0[k], x0, fmaf(-row0[k + 1], x1, fmaf(-row0[k + 2], x2, fmaf(-row0[k + 3], x3, b0))));
    if (lane + 32 < k) b1 = fmaf(-row1[k], x0, fmaf(-row1[k + 1], x1, fmaf(-row1[k + 2], x2, fmaf(-row1[k + 3], x3, b1))));
    if (at >= 0 && at < 4) {
      if (hi) b1 = x;
      else b0 = x;
    }
  }
}

// Sums over the columns of an n x n matrix (n <= 64): s0 of row `lane` and s1
// of row lane + 32, both taken on from their values at entry; term(i, j, v) is
// v with the term of (i, j) added.  A lane has a row; the rows from 32 on would
// leave most lanes idle at full price, so up to four lanes share one of them
// (CO's 41 rows: 57 FP64 instructions in place of 82).
template <class Term>
__device__ __forceinline__ void row_sums(int n, Term term, double &s0, double &s1) {
  const int lane = threadIdx.x & 31, extra = n - 32;
  const int i0 = min(lane, n - 1);
#pragma unroll 4
  for (int j = 0; j < n; j++) s0 = term(i0, j, s0);
  if (extra <= 0) return;
  const int parts = min(4, 32 / extra), len = (n + parts - 1) / parts;
  const int r = lane / parts, j0 = (lane - r * parts) * len, j1 = min(n, j0 + len);
  const int i1 = 32 + min(r, extra - 1);
  double t = 0.0;
#pragma unroll 4
  for (int k = 0; k < len; k++)
    if (j0 + k < j1) t = term(i1, j0 + k, t);
  for (int k = 0; k < parts; k++) s1 += __shfl_sync(FULL, t, (lane * parts + k) & 31);
}

template <bool MIXED>
__global__ void __launch_bounds__(256) levpop_kernel(const __grid_constant__ CoolantTables C,
                                                     const __grid_constant__ LevArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int n = C.nlev, nn = n * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LevLayout L = levpop_layout(n, C.nrad, MIXED);
  unsigned char *base = smem + L.total * warp;
  double *R = reinterpret_cast<double *>(base + L.R);          // rates, then the solvlevpop matrix
  double *lines = reinterpret_cast<double *>(base + L.lines);  // line values of the radiative pairs
  double *b = reinterpret_cast<double *>(base + L.b);
  double *sp = reinterpret_cast<double *>(base + L.sp);
  double *x = reinterpret_cast<double *>(base + L.x);
  double *rs = reinterpret_cast<double *>(base + L.rs);        // multipliers of the elimination
  int *act = reinterpret_cast<int *>(base + L.act);            // its active columns
  const int wpb = blockDim.x >> 5;
  for (int cell = blockIdx.x * wpb + warp; cell < A.ncell; cell += gridDim.x * wpb) {
    const double T = A.T[cell], Td = A.Td[cell], rho = A.density[cell];
    const double *p5 = A.partner5 + (size_t)cell * 5;
    for (int i = lane; i < n; i += 32) sp[i] = A.spop[(size_t)cell * n + i];
    // ---- escape probabilities and the radiative terms ----
    // every (pair, ray) has a lane of its own, the values (in the matrix's
    // memory, a chunk of the rays at a time) are then added in ray order.  The
    // pairs with no radiative coupling in either direction (A = B = 0) leave R
    // unchanged and their line term zero: only the radiative pairs are visited
    const double ngrain = 2.0e-12 * rho * A.metallicity * 100. / A.g2d;
    const double *tau = A.tau + (size_t)cell * C.nlin * A.nrays;
    double *radd = lines + C.nrad, *radu = radd + C.nrad;   // ray sums, then the radiative rates
    const int nrad = C.nrad, chunk = max(1, min(A.nrays, nn / max(nrad, 1)));
    for (int r0 = 0; r0 < A.nrays; r0 += chunk) {
      const int nr = min(chunk, A.nrays - r0);
      const float inv = 1.0f / (float)nr;
      for (int e = lane; e < nrad * nr; e += 32) {
        const int pe = __float2int_rz(__fmul_rn((float)e + 0.5f, inv)), r = r0 + e - pe * nr;
        const int li = (C.pair_ij[pe] >> 16) - 1;
        R[e] = escape_ray((A.pseudo1d && r != 6) ? 1.0e50 : (li >= 0 ? tau[li * A.nrays + r] : 0.0));
      }
      __syncwarp();
      for (int pe = lane; pe < nrad; pe += 32) {
        double bsum = r0 ? radd[pe] : 0.0;
        for (int r = 0; r < nr; r++) bsum += R[pe * nr + r];
        radd[pe] = bsum;
      }
      __syncwarp();
    }
    for (int pe = lane; pe < nrad; pe += 32) {
      const int ij = C.pair_ij[pe];
      double line, down, up;
      radiative_pair(C, pe, Td, ngrain, sp[ij & 0xff], sp[(ij >> 8) & 0xff], radd[pe], A.nrays, A.pseudo1d != 0, line,
                     down, up);
      lines[pe] = line;
      radd[pe] = down;
      radu[pe] = up;
    }
    __syncwarp();
    // ---- rates: the partners' interpolated collision rates, then the
    // radiative ones; each partner's bracket is found by one lane ----
    {
      int row = 0;
      double step = 0.0, dens = 0.0;
      if (lane < C.npart) partner_at(C, lane, T, p5, row, step, dens);
      for (int q = 0; q < C.npart; q++) {
        const size_t at = ((size_t)q * C.ntemp + __shfl_sync(FULL, row, q)) * nn;
        const double st = __shfl_sync(FULL, step, q), dq = __shfl_sync(FULL, dens, q);
        const double *lo = C.col + at, *df = C.dcol + at;
        const bool first = q == 0, last = q == C.npart - 1;
#pragma unroll 2
        for (int e = lane; e < nn; e += 32) {
          double v = fma(fma(__ldg(&df[e]), st, __ldg(&lo[e])), dq, first ? 0.0 : R[e]);
          // the radiative entries get their term, and the threshold, below
          if (last && !(nrad && __ldg(&C.pair_of[e])) && mag_bits(v) < 0x358dee7a4ad4b81fll) v = 0.0;   // 1e-50
          R[e] = v;
        }
      }
      __syncwarp();
      // the radiative entries, two a pair: added as they are made they would
      // cost nearly every warp of entries an FP64 add
      if (C.npart > 0)
        for (int k = lane; k < 2 * nrad; k += 32) {
          const int pe = k >> 1, ij = C.pair_ij[pe], i = ij & 0xff, j = (ij >> 8) & 0xff;
          const int e = (k & 1) ? j * n + i : i * n + j;
          const double v = ((k & 1) ? radu[pe] : radd[pe]) + R[e];
          R[e] = mag_bits(v) < 0x358dee7a4ad4b81fll ? 0.0 : v;
        }
      if (C.npart == 0)
        for (int e = lane; e < nn; e += 32) {
          const int po = nrad ? __ldg(&C.pair_of[e]) : 0;
          const double v = po ? (po > 0 ? radd[po - 1] : radu[-po - 1]) : 0.0;
          R[e] = fabs(v) < 1.0e-50 ? 0.0 : v;
        }
    }
    __syncwarp();
    // the cooling rate: the sum of the line values (the non-radiative pairs
    // contribute zeros), by all lanes: an FP64 add costs a warp the same
    // whatever its lanes, and one lane's 40 of CO were a twentieth of the kernel
    {
      double cool = 0.0;
      for (int pe = lane; pe < C.nrad; pe += 32) cool += lines[pe];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) cool += __shfl_xor_sync(FULL, cool, o);
      if (lane == 0) A.cooling[cell] = cool;
    }
    if (A.line) {
      double *lo = A.line + (size_t)cell * nn;
      for (int e = lane; e < nn; e += 32) lo[e] = 0.0;
      __syncwarp();
      for (int pe = lane; pe < C.nrad; pe += 32) lo[C.rad_pairs[pe]] = lines[pe];
    }
    __syncwarp();
    // ---- solvlevpop matrix: transpose, diagonal -sum, conservation row ----
    {
      double s0 = 0.0, s1 = 0.0;
      row_sums(n, [&](int i, int j, double v) { return v + R[i * n + j]; }, s0, s1);
      if (lane < n) b[lane] = s0;
      if (lane + 32 < n) b[lane + 32] = s1;
    }
    __syncwarp();
    for (int e = lane; e < nn; e += 32) {
      const int i = e / n, j = e - i * n;
      if (j > i) { const double t = R[e]; R[e] = R[j * n + i]; R[j * n + i] = t; }
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) R[i * n + i] = -b[i];
    __syncwarp();
    for (int i = lane; i < n; i += 32) { R[(n - 1) * n + i] = 1.0e-8; b[i] = 0.0; }
    __syncwarp();
    const double dens = A.cdens[cell];
    if (lane == 0) b[n - 1] = dens * 1.0e-8;
    __syncwarp();
    bool ok, redo = false;
    if constexpr (!MIXED) {
      ok = gauss_full(R, b, n, rs, act, x);
    } else {
      // FP32 copy of the matrix with its rows equilibrated in FP32 (D M, D =
      // 1 / row maximum), its LU factors, then x = inv(DM) D b and up to two
      // refinement steps x += inv(DM) D (b - M x) with the residual in FP64
      // and the correction in FP32.  Each step is accepted by the size of the
      // correction the next would make (refine_ok); otherwise, and where the
      // matrix has entries that FP32 cannot hold (2^127 and beyond, NaN), the
      // cell is re-solved by the FP64 elimination (R is intact).
      float *Mf = reinterpret_cast<float *>(base + L.Mf);
      const int n4 = (n + 3) & ~3, ld = n4 | 1;
      float *upan = reinterpret_cast<float *>(base + L.upan), *dinv = upan + 4 * n4;
      int *perm = reinterpret_cast<int *>(dinv + n4);
      // rows as columns of R^T would be: lane i scales rows i and i + 32
      float s0 = 1.0f, s1 = 1.0f;
      int top = 0;   // the largest magnitude's upper word
      for (int i = lane; i < n4; i += 32) {
        float mx = 0.0f;
        for (int l = 0; l < n4; l++) {
          const double r = (i < n && l < n) ? R[i * n + l] : (i == l ? 1.0 : 0.0);
          const float v = fp64::d2f(r);
          top = max(top, fp64::hi32(r) & 0x7fffffff);
          Mf[i * ld + l] = v;
          mx = fmaxf(mx, fabsf(v));
        }
        const float sc = (mx > 0.0f) ? 1.0f / mx : 1.0f;
        for (int l = 0; l < n4; l++) Mf[i * ld + l] *= sc;
        if (i < 32) s0 = sc;
        else s1 = sc;
      }
      __syncwarp();
      ok = __all_sync(FULL, top < 0x47e00000);   // 2^127
      bool good = false;
      if (ok) {
        ok = lu_pp(Mf, n4, ld, upan, perm, dinv);
        // b is zero but for its last entry
        float c0 = lane == n - 1 ? s0 : 0.0f, c1 = lane + 32 == n - 1 ? s1 : 0.0f;
        lu_pp_solve(Mf, n4, ld, perm, dinv, c0, c1);
        const double bl = b[n - 1];
        if (lane < n) x[lane] = (double)c0 * bl;
        if (lane + 32 < n) x[lane + 32] = (double)c1 * bl;
        float prev0 = 0.0f, prev1 = 0.0f;
        for (int it = 0; it < 3 && ok && !good; it++) {
          __syncwarp();
          double d0 = lane < n ? b[lane] : 0.0, d1 = lane + 32 < n ? b[lane + 32] : 0.0;
          row_sums(n, [&](int i, int l, double v) { return fma(-R[i * n + l], x[l], v); }, d0, d1);
          __syncwarp();
          c0 = lane < n ? (float)d0 * s0 : 0.0f;
          c1 = lane + 32 < n ? (float)d1 * s1 : 0.0f;
          lu_pp_solve(Mf, n4, ld, perm, dinv, c0, c1);
          bool bad = false;
          auto step = [&](int i, float c, float &prev) {
            const double sd = (double)c;
            // from the second correction on, the correction is also the test of
            // the previous one
            if (it > 0 && (!(fabsf(c) < INFINITY) || !refine_ok(fabs(x[i]), fabs(sd), (double)prev, dens))) bad = true;
            if (it < 2) {
              x[i] += sd;
              prev = fabsf(c);
            }
          };
          if (lane < n) step(lane, c0, prev0);
          if (lane + 32 < n) step(lane + 32, c1, prev1);
          good = (it > 0) && !__any_sync(FULL, bad);
        }
      }
      if (!ok || !good) {
        __syncwarp();
        for (int i = lane; i < n; i += 32) b[i] = 0.0;
        __syncwarp();
        if (lane == 0) b[n - 1] = dens * 1.0e-8;
        __syncwarp();
        ok = gauss_full(R, b, n, rs, act, x);
        redo = true;
      }
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
      double v = x[i];
      if (v < 0.0) v = 0.0;
      A.pop[(size_t)cell * n + i] = v;
    }
    if (lane == 0 && A.status) A.status[cell] = ok ? (redo ? 2 : 0) : 1;
    __syncwarp();
  }
}

// ---- coolants of at most 8 levels ----

constexpr int SMALL_LEVELS = 8, SMALL_THREADS = 128;

// per-cell shared memory of the small kernel, in doubles (odd, so that cells
// side by side fall in distinct banks)
struct SmallLayout {
  int R, b, sp, lines, down, up, step, dens, total;
};
__host__ __device__ inline SmallLayout small_layout(int n, int nrad, int npart) {
  SmallLayout L;
  int o = 0;
  L.R = o; o += n * n;
  L.b = o; o += n;
  L.sp = o; o += n;
  L.lines = o; o += nrad;
  L.down = o; o += nrad;
  L.up = o; o += nrad;
  L.step = o; o += npart;
  L.dens = o; o += npart;
  L.total = o | 1;
  return L;
}

// The reference's Gauss-Jordan elimination by one thread: the pivot order and
// the reference's unfused products, on the columns still to be pivoted.
__device__ __forceinline__ bool gauss_jordan_thread(double *a, double *b, int n) {
  unsigned used = 0;
  for (int it = 0; it < n; it++) {
    long long best = -1;
    int irow = -1, icol = -1;
    for (int i = 0; i < n; i++) {
      if ((used >> i) & 1u) continue;
      for (int j = 0; j < n; j++)
        if (!((used >> j) & 1u)) {
          const long long v = mag_bits(a[i * n + j]);
          if (v >= best) { best = v; irow = i; icol = j; }
        }
    }
    used |= 1u << icol;
    if (irow != icol) {
      for (int l = 0; l < n; l++)
        if (l == icol || !((used >> l) & 1u)) {
          const double d = a[irow * n + l];
          a[irow * n + l] = a[icol * n + l];
          a[icol * n + l] = d;
        }
      const double d = b[irow];
      b[irow] = b[icol];
      b[icol] = d;
    }
    const double piv = a[icol * n + icol];
    if (piv == 0.0) return false;
    const double pivinv = fp64::div_any(1.0, piv);
    for (int l = 0; l < n; l++)
      if (!((used >> l) & 1u)) a[icol * n + l] = a[icol * n + l] * pivinv;
    const double bp = b[icol] * pivinv;
    b[icol] = bp;
    for (int ll = 0; ll < n; ll++) {
      if (ll == icol) continue;
      const double dum = a[ll * n + icol];
      for (int l = 0; l < n; l++)
        if (!((used >> l) & 1u)) a[ll * n + l] = __dsub_rn(a[ll * n + l], __dmul_rn(a[icol * n + l], dum));
      b[ll] = __dsub_rn(b[ll], __dmul_rn(bp, dum));
    }
  }
  return true;
}

// A batch of cells per block: a lane per (cell, partner), (cell, pair), (cell,
// entry), (cell, row) and, for the elimination, per cell.  What bounds it: the
// FP64 pipe.  One warp per cell left 23 of 32 lanes idle in the escape
// probabilities of C+'s nine pairs and all but one row's worth in the 5 x 5
// elimination.  100,000 C+ cells, 12 rays, with the
// line output: 4.23 -> 0.62 ms.
__global__ void __launch_bounds__(SMALL_THREADS, 6) levpop_small_kernel(const __grid_constant__ CoolantTables C,
                                                                       const __grid_constant__ LevArgs A, int batch) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int n = C.nlev, nn = n * n, nrad = C.nrad, npart = C.npart, tid = threadIdx.x;
  const SmallLayout L = small_layout(n, nrad, npart);
  double *cells = reinterpret_cast<double *>(smem);
  int *rows = reinterpret_cast<int *>(cells + (size_t)batch * L.total);   // [batch][npart]
  for (long long base = (long long)blockIdx.x * batch; base < A.ncell; base += (long long)gridDim.x * batch) {
    const int nb = (int)min((long long)batch, A.ncell - base);
    for (int i = tid; i < nb * n; i += SMALL_THREADS) cells[(i / n) * L.total + L.sp + i % n] = A.spop[base * n + i];
    for (int i = tid; i < nb * npart; i += SMALL_THREADS) {
      const int c = i / npart, q = i - c * npart;
      double *S = cells + c * L.total;
      partner_at(C, q, A.T[base + c], A.partner5 + (size_t)(base + c) * 5, rows[i], S[L.step + q], S[L.dens + q]);
    }
    __syncthreads();
    for (int i = tid; i < nb * nrad; i += SMALL_THREADS) {
      const int c = i / nrad, pe = i - c * nrad, ij = C.pair_ij[pe], li = (ij >> 16) - 1;
      double *S = cells + c * L.total;
      const double *tau = A.tau + ((size_t)(base + c) * C.nlin + (li >= 0 ? li : 0)) * A.nrays;
      double bsum = 0.0;
      for (int r = 0; r < A.nrays; r++)
        bsum += escape_ray((A.pseudo1d && r != 6) ? 1.0e50 : (li >= 0 ? tau[r] : 0.0));
      const double ngrain = 2.0e-12 * A.density[base + c] * A.metallicity * 100. / A.g2d;
      radiative_pair(C, pe, A.Td[base + c], ngrain, S[L.sp + (ij & 0xff)], S[L.sp + ((ij >> 8) & 0xff)], bsum, A.nrays,
                     A.pseudo1d != 0, S[L.lines + pe], S[L.down + pe], S[L.up + pe]);
    }
    __syncthreads();
    for (int i = tid; i < nb * nn; i += SMALL_THREADS) {
      const int c = i / nn, e = i - c * nn;
      double *S = cells + c * L.total;
      double v = 0.0;
      for (int q = 0; q < npart; q++) {
        const size_t at = ((size_t)q * C.ntemp + rows[c * npart + q]) * nn + e;
        v = fma(fma(__ldg(&C.dcol[at]), S[L.step + q], __ldg(&C.col[at])), S[L.dens + q], v);
      }
      const int po = nrad ? __ldg(&C.pair_of[e]) : 0;
      if (po) v = S[po > 0 ? L.down + po - 1 : L.up - po - 1] + v;
      if (mag_bits(v) < 0x358dee7a4ad4b81fll) v = 0.0;   // 1e-50
      S[L.R + e] = v;
      // the line emission, zero but for the radiative pairs
      if (A.line) A.line[(size_t)base * nn + i] = po > 0 ? S[L.lines + po - 1] : 0.0;
    }
    __syncthreads();
    for (int i = tid; i < nb * n; i += SMALL_THREADS) {
      const int c = i / n, r = i - c * n;
      double *S = cells + c * L.total;
      double out = 0.0;
      for (int j = 0; j < n; j++) out = out + S[L.R + r * n + j];
      S[L.b + r] = out;
    }
    __syncthreads();
    for (int c = tid; c < nb; c += SMALL_THREADS) {
      double *S = cells + c * L.total, *R = S + L.R, *b = S + L.b;
      // the cooling rate: the line values in row-major order
      double cool = 0.0;
      for (int pe = 0; pe < nrad; pe++) cool = cool + S[L.lines + pe];
      A.cooling[base + c] = cool;
      // the solvlevpop matrix: transpose, diagonal -sum, conservation row
      for (int i = 0; i < n; i++) {
        for (int j = i + 1; j < n; j++) {
          const double t = R[i * n + j];
          R[i * n + j] = R[j * n + i];
          R[j * n + i] = t;
        }
        R[i * n + i] = -b[i];
      }
      for (int j = 0; j < n; j++) {
        R[(n - 1) * n + j] = 1.0e-8;
        b[j] = 0.0;
      }
      b[n - 1] = A.cdens[base + c] * 1.0e-8;
      const bool ok = gauss_jordan_thread(R, b, n);
      if (A.status) A.status[base + c] = ok ? 0 : 1;
    }
    __syncthreads();
    for (int i = tid; i < nb * n; i += SMALL_THREADS) {
      double v = cells[(i / n) * L.total + L.b + i % n];
      if (v < 0.0) v = 0.0;
      A.pop[base * n + i] = v;
    }
    __syncthreads();
  }
}

}  // namespace

size_t levpop_smem_per_warp(int n, int nrad, bool mixed) { return levpop_layout(n, nrad, mixed).total; }

namespace {
// LTE populations of one cell per thread: CALCULATE_PARTITION_FUNCTION and
// CALCULATE_LTE_POPULATIONS (3DPDR.F90:1847-1894), the same operation order;
// the reference STOPs when the populations do not add up to the density
// within 1e-3 -- here the cell's status is set to 1 instead.
__global__ void lte_kernel(CoolantTables C, int ncell, const double *__restrict__ T,
                           const double *__restrict__ density, double *__restrict__ pop, int *status) {
  for (int cell = blockIdx.x * blockDim.x + threadIdx.x; cell < ncell; cell += gridDim.x * blockDim.x) {
    const double t = T[cell], d = density[cell];
    double z = 0.0;
    for (int i = 0; i < C.nlev; i++) z = z + C.weights[i] * exp(-C.energies[i] / KB / t);
    double tot = 0.0;
    for (int i = 0; i < C.nlev; i++) {
      const double p = d * C.weights[i] * exp(-C.energies[i] / KB / t) / z;
      pop[(size_t)cell * C.nlev + i] = p;
      tot = tot + p;
    }
    if (status) status[cell] = (fabs(tot - d) / d > 1.0e-3) ? 1 : 0;
  }
}
}  // namespace

int launch_lte(const pdr_coolant *c, int ncell, const double *T, const double *density, double *pop, int *status,
               int sm_count, cudaStream_t st) {
  const int blocks = std::min((ncell + 127) / 128, sm_count * 8);
  lte_kernel<<<blocks, 128, 0, st>>>(c->dev, ncell, T, density, pop, status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "lte_kernel launch");
}

int launch_levpop(const pdr_coolant *c, const LevArgsHost &h, bool mixed, int sm_count, cudaStream_t st) {
  LevArgs A;
  A.ncell = h.ncell; A.nrays = h.nrays; A.pseudo1d = h.pseudo1d;
  A.metallicity = h.metallicity; A.g2d = h.g2d;
  A.density = h.density; A.T = h.T; A.Td = h.Td; A.partner5 = h.partner5; A.cdens = h.cdens;
  A.spop = h.spop; A.tau = h.tau; A.pop = h.pop; A.cooling = h.cooling; A.line = h.line; A.status = h.status;
  const int n = c->dev.nlev;
  if (n > 64) {   // the elimination gives a lane two rows at most
    set_error("pdr_levpop_batched: coolants with more than 64 levels are not supported");
    return PDR_E_ARG;
  }
  // the fine-structure coolants, in both forms: a batch of cells per block, up
  // to a warp's worth of them for the elimination, fewer where that leaves SMs
  // idle (at 8 levels the cells' arrays still leave several blocks per SM)
  if (n <= SMALL_LEVELS) {
    const size_t per_cell = 8 * (size_t)small_layout(n, c->dev.nrad, c->dev.npart).total + 4 * (size_t)c->dev.npart;
    const long long per_sm = 6;
    const long long want = ((long long)h.ncell + sm_count * per_sm - 1) / (sm_count * per_sm);
    const int batch = (int)std::max(1ll, std::min({32ll, want, (long long)(48 * 1024 / per_cell)}));
    const long long grid = std::min(((long long)h.ncell + batch - 1) / batch, sm_count * per_sm);
    levpop_small_kernel<<<(int)grid, SMALL_THREADS, per_cell * batch, st>>>(c->dev, A, batch);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : cuda_fail(e, "levpop_small_kernel launch");
  }
  const size_t pw = levpop_smem_per_warp(n, c->dev.nrad, mixed);
  // the block size (1..8 warps) that keeps the most warps resident per SM
  // (the shared memory of one warp bounds it for the 41-level coolant),
  // chosen once per device and warp size; the attribute is set to the largest
  // candidate and never lowered, so concurrent launches cannot undercut it
  auto kern = mixed ? levpop_kernel<true> : levpop_kernel<false>;
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  struct Shape { int dev; size_t pw; bool mixed; int wpb, per_sm; };
  static std::mutex mu;
  static std::vector<Shape> shapes;
  static size_t attr[64][2] = {};
  int wpb = 0, per_sm = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    for (const Shape &sh : shapes)
      if (sh.dev == dev && sh.pw == pw && sh.mixed == mixed) { wpb = sh.wpb; per_sm = sh.per_sm; }
    if (wpb == 0) {
      const size_t top = std::min((size_t)optin, pw * 8);
      if (top > attr[dev & 63][mixed]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)top);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(levpop)");
        attr[dev & 63][mixed] = top;
      }
      for (int w = 8; w >= 1; w--) {
        if (pw * w > top) continue;
        int b = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, w * 32, pw * w);
        if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor(levpop)");
        if (b * w > per_sm * wpb) { wpb = w; per_sm = b; }
      }
      if (wpb < 1) {
        set_error("pdr_levpop_batched: one warp's shared memory exceeds a block's");
        return PDR_E_ARG;
      }
      shapes.push_back({dev, pw, mixed, wpb, per_sm});
    }
  }
  const size_t smem = pw * wpb;
  long long blocks = ((long long)h.ncell + wpb - 1) / wpb;
  if (blocks > (long long)sm_count * per_sm) blocks = (long long)sm_count * per_sm;
  if (blocks < 1) blocks = 1;
  kern<<<(int)blocks, wpb * 32, smem, st>>>(c->dev, A);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "levpop_kernel launch");
}

}  // namespace pdr
