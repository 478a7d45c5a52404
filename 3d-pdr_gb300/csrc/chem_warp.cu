// chem_warp.cu -- batched BDF chemistry integrator, one warp per cell.
//
// Replaces the per-cell CVODE solve of calculate_abundances.c:124-326 for
// networks with at most 32 ODE species (the reduced network has exactly 32):
// lane i owns species i -- its Nordsieck row z[0..5][i], error weight and
// correction -- and row i of the Newton matrix, held in registers.
//
// The integrator restates the published CVODE method step for step (the same
// algorithm as the CPU oracle; constants and formulas are listed there):
// fixed-leading-coefficient BDF of order 1..5 in Nordsieck form, Newton
// iteration with at most 3 corrections, WRMS local error test, CVODE's step
// and order heuristics, initial-step estimate, tout ladder of
// calculate_abundances.c:214,302-303 with its retry rules, clamping of
// outputs below abstol and the x_e of the last RHS call in the electron slot.
//
// Per cell, the warp also builds the RHS and the analytic Jacobian from the
// network tables (pdr_net.cpp):
//   RHS  f_i = sum_r nu_ir phi_r,  phi_r = kn_r x_a x_b  (kn = k or k n_H),
//        fluxes computed reaction-parallel, then the stoichiometric terms are
//        summed in 32 balanced chunks with deterministic partial sums;
//   Jac  J_ij = sum_r nu_ir dphi_r/dx_j plus the chain rule through
//        x_e = sum_j c_j x_j (the generated Jac() of the reference omits it).
//
// Precision modes:
//   PDR_FP64  : M = I - gamma J in FP64, partial-pivot LU (CVDense semantics).
//   PDR_MIXED : M is formed and factorised in FP32 after the similarity
//               scaling W M W^-1 with W = diag(1/(rtol|y|+atol)) taken at
//               setup, and the Nordsieck columns z2..z5 are FP32; the state,
//               z1, RHS, Newton residual and error test stay FP64.  A cell
//               whose Newton iteration keeps failing with a fresh FP32 matrix
//               is queued and re-solved from its inputs in FP64.
#include <cstdint>
#include <mutex>
#include <type_traits>

#include "bdf_core.cuh"
#include "fp64_fast.cuh"
#include "launch_shape.h"
#include "pdr_internal.h"

namespace pdr {

namespace {

using namespace bdf;
constexpr unsigned FULL = 0xffffffffu;

struct ChemArgs {
  WarpTables tab;
  int ncell, nspec, nreac;
  double *abundance;
  const double *rate;
  const double *density;
  const double *t_end_yr;
  double t_end_default_yr, start_time_yr, reltol, abstol;
  long long mxstep, max_total_steps;
  int *status;
  int *stats;
  const int *cell_list;     // optional indirection (FP64 redo pass)
  int *queue;               // work-queue cursor
  int *fallback_list;       // mixed mode: cells to redo in FP64
  int *fallback_count;
  int refill_static;        // 1: warp w takes cells w, w+W, ... ; 0: atomic work queue
  // work-queue mode: SMs the launch may keep (device word, read between
  // cells; null: all).  Blocks beyond limit * gridDim.x / grid_sms take no
  // further cells, so a later launch on another stream gets their SMs.
  const int *sm_limit;
  int grid_sms;             // SMs the grid was sized for
  int stage;                // 1: the blocks copy the packed term tables to shared memory
};

// true when this block is beyond the launch's current SM allowance
__device__ __forceinline__ bool over_sm_limit(const int *sm_limit, int grid_sms) {
  if (!sm_limit) return false;
  const int lim = *reinterpret_cast<const volatile int *>(sm_limit);
  return (long long)blockIdx.x * grid_sms >= (long long)lim * gridDim.x;
}

// byte offsets of one warp's shared arrays (host and device agree)
struct WarpLayout {
  size_t kn, work, xs, part, slots, jrow, sig, tri, ws, total;
};

__host__ __device__ inline WarpLayout warp_layout(int nsp, const WarpTables &T, bool mixed, bool zsh) {
  auto al = [](size_t x) { return (x + 15) & ~size_t(15); };
  const size_t mt = mixed ? 4 : 8;
  WarpLayout L;
  size_t o = 0;
  L.kn = o; o += al(8 * (size_t)(T.nkn + 1));   // rate constants, extras, a zero
  // work: one after the other, the RHS operands and partial sums (FP64), the
  // Jacobian's two scatter buffers and boundary slots, the LU's panel and
  // pivot order
  L.work = o;
  const size_t rhs = 8 * (size_t)T.nop + 8 * (size_t)(T.nparts + 1);
  const size_t jac = 2 * mt * (size_t)T.nreac + mt * (size_t)T.nslots;
  const size_t lu = 4 * mt * nsp + 4 * (size_t)nsp;
  L.part = o + 8 * (size_t)T.nop;
  L.slots = o + 2 * mt * (size_t)T.nreac;
  o += al(rhs > jac ? (rhs > lu ? rhs : lu) : (jac > lu ? jac : lu));
  L.xs = o; o += mixed ? 0 : al(8 * (size_t)(nsp + 2));   // FP64: the slot values of the assembly
  L.jrow = o; o += al(mt * (size_t)nsp * (nsp + 1));
  // mixed: the column scales and FP32 slot values of the assembly, then the
  // triangles of the four-column solve
  L.sig = L.tri = o;
  o += mixed ? al(4 * (size_t)(2 * (nsp + 2) > (nsp / 4) * 20 ? 2 * (nsp + 2) : (nsp / 4) * 20)) : 0;
  // the Nordsieck rows when they live in shared memory: six FP64 columns, or
  // in the mixed form two FP64 and four FP32 columns
  L.ws = o; o += al(sizeof(CoefShared) + (zsh ? (mixed ? 2 * 8 + 4 * 4 : 8 * (QMAX + 1)) * kWarp : 0));
  L.total = o;
  return L;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, o));
  return v;
}

template <class T>
__device__ __forceinline__ T bcast(T v, int src) { return __shfl_sync(FULL, v, src); }

// index of the lane with the largest candidate value (lowest lane on ties);
// returns -1 when every candidate is zero
__device__ __forceinline__ int argmax_lane(float v, bool cand) {
  unsigned bits = cand ? __float_as_uint(v) : 0u;
  unsigned mx = __reduce_max_sync(FULL, bits);
  unsigned b = __ballot_sync(FULL, cand && bits == mx);
  return (mx == 0u) ? -1 : __ffs(b) - 1;
}
__device__ __forceinline__ int argmax_lane(double v, bool cand) {
  unsigned long long u = cand ? (unsigned long long)__double_as_longlong(v) : 0ull;
  unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
  unsigned mh = __reduce_max_sync(FULL, hi);
  unsigned ml = __reduce_max_sync(FULL, (hi == mh) ? lo : 0u);
  unsigned b = __ballot_sync(FULL, cand && hi == mh && lo == ml);
  return (mh == 0u && ml == 0u) ? -1 : __ffs(b) - 1;
}

// LU with partial pivoting of the rows held in shared memory, lane i = row i
// at a + i*ld.  Rows stay in place: on exit row i holds its multipliers in
// the columns before the step at which it was the pivot (mystep) and its U
// row from there on; invd = 1/diagonal, perm[k] = pivot row of step k.
// Right-looking in panels of four columns: a lane keeps its row's panel entries
// in registers (the pivot row's come by shuffle), then the pivot rows' entries
// right of the panel are finished column by column (lane = column), and each
// remaining row takes the four updates of a column at once, one load and one
// store of the entry instead of four.  Every entry sees the same updates in
// the same order as column by column.  upan: 4 N values, 16-byte aligned.
template <int N, class MT>
__device__ __forceinline__ bool lu_rows(MT *a, int ld, int lane, int &mystep, MT &invd, int *perm, MT *upan) {
  static_assert(N % 4 == 0 && N <= 32, "panels of four, a lane per row");
  mystep = (lane < N) ? -1 : N;
  MT *row = a + (lane < N ? lane : 0) * ld;
  bool ok = true;
#pragma unroll 1
  for (int k0 = 0; k0 < N; k0 += 4) {
    MT r[4];
    int pt[4];
#pragma unroll
    for (int t = 0; t < 4; t++) r[t] = row[k0 + t];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const bool cand = (mystep < 0);
      int p = argmax_lane(cand ? fabs(r[t]) : MT(0), cand);
      if (p < 0) { ok = false; p = 0; }   // singular: finish on any row, the caller discards the factors
      pt[t] = p;
      MT u[4];
#pragma unroll
      for (int j = t; j < 4; j++) u[j] = bcast(r[j], p);
      MT rinv;
      if constexpr (sizeof(MT) == 8) rinv = fp64::rcp_near(u[t]);
      else rinv = __frcp_rn(u[t]);
      if (lane == p) { mystep = k0 + t; invd = rinv; perm[k0 + t] = p; }
      if (mystep < 0) {
        r[t] = r[t] * rinv;
#pragma unroll
        for (int j = t + 1; j < 4; j++) r[j] = fma(-r[t], u[j], r[j]);
      }
    }
    if (lane < N) {
#pragma unroll
      for (int t = 0; t < 4; t++) row[k0 + t] = r[t];
    }
    if (k0 + 4 >= N) break;
    const MT m10 = bcast(r[0], pt[1]), m20 = bcast(r[0], pt[2]), m21 = bcast(r[1], pt[2]);
    const MT m30 = bcast(r[0], pt[3]), m31 = bcast(r[1], pt[3]), m32 = bcast(r[2], pt[3]);
    __syncwarp();   // the last panel's updates of these rows
    if (lane >= k0 + 4 && lane < N) {
      MT *c = a + lane;
      const MT u0 = c[pt[0] * ld];
      const MT u1 = fma(-m10, u0, c[pt[1] * ld]);
      const MT u2 = fma(-m21, u1, fma(-m20, u0, c[pt[2] * ld]));
      const MT u3 = fma(-m32, u2, fma(-m31, u1, fma(-m30, u0, c[pt[3] * ld])));
      c[pt[1] * ld] = u1;
      c[pt[2] * ld] = u2;
      c[pt[3] * ld] = u3;
      MT *q = upan + 4 * lane;
      q[0] = u0; q[1] = u1; q[2] = u2; q[3] = u3;
    }
    __syncwarp();
    if (mystep < 0) {
#pragma unroll 1
      for (int j = k0 + 4; j < N; j += 4) {
        MT s[4], u[4][4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          s[c] = row[j + c];
          if constexpr (sizeof(MT) == 4) {
            const float4 v = reinterpret_cast<const float4 *>(upan)[j + c];
            u[c][0] = v.x; u[c][1] = v.y; u[c][2] = v.z; u[c][3] = v.w;
          } else {
            const double2 v = reinterpret_cast<const double2 *>(upan)[2 * (j + c)];
            const double2 w = reinterpret_cast<const double2 *>(upan)[2 * (j + c) + 1];
            u[c][0] = v.x; u[c][1] = v.y; u[c][2] = w.x; u[c][3] = w.y;
          }
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
          for (int t = 0; t < 4; t++) s[c] = fma(-r[t], u[c][t], s[c]);
          row[j + c] = s[c];
        }
      }
    }
    __syncwarp();
  }
  __syncwarp();
  return ok;
}

// The triangular solves work in pivot order: lane k takes row perm[k], so that
// step k's value sits in lane k.  b and the result are in species order.
//
// FP64: one step per column.
template <int N>
__device__ __forceinline__ double lu_solve_rows(const double *a, int ld, int lane, int rowk, double invd, double b) {
  const double *row = a + rowk * ld;
  b = bcast(b, rowk);
#pragma unroll 4
  for (int k = 0; k < N; k++) {
    const double yk = bcast(b, k);
    if (lane > k) b = fma(-row[k], yk, b);
  }
  double x = 0.0;
#pragma unroll 4
  for (int k = N - 1; k >= 0; k--) {
    const double xk = bcast(b * invd, k);
    if (lane == k) x = xk;
    if (lane < k) b = fma(-row[k], xk, b);
  }
  return x;
}

// FP32: four columns per step.  Every lane finds the four values of a step from
// the four lanes' entries by the 4 x 4 triangle (the same operations as the
// owning lanes would do one after the other), so a step waits for one round
// of shuffles instead of four.  tri[5*b]: the triangles of block b -- L10 L20
// L21 L30 | L31 L32 | U23 U13 U03 U12 | U02 U01 | 1/d0..3, see setup().
constexpr int TRI = 20;
__device__ __forceinline__ int tri_row(int q) { return (0x46fe9u >> (2 * q)) & 3; }   // (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
__device__ __forceinline__ int tri_col(int q) { return (0x6bf910u >> (2 * q)) & 3; }   // (2,3) (1,3) (0,3) (1,2) (0,2) (0,1)
template <int N>
__device__ __forceinline__ float lu_solve_rows4(const float *a, int ld, int lane, int rowk, const float *tri, float b) {
  const float *row = a + rowk * ld;
  b = bcast(b, rowk);
#pragma unroll 1
  for (int k = 0; k < N; k += 4) {
    const float4 l = *reinterpret_cast<const float4 *>(tri + k * (TRI / 4));
    const float2 m = *reinterpret_cast<const float2 *>(tri + k * (TRI / 4) + 4);
    const float r0 = row[k], r1 = row[k + 1], r2 = row[k + 2], r3 = row[k + 3];
    const float y0 = bcast(b, k);
    const float b1 = bcast(b, k + 1), b2 = bcast(b, k + 2), b3 = bcast(b, k + 3);
    const float y1 = fmaf(-l.x, y0, b1);
    const float y2 = fmaf(-l.z, y1, fmaf(-l.y, y0, b2));
    const float y3 = fmaf(-m.y, y2, fmaf(-m.x, y1, fmaf(-l.w, y0, b3)));
    if (lane > k) b = fmaf(-r0, y0, b);
    if (lane > k + 1) b = fmaf(-r1, y1, b);
    if (lane > k + 2) b = fmaf(-r2, y2, b);
    if (lane > k + 3) b = fmaf(-r3, y3, b);
  }
  float x = 0.0f;
#pragma unroll 1
  for (int k = N - 4; k >= 0; k -= 4) {
    const float4 u = *reinterpret_cast<const float4 *>(tri + k * (TRI / 4) + 8);
    const float2 v = *reinterpret_cast<const float2 *>(tri + k * (TRI / 4) + 12);
    const float4 d = *reinterpret_cast<const float4 *>(tri + k * (TRI / 4) + 16);
    const float r0 = row[k], r1 = row[k + 1], r2 = row[k + 2], r3 = row[k + 3];
    const float b0 = bcast(b, k), b1 = bcast(b, k + 1), b2 = bcast(b, k + 2), b3 = bcast(b, k + 3);
    const float x3 = b3 * d.w;
    const float x2 = fmaf(-u.x, x3, b2) * d.z;
    const float x1 = fmaf(-u.w, x2, fmaf(-u.y, x3, b1)) * d.y;
    const float x0 = fmaf(-v.y, x1, fmaf(-v.x, x2, fmaf(-u.z, x3, b0))) * d.x;
    if (lane == k) x = x0;
    if (lane == k + 1) x = x1;
    if (lane == k + 2) x = x2;
    if (lane == k + 3) x = x3;
    if (lane < k) b = fmaf(-r0, x0, fmaf(-r1, x1, fmaf(-r2, x2, fmaf(-r3, x3, b))));
  }
  return x;
}

// One cell integrated by one warp: lane = species = Newton-matrix row.
// ZSH: Nordsieck rows in shared memory instead of registers.
template <int NSP, bool MIXED, bool ZSH>
struct WarpCell : Core<WarpCell<NSP, MIXED, ZSH>, ZSH, MIXED> {
  using MT = typename std::conditional<MIXED, float, double>::type;
  // Newton-matrix row stride: the species columns and the x_e column (odd, so
  // the rows of a warp fall in distinct banks)
  static constexpr int LDJ = NSP + 1;
  const ChemArgs &A;
  const int lane;
  const bool owns;
  const double inv_n = 1.0 / NSP;
  // shared-memory views of this warp
  double *kn, *scr, *xs, *part;
  const int *rt, *ht, *pk, *bnd;   // the packed term tables, in shared memory or global
  const unsigned char *pl;
  const unsigned short *rab;
  MT *slots;      // partials of the Jacobian entries whose runs cross chunks
  MT *jrow;       // [NSP][NSP+1] Newton matrix rows / their LU factors
  float *sig;     // [NSP+2] column scales (mixed)
  int *perm;      // [NSP] pivot lane of each elimination step
  float *xs32;    // [NSP+2] FP32 copy of the slot values at setup (mixed)
  double cx;      // electron-sum coefficient of species `lane`
  int cxi;        // the same as an integer
  float cxf;      //   and in FP32
  bool cx_unit;   // every coefficient of the network is -1, 0 or 1 (warp-uniform)
  unsigned cx_any;   // the species with a nonzero coefficient
  int rowk;       // pivot row of elimination step `lane`
  float *tri;     // [NSP/4][20] 4 x 4 triangles of the factors' diagonal blocks (mixed)
  MT invd;        // reciprocal pivot of that row
  double wsc, ssc;      // FP64 form: setup-time weight and its inverse
  float wsc32, ssc32;   // mixed form: the same in FP32 (the scaling of the FP32 matrix)

  __device__ __forceinline__ WarpCell(const ChemArgs &a, int ln) : A(a), lane(ln), owns(ln < NSP) {}
  __device__ __forceinline__ bool leader() const { return lane == 0; }
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ double sum_all(double v) const { return warp_sum(v); }
  __device__ __forceinline__ float sum_all(float v) const { return warp_sum(v); }
  __device__ __forceinline__ double max_all(double v) const { return warp_max(v); }

  __device__ __forceinline__ void set_xe_coef() {
    cx = owns ? __ldg(&A.tab.xe_coef[lane]) : 0.0;
    cxi = (int)cx;
    cxf = owns ? __ldg(&A.tab.xe_coef_f[lane]) : 0.0f;
    cx_unit = __all_sync(FULL, cx == (double)cxi && cxi >= -1 && cxi <= 1);
    cx_any = __ballot_sync(FULL, cx != 0.0);
  }
  // this lane's term c_i x_i of x_e: a sign select when the coefficients are
  // -1, 0 or 1 (every FP64 warp instruction costs an FP64 issue slot)
  __device__ __forceinline__ double xe_term(double yv) const {
    if (cx_unit) {
      const unsigned long long b = (unsigned long long)__double_as_longlong(yv);
      return (!owns || cxi == 0) ? 0.0 : __longlong_as_double((long long)(cxi < 0 ? (b ^ 0x8000000000000000ull) : b));
    }
    return owns ? cx * yv : 0.0;
  }

  // point the warp's arrays into its shared-memory slice
  __device__ __forceinline__ void bind(unsigned char *base, const WarpLayout &L) {
    kn = reinterpret_cast<double *>(base + L.kn);
    scr = reinterpret_cast<double *>(base + L.work);
    xs = reinterpret_cast<double *>(base + L.xs);
    part = reinterpret_cast<double *>(base + L.part);
    slots = reinterpret_cast<MT *>(base + L.slots);
    jrow = reinterpret_cast<MT *>(base + L.jrow);
    sig = reinterpret_cast<float *>(base + L.sig);
    xs32 = sig + NSP + 2;
    perm = reinterpret_cast<int *>(reinterpret_cast<MT *>(scr) + 4 * NSP);
    tri = reinterpret_cast<float *>(base + L.tri);
    this->ws = reinterpret_cast<CoefShared *>(base + L.ws);
  }

  // the packed term tables: `t` in shared memory or global
  __device__ __forceinline__ void bind_tables(const int *t) {
    const WarpTables &T = A.tab;
    rt = t + T.wt_rt;
    ht = t + T.wt_h;
    pk = t + T.wt_pk;
    bnd = t + T.wt_bnd;
    pl = reinterpret_cast<const unsigned char *>(t + T.wt_pl);
    rab = reinterpret_cast<const unsigned short *>(t + T.wt_rab);
  }

  // per-cell rate constants kn_r = k_r (times n_H for the terms that carry
  // it), the extras |nu| kn_r of the RHS terms with |nu| > 1, a zero for the
  // padding terms, and the constants of the slot and partial-sum arrays
  __device__ __forceinline__ void load_rates(const double *rate, double n_H) {
    const WarpTables &T = A.tab;
    for (int r = lane; r < T.nreac; r += kWarp) kn[r] = __ldg(&rate[r]) * (__ldg(&T.nh_mask[r]) != 0.0 ? n_H : 1.0);
    if (lane == 0) kn[T.nkn] = 0.0;
    __syncwarp();
    for (int e = lane; e < T.nkext; e += kWarp) {
      double k = 0.0;
      for (int q = __ldg(&T.kext_ptr[e]); q < __ldg(&T.kext_ptr[e + 1]); q++) {
        const int2 rn = __ldg(&T.kext_rn[q]);
        k = fma((double)rn.y, kn[rn.x], k);
      }
      kn[T.nreac + e] = k;
    }
    __syncwarp();
  }

  // f(y): returns f_lane, records x_e of this call (lane 0).  The operands are
  // this state's slot values and the products x_a x_b of the two-body reactant
  // pairs (one FP64 multiply per pair instead of two per reaction); every
  // stoichiometric term is then one FMA with the signed rate constant.
  //
  // x_e is summed as a tree over the lower lanes (the lane pairs and order of
  // the butterfly, so the same sum), and the lanes that each level leaves idle
  // form pair products in the same FP64 instruction: v*1 + w is the sum, x_a x_b
  // + (-0) the product, both rounded as the add and the multiply.  196 pairs
  // and the sum take 8 instructions instead of 12.
  __device__ __forceinline__ double rhs(double yv) {
    const WarpTables &T = A.tab;
    double *P = scr;
    if (owns) P[lane] = yv;
    if (lane == 0) {
      P[NSP + 1] = 1.0;
      part[T.nparts] = 0.0;
    }
    double v = xe_term(yv);
    __syncwarp();
    PairWord d(pk[lane]);
#pragma unroll 1
    for (int k = 0; k < T.pk_len; k++) {
      const int o = 16 >> k;   // 0 from round 5 on
      if (k == 5) {
        if (lane == 0) P[NSP] = v;
        __syncwarp();
      }
      const double x = P[d.a()], y = P[d.b()];
      const int at = d.operand();
      d = PairWord(pk[min(k + 1, T.pk_len - 1) * kWarp + lane]);
      const double w = __shfl_down_sync(FULL, v, o);
      const bool sum = lane < o;
      const double r = fma(sum ? v : x, sum ? 1.0 : y, sum ? w : -0.0);
      if (sum) v = r;
      else if (at) P[at] = r;
    }
    this->xe_last = v;
    __syncwarp();
    // the terms in groups of four, every load of a group before its stores (the
    // compiler cannot tell the partial sums from the tables and operands, and
    // one term at a time the chain of two loads, FMA and store took 240 cycles)
    double s = 0.0;
    double *pp = part + pl[lane];
#pragma unroll 1
    for (int t = 0; t < T.rhs_len4; t += 4) {
      unsigned d4[4];
      double k[4], o[4];
#pragma unroll
      for (int u = 0; u < 4; u++) d4[u] = (unsigned)rt[(t + u) * kWarp + lane];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        k[u] = *reinterpret_cast<const double *>(reinterpret_cast<const char *>(kn) + TermWord(d4[u]).rate_at());
        o[u] = *reinterpret_cast<const double *>(reinterpret_cast<const char *>(P) + TermWord(d4[u]).operand_at());
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        // nu kn_r with nu = +-1 (|nu| > 1 reads its extra constant): the sign
        // bit of kn_r flipped in the integer pipe
        s = fma(__hiloint2double(__double2hiint(k[u]) ^ (int)TermWord(d4[u]).sign(), __double2loint(k[u])), o[u], s);
        if (TermWord(d4[u]).last()) {
          *pp++ = s;
          s = 0.0;
        }
      }
    }
    __syncwarp();
    double f = part[pl[kWarp + lane]];
#pragma unroll 1
    for (int k = 2; k <= T.plist_len; k++) f += part[pl[k * kWarp + lane]];
    __syncwarp();
    this->nfe++;
    return owns ? f : 0.0;
  }

  // Jacobian rows at y, times rf, plus the identity when `identity`:
  // FP64 m = rf*J (+I); mixed m = rf * W J W^-1 (+I), W = diag(1/(rtol|y|+atol))
  // same_y: rhs() was called for this y just before, and its x_e still holds
  __device__ __forceinline__ void assemble(double yv, double rf_d, bool identity, bool same_y) {
    const WarpTables &T = A.tab;
    const double xe = same_y ? this->xe_last : warp_sum(xe_term(yv));
    __syncwarp();   // the work area changes hands
    if constexpr (!MIXED) {
      if (owns) xs[lane] = yv;
      if (lane == 0) {
        xs[NSP] = xe;
        xs[NSP + 1] = 1.0;
      }
    }
    if constexpr (MIXED) {
      // column scales 1/w_j = rtol|y_j|+atol, normalised by atol so they fit
      // FP32, formed in FP32 (the matrix is FP32; y and x_e converted once)
      const float y32 = (float)yv;
      ssc32 = fmaf(this->rtol32, fabsf(y32), this->atol32);
      wsc32 = __frcp_rn(ssc32);
      if (owns) {
        sig[lane] = ssc32 * __frcp_rn(this->atol32);
        xs32[lane] = y32;
      }
      if (lane == 0) {
        sig[NSP] = 1.0f;
        sig[NSP + 1] = 0.0f;
        xs32[NSP] = (float)xe;
        xs32[NSP + 1] = 1.0f;
      }
    }
    __syncwarp();
    MT *Da = reinterpret_cast<MT *>(scr);
    MT *Db = Da + T.nreac;
#pragma unroll 1
    for (int r = lane; r < T.nreac; r += kWarp) {
      const int ab = rab[r], sa = ab & 0xff, sb = ab >> 8;
      if constexpr (MIXED) {
        // dphi_r/dx_a and dphi_r/dx_b, column-scaled, in FP32: one conversion
        // of the rate constant per reaction
        const float k32 = (float)kn[r];
        Da[r] = k32 * (xs32[sb] * sig[sa]);
        Db[r] = k32 * (xs32[sa] * sig[sb]);
      } else {
        const double k = kn[r];
        Da[r] = k * xs[sb];
        Db[r] = (sb == NSP + 1) ? 0.0 : k * xs[sa];
      }
    }
    MT *row = jrow + lane * (LDJ);
    {
      // the matrix is contiguous and 16-byte aligned
      static_assert(NSP * LDJ * sizeof(MT) % 16 == 0, "zeroed in 16-byte pieces");
      int4 *z = reinterpret_cast<int4 *>(jrow);
#pragma unroll 1
      for (int j = lane; j < (int)(NSP * LDJ * sizeof(MT) / 16); j += kWarp) z[j] = make_int4(0, 0, 0, 0);
    }
    __syncwarp();
    // term-parallel: the (row, column) contributions nu * dphi_r/dx_col sorted
    // by entry and cut into 32 balanced chunks; a lane sums each run of one
    // entry in a register and stores it, and a run that crosses a chunk
    // boundary leaves partials in slots that a second pass adds in chunk order.  The rows of the electron
    // and hydrogen hold most contributions: walking one row per lane left the
    // warp waiting on those two lanes.
    {
      MT s = MT(0);
      // in groups of four, every load of a group before its stores
#pragma unroll 1
      for (int t = 0; t < T.hlen4; t += 4) {
        int x[4];
        MT d[4];
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = ht[(t + u) * kWarp + lane];
#pragma unroll
        for (int u = 0; u < 4; u++) d[u] = Da[JacWord(x[u]).index()];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          // nu, a small signed integer: converted without the FP64 pipe
          const float nu = (float)JacWord(x[u]).nu();
          if constexpr (MIXED) s = fmaf(nu, d[u], s);
          else s = fma(fp64::f2d(nu), d[u], s);
          const int kind = JacWord(x[u]).kind();
          if (kind) {
            (kind == 1 ? jrow : slots)[JacWord(x[u]).target()] = s;
            s = MT(0);
          }
        }
      }
      __syncwarp();
      for (int b = lane; b < T.nbnd; b += kWarp) {
        const unsigned tt = (unsigned)bnd[b];
        MT acc = MT(0);
#pragma unroll 1
        for (unsigned q = (tt >> 11) & 0xff; q < (tt >> 19); q++) acc += slots[q];
        jrow[tt & 0x7ff] = acc;
      }
      __syncwarp();
    }
    static_assert(NSP == kWarp, "a lane for every row");
    const MT e = row[NSP];
    MT rf;
    if constexpr (MIXED) rf = (MT)rf_d * (wsc32 * this->atol32);   // row weight, normalised like the columns
    else rf = (MT)rf_d;
    // the x_e chain rule adds e c_j to the charged species' columns (c_j from its
    // lane; the FP64 form leaves the neutral ones out)
    const float cxt = cxf;
#pragma unroll 2
    for (int j = 0; j < NSP; j++) {
      MT v = row[j];
      if constexpr (MIXED) v = fmaf(e * bcast(cxt, j), sig[j], v);
      else if ((cx_any >> j) & 1u) v = fma(e, bcast(cx, j), v);
      row[j] = fma(rf, v, (identity && lane == j) ? MT(1) : MT(0));
    }
    __syncwarp();
  }

  // Newton matrix at y: FP64 M = I - gamma J, or FP32 W M W^-1, factorised
  __device__ __forceinline__ bool setup(double yv) {
    assemble(yv, -this->gamma, true, true);
    int mystep;
    bool ok = lu_rows<NSP, MT>(jrow, LDJ, lane, mystep, invd, perm, reinterpret_cast<MT *>(scr));
    const MT *row = jrow + lane * (LDJ);
    bool finite = true;
    if (owns) {
#pragma unroll 4
      for (int j = 0; j < NSP; j++) finite &= isfinite(row[j]);
    }
    ok = __all_sync(FULL, finite) && ok;
    if (ok) {
      rowk = perm[lane < NSP ? lane : 0];
      invd = bcast(invd, rowk);
      if constexpr (MIXED) {
        // entries (i, j) of each diagonal block, in the order the solves read them
#pragma unroll 1
        for (int e = lane; e < (NSP / 4) * 12; e += kWarp) {
          const int blk = e / 12, q = e - blk * 12;
          const int i = tri_row(q), j = tri_col(q);
          tri[blk * TRI + q + (q >= 6 ? 2 : 0)] = jrow[perm[4 * blk + i] * LDJ + 4 * blk + j];
        }
        if (owns) tri[(lane >> 2) * TRI + 16 + (lane & 3)] = invd;
      }
      __syncwarp();   // the pivot order's memory is the RHS's next
    }
    this->after_setup();
    return ok;
  }

  __device__ __forceinline__ double solve(double b) {
    const double x = lu_solve_rows<NSP>(jrow, LDJ, lane, rowk, invd, b);
    return owns ? x : 0.0;
  }

  // mixed form: the residual is converted once and scaled in FP32 (the
  // scaling of the FP32 matrix), the correction comes back times ssc*gscale
  __device__ __forceinline__ float solve32(double b, float gs) {
    const float xv = lu_solve_rows4<NSP>(jrow, LDJ, lane, rowk, tri, (float)b * wsc32);
    return owns ? xv * (ssc32 * gs) : 0.0f;
  }

  // calculate_abundances.c:132-317 for one cell
  __device__ __forceinline__ void run(int cell) {
    const int nspec = A.nspec;
    double *ab = A.abundance + (size_t)cell * nspec;
    this->rtol = A.reltol;
    this->atol = A.abstol;
    this->mxstep = A.mxstep;
    this->max_total_steps = A.max_total_steps;
    set_xe_coef();
    load_rates(A.rate + (size_t)cell * A.nreac, A.density[cell]);
    this->clear_row(owns ? ab[lane] : 0.0);
    this->xe_last = ab[nspec - 1];
    const double tend_yr = A.t_end_yr ? A.t_end_yr[cell] : A.t_end_default_yr;
    double yv = 0.0;
    const int status = this->integrate(A.start_time_yr, tend_yr, MIXED, &yv);
    if (status == FELL_BACK) {
      if (lane == 0) {
        const int k = atomicAdd(A.fallback_count, 1);
        A.fallback_list[k] = cell;
        A.status[cell] = FELL_BACK;
      }
      return;
    }
    if (yv < this->atol) yv = 0.0;
    if (owns) ab[lane] = yv;
    if (lane == 0) {
      ab[nspec - 1] = this->xe_last;
      A.status[cell] = status;
      if (A.stats) {
        int *s = A.stats + (size_t)cell * 8;
        s[0] = this->nst; s[1] = this->nfe; s[2] = this->nje; s[3] = this->nsetups;
        s[4] = this->nni; s[5] = this->ncfn; s[6] = this->netf; s[7] = MIXED ? 0 : (A.cell_list ? 1 : 0);
      }
    }
  }
};

// Register variants (the autotuner picks): RV 0 lets the compiler use the
// registers it wants (about 230; 8 warps/SM); RV 1 caps them at 128 for 16
// warps/SM with the Nordsieck rows in shared memory; RV 2 and 3 cap them at
// 168 for 12 warps/SM, Nordsieck rows in registers (2) or shared memory (3).
template <int RV> struct RegVariant;
template <> struct RegVariant<0> { static constexpr int threads = 256, min_blocks = 1; static constexpr bool zsh = false; };
template <> struct RegVariant<1> { static constexpr int threads = 256, min_blocks = 2; static constexpr bool zsh = true; };
template <> struct RegVariant<2> { static constexpr int threads = 384, min_blocks = 1; static constexpr bool zsh = false; };
template <> struct RegVariant<3> { static constexpr int threads = 384, min_blocks = 1; static constexpr bool zsh = true; };

// What bounds it: with 16 warps of an SM at different phases of a step, the
// instruction cache, then the FP64 pipe.  So the hot code is kept small -- one
// call site for the RHS, the setup and the solve, rolled loops, divisions side
// by side -- and the FP64 instructions few (about 75 a step in the mixed form).
// 64,000 cells, mixed: 684 -> 495 ms; 5,003: 71.3 -> 49.5 ms; 64 (latency, several
// of the cells on one SM, as the warps take them from one counter): 28.3 -> 21.1 ms;
// 1,500 cells in FP64 through host buffers: 80.9 -> 71.2 ms.  Results are the same
// bits, but for FP64 pivot reciprocals that may round the other way once in 2^35.
template <int NSP, bool MIXED, int RV>
__global__ void __launch_bounds__(RegVariant<RV>::threads, RegVariant<RV>::min_blocks)
    chem_warp_kernel(const __grid_constant__ ChemArgs A, int total_cells, const int *total_ptr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using MT = typename std::conditional<MIXED, float, double>::type;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr bool ZSH = RegVariant<RV>::zsh;
  const WarpLayout L = warp_layout(NSP, A.tab, MIXED, ZSH);
  WarpCell<NSP, MIXED, ZSH> c(A, lane);
  // the packed term tables at the start of the block's shared memory: every RHS
  // and assembly reads them, and the L1 left beside the warps' arrays misses
  unsigned char *base = smem_raw;
  if (A.stage) {
    int4 *dst = reinterpret_cast<int4 *>(smem_raw);
    const int4 *src = reinterpret_cast<const int4 *>(A.tab.wtab);
    for (int i = threadIdx.x; i < A.tab.wtab_words / 4; i += blockDim.x) dst[i] = __ldg(&src[i]);
    base += 4 * (size_t)A.tab.wtab_words;
  }
  c.bind(base + L.total * warp, L);
  c.bind_tables(A.stage ? reinterpret_cast<const int *>(smem_raw) : A.tab.wtab);
  if constexpr (ZSH) c.z.bind(reinterpret_cast<unsigned char *>(c.ws) + sizeof(CoefShared), lane, kWarp);
  __syncthreads();
  if (total_ptr) total_cells = *total_ptr;
  const int gwarp = blockIdx.x * (blockDim.x >> 5) + warp, nwarps = gridDim.x * (blockDim.x >> 5);
  for (int k = 0;; k++) {
    int idx = 0;
    if (A.refill_static) {
      idx = gwarp + k * nwarps;
    } else {
      if (lane == 0) idx = over_sm_limit(A.sm_limit, A.grid_sms) ? 0x7fffffff : atomicAdd(A.queue, 1);
      idx = __shfl_sync(FULL, idx, 0);
    }
    if (idx >= total_cells) break;
    const int cell = A.cell_list ? A.cell_list[idx] : idx;
    c.run(cell);
    __syncwarp();
  }
}

// Diagnostic evaluation of the device RHS (mode 0) or Jacobian (mode 1) on
// given states: one warp per state, the same code the integrator runs.
template <int NSP>
__global__ void __launch_bounds__(128) eval_kernel(const __grid_constant__ ChemArgs A, int nstate,
                                                   const double *x, double *out, double *xe_out, int mode) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const WarpLayout L = warp_layout(NSP, A.tab, false, false);
  WarpCell<NSP, false, false> c(A, lane);
  c.bind(smem_raw + L.total * warp, L);
  c.bind_tables(A.tab.wtab);
  c.rtol = A.reltol;
  c.mxstep = A.mxstep;
  c.max_total_steps = A.max_total_steps;
  c.atol = A.abstol;
  c.set_xe_coef();
  for (int s = blockIdx.x * (blockDim.x >> 5) + warp; s < nstate; s += gridDim.x * (blockDim.x >> 5)) {
    c.load_rates(A.rate + (size_t)s * A.nreac, A.density[s]);
    const double yv = (lane < NSP) ? x[(size_t)s * NSP + lane] : 0.0;
    if (mode == 0) {
      const double f = c.rhs(yv);
      if (lane < NSP) out[(size_t)s * NSP + lane] = f;
      if (lane == 0 && xe_out) xe_out[s] = c.xe_last;
    } else {
      c.assemble(yv, 1.0, false, false);
      if (lane < NSP)
#pragma unroll
        for (int j = 0; j < NSP; j++) out[((size_t)s * NSP + lane) * NSP + j] = c.jrow[lane * WarpCell<NSP, false, false>::LDJ + j];
    }
    __syncwarp();
  }
}

}  // namespace

size_t chem_warp_smem_per_warp(const WarpTables &T, bool mixed, bool zshared) {
  return warp_layout(T.neq, T, mixed, zshared).total;
}

// Launch the persistent warp kernel over `ncell` cells (or the cells listed in
// cell_list).  Returns 0 or a PDR_E_* code.
int launch_chem_warp(const pdr_net *net, int ncell, double *ab, const double *rate, const double *dens,
                     const double *tend, const pdr_chem_opts &o, int *status, int *stats, int *queue,
                     int *fb_list, int *fb_count, const int *cell_list, const int *total_ptr, bool mixed,
                     int sm_count, cudaStream_t st, const int *sm_limit) {
  const WarpTables &T = net->warp;
  if (T.neq != 32) return PDR_E_NET;
  ChemArgs A;
  A.tab = T;
  A.ncell = ncell;
  A.nspec = net->host.nspec;
  A.nreac = net->host.nreac;
  A.abundance = ab;
  A.rate = rate;
  A.density = dens;
  A.t_end_yr = tend;
  A.t_end_default_yr = o.end_time_yr;
  A.start_time_yr = o.start_time_yr;
  A.reltol = o.reltol;
  A.abstol = o.abstol;
  A.mxstep = o.mxstep;
  A.max_total_steps = 500000;
  A.status = status;
  A.stats = stats;
  A.cell_list = cell_list;
  A.queue = queue;
  A.sm_limit = sm_limit;
  A.grid_sms = sm_count;
  A.fallback_list = fb_list;
  A.fallback_count = fb_count;
  // refill 2 (one warp per cell, no persistence) applies to the pass over
  // all cells; the FP64 pass over a device-side list keeps the work queue
  const bool one_per_cell = (o.refill == 2) && !cell_list;
  A.refill_static = (o.refill == 1 || one_per_cell) ? 1 : 0;
  const int rv = warp_variant(o, mixed);
  const bool zsh = (rv == 1 || rv == 3);
  const size_t per_warp = chem_warp_smem_per_warp(T, mixed, zsh), tables = 4 * (size_t)T.wtab_words;
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  dev &= 63;
  const int wpb = warp_block(o, rv, per_warp, tables, (size_t)optin);
  if (wpb < 1) return PDR_E_ARG;
  const int variant = (mixed ? 4 : 0) + rv;
  using KFn = void (*)(ChemArgs, int, const int *);
  static const KFn kernels[8] = {chem_warp_kernel<32, false, 0>, chem_warp_kernel<32, false, 1>,
                                 chem_warp_kernel<32, false, 2>, chem_warp_kernel<32, false, 3>,
                                 chem_warp_kernel<32, true, 0>,  chem_warp_kernel<32, true, 1>,
                                 chem_warp_kernel<32, true, 2>,  chem_warp_kernel<32, true, 3>};
  // The dynamic shared-memory limit is an attribute of the function on each
  // device: it only ever grows (to the largest block size used so far on that
  // device), so that a launch with fewer warps never lowers it below what
  // another block size needs.  The occupancy is cached per (device, variant,
  // block size, table staging); calls made while a stream is being captured
  // then issue no attribute changes.
  static std::mutex mu;
  static size_t attr_smem[64][8] = {};
  static int cached_per_sm[64][8][WARPS_168 + 1][2] = {};
  static size_t cached_smem[64][8][WARPS_168 + 1][2] = {};
  int per_sm = 0;
  size_t smem = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    // the tables go to shared memory where that costs no resident warps
    int fit[2] = {0, 0};
    for (int stage = 0; stage < 2; stage++) {
      const size_t sm = per_warp * wpb + (stage ? tables : 0);
      if (sm + 1024 > (size_t)optin && stage) continue;
      if (sm > attr_smem[dev][variant]) {
        e = cudaFuncSetAttribute(kernels[variant], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute");
        attr_smem[dev][variant] = sm;
      }
      if (cached_smem[dev][variant][wpb][stage] != sm) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cached_per_sm[dev][variant][wpb][stage], kernels[variant],
                                                          wpb * 32, sm);
        if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        cached_smem[dev][variant][wpb][stage] = sm;
      }
      fit[stage] = cached_per_sm[dev][variant][wpb][stage];
    }
    A.stage = fit[1] > 0 && fit[1] >= fit[0];
    per_sm = fit[A.stage];
    smem = per_warp * wpb + (A.stage ? tables : 0);
  }
  if (o.blocks_per_sm > 0 && o.blocks_per_sm < per_sm) per_sm = o.blocks_per_sm;
  if (per_sm < 1) per_sm = 1;
  const int grid = one_per_cell ? (ncell + wpb - 1) / wpb : sm_count * per_sm;
  kernels[variant]<<<grid, wpb * 32, smem, st>>>(A, ncell, total_ptr);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "chem_warp_kernel launch");
}

}  // namespace pdr

namespace pdr {
int launch_chem_eval(const pdr_net *net, int nstate, const double *x, const double *rate, const double *dens,
                     double *out, double *xe_out, int mode, cudaStream_t st) {
  const WarpTables &T = net->warp;
  if (T.neq != 32) return PDR_E_NET;
  ChemArgs A{};
  A.tab = T;
  A.nspec = net->host.nspec;
  A.nreac = net->host.nreac;
  A.rate = rate;
  A.density = dens;
  A.reltol = 1e-8;
  A.abstol = 1e-30;
  const size_t smem = chem_warp_smem_per_warp(T, false, false) * 4;
  auto k = eval_kernel<32>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(eval)");
  k<<<(nstate + 3) / 4, 128, smem, st>>>(A, nstate, x, out, xe_out, mode);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "eval_kernel launch");
}
}  // namespace pdr
