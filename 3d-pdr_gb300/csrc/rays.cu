// rays.cu -- column densities and the attenuated UV field along the rays.
//
// CALC_UVFIELD (3DPDR.F90:1636-1701) and calc_columndens (3DPDR.F90:1789-1844)
// for all cells at once.  Both walk the evaluation points of every ray in
// order: each step between consecutive points has length |x_i - x_{i-1}| and
// contributes the trapezoid of the two points' densities (times an abundance
// for the species columns).  The sums keep the reference's order and its
// unfused products (explicit round-to-nearest intrinsics), so the columns
// agree with a serial evaluation bit for bit; only the UV field's exp differs
// from a CPU libm in the last place.
//
// The work is gathers: per point 3 coordinates, a grid index, the density of
// that grid point and, for the columns, its abundances.  Threads take one
// (cell, ray) (UV field) or one (cell, ray, group of 8 species) (columns) and
// walk its points sequentially; consecutive threads take consecutive rays,
// whose point lists are adjacent in memory.
#include <algorithm>

#include "fp64_fast.cuh"
#include "pdr_internal.h"

namespace pdr {
namespace {

constexpr double PC = 3.08568025e+18;   // parsec in cm (healpix_types.F90:98)
constexpr int SG = 8;                     // species per thread in the columns kernel
constexpr int UV_THREADS = 192;           // 16 cells of 12 rays
constexpr int TAU_THREADS = 256, TAU_STEPS = 8;

// |x_i - x_{i-1}| as the reference writes it: sqrt((dx^2 + dy^2) + dz^2)
__device__ __forceinline__ double step_length(const double *xyz, long long p) {
  const double dx = __dsub_rn(xyz[3 * (p - 1)], xyz[3 * p]);
  const double dy = __dsub_rn(xyz[3 * (p - 1) + 1], xyz[3 * p + 1]);
  const double dz = __dsub_rn(xyz[3 * (p - 1) + 2], xyz[3 * p + 2]);
  return fp64::sqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
}

struct UvArgs {
  int ncell, nrays, ngrid, field, uni_ray;
  long long npoint;
  const int *epray;
  const long long *offset;
  const double *xyz;
  const int *gp;
  const double *rho;
  double g_iso, g_uni, av_fac, uv_fac;
  double *colden, *AV, *rad, *uv;
};

// total-H column of one ray (NaN where an index leaves the grid)
__device__ __forceinline__ double ray_column(const UvArgs &A, size_t cj) {
  const int ne = A.epray[cj];
  const long long p0 = A.offset[cj];
  if (ne > 0 && (p0 < 0 || p0 + ne >= A.npoint)) return nan("");
  double col = 0.0;
  if (ne > 0) {
    const int g0 = A.gp[p0];
    double rho_prev = (g0 >= 0 && g0 < A.ngrid) ? A.rho[g0] : nan("");
    for (int i = 1; i <= ne; i++) {
      const long long p = p0 + i;
      const int gi = A.gp[p];
      const double rho_i = (gi >= 0 && gi < A.ngrid) ? A.rho[gi] : nan("");
      const double step = step_length(A.xyz, p);
      col = __dadd_rn(col, __dmul_rn(__dmul_rn(__dadd_rn(rho_prev, rho_i) * 0.5, step), PC));
      rho_prev = rho_i;
    }
  }
  return col;
}

// A thread per (cell, ray) -- one per cell left a lattice of 29^3 cells with
// one block per SM -- then the field of each cell is added in ray order, with
// the reference's clamp after every ray, by one of its threads.  More rays
// than a block has threads are taken in rounds.
__global__ void __launch_bounds__(UV_THREADS) uvfield_kernel(const __grid_constant__ UvArgs A) {
  __shared__ double term[UV_THREADS];
  const int per = max(1, UV_THREADS / A.nrays);   // cells per block
  for (long long base = (long long)blockIdx.x * per; base < A.ncell; base += (long long)gridDim.x * per) {
    const int nb = (int)min((long long)per, A.ncell - base);
    double uv = 0.0;
    for (int j0 = 0; j0 < A.nrays; j0 += UV_THREADS) {
      const int nj = min(A.nrays - j0, UV_THREADS);   // all rays, unless they are taken in rounds
      const int c = threadIdx.x / nj, j = j0 + threadIdx.x - c * nj;
      if (c < nb) {
        const size_t cj = (size_t)(base + c) * A.nrays + j;
        const double col = ray_column(A, cj);
        const double av = __dmul_rn(col, A.av_fac);
        double rad = 0.0;
        if (A.field == 0) rad = A.g_iso;
        else if (j == A.uni_ray) rad = A.g_uni;
        A.colden[cj] = col;
        A.AV[cj] = av;
        A.rad[cj] = rad;
        term[threadIdx.x] = __dmul_rn(rad, exp(__dmul_rn(-av, A.uv_fac)));
      }
      __syncthreads();
      if (threadIdx.x < nb)
        for (int q = 0; q < nj; q++) {
          uv = __dadd_rn(uv, term[threadIdx.x * nj + q]);
          if (uv < 1.0e-50) uv = 0.0;
        }
      __syncthreads();
    }
    if (threadIdx.x < nb) A.uv[base + threadIdx.x] = uv;
  }
}

constexpr int MAXSEL = 256;

struct ColArgs {
  int ncell, nrays, ngrid, nspec, nsel, ngroup;
  long long npoint;
  const int *epray;
  const long long *offset;
  const double *xyz;
  const int *gp;
  const double *rho, *ab;
  double *out;
  int species[MAXSEL];   // validated on the host
};

__global__ void columns_kernel(const __grid_constant__ ColArgs A) {
  const long long total = (long long)A.ncell * A.nrays * A.ngroup;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int g = (int)(t % A.ngroup);
    const long long cj = t / A.ngroup;
    const int s0 = g * SG, ns = min(SG, A.nsel - s0);
    int k[SG];
    double acc[SG];
#pragma unroll
    for (int u = 0; u < SG; u++) {
      k[u] = (u < ns) ? A.species[s0 + u] : 0;
      acc[u] = 0.0;
    }
    const int ne = A.epray[cj];
    const long long p0 = A.offset[cj];
    bool bad = (ne > 0) && (p0 < 0 || p0 + ne >= A.npoint);
    if (ne > 0 && !bad) {
      int gprev = A.gp[p0];
      if (gprev < 0 || gprev >= A.ngrid) { bad = true; gprev = 0; }
      double rprev = A.rho[gprev];
      for (int i = 1; i <= ne && !bad; i++) {
        const long long p = p0 + i;
        int gi = A.gp[p];
        if (gi < 0 || gi >= A.ngrid) { bad = true; break; }
        const double ri = A.rho[gi];
        // half the step (exact), so that the trapezoid's factor costs nothing per species
        const double sp = __dmul_rn(__dmul_rn(step_length(A.xyz, p), PC), 0.5);
        const double *xa = A.ab + (size_t)gprev * A.nspec, *xb = A.ab + (size_t)gi * A.nspec;
#pragma unroll
        for (int u = 0; u < SG; u++)
          if (u < ns) {
            const double mid = __dadd_rn(__dmul_rn(rprev, xa[k[u]]), __dmul_rn(ri, xb[k[u]]));
            acc[u] = __dadd_rn(acc[u], __dmul_rn(sp, mid));
          }
        gprev = gi;
        rprev = ri;
      }
    }
    double *o = A.out + cj * A.nsel + s0;
#pragma unroll
    for (int u = 0; u < SG; u++)
      if (u < ns) o[u] = bad ? nan("") : acc[u];
  }
}

struct TauArgs {
  int ncell, nrays, ngrid, nlev, nlin;
  long long npoint;
  const int *epray;
  const long long *offset;
  const double *xyz;
  const int *gp;
  const double *pop, *T, *weights, *rweights, *frac1;
  const int *up, *lo;
  double v2;
  double *tau;
};

// A lane per (cell, ray, line): a block takes 256 consecutive ones, the lines
// of a ray side by side.  The rays' step lengths, a square root each, are
// computed once for all their lines, eight points of every ray of the block at
// a time, in shared memory with the points' grid indices.  A point's term
// g_u n_l - g_l n_u is shared by the two steps it ends and starts.  The
// division by the lower level's weight g is the product with its rounded
// reciprocal y and one residual step, q = a y, q + (a - g q) y, which rounds as
// the division does (Markstein); the trapezoid's 1/2 is in f12 (exact).  What
// bounds it: the FP64 pipe, 11 instructions per line and step.  (One warp per
// ray with two lines per lane left 24 of 64 slots of CO's 40 lines idle and
// took 17 and the square root.)  CO, 29^3 cells, 12 rays of 8.5 points: 8.5 ->
// 2.64 ms.
__global__ void __launch_bounds__(TAU_THREADS) tau_kernel(const __grid_constant__ TauArgs A, int rays_max) {
  constexpr double KB = 1.38065040e-16, MP = 1.67262164e-24, PI = 3.141592653589793238462643383279502884197;
  extern __shared__ __align__(16) unsigned char smem[];
  double *steps = reinterpret_cast<double *>(smem);                    // [rays_max][TAU_STEPS]
  double *frac2 = steps + (size_t)rays_max * TAU_STEPS;                // [rays_max]
  int *gps = reinterpret_cast<int *>(frac2 + rays_max);                // [rays_max][TAU_STEPS], -1: outside the grid
  int *nes = gps + (size_t)rays_max * TAU_STEPS;                       // [rays_max] points of the ray, -1: bad
  const int tid = threadIdx.x;
  const long long total = (long long)A.ncell * A.nrays * A.nlin, nray_all = (long long)A.ncell * A.nrays;
  for (long long t0 = (long long)blockIdx.x * TAU_THREADS; t0 < total; t0 += (long long)gridDim.x * TAU_THREADS) {
    const long long ray0 = t0 / A.nlin;
    const int nr = (int)(min((t0 + TAU_THREADS - 1) / A.nlin, nray_all - 1) - ray0) + 1;
    int longest = 0;
    for (int i = tid; i < nr; i += TAU_THREADS) {
      const long long cj = ray0 + i;
      const int ne = A.epray[cj];
      const long long p0 = A.offset[cj];
      int n = max(ne, 0);
      if (ne > 0 && (p0 < 0 || p0 + ne >= A.npoint)) n = -1;
      nes[i] = n;
      longest = max(longest, n);
      // FRAC2 of escape_probability.F90:57 for this cell's temperature
      frac2[i] = 1.0 / __dsqrt_rn(__dadd_rn(
          __ddiv_rn(__ddiv_rn(__dmul_rn(8.0 * KB, A.T[cj / A.nrays]), PI), MP), A.v2));
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    __shared__ int most;
    if (tid == 0) most = 0;
    __syncthreads();
    if ((tid & 31) == 0 && longest > 0) atomicMax(&most, longest);
    __syncthreads();
    longest = most;
    // this thread's ray and line
    const long long t = t0 + tid;
    const bool mine = t < total;
    const long long cj = mine ? t / A.nlin : ray0;
    const int l = mine ? (int)(t - cj * A.nlin) : 0, ray = (int)(cj - ray0);
    const int u = A.up[l], d = A.lo[l], ne = mine ? nes[ray] : 0;
    const double gu = A.weights[u], gd = A.weights[d], rg = A.rweights[d];
    const double f12 = __dmul_rn(A.frac1[l], frac2[ray]) * 0.5;
    double prev = 0.0, tau = 0.0;
    bool bad = ne < 0;
    if (ne > 0) {
      const int ga = A.gp[A.offset[cj]];
      if (ga < 0 || ga >= A.ngrid) bad = true;
      else {
        const double *pa = A.pop + (size_t)ga * A.nlev;
        prev = __dsub_rn(__dmul_rn(pa[d], gu), __dmul_rn(pa[u], gd));
      }
    }
    for (int i0 = 1; i0 <= longest; i0 += TAU_STEPS) {
      for (int q = tid; q < nr * TAU_STEPS; q += TAU_THREADS) {
        const int r = q / TAU_STEPS, i = i0 + q - r * TAU_STEPS;
        if (i > nes[r]) continue;
        const long long p = A.offset[ray0 + r] + i;
        const int gb = A.gp[p];
        gps[q] = (gb >= 0 && gb < A.ngrid) ? gb : -1;
        steps[q] = step_length(A.xyz, p);
      }
      __syncthreads();
      const int m = bad ? 0 : min(TAU_STEPS, ne - i0 + 1);
      for (int i = 0; i < m; i++) {
        const int gb = gps[ray * TAU_STEPS + i];
        if (gb < 0) { bad = true; break; }
        const double *pb = A.pop + (size_t)gb * A.nlev;
        const double cur = __dsub_rn(__dmul_rn(pb[d], gu), __dmul_rn(pb[u], gd));
        const double x = __dadd_rn(prev, cur);
        const double q0 = __dmul_rn(x, rg);
        double frac3 = fma(fma(-gd, q0, x), rg, q0);
        // beyond the residual step's exponent range, or a weight it was not made for
        if ((((unsigned)__double2hiint(x) >> 20) & 0x7ff) - 128u > 1790u && (__double_as_longlong(x) << 1) != 0)
          frac3 = __ddiv_rn(x, gd);
        tau = __dadd_rn(tau, __dmul_rn(__dmul_rn(__dmul_rn(f12, frac3), steps[ray * TAU_STEPS + i]), PC));
        prev = cur;
      }
      __syncthreads();
    }
    if (mine) {
      const int c = (int)(cj / A.nrays), j = (int)(cj - (long long)c * A.nrays);
      A.tau[((size_t)c * A.nlin + l) * A.nrays + j] = bad ? nan("") : tau;
    }
    __syncthreads();
  }
}

}  // namespace

int launch_tau(const pdr_coolant *cool, const pdr_rays &r, const double *pop, const double *T, double v_turb,
               double *tau, int sm_count, cudaStream_t st) {
  TauArgs A;
  A.ncell = r.ncell;
  A.nrays = r.nrays;
  A.ngrid = r.ngrid;
  A.npoint = r.npoint;
  A.nlev = cool->dev.nlev;
  A.nlin = cool->dev.nlin;
  A.epray = r.d_epray;
  A.offset = r.d_offset;
  A.xyz = r.d_xyz;
  A.gp = r.d_gridpoint;
  A.pop = pop;
  A.T = T;
  A.weights = cool->dev.weights;
  A.rweights = cool->dev.rweights;
  A.frac1 = cool->dev.line_frac1;
  A.up = cool->dev.line_up;
  A.lo = cool->dev.line_lo;
  A.v2 = v_turb * v_turb;
  A.tau = tau;
  // the rays of a block's 256 consecutive (ray, line) pairs
  const int rays_max = (TAU_THREADS + A.nlin - 2) / A.nlin + 1;
  const size_t smem = (size_t)rays_max * (TAU_STEPS * (8 + 4) + 8 + 4);
  const long long want = ((long long)r.ncell * r.nrays * A.nlin + TAU_THREADS - 1) / TAU_THREADS;
  const int blocks = (int)std::max(1ll, std::min(want, (long long)sm_count * 16));
  tau_kernel<<<blocks, TAU_THREADS, smem, st>>>(A, rays_max);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "tau_kernel launch");
}

int launch_uvfield(const pdr_rays &r, const double *rho, int field, const double *G, const double *vectors,
                   double metallicity, double *colden, double *AV, double *rad, double *uv, int sm_count,
                   cudaStream_t st) {
  UvArgs A;
  A.ncell = r.ncell;
  A.nrays = r.nrays;
  A.ngrid = r.ngrid;
  A.npoint = r.npoint;
  A.field = field;
  A.epray = r.d_epray;
  A.offset = r.d_offset;
  A.xyz = r.d_xyz;
  A.gp = r.d_gridpoint;
  A.rho = rho;
  A.colden = colden;
  A.AV = AV;
  A.rad = rad;
  A.uv = uv;
  // Fortran default-REAL literals of input_parameters.F90:57-58
  A.av_fac = (double)6.289e-22f * metallicity;
  A.uv_fac = (double)3.02f;
  A.g_iso = G[0] / (double)r.nrays;
  A.g_uni = 0.0;
  A.uni_ray = -1;
  if (field == 1) {
    // the ray most anti-parallel to G (last one on ties, 3DPDR.F90:1672-1683)
    double best = 0.0;
    for (int j = 0; j < r.nrays; j++) {
      const double d = -(G[0] * vectors[3 * j] + G[1] * vectors[3 * j + 1] + G[2] * vectors[3 * j + 2]);
      if (d >= best) { best = d; A.uni_ray = j; }
    }
    if (A.uni_ray >= 0) A.g_uni = best;
  }
  const int per = std::max(1, UV_THREADS / r.nrays);
  const int blocks = std::max(1, std::min((r.ncell + per - 1) / per, sm_count * 16));
  uvfield_kernel<<<blocks, UV_THREADS, 0, st>>>(A);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "uvfield_kernel launch");
}

int launch_columns(const pdr_rays &r, const double *rho, const double *ab, int nspec, const int *species, int nsel,
                   double *out, int sm_count, cudaStream_t st) {
  ColArgs A;
  A.ncell = r.ncell;
  A.nrays = r.nrays;
  A.ngrid = r.ngrid;
  A.npoint = r.npoint;
  A.nspec = nspec;
  A.nsel = nsel;
  A.ngroup = (nsel + SG - 1) / SG;
  A.epray = r.d_epray;
  A.offset = r.d_offset;
  A.xyz = r.d_xyz;
  A.gp = r.d_gridpoint;
  A.rho = rho;
  A.ab = ab;
  A.out = out;
  if (nsel > MAXSEL) return PDR_E_ARG;
  for (int s = 0; s < nsel; s++) {
    A.species[s] = species ? species[s] : s;
    if (A.species[s] < 0 || A.species[s] >= nspec) {
      set_error("pdr_column_densities_batched: species index out of range");
      return PDR_E_ARG;
    }
  }
  const long long total = (long long)r.ncell * r.nrays * A.ngroup;
  const long long want = (total + 127) / 128;
  const int blocks = (int)std::max(1ll, std::min(want, (long long)sm_count * 16));
  columns_kernel<<<blocks, 128, 0, st>>>(A);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "columns_kernel launch");
}

}  // namespace pdr
