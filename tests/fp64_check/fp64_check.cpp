// Host checks of fp64_fast.cuh, compiled with the intrinsics of cuda_runtime.h
// beside this file.
//  rounding  sqrt_rn rounds as the IEEE operation and rcp_near is within 0.5 + 2^-35 ulp,
//            whatever the FP32 unit's start value (moved by up to 2 ulp) -- on random operands
//            and on those whose results lie nearest to the midpoint of two doubles
//  tables    every row of fp64_tables.inc against its definition
//  functions the errors stated in fp64_fast.cuh, over the ranges the kernels use and at
//            their ends; "ulp" is 2^-52 of the result
// Usage: fp64_check rounding|tables|functions; exit 0 when every check holds.
#include "../../3d-pdr_gb300/csrc/fp64_fast.cuh"

#include <quadmath.h>

#include <cstdio>
#include <random>
#include <string>
#include <vector>

using namespace pdr::fp64;
typedef unsigned __int128 U128;

static std::mt19937_64 rng(20261206);
static double uniform(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }

// operands whose square root lies within about 2^-50 ulp of a midpoint: with
// 53-bit x and n = 2 m + 1 the (odd, 54-bit) midpoint, 4 x = n^2 - c for a small
// c = 1 mod 8, so n is a square root of c modulo 2^54 (2^55 in the upper binade)
static std::vector<double> hard_squares() {
  std::vector<double> out;
  for (int k = 54; k <= 55; k++)
    for (long long c = -4095; c <= 4097; c += 8) {
      uint64_t s = 1;   // 2-adic square root of c, a bit at a time
      for (int b = 3; b < k; b++)
        if (((U128)s * s - (U128)(__int128)c) >> b & 1) s += 1ull << (b - 1);
      const uint64_t mask = (uint64_t(1) << k) - 1;
      for (uint64_t r : {s & mask, (0 - s) & mask, (s + (uint64_t(1) << (k - 1))) & mask, (0 - s + (uint64_t(1) << (k - 1))) & mask}) {
        const uint64_t n = r & ((1ull << 54) - 1);
        if (n < (1ull << 53)) continue;
        const U128 x4 = (U128)n * n - (U128)(__int128)c;
        if (x4 & ((U128)mask)) continue;
        const double x = (double)(uint64_t)(x4 >> k);   // at most 53 bits
        if ((U128)(uint64_t)x << k != x4) continue;
        for (int e : {-60, 0, 44}) out.push_back(std::ldexp(x, k - 2 - 104 + e));
      }
    }
  return out;
}

static int check_rounding() {
  long bad = 0, n = 0;
  auto same = [&](const char *what, double x, double got, double want) {
    n++;
    if (__double_as_longlong(got) == __double_as_longlong(want)) return;
    if (bad++ < 10) std::printf("%s(%.17g) with the start value %+d ulp: %.17g, not %.17g\n", what, x, g_seed_ulps, got, want);
  };
  // the nearest double, or the other neighbour where the exact value is within 2^-35 ulp of their midpoint
  auto near_rcp = [&](double x, double got) {
    n++;
    if (__double_as_longlong(got) == __double_as_longlong(1.0 / x)) return;
    // in ulps of the result (distances from a midpoint are exact to 2^-60 ulp in 113 bits)
    const __float128 off = fabsq((1 / (__float128)x - got) / std::ldexp(1.0, std::ilogb(1.0 / x) - 52)) - 0.5Q;
    if (fabsq(off) <= ldexpq(1.0Q, -35)) return;
    if (bad++ < 10) std::printf("rcp_near(%.17g) with the start value %+d ulp: %.17g\n", x, g_seed_ulps, got);
  };
  std::vector<double> sq = hard_squares(), rc;
  std::printf("%zu hard square roots\n", sq.size());
  if (sq.size() < 1000) bad++;
  // 1/(2^53 - k) is k^2 2^-54 ulp above a midpoint for odd k
  for (int k = 1; k < 8000; k += 2)
    for (int e : {-1000, -53, 0, 900}) rc.push_back(std::ldexp(9007199254740992.0 - k, e) * (k & 2 ? 1 : -1));
  for (int i = 0; i < 400000; i++) {
    rc.push_back(std::ldexp(uniform(1.0, 2.0) * (i & 1 ? 1 : -1), (int)(rng() % 2040) - 1020));
    sq.push_back(std::ldexp(uniform(1.0, 4.0), 2 * ((int)(rng() % 120) - 60)));
  }
  // the ends of a binade, the ends of the range, and what the library takes
  for (int k = 0; k < 60; k++)
    for (double x : {1.0 + std::ldexp(k, -52), 2.0 - std::ldexp(k, -52), 4.0 - std::ldexp(k, -51)})
      for (int e : {-1030, -1022, -126, -60, 0, 60, 126, 1021}) {
        rc.push_back(std::ldexp(x, e));
        sq.push_back(std::ldexp(x, e));
      }
  for (double x : {0.0, 5e-324, 1e-310, (double)INFINITY}) {
    rc.push_back(x);
    sq.push_back(x);
  }
  for (g_seed_ulps = -2; g_seed_ulps <= 2; g_seed_ulps++) {
    if (g_seed_ulps != -2 && g_seed_ulps != 2)
      for (double x : rc) near_rcp(x, rcp_near(x));
    for (double x : sq) same("sqrt_rn", x, sqrt_rn(x), std::sqrt(x));
  }
  std::printf("%ld of %ld misrounded\n", bad, n);
  return bad != 0;
}

typedef __float128 Q;

static int check_tables() {
  int bad = 0;
  auto expect = [&](const char *what, int j, bool ok) {
    if (!ok && bad++ < 10) std::printf("%s, row %d\n", what, j);
  };
  for (int j = 0; j < 1024; j++) {
    const Q v = exp2q((Q)j / 1024);
    expect("2^(j/1024) rounded", j, kExp2Tab[j].t == (double)v);
    // the row's relative error, to nine digits
    const Q d = v / kExp2Tab[j].t - 1;
    expect("its relative error", j, fabsq(kExp2Tab[j].d - d) <= 1e-8Q * fabsq(d) + 1e-30Q);
  }
  Q rmax = 0;
  for (int j = 0; j < 512; j++) {
    const LogRow &r = kLogTab[j];
    const Q v = -1024 * log2q((Q)r.c), grid = (Q)r.hi * 4294967296.0Q;
    expect("hi on the 2^-32 grid", j, grid == floorq(grid));
    expect("hi + lo", j, fabsq((Q)r.hi + r.lo - v) <= 1e-17Q);
    // m c - 1 over the row's mantissas
    for (int k = 0; k < 2; k++) rmax = fmaxq(rmax, fabsq((1 + (Q)(j + k) / 512) * r.c - 1));
    expect("c of twelve bits", j, r.c * 4096.0f == std::floor(r.c * 4096.0f));
  }
  std::printf("largest |m c - 1|: %.3g\n", (double)rmax);
  expect("m c - 1", 0, rmax < 1.0Q / 400);
  return bad != 0;
}

static int check_functions() {
  const int N = 300000;
  const double U = 2.220446049250313e-16;
  int bad = 0;
  auto expect = [&](const char *what, double worst, double bound) {
    std::printf("%-12s %.4g (bound %.4g)\n", what, worst, bound);
    if (!(worst <= bound)) bad++;
  };
  auto rel = [](double got, Q want) { return (double)fabsq(((Q)got - want) / want); };
  double e = 0, l = 0, l1 = 0, la = 0, p = 0, x2 = 0;
  for (int i = 0; i < N; i++) {
    const double x = i % 7 == 0 ? uniform(-1e-3, 1e-3) : (i & 1) ? uniform(-40, 5) : uniform(-690, 690);
    e = std::fmax(e, rel(exp_fast(x), expq(x)) / U);
    // the rates' T/300 and T, columns, optical depths; near 1 the logarithm's leading bits cancel
    const double y = i % 5 == 0 ? 1 + uniform(-0.01, 0.01) : i % 11 == 0 ? std::ldexp(uniform(1, 2), i % 2000 - 1000)
                                                                              : std::exp(uniform(-60, 60));
    const Q lq = 1024 * log2q(y);
    const Log2 L = log2k(y);
    l = std::fmax(l, (double)fabsq((Q)L.h + L.l - lq));
    // its use: log10 of columns, which the shielding clamps at 12 from below
    const double n = std::exp(uniform(std::log(1e12), std::log(1e30)));
    l1 = std::fmax(l1, rel(log10_fast(n), log10q(n)) / U);
    const double n1 = 1 + std::exp(uniform(-40, 28));
    la = std::fmax(la, (double)fabsq(log10_fast(n1) - log10q(n1)));
    const double b = uniform(-6, 6);
    if (std::fabs(b * std::log2(y)) < 990) p = std::fmax(p, rel(powk(L, b), powq(y, b)) / U);
    const int k = (int)(rng() % 1800000) - 900000;
    const double r = uniform(-2, 2), a = uniform(1, 2);
    x2 = std::fmax(x2, rel(exp2_times(a, k, r), a * exp2q(((Q)k + r) / 1024)) / U);
  }
  expect("exp_fast", e, 0.502);
  expect("log2k", l, 1.5e-14);
  expect("log10_fast", l1, 0.545);   // the last rounding, and 9.3e-18 of log10(2)/1024
  expect("its small", la, 4e-15);
  expect("powk", p, 0.70);
  // the roundings of a times the row and of the sum; at |r| = 2 the series' first term left
  // out, (2 C1)^3/60 of 2 C1^2 (0.17), and the FP32 rounding of those kept (0.1)
  expect("exp2_times", x2, 1.27);
  for (double x : {0.0, -0.0}) expect("exp_fast(0)", std::fabs(exp_fast(x) - 1), 0);
  expect("exp_fast(-800)", exp_fast(-800.0), 0);
  // f2d and d2f: exact where they have to be, truncation elsewhere
  double conv = 0;
  for (int i = 0; i < N; i++) {
    const float f = (float)(std::ldexp(uniform(1, 2), (int)(rng() % 252) - 126)) * (i & 1 ? 1.0f : -1.0f);
    if (f2d(f) != (double)f || d2f((double)f) != f) conv++;
    const double d = std::ldexp(uniform(1, 2), (int)(rng() % 240) - 120);
    const float t = d2f(d);
    if (!((double)t <= d && d < (double)std::nextafter(t, INFINITY))) conv++;
  }
  if (f2d(0.0f) != 0 || d2f(0.0) != 0 || d2f(1e-40) != 0 || d2f(-1e-300) != 0) conv++;
  expect("f2d, d2f", conv, 0);
  double rs = 0, dv = 0, any = 0;
  for (g_seed_ulps = -1; g_seed_ulps <= 1; g_seed_ulps++)
    for (int i = 0; i < N / 3; i++) {
      const double w = std::ldexp(uniform(1, 4), 2 * ((int)(rng() % 60) - 30));
      rs = std::fmax(rs, rel(rsqrt_fast(w), 1 / sqrtq(w)) / U);
      const double a = std::ldexp(uniform(1, 2), (int)(rng() % 280) - 140) * (i & 1 ? 1 : -1);
      double b = std::ldexp(uniform(1, 2), (int)(rng() % 280) - 140) * (i & 2 ? 1 : -1);
      if (i % 9 == 0) b = 1 + std::ldexp((double)(i % 50), -52);
      if (i % 13 == 0) b = 2 - std::ldexp((double)(1 + i % 50), -52);
      const Q q = (Q)a / b;
      const double got = div_fast(a, b);
      dv = std::fmax(dv, (double)(fabsq(got - q) / std::ldexp(1.0, std::ilogb(a / b) - 52)));
      const double c = std::ldexp(uniform(1, 2), (int)(rng() % 2040) - 1020), d = std::ldexp(uniform(1, 2), (int)(rng() % 2040) - 1020);
      if (div_any(c, d) != c / d) any++;
    }
  expect("rsqrt_fast", rs, 0.64);
  expect("div_fast", dv, 0.5 + std::ldexp(1.0, -35));
  for (double c : {0.0, 1.0, -3.0, 5e-324, 1e308, (double)INFINITY})
    for (double d : {0.0, 7.0, -2.0, 5e-324, 1e308, (double)INFINITY}) {
      const double g = div_any(c, d), w = c / d;
      if (__double_as_longlong(g) != __double_as_longlong(w) && !(std::isnan(g) && std::isnan(w))) any++;
    }
  expect("div_any", any, 0);
  return bad != 0;
}

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "rounding") return check_rounding();
  if (what == "tables") return check_tables();
  if (what == "functions") return check_functions();
  std::printf("usage: fp64_check rounding|tables|functions\n");
  return 2;
}
