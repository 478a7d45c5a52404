// Host checks of fp64_fast.cuh, compiled with the intrinsics of cuda_runtime.h
// beside this file.
//  rounding  sqrt_rn rounds as the IEEE operation and rcp_near is within 0.5 + 2^-35 ulp,
//            whatever the FP32 unit's start value (moved by up to 2 ulp) -- on random operands
//            and on those whose results lie nearest to the midpoint of two doubles
// Usage: fp64_check rounding; exit 0 when every check holds.
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

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "rounding") return check_rounding();
  std::printf("usage: fp64_check rounding\n");
  return 2;
}
