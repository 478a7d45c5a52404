// The device intrinsics that fp64_fast.cuh uses, for a host build of it; the
// FP32 unit's approximations are the rounded values moved by g_seed_ulps.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline

struct alignas(8) float2 { float x, y; };
struct alignas(16) double2 { double x, y; };

template <class To, class From>
inline To bits_as(From v) {
  static_assert(sizeof(To) == sizeof(From), "same size");
  To t;
  std::memcpy(&t, &v, sizeof t);
  return t;
}
inline double __hiloint2double(int h, int l) { return bits_as<double>((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
inline int __double2hiint(double d) { return (int)(bits_as<uint64_t>(d) >> 32); }
inline int __double2loint(double d) { return (int)bits_as<uint64_t>(d); }
inline long long __double_as_longlong(double d) { return bits_as<long long>(d); }
inline double __longlong_as_double(long long b) { return bits_as<double>(b); }
inline unsigned __float_as_uint(float f) { return bits_as<unsigned>(f); }
inline int __float_as_int(float f) { return bits_as<int>(f); }
inline float __uint_as_float(unsigned u) { return bits_as<float>(u); }
inline unsigned __funnelshift_l(unsigned lo, unsigned hi, int s) { return (hi << s) | (lo >> (32 - s)); }
inline int __float2int_rn(float f) { return (int)std::lrint(f); }
inline double __drcp_rn(double x) { return 1.0 / x; }
inline double __dsqrt_rn(double x) { return std::sqrt(x); }
template <class T>
inline T __ldg(const T *p) { return *p; }

inline int g_seed_ulps = 0;
namespace pdr {
namespace fp64 {
inline float moved(float y) { return __uint_as_float(__float_as_uint(y) + g_seed_ulps); }
inline float rcp_approx(float x) { return moved((float)(1.0 / (double)x)); }
inline float rsqrt_approx(float x) { return moved((float)(1.0 / std::sqrt((double)x))); }
}  // namespace fp64
}  // namespace pdr
