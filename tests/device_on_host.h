// Stand-ins for the CUDA built-ins that the table query headers use, so that a
// host compiler can build the headers and a test can call them on the CPU:
// the same integer and rounded arithmetic, one thread.
#pragma once

#include <cuda_runtime.h>

#include <cfenv>
#include <cmath>
#include <cstring>

template <class F>
inline auto rounded(int mode, F f) {
  const int before = fegetround();
  fesetround(mode);
  const auto r = f();
  fesetround(before);
  return r;
}

template <class T> inline T __ldg(const T* p) { return *p; }
inline float __fadd_rd(float a, float b) { return rounded(FE_DOWNWARD, [&] { volatile float x = a, y = b; return x + y; }); }
inline float __fmaf_rd(float a, float b, float c) { return rounded(FE_DOWNWARD, [&] { return fmaf(a, b, c); }); }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
inline float __fdividef(float a, float b) { return a / b; }
inline float __expf(float a) { return expf(a); }
inline int __float_as_int(float f) {
  int i;
  memcpy(&i, &f, sizeof i);
  return i;
}
inline long long __float2ll_rn(float f) { return llrintf(f); }
inline long long __double2ll_rn(double d) { return llrint(d); }
inline unsigned __float2uint_rn(float f) { return (unsigned)llrintf(f); }
inline int __float2int_rz(float f) { return (int)f; }
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((unsigned long long)a * b) >> 32); }
template <class T> inline T __shfl_sync(unsigned, T v, int, int = 32) { return v; }
inline void atomicAdd(unsigned long long* p, unsigned long long v) { *p += v; }
inline int max(int a, int b) { return a > b ? a : b; }
inline int min(int a, int b) { return a < b ? a : b; }
static const uint3 threadIdx{0u, 0u, 0u};
