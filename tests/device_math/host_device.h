// CUDA's integer and rounding intrinsics in plain C++, so that the device
// headers that use nothing else (hexo_ds.cuh, hexo_f64.cuh) compile for the
// host and can be held against long double there.  Include before them.
//
// The two approximate instructions are modelled by the correctly rounded
// result moved by `mufu_ulp` units of its last place; their documented errors
// are 2^-23 (rcp) and 2^-22.9 (rsqrt) relative, up to one unit either way.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline
#define __noinline__
using std::max;
using std::min;

template <class To, class From> inline To bits_of(From x) {
    static_assert(sizeof(To) == sizeof(From), "");
    To r;
    std::memcpy(&r, &x, sizeof r);
    return r;
}
inline uint32_t __float_as_uint(float f) { return bits_of<uint32_t>(f); }
inline float __uint_as_float(uint32_t u) { return bits_of<float>(u); }
inline long long __double_as_longlong(double d) { return bits_of<long long>(d); }
inline double __longlong_as_double(long long x) { return bits_of<double>(x); }
inline int __double2hiint(double d) { return (int)(bits_of<uint64_t>(d) >> 32); }
inline int __double2loint(double d) { return (int)(uint32_t)bits_of<uint64_t>(d); }
inline double __hiloint2double(int h, int l) {
    return bits_of<double>((uint64_t)(uint32_t)h << 32 | (uint64_t)(uint32_t)l);
}
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) {
    return (uint32_t)((((uint64_t)hi << 32 | lo) << (s & 31u)) >> 32);
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    return (uint32_t)(((uint64_t)hi << 32 | lo) >> (s & 31u));
}
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
inline int __mulhi(int a, int b) { return (int)((long long)a * b >> 32); }
inline int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fdividef(float a, float b) { return a / b; }
inline float __log2f(float a) { return std::log2(a); }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline double __dsqrt_rn(double a) { return std::sqrt(a); }
inline float __double2float_rn(double a) { return (float)a; }
inline float __uint2float_rn(uint32_t a) { return (float)a; }
inline float __uint2float_rz(uint32_t a) {   // a < 2^24 wherever it is used: exact
    return (float)a;
}
inline float __int2float_rn(int a) { return (float)a; }
inline int __float2int_rn(float a) {   // saturates, NaN is 0
    return std::isnan(a) ? 0 : a >= 2147483648.0f ? 2147483647 : a <= -2147483648.0f ? (int)0x80000000 : (int)std::nearbyint(a);
}
inline double __ull2double_rn(uint64_t a) { return (double)a; }

static int mufu_ulp = 0;
inline float mufu(const char *ins, float x) {   // .ftz: a subnormal operand or result counts as zero
    const float t = std::fabs(x) < 0x1p-126f ? std::copysign(0.0f, x) : x;
    const long double v = std::strstr(ins, "rsqrt") ? 1.0L / std::sqrt((long double)t) : 1.0L / (long double)t;
    const float r = (float)v;
    if (!std::isfinite(r) || r == 0.0f) return r;
    const float m = __uint_as_float(__float_as_uint(r) + (uint32_t)mufu_ulp);
    return std::fabs(m) < 0x1p-126f ? std::copysign(0.0f, m) : m;
}
// the headers' asm statements: `r` is the result, `x` the operand
#define asm(...) r = mufu(#__VA_ARGS__, x)
