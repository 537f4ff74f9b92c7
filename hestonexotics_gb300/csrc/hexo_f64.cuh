// Double-precision pieces of the FP64 path kernel that keep off the FP64 pipe.
//
// GB300 runs one FP64 warp instruction per 64 cycles and SM sub-partition
// (2 lanes per cycle and SM, conversions between float, integer and double
// included), against 64 FP32 or integer instructions in the same time.  The
// FP64 step written with double divisions, square roots, log and exp issues
// about 100 FP64 instructions and leaves nine tenths of the other issue slots
// idle.  Here a quotient or root starts as a double-single value (hexo_ds.cuh:
// about 2^-46, FP32 instructions only), becomes a double by integer packing,
// and its remainder is then computed exactly from the low halves of the
// significands in 64-bit integer arithmetic: the value and the product that
// approximates it agree to more than 40 bits, so their difference fits in a
// 64-bit word and only the products' lower words are needed.  One Newton
// correction with that remainder gives a result within 2^-53 of the exact
// one, and the correction itself is small enough for FP32.  FP64 instructions
// are left for sums and products that need all 53 bits.
#pragma once
#include <stdint.h>
#include "hexo_ds.cuh"

namespace hexo {
namespace f64 {

__device__ __forceinline__ uint32_t hi32(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ uint32_t lo32(double x) { return (uint32_t)__double2loint(x); }
__device__ __forceinline__ double from_words(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }

// The 24 leading bits of x, 2^-126 <= x < 2^128: sign 0, exponent rebiased by flipping its top bit.
__device__ __forceinline__ float head(double x) {
    return __uint_as_float((__funnelshift_l(lo32(x), hi32(x), 3) & 0x7fffffffu) ^ 0x40000000u);
}
// 2^e, e the exponent of x (2^-126 <= x < 2^128).
__device__ __forceinline__ float pow2_of(double x) {
    return __uint_as_float(((hi32(x) << 3) & 0x7f800000u) ^ 0x40000000u);
}
// f as a double: exact for normal f; 0 and subnormals become values below 2^-126.
__device__ __forceinline__ double to_double(float f) {
    const uint32_t b = __float_as_uint(f);
    return from_words(((uint32_t)((int32_t)b >> 3) & 0x8fffffffu) + 0x38000000u, b << 29);
}
// x as a double-single value, 2^-74 <= x < 2^100: head and the other 29 bits.
__device__ __forceinline__ ds::F2 split(double x) {
    const float h = head(x);
    const float e = __uint_as_float(__float_as_uint(h) & 0x7f800000u);
    return ds::F2{h, __fmul_rn(__fmul_rn(__uint2float_rn(lo32(x) & 0x1fffffffu), 0x1p-52f), e)};
}

// h + l as a double, 2^-74 <= h < 2^74 and |l| <= 2^-23 h: l is rounded to
// units of the double's last place and added to the bits of h.  The units are
// those of the binade that h + l lies in (below h's when h is a power of two
// and l negative).
__device__ __forceinline__ double join(ds::F2 x) {
    const uint32_t hb = __float_as_uint(x.h);
    const uint32_t eb = (hb + (uint32_t)((int32_t)__float_as_uint(x.l) >> 31)) & 0x7f800000u;
    const int32_t k = __float2int_rn(__fmul_rn(x.l, __uint_as_float(0x7f000000u + (52u << 23) - eb)));
    return __longlong_as_double((long long)((uint64_t)hb * 0x20000000ull + 0x3800000000000000ull) + (long long)k);
}

// x - a b for doubles with |x - a b| < 2^-33 2^(ea+eb) (ea, eb the exponents
// of a and b): words 1 and 2 of the significands' product taken from x's,
// cut at 2^-64 of 2^(ea+eb) (the unit of the integer forms).
__device__ __forceinline__ int32_t remainder_mul_units(double x, double a, double b) {
    const uint32_t al = lo32(a), bl = lo32(b), ah = hi32(a), bh = hi32(b), xl = lo32(x), xh = hi32(x);
    const uint32_t am = (ah & 0x000fffffu) | 0x00100000u, bm = (bh & 0x000fffffu) | 0x00100000u;
    uint64_t p = (uint64_t)al * bm + __umulhi(al, bl);
    p += (uint64_t)bl * am;
    p += (uint64_t)(am * bm) << 32;
    const uint32_t s = 20u + 1023u + (xh >> 20) - (ah >> 20) - (bh >> 20);   // 19 to 22
    const uint64_t d = (((uint64_t)__funnelshift_l(xl, xh, s) << 32) | (uint64_t)(uint32_t)(xl << s)) - p;
    return (int32_t)__funnelshift_r((uint32_t)d, (uint32_t)(d >> 32), 8);
}
__device__ __forceinline__ float remainder_mul(double x, double a, double b) {
    const float r = __int2float_rn(remainder_mul_units(x, a, b));
    return __fmul_rn(__fmul_rn(__fmul_rn(r, 0x1p-64f), pow2_of(a)), pow2_of(b));
}
// x - q^2
__device__ __forceinline__ int32_t remainder_sqr_units(double x, double q) {
    const uint32_t ql = lo32(q), qh = hi32(q), xl = lo32(x), xh = hi32(x);
    const uint32_t qm = (qh & 0x000fffffu) | 0x00100000u;
    uint64_t p = (uint64_t)ql * (qm + qm) + __umulhi(ql, ql);
    p += (uint64_t)(qm * qm) << 32;
    const uint32_t s = 20u + 1023u + (xh >> 20) - 2u * (qh >> 20);
    const uint64_t d = (((uint64_t)__funnelshift_l(xl, xh, s) << 32) | (uint64_t)(uint32_t)(xl << s)) - p;
    return (int32_t)__funnelshift_r((uint32_t)d, (uint32_t)(d >> 32), 8);
}
__device__ __forceinline__ float remainder_sqr(double x, double q) {
    const float r = __int2float_rn(remainder_sqr_units(x, q)), e = pow2_of(q);
    return __fmul_rn(__fmul_rn(__fmul_rn(r, 0x1p-64f), e), e);
}

// ------------------------------------------------------------------ tables
//
// 2^(j/256) and, for the logarithm, 512 short reciprocals with their logarithms,
// computed at compile time in double-double arithmetic (Dekker's splitting
// and Knuth's TwoSum, as in hexo_ds.cuh) from the exponential and inverse
// hyperbolic tangent series.

struct DD {
    double h, l;
};
constexpr DD dd_two_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return DD{s, (a - (s - t)) + (b - t)};
}
constexpr DD dd_two_prod(double a, double b) {
    const double ta = 134217729.0 * a, tb = 134217729.0 * b;
    const double ah = ta - (ta - a), bh = tb - (tb - b), al = a - ah, bl = b - bh, p = a * b;
    return DD{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr DD dd_add(DD a, DD b) {
    const DD s = dd_two_sum(a.h, b.h);
    return dd_two_sum(s.h, s.l + (a.l + b.l));
}
constexpr DD dd_mul(DD a, DD b) {
    const DD p = dd_two_prod(a.h, b.h);
    return dd_two_sum(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr DD dd_div(DD a, DD b) {
    const double q = a.h / b.h;
    const DD p = dd_mul(b, DD{q, 0.0});
    const DD r = dd_add(a, DD{-p.h, -p.l});
    return dd_two_sum(q, r.h / b.h);
}
constexpr DD dd_exp(DD x) {   // |x| < 1
    DD s{1.0, 0.0}, t{1.0, 0.0};
    for (int n = 1; n < 30; ++n) {
        t = dd_div(dd_mul(t, x), DD{(double)n, 0.0});
        s = dd_add(s, t);
    }
    return s;
}
constexpr DD dd_log_ratio(DD num, DD den) {   // log((den + num) / (den - num)) = 2 atanh(num / den)
    const DD z = dd_div(num, den), z2 = dd_mul(z, z);
    DD s{0.0, 0.0}, t = z;
    for (int n = 1; n < 80; n += 2) {
        s = dd_add(s, dd_div(t, DD{(double)n, 0.0}));
        t = dd_mul(t, z2);
    }
    return DD{2.0 * s.h, 2.0 * s.l};
}
constexpr DD kLn2 = dd_log_ratio(DD{1.0, 0.0}, DD{3.0, 0.0});

// A double-double value's x.h + x.l, 0 <= x < 4, in units of 2^-62 (to nearest).
constexpr uint64_t dd_fixed62(DD x) {
    const double s = 4611686018427387904.0;                  // 2^62
    const uint64_t h = (uint64_t)(x.h * s);                  // exact: x.h has 53 bits
    const double r = x.h * s - (double)h + x.l * s;
    return h + (uint64_t)(int64_t)(r < 0.0 ? r - 0.5 : r + 0.5);
}

constexpr int kExpTab = 256;   // a CTA's copy in shared memory: kExpTab * 8 bytes
struct ExpTab {
    uint64_t t[kExpTab];       // 2^(j/256) in units of 2^-62
};
constexpr ExpTab make_exp_tab() {
    ExpTab r{};
    for (int j = 0; j < kExpTab; ++j) r.t[j] = dd_fixed62(dd_exp(dd_mul(kLn2, DD{(double)j / kExpTab, 0.0})));
    return r;
}
constexpr int kLogTab = 512;
struct LogEntry {
    uint64_t lg;               // -log(inv 2^-12) in units of 2^-57
    uint32_t inv, pad;         // round(2^12 / c_j), c_j the middle of the j-th of 512 parts of [1, 2)
};
struct LogTab {
    LogEntry e[kLogTab];
};
constexpr LogTab make_log_tab() {
    LogTab r{};
    for (int j = 0; j < kLogTab; ++j) {
        const uint32_t inv = (uint32_t)(4096.0 / (1.0 + (j + 0.5) / kLogTab) + 0.5);
        const DD lg = dd_log_ratio(DD{4096.0 - inv, 0.0}, DD{4096.0 + inv, 0.0});
        r.e[j] = LogEntry{(dd_fixed62(lg) + 16u) >> 5, inv, 0u};
    }
    return r;
}
constexpr int kTurnTab = 256;  // sin and cos of 2 pi j / 256
struct TurnTab {
    double s[kTurnTab], c[kTurnTab];
};
constexpr DD kPi = {0x1.921fb54442d18p+1, 0x1.1a62633145c07p-53};
constexpr TurnTab make_turn_tab() {
    TurnTab r{};
    for (int j = 0; j < kTurnTab; ++j) {   // Taylor series at the angle within (-pi, pi]
        const DD x = dd_mul(kPi, DD{(j <= kTurnTab / 2 ? j : j - kTurnTab) * (2.0 / kTurnTab), 0.0});
        DD s{0.0, 0.0}, c{0.0, 0.0}, t{1.0, 0.0};
        for (int n = 0; n < 48; n += 2) {
            c = dd_add(c, t);
            t = dd_div(dd_mul(t, x), DD{n + 1.0, 0.0});
            s = dd_add(s, t);
            t = dd_div(dd_mul(t, x), DD{-(n + 2.0), 0.0});
        }
        r.s[j] = s.h;
        r.c[j] = c.h;
    }
    return r;
}
__device__ constexpr TurnTab kTurnTabDev = make_turn_tab();
__device__ constexpr ExpTab kExpTabInit = make_exp_tab();
__device__ constexpr LogTab kLogTabDev = make_log_tab();

// A CTA's copy of the exponential's table, visible after the next barrier.
__device__ __forceinline__ void exp_table_init(ExpTab *t, uint32_t tid, uint32_t nthreads) {
    for (uint32_t j = tid; j < (uint32_t)kExpTab; j += nthreads) t->t[j] = kExpTabInit.t[j];
}

// ----------------------------------------------------------- exp, log, root

__device__ __forceinline__ uint32_t hi(uint64_t x) { return (uint32_t)(x >> 32); }
__device__ __forceinline__ uint32_t lo(uint64_t x) { return (uint32_t)x; }
// a b 2^-64, at most 3 too small (the low words' product is left out).
__device__ __forceinline__ uint64_t mul_hi(uint64_t a, uint64_t b) {
    return (uint64_t)hi(a) * hi(b) + __umulhi(hi(a), lo(b)) + __umulhi(lo(a), hi(b));
}
// r^2 2^64 of r 2^-64, at most 1 too small.
__device__ __forceinline__ uint64_t sqr_hi(uint64_t r) {
    return (uint64_t)hi(r) * hi(r) + 2ull * __umulhi(hi(r), lo(r));
}

// exp(x) in integer arithmetic, within 0.57 ulp for |x| < 32 and 0.63 up to 512
// (ln2/256 is kept to 2^-71): x in units of 2^-54 is n ln2/256 + r, 0 <= r <
// ln2/256 (1 + 2^-11), r in units of 2^-71 with what x has below 2^-54, and the
// result 2^(n/256) (1 + r + r^2/2 + r^3 (1/6 + r/24 + r^2/120)) in units of
// 2^-62.  No FP64 instruction (the library's exp takes the time of 18).
__device__ __forceinline__ double exp_tab(double x, const ExpTab *tab) {
    const uint32_t xh = hi32(x), a = xh & 0x7fffffffu;
    if (a >= 0x40800000u) return exp(x);   // |x| >= 512, infinite or NaN
    const uint64_t M = ((uint64_t)((a << 10 & 0x3fffffffu) | 0x40000000u) << 32 | (uint64_t)(lo32(x) >> 22) << 32) |
                       (uint64_t)(lo32(x) << 10);
    const uint32_t sh = 1031u - (a >> 20);
    uint64_t F = M >> min(sh, 63u), R = F << 17;                     // units of 2^-54, 2^-71
    if (sh - 11u < 53u) R |= ((M << 1) << (63u - sh)) >> 47;         // |x| < 1/4: bits below 2^-54
    if ((int32_t)xh < 0) {
        F = 0ull - F;
        R = 0ull - R;
    }
    const int32_t n = __mulhi((int32_t)hi(F) - 2, (int32_t)(kExpTab / kLn2.h * 0x1p22)) >> 12;
    constexpr uint64_t L71 = (uint64_t)(kLn2.h / kExpTab * 0x1p71) + (uint64_t)(int64_t)(kLn2.l / kExpTab * 0x1p71 + 0.5);
    const uint64_t r = R - (uint64_t)(int64_t)n * L71;
    const uint32_t rh = hi(r);
    const uint32_t p = 2863311531u + __umulhi(rh, 5592405u + __umulhi(rh, 8738u));   // 1/6 + r/24 + r^2/120, 2^-34
    const uint32_t q = __umulhi(rh << 1, p) << 1;                                    // r p, 2^-43
    const uint64_t r2 = sqr_hi(r);                                                   // r^2, 2^-78
    const uint64_t u = (r >> 7) + (r2 >> 15) + (uint64_t)__umulhi((uint32_t)(r2 >> 29), q) * 16ull;   // 2^-64
    const uint64_t T = tab->t[n & (kExpTab - 1)];
    uint64_t y = T + mul_hi(T, u);
    const uint32_t s = hi(y) >> 31;        // 2^63 or more: the next binade
    y >>= s;
    return __longlong_as_double((long long)(((uint64_t)(1022u + (uint32_t)(n >> 8) + s) << 52) + ((y + 512ull) >> 10)));
}

// sin(x) and cos(x), within 1.3 ulp of 1: x = n 2 pi / 256 + d, |d| <= pi /
// 256, the table's sine and cosine turned by d (sin d to d^5, cos d - 1 to
// d^6).  15 FP64 instructions (the library's sincos: about 45).
__device__ __forceinline__ void sincos_tab(double x, double *sn, double *cs) {
    if ((hi32(x) & 0x7fffffffu) >= 0x41600000u) {   // |x| >= 2^23, infinite or NaN
        sincos(x, sn, cs);
        return;
    }
    constexpr double H = kPi.h / (kTurnTab / 2), L = kPi.l / (kTurnTab / 2);
    const double t = __fma_rn(x, 1.0 / H, 0x1.8p52), n = __dsub_rn(t, 0x1.8p52);
    const uint32_t j = lo32(t) & (uint32_t)(kTurnTab - 1);
    const double d = __fma_rn(-n, L, __fma_rn(-n, H, x)), d2 = __dmul_rn(d, d);
    const float f2 = __double2float_rn(d2);
    const double q = __dadd_rn(-1.0 / 6.0, to_double(__fmul_rn(f2, 1.0f / 120.0f)));
    const double s = __fma_rn(__dmul_rn(d, d2), q, d);                                        // sin d
    const double u = __dmul_rn(d2, __dadd_rn(-0.5, to_double(__fmul_rn(f2, __fmaf_rn(f2, -1.0f / 720.0f, 1.0f / 24.0f)))));
    const double s0 = kTurnTabDev.s[j], c0 = kTurnTabDev.c[j];
    *sn = __fma_rn(c0, s, __fma_rn(s0, u, s0));
    *cs = __fma_rn(-s0, s, __fma_rn(c0, u, c0));
}

// -log(x) in units of 2^-57 of x = P 2^(k-63), 2^63 <= P < 2^64, -80 < k < 0,
// plus what a relative error d of x and of the result puts on it (log(x (1 +
// d)) (1 + d) to first order, |d| < 2^-40): r = P inv - 1, |r| < 2^-9.6, exact
// in units of 2^-71, log x = k ln2 + log c_j + r - r^2/2 + r^3/3 - r^4/4 +
// r^5/5, the last three in float (below 2^-30; 1/3 rounded up by what cutting
// r to 24 bits takes on average).
__device__ __forceinline__ uint64_t neg_log_fixed(uint64_t P, int k, float d) {
    const LogEntry e = kLogTabDev.e[(uint32_t)(P >> 54) & (uint32_t)(kLogTab - 1)];
    const int64_t r = (int64_t)((P >> 4) * (uint64_t)e.inv);
    const uint64_t ra = (uint64_t)(r < 0 ? -r : r);
    const float rf = __fmul_rn(__int2float_rn((int32_t)(r >> 32)), 0x1p-39f);
    const float c3 = __fmul_rn(__fmul_rn(rf, rf), __fmul_rn(rf, __fmaf_rn(rf, __fmaf_rn(rf, 0.2f, -0.25f), 0x1.555556p-2f)));
    const float lf = __fmul_rn(0.6931472f, __fadd_rn((float)k, __log2f(__uint_as_float((hi(P) >> 8 & 0x007fffffu) | 0x3f800000u))));
    const int32_t c = __float2int_rn(__fmul_rn(__fmaf_rn(d, __fadd_rn(1.0f, lf), c3), 0x1p57f));
    constexpr uint64_t L57 = (uint64_t)(kLn2.h * 0x1p57) + (uint64_t)(int64_t)(kLn2.l * 0x1p57 + 0.5);
    const uint64_t l = (uint64_t)(int64_t)k * L57 + e.lg + (uint64_t)(r >> 14) - (sqr_hi(ra) >> 22) + (uint64_t)(int64_t)c;
    return (int64_t)l < 0 ? 0ull - l : 0ull;
}

// Whether a joined value lies within 2^-20 of a power of two.  There the unit
// of its last place need not be the seed's, and a correction can carry it over
// into the next binade, where the same bits count twice or half as much: the
// root and the reciprocal below take the plain operation for these.
__device__ __forceinline__ bool near_binade(double y) { return (hi32(y) << 12) + 0x1000u <= 0x1000u; }

// sqrt(x), within 0.51 ulp from 2^-113 on: the remainder's correction is added
// to the bits of the joined root in units of its last place.  Below, the seed's
// float remainder runs out of bits (relative error 2^-31 at 2^-119), and x
// below 2^-120, 0 included, gives a root of about 2^-60.  No FP64 instruction
// but for one value in 2^19 (the library's root takes the time of 7).
__device__ __forceinline__ double root(double x) {
    const uint32_t h = (uint32_t)max((int)hi32(x), 0x38700800);   // not a power of two: 0 is common
    const double xc = from_words(h, lo32(x));
    const ds::F2 xs = split(xc);
    const float hr = __fmul_rn(0.5f, ds::rsqrt_approx(xs.h));
    const float s0 = __fmul_rn(__fadd_rn(xs.h, xs.h), hr);
    const double S = join(ds::fast_two_sum(s0, __fmul_rn(__fadd_rn(__fmaf_rn(-s0, s0, xs.h), xs.l), hr)));
    if ((int)hi32(x) >= 0x46300000 || near_binade(S)) return __dsqrt_rn(x);   // x >= 2^100, infinite or NaN
    const float u = __fmul_rn(__fmul_rn(pow2_of(S), hr), 0x1p-12f);           // 2^-64 of the remainder's unit, in ulp of S
    const int32_t k = __float2int_rn(__fmul_rn(__int2float_rn(remainder_sqr_units(xc, S)), u));
    return __longlong_as_double(__double_as_longlong(S) + (long long)k);
}

// z k within 0.51 ulp, z a float (0 gives a value below 2^-126 k) and k >= 0
// normal, |z k| within the normal range: the 24- and 53-bit significands
// multiplied in integers.
__device__ __forceinline__ double mul_float(float z, double k) {
    const uint32_t zb = __float_as_uint(z), kh = hi32(k), kl = lo32(k);
    const uint32_t zm = zb << 8 | 0x80000000u;
    uint64_t P = (uint64_t)zm * ((kh << 11 | kl >> 21) | 0x80000000u) + __umulhi(zm, kl << 11);
    const uint32_t s = ~hi(P) >> 31;
    P <<= s;
    const uint32_t e = (kh >> 20) + (zb >> 23 & 0xffu) - 127u - s;   // the exponent field less one, which the leading bit adds
    return __longlong_as_double((long long)((((uint64_t)(zb & 0x80000000u)) << 32) + ((uint64_t)e << 52) + ((P + 1024ull) >> 11)));
}

// 1 / x within 0.51 ulp, 2^-60 <= x < 2^60, like root without an FP64 instruction.
__device__ __forceinline__ double recip(double x) {
    const ds::F2 xs = split(x);
    const float r = ds::rcp_approx(xs.h);
    const ds::F2 y = ds::fast_two_sum(r, __fmul_rn(__fmaf_rn(-r, xs.l, __fmaf_rn(-r, xs.h, 1.0f)), r));
    const double Y = join(y);
    if (near_binade(Y)) return 1.0 / x;
    const float u = __fmul_rn(__fmul_rn(pow2_of(x), r), 0x1p-12f);
    const int32_t k = __float2int_rn(__fmul_rn(__int2float_rn(remainder_mul_units(1.0, x, Y)), u));
    return __longlong_as_double(__double_as_longlong(Y) + (long long)k);
}

// The same for any x > 0, and sqrt(x) for any x >= 0 (the ranges [2^-60, 2^60)
// and [2^-60, 2^100) tested on the exponent: a comparison is an FP64
// instruction too).
__device__ __forceinline__ double recip_any(double x) {
    return hi32(x) - 0x3c300000u < 0x07800000u ? recip(x) : 1.0 / x;
}
__device__ __forceinline__ double root_any(double x) {
    return hi32(x) - 0x3c300000u < 0x0a000000u ? root(x) : sqrt(x);
}

// x / y from r = 1 / y rounded (0: not given): the product corrected by its
// remainder, as exact as a division.
__device__ __forceinline__ double div_by(double x, double y, double r) {
    if (r == 0.0) return __ddiv_rn(x, y);
    const double q = __dmul_rn(x, r), c = __fma_rn(__fma_rn(-q, y, x), r, q);
    return (hi32(q) & 0x7ff00000u) == 0x7ff00000u ? q : c;   // infinite stays infinite
}

// ---------------------------------------------------------------- QE step

// m within [2^-30, 2^30), s2 within [2^-60, 2^60) and s2 / m^2 above about
// 2^-40, where the functions below are used: no double-single intermediate
// leaves the float range, and the variance is not the mean to nearly all of
// its bits (a vol-of-vol so small that rho / sigma magnifies the last bit).
__device__ __forceinline__ bool in_range(double m, double s2) {
    const uint32_t hm = hi32(m), hs = hi32(s2);
    return hm - 0x3e100000u < 0x03c00000u && hs - 0x3c300000u < 0x07800000u && (int32_t)(hs - 2u * hm + 0x42700000u) >= 0;
}

// Whether the step takes the quadratic branch, s2 < 1.5 m^2 (Psi < PSI_C,
// HSimulation.tpp:61-63), while in range: in float unless the two are within
// 2^-20.  The exact comparison is a call so that it is not computed ahead of
// the branch (three FP64 instructions in every step).
static __device__ __noinline__ bool quadratic_exact(double m, double s2) {
    return s2 < __dmul_rn(1.5, __dmul_rn(m, m));
}
__device__ __forceinline__ bool quadratic(double m, double s2) {
    const float mf = head(m), sf = head(s2);
    const float t = __fmul_rn(__fmul_rn(1.5f, mf), mf);
    bool quad = sf < t;
    if (!(fabsf(__fsub_rn(sf, t)) > __fmul_rn(0x1p-20f, sf))) quad = quadratic_exact(m, s2);
    return quad;
}
// The same outside in_range, on the mean in the reference's order of
// operations, as variance_wide takes it (where exp(-kappa dt) rounds to 1 the
// two means can differ by all of v).
static __device__ __noinline__ bool quadratic_wide(double v, double theta, double disc, double s2) {
    return quadratic_exact(__fma_rn(__dsub_rn(v, theta), disc, theta), s2);
}

// The quadratic branch a (b + z)^2 (HSimulation.tpp:64-68).  Its a and b
// satisfy a + a b^2 = m and 2 a^2 + 4 a (a b^2) = s^2, so a b^2 = c =
// sqrt(m^2 - s^2/2), a = (s^2/2) / (m + c), and
//   a (b + z)^2 = (sqrt(c) + z sqrt(a))^2:
// no difference of nearby values, and two roots, a division and a root in a
// chain instead of two divisions and two roots.  The chain runs in
// double-single; c^(1/2) and a^(1/2) are then corrected against m^2 - s^2/2
// and s^2/2 with exact remainders.  Six FP64 instructions.
__device__ __forceinline__ double variance_quadratic(double m, double s2, float z) {
    const double hs = from_words(hi32(s2) - 0x00100000u, lo32(s2));   // s^2 / 2
    const double D = __fma_rn(m, m, -hs);                             // > m^2 / 4
    const ds::F2 Df = split(D), mf = split(m), hf = split(hs);
    // c = sqrt(D), sc = sqrt(c), a = hs / (m + c), sa = sqrt(a); the last two roots normalised for join
    const float r1 = __fmul_rn(0.5f, ds::rsqrt_approx(Df.h));
    const float c0 = __fmul_rn(__fadd_rn(Df.h, Df.h), r1);
    const float cl = __fmul_rn(__fadd_rn(__fmaf_rn(-c0, c0, Df.h), Df.l), r1);
    const float r2 = __fmul_rn(0.5f, ds::rsqrt_approx(c0));
    const float sc0 = __fmul_rn(__fadd_rn(c0, c0), r2);
    const ds::F2 sc = ds::fast_two_sum(sc0, __fmul_rn(__fadd_rn(__fmaf_rn(-sc0, sc0, c0), cl), r2));
    const ds::F2 g = ds::fast_two_sum(mf.h, c0);
    const float gl = __fadd_rn(g.l, __fadd_rn(mf.l, cl)), rg = ds::rcp_approx(g.h);
    const float a0 = __fmul_rn(hf.h, rg);
    const float al = __fmul_rn(__fmaf_rn(-a0, gl, __fadd_rn(__fmaf_rn(-a0, g.h, hf.h), hf.l)), rg);
    const float r3 = __fmul_rn(0.5f, ds::rsqrt_approx(a0));
    const float sa0 = __fmul_rn(__fadd_rn(a0, a0), r3);
    const ds::F2 sa = ds::fast_two_sum(sa0, __fmul_rn(__fadd_rn(__fmaf_rn(-sa0, sa0, a0), al), r3));
    const double SC = join(sc), SA = join(sa);
    const double q = __dmul_rn(SC, SC);                               // c, to double-single accuracy
    const float dc = __fmul_rn(remainder_sqr(D, q), r1);              // c - q
    const double gd = __dadd_rn(m, q), u = __dmul_rn(SA, SA);
    const float da = __fmul_rn(__fmaf_rn(-a0, dc, remainder_mul(hs, u, gd)), rg);   // a - u
    const float cor = __fmaf_rn(z, __fmul_rn(da, r3), __fmul_rn(dc, r2));
    const double w = __fma_rn(to_double(z), SA, SC);
    const float wf = __fmaf_rn(z, sa0, sc0);
    return __fma_rn(w, w, to_double(__fmul_rn(__fadd_rn(wf, wf), cor)));
}

// The exponential branch (HSimulation.tpp:70-73) with Y = (s^2 + m^2) /
// (2 m^2) = 1 / (1 - p) = 1 / (beta m): log((1-p)/(1-U)) / beta = -m Y
// log(Y (1 - U)), positive exactly when p < U.  Y is one quotient in
// double-single, its remainder exact, and the product is taken in integers;
// two FP64 instructions instead of five divisions and a logarithm.
__device__ __forceinline__ double variance_exponential(double m, double s2, uint64_t uw) {
    const double mm = __dmul_rn(m, m), W = __fma_rn(m, m, s2);
    const double mm2 = from_words(hi32(mm) + 0x00100000u, lo32(mm));
    const ds::F2 Wf = split(W), Mf = split(mm2);
    const float rm = ds::rcp_approx(Mf.h);
    const float y0 = __fmul_rn(Wf.h, rm);
    float e = __fmaf_rn(-y0, Mf.h, Wf.h);
    e = __fmaf_rn(-y0, Mf.l, __fadd_rn(e, Wf.l));
    const ds::F2 Yf = ds::fast_two_sum(y0, __fmul_rn(e, rm));
    const uint64_t N = 0ull - uw;                                     // 1 - U = N 2^-64 (uw == 0: U = 0 < p)
    const double Y = join(Yf);
    // x = Y (1 - U) = P 2^(k-63)
    const uint64_t Ym = (uint64_t)__double_as_longlong(Y) << 11 | 0x8000000000000000ull;
    const int lz = __clzll((long long)N) & 63;
    uint64_t P = mul_hi(Ym, N << lz);
    const int s = (int)(~hi(P) >> 31), eY = (int)(hi32(Y) >> 20) - 1023;
    const int k = eY - lz - s;
    P <<= s;
    const float d = __fdividef(__fmul_rn(remainder_mul(W, Y, mm2), rm), y0);
    // m Y (-log x), its significand in 64 bits
    const uint64_t A = neg_log_fixed(P, k, d);
    const int la = __clzll((long long)A) & 63;
    uint64_t V = mul_hi((uint64_t)__double_as_longlong(m) << 11 | 0x8000000000000000ull, Ym);   // 2^61.99 or more
    V = mul_hi(V, A << la);
    const int lv = __clzll((long long)V) & 63;
    V <<= lv;
    const uint32_t ev = (hi32(m) >> 20) + (uint32_t)(eY + 8 - la - lv);   // the leading bit's exponent
    const double v = __longlong_as_double((long long)(((uint64_t)(ev - 1u) << 52) + ((V + 1024ull) >> 11)));
    return N != 0ull && k < 0 && A != 0ull ? v : 0.0;                 // k >= 0: p >= U
}

// The next variance outside in_range, in the reference's order of operations.
static __device__ __noinline__ double variance_wide(double v, double theta, double disc, double s2, bool quad, float z,
                                                    uint64_t uw) {
    const double m = __fma_rn(__dsub_rn(v, theta), disc, theta);
    const double mm = __dmul_rn(m, m);
    if (quad) {
        const double inv = __ddiv_rn(__dmul_rn(2.0, mm), s2);                // 2/Psi
        const double im1 = __dsub_rn(inv, 1.0);
        const double bp2 = __dadd_rn(im1, __dsqrt_rn(__dmul_rn(inv, im1)));
        const double zb = __dadd_rn(__dsqrt_rn(bp2), (double)z);
        return __dmul_rn(__dmul_rn(__ddiv_rn(m, __dadd_rn(1.0, bp2)), zb), zb);
    }
    const double Psi = __ddiv_rn(s2, mm);
    const double p = __ddiv_rn(__dsub_rn(Psi, 1.0), __dadd_rn(Psi, 1.0));
    const double beta = __ddiv_rn(2.0, __dmul_rn(m, __dadd_rn(Psi, 1.0)));
    const double U = __ull2double_rn(uw) * 0x1p-64;
    return p < U ? __ddiv_rn(log(__ddiv_rn(__dsub_rn(1.0, p), __dsub_rn(1.0, U))), beta) : 0.0;
}

} // namespace f64
} // namespace hexo
