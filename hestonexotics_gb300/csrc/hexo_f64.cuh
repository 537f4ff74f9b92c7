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
// A float near a signed x, |x| < 2^128 (24 leading bits; below 2^-126: 0).
__device__ __forceinline__ float to_float(double x) {
    const uint32_t h = hi32(x), a = h & 0x7fffffffu;
    const uint32_t b = a < 0x38100000u ? 0u : (__funnelshift_l(lo32(x), a, 3) & 0x7fffffffu) ^ 0x40000000u;
    return __uint_as_float(b | (h & 0x80000000u));
}
// f as a double: exact for normal f; 0 and subnormals become values below 2^-126.
__device__ __forceinline__ double to_double(float f) {
    const uint32_t b = __float_as_uint(f);
    return from_words(((uint32_t)((int32_t)b >> 3) & 0x8fffffffu) + 0x38000000u, b << 29);
}
// x / 2 for |x| >= 2^-1000, else 0.
__device__ __forceinline__ double half(double x) {
    const uint32_t h = hi32(x);
    const bool tiny = (h & 0x7fffffffu) < 0x01700000u;
    return from_words(tiny ? 0u : h - 0x00100000u, tiny ? 0u : lo32(x));
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
// cut at 2^-64 of 2^(ea+eb).
__device__ __forceinline__ float remainder_mul(double x, double a, double b) {
    const uint32_t al = lo32(a), bl = lo32(b), ah = hi32(a), bh = hi32(b), xl = lo32(x), xh = hi32(x);
    const uint32_t am = (ah & 0x000fffffu) | 0x00100000u, bm = (bh & 0x000fffffu) | 0x00100000u;
    uint64_t p = (uint64_t)al * bm + __umulhi(al, bl);
    p += (uint64_t)bl * am;
    p += (uint64_t)(am * bm) << 32;
    const uint32_t s = 20u + 1023u + (xh >> 20) - (ah >> 20) - (bh >> 20);   // 19 to 22
    const uint64_t d = (((uint64_t)__funnelshift_l(xl, xh, s) << 32) | (uint64_t)(uint32_t)(xl << s)) - p;
    const int32_t r = (int32_t)__funnelshift_r((uint32_t)d, (uint32_t)(d >> 32), 8);
    return __fmul_rn(__fmul_rn(__fmul_rn(__int2float_rn(r), 0x1p-64f), pow2_of(a)), pow2_of(b));
}
// x - q^2
__device__ __forceinline__ float remainder_sqr(double x, double q) {
    const uint32_t ql = lo32(q), qh = hi32(q), xl = lo32(x), xh = hi32(x);
    const uint32_t qm = (qh & 0x000fffffu) | 0x00100000u;
    uint64_t p = (uint64_t)ql * (qm + qm) + __umulhi(ql, ql);
    p += (uint64_t)(qm * qm) << 32;
    const uint32_t s = 20u + 1023u + (xh >> 20) - 2u * (qh >> 20);
    const uint64_t d = (((uint64_t)__funnelshift_l(xl, xh, s) << 32) | (uint64_t)(uint32_t)(xl << s)) - p;
    const int32_t r = (int32_t)__funnelshift_r((uint32_t)d, (uint32_t)(d >> 32), 8);
    const float e = pow2_of(q);
    return __fmul_rn(__fmul_rn(__fmul_rn(__int2float_rn(r), 0x1p-64f), e), e);
}

// ------------------------------------------------------------------ tables
//
// 2^(j/256) and, for the logarithm, 512 reciprocals with their logarithms,
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

constexpr int kExpTab = 256;   // a CTA's copy in shared memory: kExpTab * 12 bytes
struct ExpTab {
    double t[kExpTab];         // 2^(j/256), rounded
    float l[kExpTab];          // what rounding left, relative to t
};
constexpr ExpTab make_exp_tab() {
    ExpTab r{};
    for (int j = 0; j < kExpTab; ++j) {
        const DD e = dd_exp(dd_mul(kLn2, DD{(double)j / kExpTab, 0.0}));
        r.t[j] = e.h;
        r.l[j] = (float)(e.l / e.h);
    }
    return r;
}
constexpr int kLogTab = 512;
struct LogEntry {
    double inv, lg;            // 1 / c_j, c_j the middle of the j-th of 512 parts of [1, 2), and -log of it
};
struct LogTab {
    LogEntry e[kLogTab];
};
constexpr LogTab make_log_tab() {
    LogTab r{};
    for (int j = 0; j < kLogTab; ++j) {
        const double inv = 1.0 / (1.0 + (j + 0.5) / kLogTab);
        const DD lg = dd_log_ratio(DD{1.0 - inv, 0.0}, dd_two_sum(1.0, inv));
        r.e[j] = LogEntry{inv, lg.h};
    }
    return r;
}
__device__ constexpr ExpTab kExpTabInit = make_exp_tab();
__device__ constexpr LogTab kLogTabDev = make_log_tab();

// A CTA's copy of the exponential's table, visible after the next barrier.
__device__ __forceinline__ void exp_table_init(ExpTab *t, uint32_t tid, uint32_t nthreads) {
    for (uint32_t j = tid; j < (uint32_t)kExpTab; j += nthreads) {
        t->t[j] = kExpTabInit.t[j];
        t->l[j] = kExpTabInit.l[j];
    }
}

// ----------------------------------------------------------- exp, log, root

// exp(x): x = n ln2/256 + r, |r| <= ln2/512, and 2^(n/256) (1 + r + r^2/2 +
// c) with c = r^3/6 + r^4/24 + r^5/120, below 2^-31, the table's own remainder and n
// times what ln2/256 lost to rounding, all in float (1/6 rounded up by what
// to_float's truncation takes from r^3 on average).  Four FP64 instructions
// (the library's exp takes the time of 18) and an error below 1 ulp.
__device__ __forceinline__ double exp_tab(double x, const ExpTab *tab) {
    if (((hi32(x) & 0x7fffffffu) >= 0x40800000u)) return exp(x);   // |x| >= 512, infinite or NaN
    constexpr double L = kLn2.h / kExpTab;
    constexpr float Ll = (float)(kLn2.l / kExpTab), invL = (float)(kExpTab / kLn2.h);
    const float t = __fmaf_rn(to_float(x), invL, 0x1.8p23f);       // rounds to an integer, |n| < 2^18
    const int n = (int)__float_as_uint(t) - 0x4b400000;
    const float nf = __fsub_rn(t, 0x1.8p23f);
    const double r = __fma_rn(-to_double(nf), L, x);
    const uint32_t j = (uint32_t)n & (uint32_t)(kExpTab - 1);
    const float rf = to_float(r);
    const float c3 = __fmul_rn(__fmul_rn(rf, rf), __fmul_rn(rf, __fmaf_rn(rf, __fmaf_rn(rf, 0x1.111112p-7f, 0x1.555556p-5f), 0x1.555558p-3f)));
    const float c = __fadd_rn(c3, __fmaf_rn(-nf, Ll, tab->l[j]));
    const double u = __dadd_rn(__fma_rn(r, half(r), r), to_double(c));
    const double T = tab->t[j];
    const double Ts = from_words(hi32(T) + ((uint32_t)(n >> 8) << 20), lo32(T));   // T 2^(n >> 8), normal
    return __fma_rn(Ts, u, Ts);
}

// log(x) (1 + d) for 2^-80 < x < 2 and a relative correction |d| < 2^-40 of
// both x and the result (log(x (1 + d)) (1 + d) to first order): x = 2^k M, M
// in [1, 2), r = M / c_j - 1, |r| <= 2^-10, log x = k ln2 + log c_j + (r -
// r^2/2) + c, c = r^3/3 - r^4/4 + r^5/5 below 2^-31 and the corrections in
// float (1/3 rounded up as 1/6 above).  Five FP64 instructions (the library's
// log takes the time of 28).
__device__ __forceinline__ double log_tab(double x, float d) {
    const uint32_t h = hi32(x);
    const int k = (int)(h >> 20) - 1023;
    const LogEntry e = kLogTabDev.e[(h >> 11) & (uint32_t)(kLogTab - 1)];
    const double r = __fma_rn(from_words((h & 0x000fffffu) | 0x3ff00000u, lo32(x)), e.inv, -1.0);
    const float kf = (float)k, rf = to_float(r);
    const float c3 = __fmul_rn(__fmul_rn(rf, rf), __fmul_rn(rf, __fmaf_rn(rf, __fmaf_rn(rf, 0.2f, -0.25f), 0x1.555558p-2f)));
    const float lf = __logf(head(x));
    const float c = __fadd_rn(c3, __fmaf_rn(d, __fadd_rn(1.0f, lf), __fmul_rn(kf, (float)kLn2.l)));
    const double u = __dadd_rn(__fma_rn(r, -half(r), r), to_double(c));
    return __dadd_rn(__fma_rn(to_double(kf), kLn2.h, e.lg), u);
}

// sqrt(x), within 0.51 ulp (x below 2^-120, 0 included, gives a root below
// 2^-59): the remainder's correction is added to the bits of the joined root
// in units of its last place.  No FP64 instruction (the library's root takes
// the time of 7).
__device__ __forceinline__ double root(double x) {
    if ((int)hi32(x) >= 0x46300000) return __dsqrt_rn(x);   // x >= 2^100, infinite or NaN
    const uint32_t h = (uint32_t)max((int)hi32(x), 0x38700000);
    const double xc = from_words(h, lo32(x));
    const ds::F2 xs = split(xc);
    const float hr = __fmul_rn(0.5f, ds::rsqrt_approx(xs.h));
    const float s0 = __fmul_rn(__fadd_rn(xs.h, xs.h), hr);
    const double S = join(ds::fast_two_sum(s0, __fmul_rn(__fadd_rn(__fmaf_rn(-s0, s0, xs.h), xs.l), hr)));
    const float unit = __uint_as_float(0x7f000000u + (52u << 23) - (__float_as_uint(s0) & 0x7f800000u));
    const int32_t k = __float2int_rn(__fmul_rn(__fmul_rn(remainder_sqr(xc, S), hr), unit));
    return __longlong_as_double(__double_as_longlong(S) + (long long)k);
}

// ---------------------------------------------------------------- QE step

// N 2^-64, N > 0, rounded to double.
__device__ __forceinline__ double u64_2m64(uint64_t N) {
    const uint32_t lz = (uint32_t)__clzll((long long)N);
    const uint64_t n = N << lz;
    const uint64_t m = (n >> 11) + ((n >> 10) & 1ull);   // a carry moves into the exponent
    return __longlong_as_double((long long)(((uint64_t)(1021u - lz) << 52) + m));
}

// m within [2^-30, 2^30), s2 within [2^-60, 2^60) and s2 / m^2 above about
// 2^-40, where the functions below are used: no double-single intermediate
// leaves the float range, and the variance is not the mean to nearly all of
// its bits (a vol-of-vol so small that rho / sigma magnifies the last bit).
__device__ __forceinline__ bool in_range(double m, double s2) {
    const uint32_t hm = hi32(m), hs = hi32(s2);
    return hm - 0x3e100000u < 0x03c00000u && hs - 0x3c300000u < 0x07800000u && (int32_t)(hs - 2u * hm + 0x42700000u) >= 0;
}

// Whether the step takes the quadratic branch, s2 < 1.5 m^2 (Psi < PSI_C,
// HSimulation.tpp:61-63): in float unless the two are within 2^-20.
__device__ __forceinline__ bool quadratic(double m, double s2) {
    const float mf = head(m), sf = head(s2);
    const float t = __fmul_rn(__fmul_rn(1.5f, mf), mf);
    if (fabsf(__fsub_rn(sf, t)) > __fmul_rn(0x1p-20f, sf)) return sf < t;
    return s2 < __dmul_rn(1.5, __dmul_rn(m, m));
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
// double-single, its remainder exact; ten FP64 instructions instead of five
// divisions and a logarithm.
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
    if (N == 0ull) return 0.0;
    const double Y = join(Yf), om = u64_2m64(N);
    const double x = __dmul_rn(Y, om);
    if (hi32(x) >= 0x3ff00000u) return 0.0;                           // p >= U
    const float d = __fdividef(__fmul_rn(remainder_mul(W, Y, mm2), rm), y0);
    return __dmul_rn(__dmul_rn(-m, Y), log_tab(x, d));
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
