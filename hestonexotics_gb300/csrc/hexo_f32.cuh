// The next variance of the FP32 form's step, in double-single arithmetic.
#pragma once
#include <stdint.h>
#include "hexo_ds.cuh"

namespace hexo {
namespace f32 {

// The two branches take m and hs = s^2/2 in double-single and m^2 = p + e.
// As in the FP64 form (hexo_f64.cuh) the quadratic branch is (sqrt(c) + z
// sqrt(a))^2 with c = sqrt(m^2 - hs) and a = hs / (m + c): 57 instructions and
// four MUFU, against 95 for a (b + z)^2 in the reference's order.  What comes
// between stays unnormalised, the square taking its low part's square along.  A
// correction's own error is the square of what it corrects, 2^-24.5 of a
// MUFU's product: c and sqrt(c), which every result is made of, are corrected
// once as floats first.  Error, rms of the result's terms, measured on the device
// against 113 bits: 2^-47.34 for small Psi, 2^-47.60 up to 1, 2^-47.49 beyond
// (without the corrections 2^-46.55, 2^-46.92 and 2^-46.90; the reference's order
// in normalised double-single steps 2^-46.68, 2^-47.11 and 2^-47.25).
__device__ __forceinline__ ds::F2 variance_quadratic(ds::F2 m, ds::F2 hs, float p, float e, float z) {
    const float D = __fsub_rn(p, hs.h);                                  // m^2 - hs > m^2 / 4
    const float Dl = __fadd_rn(__fsub_rn(__fsub_rn(p, D), hs.h), __fsub_rn(e, hs.l));
    const float r1 = ds::rsqrt_approx(D), h1 = __fmul_rn(0.5f, r1), c0 = __fmul_rn(D, r1);
    const float c = __fmaf_rn(__fadd_rn(__fmaf_rn(-c0, c0, D), Dl), h1, c0);
    const float cl = __fmul_rn(__fadd_rn(__fmaf_rn(-c, c, D), Dl), h1);
    const float r2 = ds::rsqrt_approx(c), h2 = __fmul_rn(0.5f, r2), b0 = __fmul_rn(c, r2);
    const float b = __fmaf_rn(__fmaf_rn(-b0, b0, c), h2, b0);            // sqrt(c)
    const float bl = __fmul_rn(__fadd_rn(__fmaf_rn(-b, b, c), cl), h2);
    const float g = __fadd_rn(m.h, c);                                   // m + c, m >= c
    const float gl = __fadd_rn(__fsub_rn(c, __fsub_rn(g, m.h)), __fadd_rn(m.l, cl));
    const float rg = ds::rcp_approx(g), a = __fmul_rn(hs.h, rg);
    const float al = __fmul_rn(__fmaf_rn(-a, gl, __fadd_rn(__fmaf_rn(-a, g, hs.h), hs.l)), rg);
    const float r3 = ds::rsqrt_approx(a), s = __fmul_rn(a, r3);          // sqrt(a)
    const float sl = __fmul_rn(__fadd_rn(__fmaf_rn(-s, s, a), al), __fmul_rn(0.5f, r3));
    const float q = __fmul_rn(z, s), ql = __fmaf_rn(z, sl, __fmaf_rn(z, s, -q));
    const ds::F2 w = ds::two_sum(b, q);
    const float wl = __fadd_rn(w.l, __fadd_rn(bl, ql)), v = __fmul_rn(w.h, w.h);
    return ds::fast_two_sum(v, __fmaf_rn(__fmaf_rn(2.0f, w.h, wl), wl, __fmaf_rn(w.h, w.h, -v)));
}

// -m Y log(Y (1 - U)), Y = (hs + m^2/2) / m^2, 1 - U = (2^64 - w) 2^-64 from
// the whole word, or 0 where p >= U: that is where Y (1 - U) >= 1, since Y =
// 1 / (1 - p).  The value is continuous there, so it does not matter that the
// FP64 form may round a tie the other way.  In double-single like the
// quadratic branch: a float-size error here would move later branch
// decisions.
__device__ __forceinline__ ds::F2 variance_exponential(ds::F2 m, ds::F2 hs, float p, float e, uint64_t uw,
                                                       const ds::LogTab *ltab) {
    const float W = __fmaf_rn(0.5f, p, hs.h);                            // hs >= 0.75 m^2
    const float Wl = __fadd_rn(__fmaf_rn(0.5f, p, __fsub_rn(hs.h, W)), __fmaf_rn(0.5f, e, hs.l));
    const float rp = ds::rcp_approx(p), y = __fmul_rn(W, rp);
    const float yl = __fmul_rn(__fmaf_rn(-y, e, __fadd_rn(__fmaf_rn(-y, p, W), Wl)), rp);
    const ds::F2 om = ds::from_u64_2m64(0ull - uw);
    const float x = __fmul_rn(y, om.h);
    const ds::F2 X = ds::fast_two_sum(x, __fmaf_rn(yl, om.h, __fmaf_rn(y, om.l, __fmaf_rn(y, om.h, -x))));
    ds::F2 vn{0.0f, 0.0f};
    if (uw != 0ull && (X.h < 1.0f || (X.h == 1.0f && X.l < 0.0f))) {     // U = 0 is never above p
        const float mY = __fmul_rn(m.h, y);
        const ds::F2 M{mY, __fmaf_rn(m.l, y, __fmaf_rn(m.h, yl, __fmaf_rn(m.h, y, -mY)))};
        const ds::F2 v1 = ds::mul(M, ds::neg(ds::log(X, ltab)));
        if (v1.h > 0.0f) vn = v1;
    }
    return vn;
}

} // namespace f32
} // namespace hexo
