// hexo_f32.cuh on the host, held against long double: tests/test_device_math.py.
#include "host_device.h"
#include "hexo_f32.cuh"

using namespace hexo;

// The FP32 form's next variance over n steps of mean m and s^2 (quadratic branch
// where s^2 < 1.5 m^2), from m and s^2/2 as the kernel holds them, against the
// closed forms: rms error relative to the size of the terms it is made of.
extern "C" double f32_rms_variance(int seed_ulp, uint64_t n, const double *m, const double *s2, const float *z,
                                   const uint64_t *uw) {
    static ds::LogTab tab[ds::kLogTab];
    mufu_ulp = seed_ulp;
    ds::log_table_init(tab, 0, 1);
    long double sum = 0.0L;
    for (uint64_t i = 0; i < n; ++i) {
        const float mh = (float)m[i], ml = (float)(m[i] - (double)mh);
        const float hh = (float)(0.5 * s2[i]), hl = (float)(0.5 * s2[i] - (double)hh);
        const float p = mh * mh, e = std::fma(mh + mh, ml, std::fma(mh, mh, -p));
        const long double M = (long double)mh + ml, hs = (long double)hh + hl;
        long double want, size;
        ds::F2 v;
        if (hs < 0.75L * M * M) {
            v = f32::variance_quadratic(ds::F2{mh, ml}, ds::F2{hh, hl}, p, e, z[i]);
            const long double c = std::sqrt(M * M - hs), a = hs / (M + c), w = std::sqrt(c) + z[i] * std::sqrt(a);
            want = w * w;
            size = std::sqrt(c) + std::fabs((long double)z[i]) * std::sqrt(a);
            size *= size;
        } else {
            v = f32::variance_exponential(ds::F2{mh, ml}, ds::F2{hh, hl}, p, e, uw[i], tab);
            const long double Y = 0.5L + hs / (M * M), x = Y * std::ldexp((long double)(0ull - uw[i]), -64);
            const long double l = uw[i] != 0ull && x < 1.0L ? -std::log(x) : 0.0L;
            want = M * Y * l;
            size = M * Y * (1.0L + l);
        }
        const long double d = ((long double)v.h + v.l - want) / size;
        sum += d * d;
    }
    return (double)std::sqrt(sum / n);
}
