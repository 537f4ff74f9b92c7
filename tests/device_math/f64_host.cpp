// hexo_f64.cuh on the host, held against long double (64 bits or more of
// significand on the machines the tests run on): tests/test_device_math.py.
#include "host_device.h"
#include "hexo_f64.cuh"

using namespace hexo;

namespace {

double device(int fn, double x) {
    switch (fn) {
    case 0: return f64::recip(x);
    case 1: return f64::root(x);
    default: return f64::exp_tab(x, &f64::kExpTabInit);
    }
}
long double exact(int fn, double x) {
    switch (fn) {
    case 0: return 1.0L / (long double)x;
    case 1: return std::sqrt((long double)x);
    default: return std::exp((long double)x);
    }
}

} // namespace

// The largest error over x, in units of the last place of the exact value's
// binade; *at is the argument it occurs at.
extern "C" double f64_worst_ulp(int fn, int seed_ulp, uint64_t n, const double *x, double *at) {
    mufu_ulp = seed_ulp;
    double worst = 0.0;
    for (uint64_t i = 0; i < n; ++i) {
        const long double want = exact(fn, x[i]);
        int e;
        (void)std::frexp(want, &e);
        const double err = (double)(std::fabs((long double)device(fn, x[i]) - want) / std::ldexp(1.0L, e - 53));
        if (!(err <= worst)) {
            worst = err;
            *at = x[i];
        }
    }
    return worst;
}

// One step's next variance as the path kernel takes it, held against the closed
// forms in long double: the largest error over the n steps relative to the
// size of the terms it is made of, in units of 2^-53; *at is the step's index.
// near[i] says whether the step took this file's own functions.
extern "C" double f64_worst_variance(int seed_ulp, uint64_t n, const double *m, const double *s2, const float *z,
                                     const uint64_t *uw, uint8_t *near, uint64_t *at) {
    mufu_ulp = seed_ulp;
    double worst = 0.0;
    for (uint64_t i = 0; i < n; ++i) {
        near[i] = f64::in_range(m[i], s2[i]);
        const bool quad = near[i] ? f64::quadratic(m[i], s2[i]) : f64::quadratic_wide(m[i], 0.0, 1.0, s2[i]);
        const double got = !near[i] ? f64::variance_wide(m[i], 0.0, 1.0, s2[i], quad, z[i], uw[i])
                           : quad   ? f64::variance_quadratic(m[i], s2[i], z[i])
                                    : f64::variance_exponential(m[i], s2[i], uw[i]);
        const long double M = m[i], hs = 0.5L * s2[i];
        long double want, size;
        if (quad) {   // (sqrt(c) + z sqrt(a))^2
            const long double c = std::sqrt(M * M - hs), a = hs / (M + c), w = std::sqrt(c) + z[i] * std::sqrt(a);
            want = w * w;
            size = std::sqrt(c) + std::fabs((long double)z[i]) * std::sqrt(a);
            size *= size;
        } else {      // -m Y log(Y (1 - U)), Y (1 - U) < 1
            const long double Y = 0.5L + hs / (M * M), x = Y * std::ldexp((long double)(0ull - uw[i]), -64);
            const long double l = uw[i] != 0ull && x < 1.0L ? -std::log(x) : 0.0L;
            want = M * Y * l;
            size = M * Y * (1.0L + l);
        }
        const double err = (double)(std::fabs((long double)got - want) / size * 0x1p53L);
        if (!(err <= worst)) {
            worst = err;
            *at = i;
        }
    }
    return worst;
}
