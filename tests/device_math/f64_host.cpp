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
