// SWIFT European call pricer on the GPU: prices and their gradients in the
// Heston parameters, for batches of option chains.
//
// The reference prices European calls with the SWIFT method (Ortiz-Gracia &
// Oosterlee, SIAM J. Sci. Comput. 38, 2016) in src/SWIFT.cpp:18-118, using the
// characteristic function and gradient of src/HDistribution.cpp:8-113 (the
// form of Cui, del Bano Rollin & Germano, EJOR 263, 2017); its calibration
// evaluates them for every chain at every Levenberg-Marquardt step
// (src/HCalibration.cpp:35-57).  Per expiry, with J frequencies
// u_j = pi (2j+1) 2^m / (2J) and k in [k1, k2]:
//   h_j  = H(upper) - H(max(lower, 0)),  H(y) = -i e^{-i u_j y} (1/u_j - e^y/(i + u_j))
//   V_k  = Re(sum_j h_j w^{k(2j+1)}) sqrt(2^m) / J                 (SWIFT.cpp:54-68)
//   c_j  = sum_k V_k w^{k(2j+1)} sqrt(2^m) / J                      (SWIFT.cpp:69-72)
//   price_i (and gradient) = Re sum_j phi(u_j) c_j disc K_i e^{-i u_j x_i}  (SWIFT.cpp:102-118)
// with w = e^{i pi / (2J)} and x_i = r tau + log(S / K_i).  The reference
// evaluates the two transforms with FFTW; here they are FFTs in shared memory
// (fft_part), or the direct sums where the caller asks for them or J is tiny.  Everything is FP64, since the results must match the reference's
// known answers to 1e-9, and the FP64 pipe (2 lanes per cycle and SM) bounds
// every kernel.
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "hexo_mc.h"
#include "hexo_runtime.h"
#include "hexo_f64.cuh"

namespace hexo {
namespace swift {

// ---------------------------------------------------------------- complex

struct cplx {
    double re, im;
};
__host__ __device__ inline cplx C(double r, double i = 0.0) { return cplx{r, i}; }
__host__ __device__ inline cplx operator+(cplx a, cplx b) { return C(a.re + b.re, a.im + b.im); }
__host__ __device__ inline cplx operator-(cplx a, cplx b) { return C(a.re - b.re, a.im - b.im); }
__host__ __device__ inline cplx operator-(cplx a) { return C(-a.re, -a.im); }
__host__ __device__ inline cplx operator*(cplx a, cplx b) {
    return C(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
__host__ __device__ inline cplx operator*(double s, cplx a) { return C(s * a.re, s * a.im); }
__host__ __device__ inline cplx operator*(cplx a, double s) { return C(s * a.re, s * a.im); }
__host__ __device__ inline cplx operator+(cplx a, double s) { return C(a.re + s, a.im); }
__host__ __device__ inline cplx operator+(double s, cplx a) { return C(a.re + s, a.im); }
__host__ __device__ inline cplx operator-(double s, cplx a) { return C(s - a.re, -a.im); }
__host__ __device__ inline cplx operator-(cplx a, double s) { return C(a.re - s, a.im); }
// a / b by Smith's method (scaled, no overflow for the magnitudes met here)
__host__ __device__ inline cplx operator/(cplx a, cplx b) {
    if (fabs(b.re) >= fabs(b.im)) {
        const double t = b.im / b.re, d = b.re + b.im * t;
        return C((a.re + a.im * t) / d, (a.im - a.re * t) / d);
    }
    const double t = b.re / b.im, d = b.re * t + b.im;
    return C((a.re * t + a.im) / d, (a.im * t - a.re) / d);
}
__host__ __device__ inline cplx operator/(cplx a, double s) { return C(a.re / s, a.im / s); }
__host__ __device__ inline cplx operator/(double s, cplx b) { return C(s) / b; }
__host__ __device__ inline double cabs_(cplx a) { return hypot(a.re, a.im); }
__host__ __device__ inline cplx cexp_(cplx a) {
    const double e = exp(a.re);
    return C(e * cos(a.im), e * sin(a.im));
}
// principal logarithm
__host__ __device__ inline cplx clog_(cplx a) { return C(log(cabs_(a)), atan2(a.im, a.re)); }
// principal square root
__host__ __device__ inline cplx csqrt_(cplx a) {
    const double r = cabs_(a);
    if (r == 0.0) return C(0.0, a.im);
    if (a.re >= 0.0) {
        const double t = sqrt(0.5 * (r + a.re));
        return C(t, a.im / (2.0 * t));
    }
    const double t = sqrt(0.5 * (r - a.re));
    return C(fabs(a.im) / (2.0 * t), copysign(t, a.im));
}
__host__ __device__ inline cplx csinh_(cplx a) { return C(sinh(a.re) * cos(a.im), cosh(a.re) * sin(a.im)); }
__host__ __device__ inline cplx ccosh_(cplx a) { return C(cosh(a.re) * cos(a.im), sinh(a.re) * sin(a.im)); }

// ------------------------------------------------ characteristic function

struct HP {
    double v0, vm, rho, kappa, sigma;
};

// Helper quantities of one frequency (HDistribution.cpp:13-26).
struct Aux {
    cplx xi, d, A1, A2, A, B, D, sh, ch;
    double ekt;
};

__host__ __device__ inline Aux aux(const HP &p, cplx u, double tau) {
    const cplx I = C(0.0, 1.0);
    Aux a;
    a.xi = p.kappa + p.sigma * p.rho * (I * u);
    const cplx f = u * u - I * u;
    a.d = csqrt_(a.xi * a.xi + p.sigma * p.sigma * f);
    a.sh = csinh_(a.d * (tau * 0.5));
    a.ch = ccosh_(a.d * (tau * 0.5));
    a.A1 = f * a.sh;
    a.A2 = a.d / p.v0 * a.ch + a.xi / p.v0 * a.sh;
    a.A = a.A1 / a.A2;
    a.ekt = exp(p.kappa * tau * 0.5);
    a.B = a.d * a.ekt / (p.v0 * a.A2);
    a.D = clog_((2.0 * a.d) / (a.d + a.xi + (a.d - a.xi) * cexp_(-(a.d * tau)))) + (p.kappa - a.d) * (tau * 0.5);
    return a;
}

// phi(u) of the log-return without drift (HDistribution.cpp:31-37)
__host__ __device__ inline cplx chf(const HP &p, double tau, cplx u, const Aux &a) {
    const cplx I = C(0.0, 1.0);
    return cexp_((p.kappa * p.vm * p.rho * tau) * (u * I) / p.sigma - a.A + (2.0 * p.kappa * p.vm) * a.D / (p.sigma * p.sigma));
}

// phi and its partial derivatives in (v0, vm, rho, kappa, sigma), in the
// reference's order of operations (HDistribution.cpp:48-84).
__host__ __device__ inline void chf_grad_reference(const HP &p, double tau, cplx u, cplx out[6]) {
    const cplx I = C(0.0, 1.0);
    const Aux a = aux(p, u, tau);
    const cplx c = chf(p, tau, u, a);
    const cplx iu = I * u;
    const cplx d_rho = a.xi * p.sigma * iu / a.d;
    const cplx A2_rho = p.sigma * iu * (2.0 + a.xi * tau) / (2.0 * a.d * p.v0) * (a.xi * a.ch + a.d * a.sh);
    const cplx B_rho = a.ekt / p.v0 * (d_rho / a.A2 - a.d / (a.A2 * a.A2) * A2_rho);
    const cplx A1_rho = (iu * (u * u - iu) * tau * a.xi * p.sigma) / (2.0 * a.d) * a.ch;
    const cplx A_rho = A1_rho / a.A2 - a.A / a.A2 * A2_rho;
    const cplx B_kappa = -I / (p.sigma * u) * B_rho + a.B * (tau * 0.5);
    const cplx d_sigma = (p.rho / p.sigma - 1.0 / a.xi) * d_rho + p.sigma * u * u / a.d;
    const cplx A1_sigma = (u * u - iu) * (0.5 * tau) * d_sigma * a.ch;
    const cplx A2_sigma = p.rho / p.sigma * A2_rho + (2.0 + tau * a.xi) / (p.v0 * tau * a.xi * iu) * A1_rho +
                          p.sigma * tau * a.A1 / p.v0 * 0.5;
    const cplx A_sigma = A1_sigma / a.A2 - a.A / a.A2 * A2_sigma;
    const cplx t_iu_vm_s = p.vm * tau * iu / p.sigma;
    const double s2 = p.sigma * p.sigma;
    const double k2 = 2.0 * p.kappa * p.vm / s2;
    const cplx g_v0 = -a.A / p.v0;
    const cplx g_vm = 2.0 * p.kappa / s2 * a.D + p.kappa * p.rho * tau * iu / p.sigma;
    const cplx g_sigma = -A_sigma - 2.0 * k2 / p.sigma * a.D + k2 / a.d * (d_sigma - a.d / a.A2 * A2_sigma) -
                         t_iu_vm_s / p.sigma * p.rho * p.kappa;
    const cplx g_kappa = -A_rho / (p.sigma * iu) + 2.0 * p.vm / s2 * a.D + k2 / a.B * B_kappa + t_iu_vm_s * p.rho;
    const cplx g_rho = -A_rho + k2 / a.d * (d_rho - a.d / a.A2 * A2_rho) + t_iu_vm_s * p.kappa;
    out[0] = c;
    out[1] = c * g_v0;
    out[2] = c * g_vm;
    out[3] = c * g_rho;
    out[4] = c * g_kappa;
    out[5] = c * g_sigma;
}

// phi and its partial derivatives in (v0, vm, rho, kappa, sigma) at a real
// frequency u (HDistribution.cpp:48-84).  The reference's A1, A2 and B hold
// sinh and cosh of d tau / 2; here both are taken out as T = tanh(d tau / 2),
// so A2 = cosh Q / v0 with Q = d + xi T, every logarithmic derivative is a
// polynomial in f, xi, d, T and the two reciprocals 1/d and 1/Q:
//   A = v0 f T / Q, D = log(2 d / ((1 + E) Q)) + (kappa - d) tau / 2, E = e^{-d tau},
//   a2r = A2_rho / A2 = W (2 + xi tau) (xi + d T) / (2 d Q),  W = i sigma u,
//   A_rho = fv d_rho - A a2r,  fv = v0 tau f / (2 Q),  d_rho = xi W / d, and so on.
// With T = (1 - E) / (1 + E) everything stands over (1 + E) Q = 2 d - (d - xi)
// (1 - E); 1 - E comes from expm1 and half angles, d - xi from sigma^2 f / (d +
// xi) and the logarithm from log1p, so nothing cancels at low frequencies,
// where D goes to 0 and most of a price comes from.  One exp, one expm1, two
// sincos, one log1p, one atan2 and about 45 complex products: some 320 FP64
// instructions, against 1,400 with the
// two dozen complex quotients of the reference's form.  False, for that form,
// from d tau / 2 = 300 on, where sinh, cosh and the squares of A2 come near the
// end of the double range: what it gives there (phi is below e^{-300}, and
// beyond the range the result is NaN) is what it gave before.
__device__ __forceinline__ double norm(cplx a) { return a.re * a.re + a.im * a.im; }
__device__ __forceinline__ cplx conj(cplx a) { return C(a.re, -a.im); }

struct ChfConst {   // of one expiry
    double is, k2, rs;   // 1 / sigma, 2 kappa vm / sigma^2, rho / sigma
};

__device__ __forceinline__ bool chf_grad(const HP &p, const ChfConst &q, double tau, double u, cplx out[6]) {
    const double su = p.sigma * u;
    const cplx xi = C(p.kappa, su * p.rho), f = C(u * u, -u);
    // d = sqrt(xi^2 + sigma^2 f), principal
    const cplx d2 = C(xi.re * xi.re - xi.im * xi.im + su * su, 2.0 * xi.re * xi.im - p.sigma * su);
    const double r = f64::root_any(norm(d2)), t0 = f64::root_any(0.5 * (r + fabs(d2.re))), t1 = 0.5 * fabs(d2.im) * f64::recip_any(t0);
    const bool right = __double2hiint(d2.re) >= 0;
    const cplx d = C(right ? t0 : t1, copysign(right ? t1 : t0, d2.im));
    if (!(d.re * tau < 600.0) || p.v0 < 1e-12) return false;
    // E = e^{-d tau}: 1 - E and 1 + E without cancellation, from expm1 and the half angle
    double hs, hc;
    f64::sincos_tab(0.5 * (d.im * tau), &hs, &hc);
    const double em = expm1(-(d.re * tau)), a = 1.0 + em, v = 2.0 * hs * hs, sn = a * (2.0 * hs * hc);
    const cplx oE = C(a * v - em, sn), pE = C(1.0 + a * (1.0 - v), -sn);
    const cplx dp = d + xi, dm = (p.sigma * p.sigma * f64::recip_any(norm(dp))) * (f * conj(dp));   // d - xi = sigma^2 f / (d + xi)
    const cplx dE = dm * oE, zd = 2.0 * d - dE;              // (1 + E) Q
    const cplx iz = conj(zd) * f64::recip_any(norm(zd)), id = conj(d) * f64::recip_any(norm(d));
    const cplx fz = f * iz, fq = fz * pE, fT = fz * oE;      // f / Q and f T / Q
    const cplx A = p.v0 * fT, w = dE * iz;                   // 1 + w = 2 d / ((1 + E) Q)
    const cplx D = C(0.5 * (log1p(2.0 * w.re + norm(w)) - tau * dm.re), atan2(w.im, 1.0 + w.re) - 0.5 * tau * (dm.im + xi.im));
    const double vt = p.vm * tau * u * q.is;   // t = vm tau i u / sigma
    const double er = q.k2 * D.re - A.re, ei = p.kappa * p.rho * vt + q.k2 * D.im - A.im;
    double ps, pc;
    f64::sincos_tab(ei, &ps, &pc);
    const double ea = f64::exp_tab(er, &f64::kExpTabInit);
    const cplx c = C(ea * pc, ea * ps);
    const cplx W = C(0.0, su), h = C(2.0 + xi.re * tau, xi.im * tau);
    const cplx xw = xi * W, d_rho = xw * id;
    const cplx a2r = (0.5 * (W * h)) * id * ((xi * pE + d * oE) * iz);
    const cplx fv = (0.5 * tau * p.v0) * fq;
    const cplx A_rho = fv * d_rho - A * a2r;
    const cplx br = d_rho * id - a2r;                        // B_rho / B
    const cplx d_sigma = (q.rs * xw - W + su * u) * id;
    const cplx a2s = q.rs * a2r + (0.5 * p.sigma) * (fq * (h * id) + tau * fT);
    const cplx A_sigma = fv * d_sigma - A * a2s;
    const double iw = -q.is / u;                              // 1 / W = i iw
    const cplx i_br = C(-iw * br.im, iw * br.re), i_ar = C(-iw * A_rho.im, iw * A_rho.re);
    out[0] = c;
    out[1] = -(c * fT);
    out[2] = c * ((2.0 * p.kappa * q.is * q.is) * D + C(0.0, p.kappa * p.rho * tau * u * q.is));
    out[3] = c * (q.k2 * br - A_rho + C(0.0, vt * p.kappa));
    out[4] = c * (q.k2 * (i_br + 0.5 * tau) - i_ar + (2.0 * p.vm * q.is * q.is) * D + C(0.0, vt * p.rho));
    out[5] = c * (q.k2 * (d_sigma * id - a2s) - A_sigma - (2.0 * q.k2 * q.is) * D - C(0.0, vt * p.rho * p.kappa * q.is));
    return true;
}

static __device__ __noinline__ void chf_grad_far(const HP &p, double tau, double u, cplx out[6]) {
    chf_grad_reference(p, tau, C(u), out);
}

// ------------------------------------------------ dynamic wavelet parameters

// Every operation is odd or even in the sign of the frequency, so phi(-u) is
// the conjugate of phi(u) bit for bit and |phi(u) + phi(-u)| = 2 |Re phi(u)|;
// phi alone needs neither B nor the hyperbolic functions twice.
double int_error(const HP &p, double tau, unsigned m) {   // HDistribution.cpp:8-11
    const double e = std::exp2((double)m);
    const cplx u = C(e * M_PI), I = C(0.0, 1.0);
    Aux a;
    a.xi = p.kappa + p.sigma * p.rho * (I * u);
    const cplx f = u * u - I * u;
    a.d = csqrt_(a.xi * a.xi + p.sigma * p.sigma * f);
    const cplx dt = a.d * (tau * 0.5);
    const double sh = sinh(dt.re), ch = cosh(dt.re), sn = sin(dt.im), cs = cos(dt.im);
    a.sh = C(sh * cs, ch * sn);
    a.ch = C(ch * cs, sh * sn);
    a.A1 = f * a.sh;
    a.A2 = a.d / p.v0 * a.ch + a.xi / p.v0 * a.sh;
    a.A = a.A1 / a.A2;
    a.D = clog_((2.0 * a.d) / (a.d + a.xi + (a.d - a.xi) * cexp_(-(a.d * tau)))) + (p.kappa - a.d) * (tau * 0.5);
    const cplx c = chf(p, tau, u, a);
    const double s = std::isfinite(c.im) ? std::fabs(2.0 * c.re) : std::isinf(c.re) ? HUGE_VAL : std::nan("");
    return s / (4.0 * e * M_PI * M_PI * tau);
}

// Cumulants (HDistribution.cpp:86-113).  The reference binds its parameter
// struct positionally as (v, s2, r, kappa, k) = (v0, vm, rho, kappa, sigma),
// so in these formulas "s2" is vm and "r" is rho.
double cum1(const HP &p, double tau) { return -0.5 * p.vm * tau; }
double cum2(const HP &p, double t) {
    const double s2 = p.vm, r = p.rho, kap = p.kappa, k = p.sigma;
    const double kap2 = kap * kap, kap3 = kap2 * kap, k2 = k * k;
    return s2 / (8 * kap3) *
           (-k2 * std::exp(-2 * kap * t) + 4 * k * std::exp(-kap * t) * (k - 2 * kap * r) +
            2 * kap * t * (4 * kap2 + k2 - 4 * kap * k * r) + k * (8 * kap * r - 3 * k));
}
double cum4(const HP &p, double t) {
    const double s2 = p.vm, r = p.rho, a = p.kappa, k = p.sigma;
    const double a2 = a * a, a3 = a2 * a, a4 = a3 * a, k2 = k * k, k3 = k2 * k, k4 = k3 * k;
    const double t2 = t * t, r2 = r * r, km = k - 2 * a * r;
    return (3 * k2 * s2) / (64 * std::pow(a, 7)) *
           (-3 * k4 * std::exp(-4 * a * t)
            - 8 * k2 * std::exp(-3 * a * t) * (2 * a * k * t * km + 4 * a2 + k2 - 6 * a * k * r)
            - 4 * std::exp(-2 * a * t) *
                  (4 * a2 * k2 * t2 * km * km +
                   2 * a * k * t * (k3 - 16 * a3 * r - 12 * a * k2 * r + 4 * a2 * k * (3 + 4 * r2)) + 8 * a4 -
                   3 * k4 - 32 * a3 * k * r + 8 * a * k3 * r + 16 * a2 * k2 * r2)
            - 8 * std::exp(-a * t) *
                  (-2 * a2 * k * t2 * km * km * km -
                   8 * a * t * (k4 - 7 * a * k3 * r + 4 * a4 * r2 - 8 * a3 * k * r * (1 + r2) + a2 * k2 * (3 + 14 * r2)) -
                   9 * k4 + 70 * a * k3 * r + 32 * a3 * k * r * (4 + 3 * r2) - 16 * a4 * (1 + 4 * r2) -
                   4 * a2 * k2 * (9 + 40 * r2))
            + 4 * a * t *
                  (5 * k4 - 40 * a * k3 * r - 32 * a3 * k * r * (3 + 2 * r2) + 16 * a4 * (1 + 4 * r2) +
                   24 * a2 * k2 * (1 + 4 * r2))
            - 73 * k4 + 544 * a * k3 * r + 128 * a3 * k * r * (7 + 6 * r2) - 32 * a4 * (3 + 16 * r2) -
            64 * a2 * k2 * (4 + 19 * r2));
}

// ------------------------------------------------------------------ kernels

constexpr uint32_t kMaxJ = 1u << 16;
constexpr int kLogParts = 3, kLogMaxPart = 13;   // parts of an FFT, and the points of one (128 KB) at most

struct Exp {                 // one expiry of one request
    HP p;
    ChfConst q;
    double tau, r, S, sqrt2m, lower, upper, du;   // du = pi 2^m / (2J): u_j = (2j + 1) du
    int32_t k1, k2;
    uint32_t J, n_opt;
    uint64_t tw_off, h_off, v_off, w_off, o_off;  // element offsets into the work buffers
    uint32_t logN, logR;     // N = 2J in R parts (the transforms by FFT), or logN = 0: direct sums
    uint64_t y_off;          // its N results of a transform's parts
    uint32_t stiff, logL;    // see kStiff; folded segments of 2^logL frequencies (price_kernel), or 0
};

// Expiries with fewer frequencies than this use the direct sums (automatic
// method).
constexpr uint32_t kFftMinJ = 16, kFftMinStiffJ = 1024;

// An expiry whose range of log prices ends above this is stiff: its payoff
// terms grow as e^upper and cancel to a price of order K, so the last bits of
// every factor reach the result e^upper times larger.  A change of rounding there
// moves prices by 3e-10 to 1e-7 relative at upper = 17 and 2e-5 to 4e-5 at 25 (long
// maturities, high vol-of-vol; both forms measured against each other), from
// 10 up to the line by 4e-10 at most (300 expiries), where the other form is also
// nearer to the exact result (0.55 times the error).  Stiff expiries keep the
// reference's order of operations throughout, so that their results do not
// move: its characteristic function, a sincos for every phase, and the direct
// sums below kFftMinStiffJ frequencies.
constexpr double kStiff = 12.0;

struct Item {                // a block's piece of one expiry: outputs from first on, or an FFT part
    uint32_t e, first;
};

struct TwiddleAt {
    uint64_t off[17];        // element offset of the table of J = 2^i frequencies
};

// What an option needs of its strike: x, disc K, and its phase's turn over 32 frequencies.
struct Opt {
    double x, f, ts, tc;
};

// A call's kernels follow one another within microseconds, so each may be
// launched while the one before runs (Launches) and waits here, before it
// touches memory, until that one has ended and its results are visible; every
// kernel waits, so the ones before that have ended too.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The tables of a call in one launch, n_tw + n_h + n_o blocks of 128 threads:
// w^n = e^{i pi n / (2J)} for n < 4J, one table per distinct J (items: log2 J,
// first n); the payoff terms h_j, one thread per j; and the options' terms,
// one thread per option (a warp each in price_kernel would spend as many FP64
// instructions on them as on a third of its sum).
__global__ void __launch_bounds__(128) setup_kernel(const Exp *ex, const Item *items, uint32_t n_tw, uint32_t n_h,
                                                    const TwiddleAt at, const double *strikes, double2 *tw, double2 *h,
                                                    Opt *opts) {
    after_previous();
    const Item it = items[blockIdx.x];
    const uint32_t n = it.first + threadIdx.x;
    if (blockIdx.x < n_tw) {
        const uint32_t J = 1u << it.e;
        if (n >= 4 * J) return;
        double s, c;
        sincospi((double)n / (double)(2 * J), &s, &c);
        tw[at.off[it.e] + n] = make_double2(c, s);
        return;
    }
    const Exp &E = ex[it.e];
    if (blockIdx.x < n_tw + n_h) {
        if (n >= E.J) return;
        const double u = (2.0 * n + 1.0) * E.du;
        auto H = [&](double y, double ey) {     // -i e^{-i u y} (1/u - ey/(i + u))
            double sy, cy;
            sincos(u * y, &sy, &cy);
            const double q = 1.0 + u * u;
            const double A = 1.0 / u - ey * u / q, B = ey / q;
            return C(cy * B - sy * A, -(cy * A + sy * B));
        };
        const double lo = fmax(E.lower, 0.0);
        cplx v;
        if (E.stiff) {
            v = H(E.upper, exp(E.upper)) - H(lo, exp(lo));
        } else {   // by table, with 1/u and 1/q taken once: 0.27 -> 0.12 ms for 2,048 chains' 0.97 M terms, 8.2 -> 6.5 us for eight
            const double iu = f64::recip_any(u), iq = f64::recip_any(1.0 + u * u);
            double s1, c1, s0, c0;
            f64::sincos_tab(u * E.upper, &s1, &c1);
            f64::sincos_tab(u * lo, &s0, &c0);
            const double B1 = f64::exp_tab(E.upper, &f64::kExpTabInit) * iq, B0 = f64::exp_tab(lo, &f64::kExpTabInit) * iq;
            const double A1 = iu - B1 * u, A0 = iu - B0 * u;
            v = C(c1 * B1 - s1 * A1, -(c1 * A1 + s1 * B1)) - C(c0 * B0 - s0 * A0, -(c0 * A0 + s0 * B0));
        }
        h[E.h_off + n] = make_double2(v.re, v.im);
        return;
    }
    if (n >= E.n_opt) return;
    const double K = strikes[E.o_off + n];
    Opt o;
    o.x = E.r * E.tau + log(E.S / K);
    o.f = exp(-E.r * E.tau) * K;
    if (!E.stiff && E.logL == 0u) sincos(64.0 * E.du * o.x, &o.ts, &o.tc);
    opts[E.o_off + n] = o;
}

// ------------------------------------------------------------- transforms
//
// Both transforms are inverse DFTs of length N = 2J: with w = e^{i pi/(2J)},
// w^{k(2j+1)} = w^k e^{2 pi i k j / N}, so
//   V_k = Re(w^k F[k mod N]) sqrt(2^m)/J,  F = IDFT_N(h_0 .. h_{J-1}, 0 .. 0),
//   c_j = w^{2 k1 j} G[j] sqrt(2^m)/J,     G = IDFT_N(g folded mod N),
//         g_m = V_{k1+m} w^{k1+m},  m in [0, k2 - k1].
// The IDFT is the radix-2 decimation in time of Cooley and Tukey (1965), in R
// parts: part r runs the n = N / R points r, r + R, ... through log2 n passes
// in shared memory (fft_terms_kernel for F, fft_payoff_kernel for G, a block
// each), and the log2 R passes that join the parts run in the registers of
// whoever reads them: all R outputs q, q + n, ... of a point when the next
// transform loads its part (they are one residue mod R, the part's own input),
// one output in density_kernel.  The parts spread an expiry over R SMs, since
// the FP64 pipe is 2 lanes per cycle and SM; 16 J log2 N FP64 instructions
// take the place of the direct sums' 4 J (k2 - k1), and two launches that of
// two per pass.
__device__ __forceinline__ double2 cmul(double2 a, double2 w) {
    return make_double2(fma(a.x, w.x, -(a.y * w.y)), fma(a.x, w.y, a.y * w.x));
}

// A part's passes over n = 2^ln points, in bit-reversed order on entry.
__device__ __forceinline__ void fft_part(double2 *s, uint32_t ln, const double2 *T, uint32_t J) {
    for (uint32_t p = 0; p < ln; ++p) {
        __syncthreads();
        const uint32_t Ns = 1u << p;
        for (uint32_t b = threadIdx.x; b < (1u << ln) / 2; b += blockDim.x) {
            const uint32_t k = b & (Ns - 1u), i = ((b - k) << 1) + k;
            const double2 x = s[i], z = cmul(s[i + Ns], T[k * ((2u * J) >> p)]);   // e^{i pi k / Ns}
            s[i] = make_double2(x.x + z.x, x.y + z.y);
            s[i + Ns] = make_double2(x.x - z.x, x.y - z.y);
        }
    }
    __syncthreads();
}
__device__ __forceinline__ uint32_t bit_reverse(uint32_t i, uint32_t ln) { return ln ? __brev(i) >> (32u - ln) : 0u; }

// y_r of F's part r: the points h_{r + R l}.
__global__ void __launch_bounds__(128) fft_terms_kernel(const Exp *ex, const Item *items, const double2 *tw,
                                                        const double2 *h, double2 *y) {
    extern __shared__ double2 s[];
    after_previous();
    const Exp &E = ex[items[blockIdx.x].e];
    const uint32_t r = items[blockIdx.x].first, J = E.J, ln = E.logN - E.logR, n = 1u << ln;
    for (uint32_t l = threadIdx.x; l < n; l += blockDim.x) {
        const uint32_t j = (l << E.logR) + r;
        s[bit_reverse(l, ln)] = j < J ? h[E.h_off + j] : make_double2(0.0, 0.0);
    }
    fft_part(s, ln, tw + E.tw_off, J);
    for (uint32_t l = threadIdx.x; l < n; l += blockDim.x) y[E.y_off + r * n + l] = s[l];
}

// F[q + c n], c < R, from the parts' y[q].
template <int LR>
__device__ __forceinline__ void fft_join(const double2 *y, uint32_t q, uint32_t ln, const double2 *T, uint32_t J,
                                         double2 (&v)[1 << LR]) {
    constexpr int R = 1 << LR;
    const uint32_t n = 1u << ln;
#pragma unroll
    for (int b = 0; b < R; ++b) v[b] = y[(uint32_t)b * n + q];
#pragma unroll
    for (int p = 0; p < LR; ++p) {   // v[b 2^p + c]: part b of R / 2^p at q + c n
        double2 t[R];
        const int w = 1 << p, half = R >> (p + 1);
#pragma unroll
        for (int b = 0; b < half; ++b)
#pragma unroll
            for (int c = 0; c < w; ++c) {
                const double2 x = v[b * w + c];
                const double2 z = cmul(v[(b + half) * w + c], T[(q + (uint32_t)c * n) * ((2u * J) >> (ln + (uint32_t)p))]);
                t[b * 2 * w + c] = make_double2(x.x + z.x, x.y + z.y);
                t[b * 2 * w + c + w] = make_double2(x.x - z.x, x.y - z.y);
            }
#pragma unroll
        for (int b = 0; b < R; ++b) v[b] = t[b];
    }
}

// z_r of G's part r: the points g_m, m = r + R l, from F at k1 + m (mod N).
template <int LR>
__device__ __forceinline__ void load_payoffs(const Exp &E, uint32_t r, double2 *s, const double2 *T, const double2 *y) {
    constexpr uint32_t R = 1u << LR;
    const uint32_t J = E.J, ln = E.logN - (uint32_t)LR, n = 1u << ln, N = 2 * J, mask = 4 * J - 1;
    const uint32_t K = (uint32_t)(E.k2 - E.k1) + 1u;
    for (uint32_t q = ((r + (uint32_t)E.k1) & (R - 1u)) + (threadIdx.x << LR); q < n; q += blockDim.x << LR) {
        double2 f[1 << LR];
        fft_join<LR>(y, q, ln, T, J, f);
#pragma unroll
        for (uint32_t c = 0; c < R; ++c) {
            const uint32_t m = (q + c * n - (uint32_t)E.k1) & (N - 1u);
            double re = 0.0, im = 0.0;
            if (m < K) {
                const double2 t = T[((uint32_t)E.k1 + m) & mask];
                const double v = fma(f[c].x, t.x, -f[c].y * t.y) * E.sqrt2m / (double)J;
                re = fma(v, t.x, re);
                im = fma(v, t.y, im);
                if (m + N < K) {   // V_{k+N} = -V_k and w^{k+N} = -w^k: the same term again
                    re = fma(v, t.x, re);
                    im = fma(v, t.y, im);
                }
            }
            s[bit_reverse(m >> LR, ln)] = make_double2(re, im);
        }
    }
}
__global__ void __launch_bounds__(128) fft_payoff_kernel(const Exp *ex, const Item *items, const double2 *tw,
                                                         const double2 *y, double2 *z) {
    extern __shared__ double2 s[];
    after_previous();
    const Exp &E = ex[items[blockIdx.x].e];
    const uint32_t r = items[blockIdx.x].first, ln = E.logN - E.logR, n = 1u << ln;
    const double2 *T = tw + E.tw_off, *Y = y + E.y_off;
    if (E.logR == kLogParts) load_payoffs<kLogParts>(E, r, s, T, Y);
    else if (E.logR == kLogParts + 1) load_payoffs<kLogParts + 1>(E, r, s, T, Y);
    else load_payoffs<0>(E, r, s, T, Y);
    fft_part(s, ln, T, E.J);
    for (uint32_t l = threadIdx.x; l < n; l += blockDim.x) z[E.y_off + r * n + l] = s[l];
}

// G[j] from its parts.
template <int LR>
__device__ __forceinline__ double2 fft_output(const double2 *z, uint32_t j, uint32_t ln, const double2 *T, uint32_t J) {
    constexpr int R = 1 << LR;
    double2 v[R];
#pragma unroll
    for (int b = 0; b < R; ++b) v[b] = z[((uint32_t)b << ln) + (j & ((1u << ln) - 1u))];
#pragma unroll
    for (int p = 0; p < LR; ++p) {
        const uint32_t Ns = 1u << (ln + (uint32_t)p);
        const double2 w = T[(j & (Ns - 1u)) * ((2u * J) >> (ln + (uint32_t)p))];
        const bool up = (j & Ns) != 0u;
#pragma unroll
        for (int b = 0; b < (R >> (p + 1)); ++b) {
            const double2 x = v[b], t = cmul(v[b + (R >> (p + 1))], w);
            v[b] = up ? make_double2(x.x - t.x, x.y - t.y) : make_double2(x.x + t.x, x.y + t.y);
        }
    }
    return v[0];
}

// V_k by the direct sum, one lane per k
__global__ void payoff_kernel(const Exp *ex, const Item *items, const double2 *tw, const double2 *h, double *V) {
    after_previous();
    const Exp &E = ex[items[blockIdx.x].e];
    const int32_t k = E.k1 + (int32_t)(items[blockIdx.x].first + threadIdx.x);
    if (k > E.k2) return;
    const uint32_t mask = 4 * E.J - 1;
    const double2 *T = tw + E.tw_off;
    const double2 *Hh = h + E.h_off;
    double acc = 0.0;
    uint32_t idx = (uint32_t)k & mask, step = ((uint32_t)(2 * k)) & mask;   // k (2j + 1) mod 4J
    for (uint32_t j = 0; j < E.J; ++j) {
        const double2 a = Hh[j], t = T[idx];
        acc = fma(a.x, t.x, fma(-a.y, t.y, acc));
        idx = (idx + step) & mask;
    }
    V[E.v_off + (uint32_t)(k - E.k1)] = acc * E.sqrt2m / (double)E.J;
}

// c_j and phi(u_j) c_j with its gradient, one lane per j; a kernel of its own
// for stiff expiries (kStiffForm), so that the reference's expressions are
// compiled by themselves and round as they always did.
template <bool kStiffForm>
__global__ void __launch_bounds__(64) density_kernel(const Exp *ex, const Item *items, const double2 *tw,
                                                     const double *V, double2 *W, const double2 *z) {
    if constexpr (!kStiffForm) after_previous();   // the stiff form is launched the ordinary way
    const Exp E = ex[items[blockIdx.x].e];   // a copy: the stiff form's contractions depend on it
    const uint32_t j = items[blockIdx.x].first + threadIdx.x;
    if (j >= E.J) return;
    const uint32_t mask = 4 * E.J - 1;
    const double2 *T = tw + E.tw_off;
    const uint32_t odd = 2 * j + 1;
    double re = 0.0, im = 0.0;
    if (E.logN) {   // w^{2 k1 j} G[j]
        const double2 *Z = z + E.y_off;
        const uint32_t ln = E.logN - E.logR;
        const double2 g = E.logR == kLogParts ? fft_output<kLogParts>(Z, j, ln, T, E.J)
                          : E.logR == kLogParts + 1 ? fft_output<kLogParts + 1>(Z, j, ln, T, E.J)
                                                    : fft_output<0>(Z, j, ln, T, E.J);
        const double2 t = T[((uint32_t)E.k1 * 2u * j) & mask];
        re = fma(g.x, t.x, -g.y * t.y);
        im = fma(g.x, t.y, g.y * t.x);
    } else {
        const double *Vk = V + E.v_off;
        uint32_t idx = ((uint32_t)E.k1 * odd) & mask;
        for (int32_t k = E.k1; k <= E.k2; ++k) {
            const double v = Vk[k - E.k1];
            const double2 t = T[idx];
            re = fma(v, t.x, re);
            im = fma(v, t.y, im);
            idx = (idx + odd) & mask;
        }
    }
    const double sc = E.sqrt2m / (double)E.J;
    const cplx c = C(re * sc, im * sc);
    cplx g[6];
    if constexpr (kStiffForm) chf_grad_reference(E.p, E.tau, C((double)odd * E.du), g);
    else if (!chf_grad(E.p, E.q, E.tau, (double)odd * E.du, g)) chf_grad_far(E.p, E.tau, (double)odd * E.du, g);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const cplx w = g[q] * c;
        double2 *Wq = W + E.w_off + (uint64_t)q * E.J;
        if constexpr (!kStiffForm)
            if (E.logL) {   // full warps: J is a multiple of the block
                const uint32_t L = 1u << E.logL, at = j & (L - 1u), seg = j >> E.logL;
                const bool up = at >= L / 2;
                const double a = up ? w.re : w.im, b = up ? w.im : w.re;
                Wq[((((seg >> 5) << E.logL) + at) << 5) + (seg & 31u)] =
                    make_double2(a + __shfl_xor_sync(0xffffffffu, b, L - 1u),    // the partner's b is of a's part
                                 b - __shfl_xor_sync(0xffffffffu, a, L - 1u));
                continue;
            }
        Wq[j] = make_double2(w.re, w.im);
    }
}

// One warp per option: Re sum_j W_q(j) disc K e^{-i u_j x}, FP64-pipe bound.
//
// From kFoldMinJ frequencies a lane takes segments of L = 2^logL <= 32
// consecutive ones and folds each about its centre: the frequencies of a pair
// are u_c -+ b_k, b_k = (2k + 1) du, so with (x, y) the parts of W and -, + for
// the lower and the upper one, the pair's two terms are
//   cos(u_c x) [(x+ + x-) cos b_k x + (y+ - y-) sin b_k x]
// + sin(u_c x) [(y+ + y-) cos b_k x - (x+ - x-) sin b_k x].
// density_kernel stores the four sums and differences; the b_k are the same
// for all segments, a sincos in each of L/2 lanes; and what is left is the
// products themselves, 24 FP64 instructions a pair with the gradient (4
// without) and a sincos and 12 (2) a segment: 1.70 -> 1.46 ms on 2,048 chains of
// 50 strikes at J = 64 to 4096, 16.2 -> 13.3 us on a calibration's
// eight.  At J = 256 (segments of 8) both forms count 140 instructions a lane,
// and the fold's longer chain made the calibration's 19.8 us.
// Fewer frequencies, where those do not pay: a lane's terms are 32 j apart, so its
// phase turns by e^{-i 64 du x} from one to the next, one complex product
// instead of a sincos (4 FP64 instructions instead of a sincos's 45, or 15 by
// table), 32 a pair with the gradient, and a sincos every 16 terms, so that
// the products' roundings do not add up beyond the sincos argument's own.
// kGrad: the gradient too.
constexpr uint32_t kTurns = 16;
constexpr uint32_t kFoldMinJ = 512, kLogFold = 5;
template <bool kGrad>
__global__ void __launch_bounds__(128) price_kernel(const Exp *ex, const Item *items, const double2 *W,
                                                    const Opt *opts, double *price, double *grad) {
    __shared__ double2 turns[4][1u << (kLogFold - 1)];   // a warp's (cos, sin) b_k x
    after_previous();
    const Exp &E = ex[items[blockIdx.x].e];
    const uint32_t i = items[blockIdx.x].first + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (i >= E.n_opt) return;   // warp-uniform
    const Opt o = opts[E.o_off + i];
    constexpr int kQ = kGrad ? 6 : 1;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    if (E.logL) {
        const uint32_t half = 1u << (E.logL - 1u);
        double2 *b = turns[threadIdx.x >> 5];
        if (lane < half) {
            double s, c;
            f64::sincos_tab((2.0 * lane + 1.0) * E.du * o.x, &s, &c);
            b[lane] = make_double2(c, s);
        }
        __syncwarp();
        for (uint32_t seg = lane; (seg << E.logL) < E.J; seg += 32u) {
            const double2 *Ws = W + E.w_off + (((uint64_t)(seg >> 5) << E.logL) << 5) + lane;
            double s, c, P[kQ], Q[kQ];
            f64::sincos_tab(((double)seg * 2.0 + 1.0) * (double)(half << 1) * E.du * o.x, &s, &c);
#pragma unroll
            for (int q = 0; q < kQ; ++q) P[q] = Q[q] = 0.0;
#pragma unroll 2
            for (uint32_t k = 0; k < half; ++k) {
                const double2 t = b[k];
#pragma unroll
                for (int q = 0; q < kQ; ++q) {
                    const double2 w = Ws[(uint64_t)q * E.J + ((half + k) << 5)];
                    const double2 m = Ws[(uint64_t)q * E.J + ((half - 1u - k) << 5)];
                    P[q] = fma(w.x, t.x, fma(w.y, t.y, P[q]));
                    Q[q] = fma(m.x, t.x, fma(m.y, t.y, Q[q]));
                }
            }
#pragma unroll
            for (int q = 0; q < kQ; ++q) acc[q] = fma(c, P[q], fma(s, Q[q], acc[q]));
        }
    } else {
        const uint32_t span = 32u * (E.stiff ? 1u : kTurns);
        for (uint32_t j0 = lane; j0 < E.J; j0 += span) {
            double s, c;     // e^{-i u x} = c - i s
            if (E.stiff) sincos((2.0 * j0 + 1.0) * E.du * o.x, &s, &c);
            else f64::sincos_tab((2.0 * j0 + 1.0) * E.du * o.x, &s, &c);
            const uint32_t j1 = min(E.J, j0 + span);
            for (uint32_t j = j0; j < j1; j += 32) {
#pragma unroll
                for (int q = 0; q < kQ; ++q) {
                    const double2 w = W[E.w_off + (uint64_t)q * E.J + j];
                    acc[q] = fma(w.x, c, fma(w.y, s, acc[q]));
                }
                const double c1 = fma(c, o.tc, -s * o.ts);
                s = fma(c, o.ts, s * o.tc);
                c = c1;
            }
        }
    }
    if constexpr (kGrad) {   // lanes 0-15 take on the first three sums, 16-31 the others
        const bool up = lane >= 16u;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double mine = up ? acc[q + 3] : acc[q], theirs = up ? acc[q] : acc[q + 3];
            acc[q] = mine + __shfl_xor_sync(0xffffffffu, theirs, 16);
        }
    } else {
        acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 16);
    }
#pragma unroll
    for (int q = 0; q < (kGrad ? 3 : 1); ++q)
        for (int d = 8; d > 0; d >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], d);
    if ((lane & 15u) == 0u) {
        const double f = o.f;
        if (lane == 0u) price[E.o_off + i] = f * acc[0];
        if constexpr (kGrad) {
            double *g = grad + (E.o_off + i) * 5;
            if (lane == 0u) { g[0] = f * acc[1]; g[1] = f * acc[2]; }
            else { g[2] = f * acc[0]; g[3] = f * acc[1]; g[4] = f * acc[2]; }
        }
    }
}

} // namespace swift
} // namespace hexo

using namespace hexo;
using namespace hexo::swift;

namespace {

// A call's launches.  A kernel may begin while the one before it still runs
// (it starts with after_previous()), where the blocks of both find an SM each:
// a calibration's eight expiries 275 -> 260 us a step, one chain of 50 strikes
// at J = 512 134 -> 108 us.  Larger grids are launched when the one before has
// ended: early blocks share the SMs that it left free and run unevenly (one
// chain of 2,000 strikes at J = 16,384 0.50 -> 0.73 ms).
struct Launches {
    cudaStream_t st;
    uint64_t sm_count;
    uint64_t last;   // blocks of the kernel before
    template <class... P, class... A>
    void run(size_t grid, unsigned block, size_t smem, void (*k)(P...), A... a) {   // errors: cudaGetLastError
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t c{};
        c.gridDim = dim3((unsigned)grid);
        c.blockDim = dim3(block);
        c.dynamicSmemBytes = smem;
        c.stream = st;
        c.attrs = &at;
        c.numAttrs = last + grid <= sm_count ? 1u : 0u;
        last = grid;
        cudaLaunchKernelEx(&c, k, static_cast<P>(a)...);
    }
};

hexo_status params_dynamic(const HP &p, double tau, double r, double S, double K_min, double K_max, double prec,
                           hexo_swift_params &out) {
    unsigned m = 0;
    while (int_error(p, tau, m++) > prec)
        if (m > 30) return HEXO_ERR_NUMERIC;
    const double mx = r * tau + std::log(S / K_min), mn = r * tau + std::log(S / K_max);
    const double c = std::fabs(cum1(p, tau)) + 10.0 * std::sqrt(std::fabs(cum2(p, tau)) + std::sqrt(std::fabs(cum4(p, tau))));
    out.m = m;
    out.exp2_m = (uint32_t)std::exp2((double)m);
    out.sqrt_exp2_m = std::sqrt((double)out.exp2_m);
    out.lower = mn - c;
    out.upper = mx + c;
    out.k1 = (int32_t)std::ceil(out.exp2_m * out.lower);
    out.k2 = (int32_t)std::floor(out.exp2_m * out.upper);
    const double iota = std::ceil(std::log2(M_PI * std::abs(out.k1 - out.k2))) - 1;
    out.J = (uint32_t)std::exp2(iota - 1);
    return HEXO_OK;
}

// A chain to price, and its wavelet parameters.
struct Pending {
    const hexo_swift_chain *ch;
    HP p;
    double r, S, kmin, kmax;
    hexo_swift_params sp;
    hexo_status status;
};

// Chooses the wavelet parameters of chains [lo, hi) that do not bring their own.
void choose_params(Pending *q, size_t lo, size_t hi) {
    for (size_t i = lo; i < hi; ++i) {
        Pending &c = q[i];
        c.status = HEXO_OK;
        if (c.ch->params) c.sp = *c.ch->params;
        else
            c.status = params_dynamic(c.p, c.ch->tau, c.r, c.S, c.kmin, c.kmax,
                                      c.ch->trunc_precision > 0.0 ? c.ch->trunc_precision : 1e-7, c.sp);
    }
}

// The same over several threads, from 128 chains a thread on: the truncation
// loop takes 1 to 2 us a chain, and starting a thread about 20 us (a surface
// of 2,048 chains: 2.4 ms on one thread, as long as its kernels).
void choose_params_all(std::vector<Pending> &q) {
    const size_t n = q.size(), most = std::min<size_t>({8u, std::max(1u, std::thread::hardware_concurrency()), n / 128u + 1u});
    std::vector<std::thread> ts;
    size_t lo = 0;
    try {
        for (size_t t = 1; t < most; ++t) {
            const size_t hi = n * t / most;
            ts.emplace_back(choose_params, q.data(), lo, hi);
            lo = hi;
        }
    } catch (...) {   // no thread to be had: the rest runs here
    }
    choose_params(q.data(), lo, n);
    for (std::thread &t : ts) t.join();
}

bool valid_params(const hexo_swift_params &sp) {
    const uint32_t J = sp.J;
    return J >= 1 && J <= kMaxJ && (J & (J - 1)) == 0 && sp.k1 <= sp.k2 &&
           (int64_t)sp.k2 - (int64_t)sp.k1 + 1 <= 4 * (int64_t)J && sp.exp2_m >= 1 && std::isfinite(sp.lower) &&
           std::isfinite(sp.upper) && sp.sqrt_exp2_m > 0.0;
}

} // namespace

extern "C" {

hexo_status hexo_swift_params_dynamic(const hexo_params *p, double tau, double S, double K_min, double K_max,
                                      double trunc_precision, hexo_swift_params *out) {
    if (!p || !out || !(tau > 0.0) || !(S > 0.0) || !(K_min > 0.0) || !(K_max >= K_min) || !(trunc_precision > 0.0))
        return HEXO_ERR_INVALID;
    const HP hp{p->v0, p->theta, p->rho, p->kappa, p->sigma};
    if (!(hp.v0 > 0.0) || !(hp.sigma > 0.0) || !(hp.kappa > 0.0)) return HEXO_ERR_INVALID;
    return params_dynamic(hp, tau, p->r, S, K_min, K_max, trunc_precision, *out);
}

hexo_status hexo_swift_price(hexo_ctx *ctx, const hexo_swift_request *reqs, uint32_t n_reqs) {
    if (!ctx || !reqs || n_reqs == 0) return HEXO_ERR_INVALID;
    std::vector<Exp> ex;
    std::vector<double> strikes;
    std::vector<const hexo_swift_chain *> chain_of;
    uint64_t tw = 0, h = 0, v = 0, w = 0, f = 0;
    uint32_t max_part = 0;
    bool any_grad = false;
    std::vector<Item> it_set, it_h, it_o, it_fft, it_pay, it_den, it_stiff, it_pri;
    TwiddleAt tw_at;                        // ~0: no table yet
    std::fill(tw_at.off, tw_at.off + 17, ~0ull);
    // the chains up to the first that is refused, whose error is returned after theirs
    std::vector<Pending> todo;
    std::string refused;
    for (uint32_t q = 0; q < n_reqs && refused.empty(); ++q) {
        const hexo_swift_request &rq = reqs[q];
        const HP hp{rq.params.v0, rq.params.theta, rq.params.rho, rq.params.kappa, rq.params.sigma};
        if (!(hp.v0 > 0.0) || !(hp.sigma > 0.0) || !(hp.kappa > 0.0) || !(rq.S > 0.0) ||
            !std::isfinite(rq.params.r) || (rq.n_chains > 0 && !rq.chains)) {
            refused = "swift request " + std::to_string(q) + ": bad parameters";
            break;
        }
        for (uint32_t c = 0; c < rq.n_chains && refused.empty(); ++c) {
            const hexo_swift_chain &ch = rq.chains[c];
            if (ch.n == 0) continue;
            if (!ch.strikes || !ch.price_out || !(ch.tau > 0.0)) {
                refused = "swift chain: missing strikes/outputs or tau <= 0";
                break;
            }
            Pending p{&ch, hp, rq.params.r, rq.S, ch.strikes[0], ch.strikes[0], {}, HEXO_OK};
            for (uint32_t i = 0; i < ch.n; ++i) {
                if (!(ch.strikes[i] > 0.0)) refused = "swift chain: strike <= 0";
                p.kmin = std::min(p.kmin, ch.strikes[i]);
                p.kmax = std::max(p.kmax, ch.strikes[i]);
            }
            if (refused.empty()) todo.push_back(p);
        }
    }
    choose_params_all(todo);
    for (const Pending &pd : todo) {
        const hexo_swift_chain &ch = *pd.ch;
        const HP &hp = pd.p;
        const hexo_swift_params &sp = pd.sp;
        if (pd.status != HEXO_OK) return ctx_fail(ctx, pd.status, "swift: the truncation loop did not converge");
        if (!valid_params(sp))
            return ctx_fail(ctx, HEXO_ERR_UNSUPPORTED, "swift: J must be a power of two up to 65536 with k2 - k1 < 4J");
        if (ch.method > HEXO_SWIFT_FFT) return ctx_fail(ctx, HEXO_ERR_INVALID, "swift chain: unknown method");
        Exp e{};
        uint32_t logJ = 0;
        while ((1u << logJ) < sp.J) ++logJ;
        e.stiff = sp.upper > kStiff;
        if (ch.method == HEXO_SWIFT_FFT ||
            (ch.method == HEXO_SWIFT_AUTO && sp.J >= (e.stiff ? kFftMinStiffJ : kFftMinJ))) {
            e.logN = logJ + 1u;
            e.logR = e.logN < 6u ? 0u : (uint32_t)std::max(kLogParts, (int)e.logN - kLogMaxPart);
            e.y_off = f;
            f += 2ull * sp.J;
            max_part = std::max(max_part, 1u << (e.logN - e.logR));
        } else {
            e.v_off = v;
            v += (uint64_t)(sp.k2 - sp.k1 + 1);
        }
        e.logL = e.stiff || sp.J < kFoldMinJ ? 0u : std::min(logJ - 5u, kLogFold);
        if (tw_at.off[logJ] == ~0ull) {
            tw_at.off[logJ] = tw;
            for (uint32_t n = 0; n < 4 * sp.J; n += 128) it_set.push_back({logJ, n});
            tw += 4ull * sp.J;
        }
        e.tw_off = tw_at.off[logJ];
        e.p = hp;
        e.q = ChfConst{1.0 / hp.sigma, 2.0 * hp.kappa * hp.vm / (hp.sigma * hp.sigma), hp.rho / hp.sigma};
        e.tau = ch.tau;
        e.r = pd.r;
        e.S = pd.S;
        e.sqrt2m = sp.sqrt_exp2_m;
        e.lower = sp.lower;
        e.upper = sp.upper;
        e.du = M_PI * (double)sp.exp2_m / (2.0 * sp.J);
        e.k1 = sp.k1;
        e.k2 = sp.k2;
        e.J = sp.J;
        e.n_opt = ch.n;
        e.h_off = h; h += sp.J;
        e.w_off = w; w += 6ull * sp.J;
        e.o_off = strikes.size();
        strikes.insert(strikes.end(), ch.strikes, ch.strikes + ch.n);
        const uint32_t at = (uint32_t)ex.size();
        for (uint32_t j = 0; j < sp.J; j += 128) it_h.push_back({at, j});
        if (e.logN)
            for (uint32_t r = 0; r < (1u << e.logR); ++r) it_fft.push_back({at, r});
        else
            for (uint32_t k = 0; k < (uint32_t)(sp.k2 - sp.k1 + 1); k += 32) it_pay.push_back({at, k});
        for (uint32_t j = 0; j < sp.J; j += 64) (e.stiff ? it_stiff : it_den).push_back({at, j});
        for (uint32_t i = 0; i < ch.n; i += 128) it_o.push_back({at, i});
        for (uint32_t i = 0; i < ch.n; i += 4) it_pri.push_back({at, i});
        ex.push_back(e);
        chain_of.push_back(&ch);
        any_grad |= ch.grad_out != nullptr;
    }
    if (!refused.empty()) return ctx_fail(ctx, HEXO_ERR_INVALID, refused);
    if (ex.empty()) return HEXO_OK;
    const uint32_t n_tw = (uint32_t)it_set.size(), n_h = (uint32_t)it_h.size();
    it_set.insert(it_set.end(), it_h.begin(), it_h.end());
    it_set.insert(it_set.end(), it_o.begin(), it_o.end());
    const size_t n_opt = strikes.size();
    std::lock_guard<std::mutex> lk(ctx->run_mu);
    cudaSetDevice(ctx->device);
    cudaStream_t st = ctx->stream;
    // one allocation: what is uploaded (one copy), work buffers, outputs (one copy back)
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off = (off + bytes + 255) / 256 * 256; return o; };
    const size_t o_ex = take(ex.size() * sizeof(Exp));
    const size_t o_is = take(it_set.size() * sizeof(Item)), o_if = take(it_fft.size() * sizeof(Item));
    const size_t o_ip = take(it_pay.size() * sizeof(Item)), o_id = take(it_den.size() * sizeof(Item));
    const size_t o_it = take(it_stiff.size() * sizeof(Item)), o_ir = take(it_pri.size() * sizeof(Item));
    const size_t o_k = take(n_opt * sizeof(double)), up_bytes = off;
    const size_t o_o = take(n_opt * sizeof(Opt));
    const size_t o_tw = take(tw * sizeof(double2)), o_h = take(h * sizeof(double2));
    const size_t o_v = take(v * sizeof(double)), o_w = take(w * sizeof(double2));
    const size_t o_y = take(f * sizeof(double2)), o_z = take(f * sizeof(double2));
    const size_t o_p = take(n_opt * sizeof(double)), o_g = take(any_grad ? n_opt * 5 * sizeof(double) : 0);
    const size_t down_bytes = off - o_p;
    void *dmem = nullptr;   // the context's arena: no allocation once it is large enough
    cudaError_t err = ctx_scratch(ctx, off, &dmem);
    if (err != cudaSuccess) return cuda_fail(ctx, err, "cudaMalloc swift");
    char *d = static_cast<char *>(dmem);
    std::vector<char> pageable;
    char *host = static_cast<char *>(ctx_scratch_host(ctx, std::max(up_bytes, down_bytes)));
    if (host == nullptr) {
        pageable.resize(std::max(up_bytes, down_bytes));
        host = pageable.data();
    }
    auto put = [&](size_t o, const void *src, size_t bytes) { if (bytes) std::memcpy(host + o, src, bytes); };
    auto put_items = [&](size_t o, const std::vector<Item> &it) { put(o, it.data(), it.size() * sizeof(Item)); };
    put(o_ex, ex.data(), ex.size() * sizeof(Exp));
    put_items(o_is, it_set);
    put_items(o_if, it_fft);
    put_items(o_ip, it_pay);
    put_items(o_id, it_den);
    put_items(o_it, it_stiff);
    put_items(o_ir, it_pri);
    put(o_k, strikes.data(), n_opt * sizeof(double));
    if ((err = cudaMemcpyAsync(d, host, up_bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return cuda_fail(ctx, err, "upload swift");
    const Exp *dex = reinterpret_cast<const Exp *>(d + o_ex);
    auto items = [&](size_t o) { return reinterpret_cast<const Item *>(d + o); };
    double2 *dtw = reinterpret_cast<double2 *>(d + o_tw), *dh = reinterpret_cast<double2 *>(d + o_h);
    double *dv = reinterpret_cast<double *>(d + o_v);
    double2 *dw = reinterpret_cast<double2 *>(d + o_w), *dy = reinterpret_cast<double2 *>(d + o_y),
            *dz = reinterpret_cast<double2 *>(d + o_z);
    double *dp = reinterpret_cast<double *>(d + o_p), *dg = any_grad ? reinterpret_cast<double *>(d + o_g) : nullptr;
    Opt *dopt = reinterpret_cast<Opt *>(d + o_o);
    Launches go{st, ctx->sm_count, it_set.size()};
    setup_kernel<<<(unsigned)it_set.size(), 128, 0, st>>>(dex, items(o_is), n_tw, n_h, tw_at,
                                                          reinterpret_cast<const double *>(d + o_k), dtw, dh, dopt);
    if (!it_fft.empty()) {
        const size_t smem = max_part * sizeof(double2);
        if (smem > 48u << 10)
            for (const void *fn : {(const void *)fft_terms_kernel, (const void *)fft_payoff_kernel})
                if ((err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)(sizeof(double2) << kLogMaxPart))) != cudaSuccess)
                    return cuda_fail(ctx, err, "swift shared memory");
        go.run(it_fft.size(), 128, smem, fft_terms_kernel, dex, items(o_if), dtw, dh, dy);
        // Where the parts fill the GPU several times over, blocks of two warps: a part of a common
        // expiry (J = 256 to 1024: 64 to 256 points) keeps its warps busy, and at 142 registers
        // more parts are resident: 0.41 -> 0.30 ms on 2,048 chains (fft_terms_kernel, 32
        // registers: 0.13 -> 0.14).  Fewer parts want every warp that a part can use: half of
        // them would leave half of an SM's FP64 units idle.
        const unsigned width = it_fft.size() >= 4ull * ctx->sm_count ? 64u : 128u;
        go.run(it_fft.size(), width, smem, fft_payoff_kernel, dex, items(o_if), dtw, dy, dz);
    }
    if (!it_pay.empty()) go.run(it_pay.size(), 32, 0, payoff_kernel, dex, items(o_ip), dtw, dh, dv);
    if (!it_den.empty())
        go.run(it_den.size(), 64, 0, density_kernel<false>, dex, items(o_id), dtw, dv, dw, dz);
    if (!it_stiff.empty()) {
        go.last = it_stiff.size();
        density_kernel<true><<<(unsigned)it_stiff.size(), 64, 0, st>>>(dex, items(o_it), dtw, dv, dw, dz);
    }
    if (any_grad) go.run(it_pri.size(), 128, 0, price_kernel<true>, dex, items(o_ir), dw, dopt, dp, dg);
    else go.run(it_pri.size(), 128, 0, price_kernel<false>, dex, items(o_ir), dw, dopt, dp, dg);
    if ((err = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, err, "swift kernels");
    if ((err = cudaMemcpyAsync(host, dp, down_bytes, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (err = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_fail(ctx, err, "swift results");
    const double *hp = reinterpret_cast<const double *>(host), *hg = reinterpret_cast<const double *>(host + (o_g - o_p));
    for (size_t e = 0; e < ex.size(); ++e) {
        const hexo_swift_chain &ch = *chain_of[e];
        std::memcpy(ch.price_out, hp + ex[e].o_off, ch.n * sizeof(double));
        if (ch.grad_out) std::memcpy(ch.grad_out, hg + ex[e].o_off * 5, ch.n * 5 * sizeof(double));
    }
    return HEXO_OK;
}

// ------------------------------------------------ calibration callbacks

// The reference's calibration data (adata_s, src/inc/HCalibration.h:13-30):
// the spot and every chain's expiry and strikes.  prices / jacobian are the
// objective and Jacobian that its Levenberg-Marquardt call evaluates
// (get_prices_for_levmar / get_jacobian_for_levmar, HCalibration.cpp:35-57):
// for a parameter vector p = (v0, vm, rho, kappa, sigma) the wavelet
// parameters of every chain are chosen for p (update_adata,
// HCalibration.cpp:11-33), then all chains are priced in one call.  The last
// p's prices and Jacobian are kept, so the pair of calls levmar makes per
// step prices once.
struct hexo_calib {
    hexo_ctx *ctx = nullptr;
    double S = 0.0, r = 0.0, trunc = 1e-7;
    std::vector<double> taus, strikes;
    std::vector<uint32_t> counts;
    bool have = false;
    double last_p[5] = {0, 0, 0, 0, 0};
    std::vector<double> prices, jac;
};

namespace {
hexo_status calib_eval(hexo_calib *c, const double *p) {
    if (c->have && std::memcmp(p, c->last_p, sizeof c->last_p) == 0) return HEXO_OK;
    const size_t n = c->strikes.size();
    c->prices.assign(n, 0.0);
    c->jac.assign(n * 5, 0.0);
    std::vector<hexo_swift_chain> chains(c->taus.size());
    size_t off = 0;
    for (size_t k = 0; k < chains.size(); ++k) {
        hexo_swift_chain &ch = chains[k];
        std::memset(&ch, 0, sizeof ch);
        ch.tau = c->taus[k];
        ch.strikes = c->strikes.data() + off;
        ch.n = c->counts[k];
        ch.params = nullptr;
        ch.trunc_precision = c->trunc;
        ch.price_out = c->prices.data() + off;
        ch.grad_out = c->jac.data() + off * 5;
        off += c->counts[k];
    }
    hexo_swift_request rq;
    std::memset(&rq, 0, sizeof rq);
    rq.params = hexo_params{p[0], p[1], p[2], p[3], p[4], c->r, 0.0};
    rq.S = c->S;
    rq.chains = chains.data();
    rq.n_chains = (uint32_t)chains.size();
    const hexo_status s = hexo_swift_price(c->ctx, &rq, 1);
    c->have = s == HEXO_OK;
    if (c->have) std::memcpy(c->last_p, p, sizeof c->last_p);
    return s;
}
} // namespace

hexo_status hexo_calib_create(hexo_ctx *ctx, double S, double r, const double *taus, const uint32_t *counts,
                              const double *strikes, uint32_t n_chains, double trunc_precision, hexo_calib **out) {
    if (!ctx || !out || !taus || !counts || !strikes || n_chains == 0 || !(S > 0.0) || !std::isfinite(r))
        return HEXO_ERR_INVALID;
    *out = nullptr;
    hexo_calib *c = new (std::nothrow) hexo_calib();
    if (!c) return HEXO_ERR_NOMEM;
    c->ctx = ctx;
    c->S = S;
    c->r = r;
    c->trunc = trunc_precision > 0.0 ? trunc_precision : 1e-7;
    size_t n = 0;
    for (uint32_t k = 0; k < n_chains; ++k) {
        if (!(taus[k] > 0.0) || counts[k] == 0) { delete c; return HEXO_ERR_INVALID; }
        c->taus.push_back(taus[k]);
        c->counts.push_back(counts[k]);
        n += counts[k];
    }
    c->strikes.assign(strikes, strikes + n);
    *out = c;
    return HEXO_OK;
}

uint32_t hexo_calib_observations(const hexo_calib *c) { return c ? (uint32_t)c->strikes.size() : 0u; }

hexo_status hexo_calib_prices(hexo_calib *c, const double *p, double *x) {
    if (!c || !p || !x) return HEXO_ERR_INVALID;
    const hexo_status s = calib_eval(c, p);
    if (s == HEXO_OK) std::memcpy(x, c->prices.data(), c->prices.size() * sizeof(double));
    return s;
}

hexo_status hexo_calib_jacobian(hexo_calib *c, const double *p, double *jac) {
    if (!c || !p || !jac) return HEXO_ERR_INVALID;
    const hexo_status s = calib_eval(c, p);
    if (s == HEXO_OK) std::memcpy(jac, c->jac.data(), c->jac.size() * sizeof(double));
    return s;
}

hexo_status hexo_calib_destroy(hexo_calib *c) {
    if (!c) return HEXO_ERR_INVALID;
    delete c;
    return HEXO_OK;
}

} // extern "C"
