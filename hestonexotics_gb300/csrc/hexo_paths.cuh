// Persistent Monte Carlo path kernel.
//
// Each CTA repeatedly takes the next tile (set, block of consecutive paths)
// from a global queue and simulates its paths, PPT paths per thread, through
// the set's step schedule up to the last maturity that block needs.  One
// path follows the reference's per-path loop (HSimulation.tpp:30-46):
//   QE step (tpp:52-86)  ->  at a pricing step, the Asian and European final
//   values (AsianContract.h:29-34, VanillaContract.h:28-31) and the call
//   payoffs of every option of that maturity  ->  trapezoid accumulation
//   (AsianContract.h:25-28) with the width in force after the pricing check.
// Payoffs are folded into exact fixed-point limb sums: per option a warp
// reduction (redux.sync) and one global atomic add per limb per warp.
//
// kF32 = false: the plain FP64 form.  kF32 = true: paths evolve in float,
// except the variance, which is kept in double-single so that the scheme's
// branch decisions match FP64 (hexo_ds.cuh); AS241 is float32 in both
// forms, so both consume bit-identical normals.
#pragma once
#include <stdint.h>
#include "hexo_types.h"
#include "hexo_device.cuh"
#include "hexo_f32.cuh"
#include "hexo_f64.cuh"

namespace hexo {


// Square root of x >= 0 from the MUFU reciprocal square root (the .ftz form:
// its operand is normal, and the other form spends three instructions on
// operands that are not).
__device__ __forceinline__ float fsqrt_fast(float x) { return __fmul_rn(x, ds::rsqrt_approx(fmaxf(x, 1e-30f))); }
// exp(x) as 2^(x log2 e) by the MUFU; results below 2^-126 are 0 (a spot so far down is 2^-78 of
// the payoffs' last unit).
__device__ __forceinline__ float exp_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__fmul_rn(x, 1.4426950408889634f)));
    return r;
}

template <bool kF32> struct Real;
template <> struct Real<false> { typedef double T; };
template <> struct Real<true> { typedef float T; };

template <bool kF32>
struct PathVars {
    typename Real<kF32>::T lx, v, X, Xp, acc;  // lx: log X (FP64); log X - log S0 - (rho/sigma) v (FP32)
    ds::F2 vd;                                  // FP32 form: the variance in double-single (v == vd.h)
};

// The path arithmetic below names every rounding (__fma_rn, __dmul_rn, ...)
// so that the compiler cannot contract or reassociate differently in
// different template instantiations: every launch shape computes the same
// bits for the same path.

// One QE step of one path (HSimulation.tpp:52-86), FP64; returns whether it
// took the quadratic branch.  As the reference writes it, a step is about 100
// FP64 instructions, and that pipe bounds it; with the roots, quotients, log
// and exp of hexo_f64.cuh it is 14 (quadratic) or 10 (exponential) with the
// trapezoid: 64-set batch at 1/128 of its paths 546 -> 90.1 ms, plain Asian
// 4.46 -> 0.73 ms.
__device__ __forceinline__ bool qe_step(PathVars<false> &pv, const SegDesc &sg, const double &theta, dev::Shishua &g,
                                        dev::RngLane &c, const dev::Ring &r, const dev::WarpScratch &ws,
                                        const f64::ExpTab *etab) {
    dev::DrawPlan dp = dev::draw_prefetch(c, r);
    const double v = pv.v;
    const double m = __fma_rn(v, sg.disc, sg.m0);                            // tpp:59
    const double s2 = fabs(__fma_rn(v, sg.cA, sg.cB));                       // tpp:60
    const bool near = f64::in_range(m, s2);
    const bool quad = near ? f64::quadratic(m, s2) : f64::quadratic_wide(v, theta, sg.disc, s2);
    if (dev::draw_prepare<false>(g, c, r, ws, quad)) dp = dev::draw_prefetch(c, r);
    float z1 = 0.0f, z2;                                                     // draw order, tpp:67,72,80
    uint64_t uw = 0;
    dev::draw_commit(g, c, r, dp, quad, z1, uw, z2);
    double vn;
    if (!near) vn = f64::variance_wide(v, theta, sg.disc, s2, quad, z1, uw);
    else if (quad) vn = f64::variance_quadratic(m, s2, z1);                  // tpp:64-68
    else vn = f64::variance_exponential(m, s2, uw);                          // tpp:70-73
    pv.v = vn;
    // tpp:80, sqrt(K3 v + K4 vn) z as sqrt(v + vn) (z sqrt(K3))
    const double t = __fma_rn(sg.K2, vn, __fma_rn(sg.K1, v, __dadd_rn(pv.lx, sg.K0)));
    pv.lx = __fma_rn(f64::root(__dadd_rn(v, vn)), f64::mul_float(z2, sg.rK3), t);
    pv.Xp = pv.X;
    pv.X = f64::exp_tab(pv.lx, etab);                                        // tpp:82
    return quad;
}

// One QE step, FP32 form: the same scheme and draws; the variance in
// double-single (m = v disc + m0 and s^2/2 = v cA/2 + cB/2, algebraically the
// reference's tpp:59-60), everything else in float; returns whether it took
// the quadratic branch.
__device__ __forceinline__ bool qe_step(PathVars<true> &pv, const SegDesc &sg, dev::Shishua &g, dev::RngLane &c,
                                        const dev::Ring &r, const dev::WarpScratch &ws, float S0, float rr,
                                        const ds::LogTab *ltab) {
    dev::DrawPlan dp = dev::draw_prefetch(c, r);
    const ds::F2 v = pv.vd;
    const ds::F2 m = ds::fma(v, ds::F2{sg.ds_disc[0], sg.ds_disc[1]}, ds::F2{sg.ds_m0[0], sg.ds_m0[1]});
    const ds::F2 hs = ds::fma(v, ds::F2{sg.ds_hA[0], sg.ds_hA[1]}, ds::F2{sg.ds_hB[0], sg.ds_hB[1]});   // s^2 / 2
    // m^2 as p + e, not normalised
    const float p = __fmul_rn(m.h, m.h);
    const float e = __fmaf_rn(__fadd_rn(m.h, m.h), m.l, __fmaf_rn(m.h, m.h, -p));
    // Psi < PSI_C, s^2/2 < 0.75 m^2; the float comparison decides unless it is within 2^-20 of the threshold
    const float t75 = __fmul_rn(0.75f, p);
    const bool quad = fabsf(__fsub_rn(hs.h, t75)) > __fmul_rn(0x1p-20f, hs.h)
                          ? hs.h < t75
                          : ds::less(hs, ds::mul_f(ds::fast_two_sum(p, e), 0.75f));
    if (dev::draw_prepare<true>(g, c, r, ws, quad)) dp = dev::draw_prefetch(c, r);
    float z1 = 0.0f, z2;
    uint64_t uw = 0;
    dev::draw_commit(g, c, r, dp, quad, z1, uw, z2);
    ds::F2 vn;
    if (quad) vn = f32::variance_quadratic(m, hs, p, e, z1);
    else vn = f32::variance_exponential(m, hs, p, e, uw, ltab);
    pv.vd = vn;
    pv.v = vn.h;
    // K1 v + K2 vn = c (v + vn) + (rho/sigma)(vn - v): the second part
    // telescopes over the steps, so it is not accumulated in float (its
    // rounding would add up step after step); lx = log X - log S0 - r v.
    float inc = __fmaf_rn(sg.f_c, __fadd_rn(v.h, vn.h), sg.f_K0);
    inc = __fmaf_rn(fsqrt_fast(__fmaf_rn(sg.f_K3, v.h, __fmul_rn(sg.f_K4, vn.h))), z2, inc);
    pv.lx = __fadd_rn(pv.lx, inc);
    pv.Xp = pv.X;
    pv.X = __fmul_rn(S0, exp_fast(__fmaf_rn(rr, vn.h, pv.lx)));
    return quad;
}

__device__ __forceinline__ float add_r(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_r(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fma_r(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_r(double a, double b, double c) { return __fma_rn(a, b, c); }

// A CTA takes one tile (blockDim * PPT consecutive paths) at a time, so its
// warps read the same set's descriptors (shared through L1); thread t holds
// paths begin + p * blockDim + t.  A tile prices its set's options in
// increasing (maturity-sorted) index order.  Each warp's sums (redux.sync)
// are stored, without atomics, in the warp's own window of kWindow
// consecutive options (one 32-bit value per option and limb, written once per
// tile); the windows are summed and flushed to this CTA's private copy of the
// global sums only when an option falls past the window and at the end of the
// tile, so the warps meet at a barrier a few times per tile rather than at
// every maturity (measured on the uneven batch: 12 % faster than a flush per
// maturity; the per-warp windows another 4 %, 17 % on a 100-strike chain).
constexpr uint32_t kWindow = 64;

// Folds the call payoffs (AsianContract.h:43-47, VanillaContract.h:37-39) of
// option oi of this warp's paths into the warp's window entry wslot: exact
// limbs per path, one warp sum per limb (redux.sync), stored by lane 0.  A
// warp whose payoffs are all 0 leaves its (cleared) window entry as it is.
// With the control variate (kCV), kind 2 folds the geometric-average call
// (G - K)^+ and kind 3 the signed difference (A - K)^+ - (G - K)^+, whose
// biased limbs are written for every counted path.
template <bool kF32, int PPT, bool kCV>
__device__ __forceinline__ void fold_option(const KernelArgs &a, const SetDesc &S, uint32_t oi, uint32_t *wslot,
                                            uint32_t lane, const bool (&active)[PPT], const uint64_t (&kpath)[PPT],
                                            const typename Real<kF32>::T (&asian)[PPT],
                                            const typename Real<kF32>::T (&euro)[PPT],
                                            const typename Real<kF32>::T (&geo)[PPT]) {
    const OptDesc &O = a.opts[S.opt_begin + oi];
    uint32_t l[kLimbs] = {0, 0, 0, 0, 0, 0};
    bool ok = true, any = false;
    const uint32_t kind = O.kind;
    const int E = S.pay_exp, eoff = S.pay_exp + 103;   // payoffs in units of 2^E
#pragma unroll
    for (int p = 0; p < PPT; ++p) {
        if (active[p] && kpath[p] < O.n_paths) {
            if constexpr (kF32) {
                const float K = O.f_strike;
                if (kCV && kind == 3u) {
                    const float d = __fsub_rn(fmaxf(0.0f, __fsub_rn(asian[p], K)), fmaxf(0.0f, __fsub_rn(geo[p], K)));
                    any = true;   // every counted path adds its 2^63 bias, zero or not
                    ok &= dev::limbs_add_signed_f32(d, eoff, l);
                } else {
                    const float f = kind == 0u ? asian[p] : (kCV && kind == 2u) ? geo[p] : euro[p];
                    const float pay = fmaxf(0.0f, __fsub_rn(f, K));
                    any |= pay != 0.0f;
                    ok &= dev::limbs_add_f32(pay, eoff, l);
                }
            } else {
                const double K = O.strike;
                if (kCV && kind == 3u) {
                    const double d = __dsub_rn(fmax(0.0, __dsub_rn(asian[p], K)), fmax(0.0, __dsub_rn(geo[p], K)));
                    any = true;   // every counted path adds its 2^63 bias, zero or not
                    ok &= dev::limbs_add_signed_f64(d, E, l);
                } else {
                    const double f = kind == 0u ? asian[p] : (kCV && kind == 2u) ? geo[p] : euro[p];
                    const double pay = __dsub_rn(f, K);
                    const int64_t bits = __double_as_longlong(pay);
                    if (bits > 0 && bits <= 0x7ff0000000000000ll) {   // positive; as max(0, pay), a NaN counts as 0
                        any = true;
                        ok &= dev::limbs_add_f64(pay, E, l);
                    }
                }
            }
        }
    }
    if (!ok) atomicOr(a.error, 1);
    if (__any_sync(0xffffffffu, any)) {
        uint32_t sum[kLimbs];
#pragma unroll
        for (int x = 0; x < kLimbs; ++x) sum[x] = __reduce_add_sync(0xffffffffu, l[x]);
        if (lane == 0u) {   // once per option and tile; 8-byte aligned (24 B per option)
            uint2 *w = reinterpret_cast<uint2 *>(wslot);
            w[0] = make_uint2(sum[0], sum[1]);
            w[1] = make_uint2(sum[2], sum[3]);
            w[2] = make_uint2(sum[4], sum[5]);
        }
    }
}

template <bool kF32, int PPT, int UNROLL, bool kCV = false>
__global__ void __launch_bounds__(512) paths_kernel(const KernelArgs a) {
    typedef typename Real<kF32>::T R;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t bd = blockDim.x, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // shared memory: raw words, normals, per-warp conversion scratch
    uint64_t *raw_all = reinterpret_cast<uint64_t *>(smem_raw);
    float *nrm_all = reinterpret_cast<float *>(raw_all + (size_t)PPT * 2 * kRngWords * bd);
    uint16_t *tq_i_all = reinterpret_cast<uint16_t *>(nrm_all + (size_t)PPT * 2 * kRngWords * bd);
    uint32_t *win = reinterpret_cast<uint32_t *>(
        smem_raw + ((size_t)PPT * 2 * kRngWords * bd * 12 + (size_t)(bd >> 5) * kWarpScratchBytes + 15) / 16 * 16);
    // after the windows: the double-single log table of the FP32 form's exponential branch, or the
    // FP64 form's exponential table; visible after the first tile's barrier
    ds::LogTab *ltab = reinterpret_cast<ds::LogTab *>(win + (size_t)(bd >> 5) * kWindow * kLimbs);
    f64::ExpTab *etab = reinterpret_cast<f64::ExpTab *>(ltab);
    if constexpr (kF32) ds::log_table_init(ltab, tid, bd);
    else f64::exp_table_init(etab, tid, bd);

    dev::Ring ring[PPT];
    dev::WarpScratch ws[PPT];
#pragma unroll
    for (int p = 0; p < PPT; ++p) {
        ring[p].raw = raw_all + (size_t)p * 2 * kRngWords * bd + tid;
        ring[p].nrm = nrm_all + (size_t)p * 2 * kRngWords * bd + tid;
        ring[p].stride = bd;
        ws[p].raw0 = ring[p].raw - lane;
        ws[p].nrm0 = ring[p].nrm - lane;
        ws[p].tq_i = tq_i_all + warp * kConvQueue;
        ws[p].lane = lane;
#ifdef HEXO_CHECKS
        ws[p].error = a.error;
        ws[p].check = a.check;
#endif
    }
    __shared__ uint32_t s_tile;
    // this CTA's private copy of the sums: CTAs never contend for one address
    unsigned long long *const acc = a.acc + (size_t)(blockIdx.x % a.n_slots) * a.acc_slot_stride;
    const uint32_t n_warps = bd >> 5;
    for (uint32_t i = tid; i < n_warps * kWindow * kLimbs; i += bd) win[i] = 0u;
    uint32_t *const wwin = win + warp * kWindow * kLimbs;   // this warp's window: one u32 per option and limb
    // adds the warps' window sums for set options [base, base + kWindow) to the global copy and clears them
    auto flush = [&](const SetDesc &S, uint32_t base) {
        __syncthreads();
        for (uint32_t i = tid; i < kWindow * kLimbs; i += bd) {
            unsigned long long v = 0ull;
            for (uint32_t w = 0; w < n_warps; ++w) {
                v += win[w * kWindow * kLimbs + i];
                win[w * kWindow * kLimbs + i] = 0u;
            }
            if (v != 0ull) {
                const uint32_t oi = S.opt_begin + base + i / kLimbs;
                if (HEXO_CHECK(oi < a.n_opts, a.error, a.check, kCheckOpt, oi)) {
                    const OptDesc &O = a.opts[oi];
                    if (HEXO_CHECK(O.out_index < a.n_out, a.error, a.check, kCheckOut, O.out_index))
                        atomicAdd(&acc[(size_t)O.out_index * kLimbs + i % kLimbs], v);
                }
            }
        }
        __syncthreads();
    };

    for (;;) {
        if (tid == 0) s_tile = atomicAdd(a.queue, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        __syncthreads();
        if (tile >= a.n_tiles) break;
        const TileDesc td = a.tiles[tile];
        if (!HEXO_CHECK(td.set < a.n_sets, a.error, a.check, kCheckSet, tile)) continue;   // CTA-uniform skips
        const SetDesc &S = a.sets[td.set];
        if (!HEXO_CHECK((uint64_t)S.seg_begin + td.seg_count <= a.n_segs && td.seg_count <= S.seg_count, a.error,
                        a.check, kCheckSegs, td.set))
            continue;
        const float S0f = S.f_S0, rf = S.f_r;
        uint32_t win_base = 0;   // first set option of the staging window

        dev::Shishua g[PPT];
        dev::RngLane c[PPT];
        PathVars<kF32> pv[PPT];
        // control variate: y = log(X / S0) now and one step back, and the
        // Asian contract's trapezoid sum on y (the geometric average's log)
        R yc[PPT], yp[PPT], accg[PPT];
        uint64_t kpath[PPT];
        bool active[PPT];
#pragma unroll
        for (int p = 0; p < PPT; ++p) {
            kpath[p] = td.path_begin + (uint64_t)p * bd + tid;
            active[p] = kpath[p] < S.n_paths;
            dev::rng_start<kF32>(g[p], c[p], ring[p], ws[p], S.seed + (uint32_t)kpath[p], S.stream);
            pv[p].vd = ds::F2{S.ds_v0[0], S.ds_v0[1]};
            pv[p].lx = kF32 ? (R)(-(float)S.f_r * S.f_v0) : (R)S.logS0;   // FP32: log X - log S0 - (rho/sigma) v
            pv[p].v = kF32 ? (R)S.f_v0 : (R)S.v0;
            pv[p].X = kF32 ? (R)S.f_S0 : (R)S.S0;
            pv[p].Xp = pv[p].X;
            pv[p].acc = (R)0;
            yc[p] = yp[p] = accg[p] = (R)0;
        }

        for (uint32_t si = 0; si < td.seg_count; ++si) {
            const SegDesc sg = a.segs[S.seg_begin + si];
            const R hdt = kF32 ? (R)sg.f_hdt : (R)sg.hdt;
            // the FP64 form's trapezoid, one instruction a step: hdt at the
            // segment's ends, dt at the spots between
            if constexpr (!kF32)
                if (sg.n_steps > 1)
#pragma unroll
                    for (int p = 0; p < PPT; ++p) pv[p].acc = __fma_rn(hdt, pv[p].X, pv[p].acc);
            // every step, then the trapezoid with this width except after the
            // last (pricing) step; one copy of the step code
#pragma unroll UNROLL
            for (uint32_t st = 1; st <= sg.n_steps; ++st) {
#pragma unroll
                for (int p = 0; p < PPT; ++p) {
                    if constexpr (kF32) qe_step(pv[p], sg, g[p], c[p], ring[p], ws[p], S0f, rf, ltab);
                    else qe_step(pv[p], sg, S.theta, g[p], c[p], ring[p], ws[p], etab);
                    if constexpr (kCV) {
                        yp[p] = yc[p];   // FP32: the exponent of X / S0 that qe_step used
                        if constexpr (kF32) yc[p] = __fmaf_rn(rf, pv[p].v, pv[p].lx);
                        else yc[p] = __dsub_rn(pv[p].lx, S.logS0);
                    }
                    if (st < sg.n_steps) {
                        if constexpr (kF32) pv[p].acc = __fmaf_rn(hdt, __fadd_rn(pv[p].X, pv[p].Xp), pv[p].acc);
                        else pv[p].acc = __fma_rn(st + 1 < sg.n_steps ? sg.dt : hdt, pv[p].X, pv[p].acc);
                        if constexpr (kCV) accg[p] = fma_r(hdt, add_r(yc[p], yp[p]), accg[p]);
                    }
                }
            }
            for (uint32_t mj = sg.mat_begin; mj < sg.mat_end; ++mj) {
                if (!HEXO_CHECK(S.mat_begin + mj < a.n_mats && mj < S.mat_count, a.error, a.check, kCheckMat, mj))
                    continue;
                const MatDesc M = a.mats[S.mat_begin + mj];
                if (!HEXO_CHECK(M.opt_end <= S.opt_count && (uint64_t)S.opt_begin + M.opt_end <= a.n_opts, a.error,
                                a.check, kCheckOpt, M.opt_end))
                    continue;
                R asian[PPT], euro[PPT], geo[PPT];
#pragma unroll
                for (int p = 0; p < PPT; ++p) {
                    R interp;
                    if constexpr (kF32) {
                        interp = __fmul_rn(__fsub_rn(pv[p].X, pv[p].Xp), M.f_w);
                        asian[p] = __fmul_rn(__fadd_rn(pv[p].acc, interp), M.f_invT);
                    } else {                                               // AsianContract.h:30-32
                        interp = __dmul_rn(__dsub_rn(pv[p].X, pv[p].Xp), M.w);
                        asian[p] = f64::div_by(__dadd_rn(pv[p].acc, interp), M.T, M.invT);
                    }
                    euro[p] = add_r(pv[p].Xp, interp);                     // VanillaContract.h:28-29
                    geo[p] = (R)0;
                    if constexpr (kCV) {   // G = S0 exp(L), L the Asian weights on y
                        if constexpr (kF32) {
                            const float L = __fmul_rn(__fadd_rn(accg[p], __fmul_rn(__fsub_rn(yc[p], yp[p]), M.f_w)),
                                                      M.f_invT);
                            geo[p] = __fmul_rn(S0f, expf(L));
                        } else {
                            const double L = f64::div_by(
                                __dadd_rn(accg[p], __dmul_rn(__dsub_rn(yc[p], yp[p]), M.w)), M.T, M.invT);
                            geo[p] = __dmul_rn(S.S0, f64::exp_tab(L, etab));
                        }
                    }
                    if (a.dbg_asian != nullptr && active[p]) {
                        const size_t at = (size_t)(kpath[p] - a.dbg_lo) * a.dbg_mats + mj;
                        a.dbg_asian[at] = (double)asian[p];
                        a.dbg_euro[at] = (double)euro[p];
                    }
                }
                // payoffs of the maturity's options, staged in the warp's window
                for (uint32_t oi = M.opt_begin; oi < M.opt_end; ++oi) {
                    if (oi >= win_base + kWindow) {           // CTA-uniform: all warps price the same options
                        flush(S, win_base);
                        win_base = oi - oi % kWindow;
                    }
                    if (!HEXO_CHECK(oi - win_base < kWindow, a.error, a.check, kCheckWindow, oi - win_base)) continue;
                    fold_option<kF32, PPT, kCV>(a, S, oi, wwin + (oi - win_base) * kLimbs, lane, active, kpath, asian,
                                                euro, geo);
                }
            }
            const R hda = kF32 ? (R)sg.f_hdt_after : (R)sg.hdt_after;
#pragma unroll
            for (int p = 0; p < PPT; ++p) {
                pv[p].acc = fma_r(hda, add_r(pv[p].X, pv[p].Xp), pv[p].acc);
                if constexpr (kCV) accg[p] = fma_r(hda, add_r(yc[p], yp[p]), accg[p]);
            }
        }
        flush(S, win_base);
        if (a.exp_steps != nullptr) {   // branch mix: each exponential-branch step drew one uniform
            uint32_t n_exp = 0;
#pragma unroll
            for (int p = 0; p < PPT; ++p)
                if (active[p]) n_exp += c[p].n_u;
            const uint32_t we = __reduce_add_sync(0xffffffffu, n_exp);
            if (lane == 0u && we != 0u) atomicAdd(a.exp_steps, (unsigned long long)we);
        }
    }
}

} // namespace hexo
