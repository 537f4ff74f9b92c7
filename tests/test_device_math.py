"""The path kernels' own arithmetic on the host (CPU): the FP64 form's roots,
reciprocals, exponential and variance, the FP32 form's variance.

csrc/hexo_f64.cuh and hexo_f32.cuh use only integer and individually rounded
operations, so they compile for the host (tests/device_math/host_device.h) and
give the device's results there but for the two approximate instructions, whose
results are the correctly rounded ones moved by -1, 0 or 1 unit of the last
place: a function has to keep its bound with each of those seeds.
"""
import ctypes as C
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

FN = {"recip": 0, "root": 1, "exp": 2}


def build(name, out):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fconstexpr-ops-limit=200000000", "-shared",
                        "-fPIC", "-I", str(ROOT / "hestonexotics_gb300" / "csrc"),
                        str(ROOT / "tests" / "device_math" / f"{name}.cpp"), "-o", str(out / f"{name}.so")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return C.CDLL(str(out / f"{name}.so"))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    lib = build("f64_host", tmp_path_factory.mktemp("device_math"))
    lib.f64_worst_ulp.restype = lib.f64_worst_variance.restype = C.c_double
    return lib


@pytest.fixture(scope="module")
def f64(lib):
    def worst(fn, seed, x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        at = C.c_double()
        w = lib.f64_worst_ulp(FN[fn], seed, C.c_uint64(len(x)), x.ctypes.data_as(C.c_void_p), C.byref(at))
        return w, at.value.hex()
    return worst


def neighbours(e_lo, e_hi, rng):
    """Powers of two and the doubles around them: the nearest 300 either way, and more up to 2^-20 away."""
    k = np.concatenate([np.arange(-300, 301), (2.0 ** rng.uniform(0, 32, 400)).astype(np.int64),
                        -(2.0 ** rng.uniform(0, 32, 400)).astype(np.int64)])
    one = np.array([1.0]).view(np.int64) + k
    return np.concatenate([np.ldexp(one.view(np.float64), e) for e in range(e_lo, e_hi)])


# 0.51 units, the functions' stated bound: half a unit of the rounding and what the correction's float product adds
@pytest.mark.parametrize("seed", [-1, 0, 1])
@pytest.mark.parametrize("fn", ["recip", "root"])
def test_recip_and_root_next_to_powers_of_two(f64, fn, seed):
    w, at = f64(fn, seed, neighbours(-58, 59, np.random.default_rng(1)))
    assert w <= 0.51, f"{w} units at {at}"


@pytest.mark.parametrize("seed", [-1, 0, 1])
@pytest.mark.parametrize("fn,lo,hi", [("recip", -59.9, 59.9), ("root", -112.9, 99.9)])
def test_recip_and_root_over_their_ranges(f64, fn, lo, hi, seed):
    w, at = f64(fn, seed, 2.0 ** np.random.default_rng(2).uniform(lo, hi, 200000))
    assert w <= 0.51, f"{w} units at {at}"


# half a unit of the rounding, 0.07 of the polynomial's 32-bit terms and the table's 2^-62, and, where |x| is
# large, n = 256 |x| / ln2 times what ln2/256 is off in units of 2^-71 (0.06 there)
@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("lo,hi,bound", [(-70, -20, 0.57), (-20, -8, 0.57), (-8, -2, 0.57), (-2, 5, 0.57), (5, 9, 0.63)])
def test_exp_over_its_range(f64, sign, lo, hi, bound):
    w, at = f64("exp", 0, sign * 2.0 ** np.random.default_rng(3).uniform(lo, hi, 200000))
    assert w <= bound, f"{w} units at {at}"


def test_exp_around_its_table(f64):
    # results around every table entry and around powers of two, arguments of either sign and zero
    n = np.arange(-5120, 5121)[:, None] * (np.log(2.0) / 256)
    x = np.concatenate([(n + np.random.default_rng(4).uniform(-1, 1, (1, 40)) * 2.0 ** -np.arange(10, 50)).ravel(),
                        [0.0, -0.0, 5e-324, -5e-324, 2.0 ** -54, -(2.0 ** -54), 511.9999, -511.9999]])
    w, at = f64("exp", 0, x)
    assert w <= 0.57, f"{w} units at {at}"


@pytest.fixture(scope="module")
def variance(lib):
    def worst(seed, m, s2, rng):
        n = len(m)
        m, s2 = np.ascontiguousarray(m), np.ascontiguousarray(s2)
        z = rng.standard_normal(n).astype(np.float32)
        # uniforms all over, near 1 and next to where x = Y (1 - U) crosses 1 (the branch's zero)
        Y = 0.5 + 0.5 * s2 / (m * m)
        x = np.where(rng.random(n) < 0.5, rng.random(n), np.exp(-2.0 ** rng.uniform(-30, 3, n))) / np.maximum(Y, 1.0)
        uw = (np.uint64(0) - np.clip(x * 2.0 ** 64, 1, 2.0 ** 64 * (1 - 2.0 ** -53)).astype(np.uint64))
        near, at = np.zeros(n, dtype=np.uint8), C.c_uint64()
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        w = lib.f64_worst_variance(seed, C.c_uint64(n), p(m), p(s2), p(z), p(uw), p(near), C.byref(at))
        i = at.value
        return w, near.astype(bool), f"m {m[i].hex()} s2 {s2[i].hex()} z {z[i]} uw {uw[i]:#x} near {near[i]}"
    return worst


# Where the step takes its own functions the error stays within 5 units of 2^-53 of the terms' size: the quadratic
# branch rounds w and w^2 and takes two roots within half a unit each, the exponential one cuts six products and
# sums at 2^-55 or finer and rounds Y and the result.  All of m's and s^2's range, in ratios s^2/m^2 from 2^-38 up.
@pytest.mark.parametrize("seed", [-1, 0, 1])
@pytest.mark.parametrize("lo,hi", [(-38, -20), (-20, -2), (-2, 3), (3, 20), (20, 60), (60, 118)])
def test_next_variance_over_its_ranges(variance, lo, hi, seed):
    rng = np.random.default_rng(5)
    lm, lr = rng.uniform(-30, 30, 120000), rng.uniform(lo, hi, 120000)
    ok = np.abs(lr + 2 * lm) < 60
    w, near, at = variance(seed, 2.0 ** lm[ok], 2.0 ** (lr + 2 * lm)[ok], rng)
    assert w <= 5.0, f"{w} units at {at}"


@pytest.fixture(scope="module")
def f32_rms(tmp_path_factory):
    lib = build("f32_host", tmp_path_factory.mktemp("device_math_f32"))
    lib.f32_rms_variance.restype = C.c_double

    def rms(seed, lo, hi):   # log2 of the error, for Psi = s^2/m^2 from 2^lo to 2^hi
        rng, n = np.random.default_rng(6), 150000
        m = 2.0 ** rng.uniform(-14, 1, n)
        s2 = 2.0 ** rng.uniform(lo, hi, n) * m * m
        z, x = rng.standard_normal(n).astype(np.float32), rng.random(n) / np.maximum(0.5 + 0.5 * s2 / (m * m), 1.0)
        uw = np.uint64(0) - np.maximum(x * 2.0 ** 64, 1.0).astype(np.uint64)
        p = lambda a: np.ascontiguousarray(a).ctypes.data_as(C.c_void_p)
        return np.log2(lib.f32_rms_variance(seed, C.c_uint64(n), p(m), p(s2), p(z), p(uw)))
    return rms


# The reference's order of operations a (b + z)^2, evaluated in normalised double-single steps, has these errors on
# the same steps (correctly rounded seeds; seeds a unit off); the branch must not be less exact.
@pytest.mark.parametrize("lo,hi,exact_seed,seed_off", [(-30, -10, -47.13, -44.54), (-10, -3, -47.24, -44.62),
                                                       (-3, 0.58, -47.51, -45.03)])
def test_fp32_quadratic_branch(f32_rms, lo, hi, exact_seed, seed_off):
    assert f32_rms(0, lo, hi) <= exact_seed
    assert f32_rms(1, lo, hi) <= seed_off
    assert f32_rms(-1, lo, hi) <= seed_off


# The exponential branch with a logarithm good to 2^-46 of 1: a unit of that from each of r's two parts, the table's
# and the sums' (2^-44.0 without r's low part in the cubic term).
@pytest.mark.parametrize("seed", [-1, 0, 1])
@pytest.mark.parametrize("lo,hi", [(0.6, 2), (2, 8), (8, 20)])
def test_fp32_exponential_branch(f32_rms, lo, hi, seed):
    assert f32_rms(seed, lo, hi) <= -45.5
