"""SWIFT expiries on both sides of the lines between its forms.

Stiff expiries (upper above 12) keep the reference's order of operations, since
their payoff terms grow as e^upper and any change of rounding shows: their
prices and gradients are held to the values recorded when every expiry was
evaluated in that order (tests/golden/swift_stiff.json, on a GB300).  The other
form would move them by 2.5e-11 (upper 12.1), 3e-10 to 1e-7 (17) and 2e-5 (25)
relative, so 1e-12 tells the two apart.  Below the line prices agree with the
oracle to the 1e-9 that the reference's known answers are good to.

Frequencies from Re(d) tau / 2 = 300 on are evaluated in the reference's form
too; phi is below e^-300 there.  Up to 350 everything is finite in every form
(cosh^2 stays below 1e308), and the result has to be.
"""
import numpy as np
import pytest

from conftest import golden
from hestonexotics_gb300 import engine as E

pytestmark = pytest.mark.gpu

K = np.array([70.0, 100.0, 130.0])
STIFF = golden("swift_stiff.json")


def unhex(a):
    return np.array([[float.fromhex(x) for x in r] if isinstance(r, list) else float.fromhex(r) for r in a])


@pytest.mark.parametrize("case", STIFF["cases"], ids=lambda c: f"{c['p5'][3]}-{c['tau']}-{c['method']}")
def test_stiff_expiries_do_not_move(engine, case):
    prm = E.Params(*case["p5"], r=STIFF["r"])
    chain = [(case["tau"], np.array(STIFF["strikes"]))]
    (price, grad), = engine.swift(prm, STIFF["S"], chain, grad=True, method=case["method"])
    only, = engine.swift(prm, STIFF["S"], chain, grad=False, method=case["method"])
    np.testing.assert_allclose(price, unhex(case["price"]), rtol=1e-12)
    np.testing.assert_allclose(only, unhex(case["price"]), rtol=1e-12)
    np.testing.assert_allclose(grad, unhex(case["grad"]), rtol=1e-12)


@pytest.mark.parametrize("method", [0, 1, 2])
@pytest.mark.parametrize("J", [256, 512, 1024])
def test_just_below_the_stiff_line(engine, oracle, J, method):
    p5, sp = [0.04, 0.05, -0.6, 1.5, 0.5], (4, 16, 4.0, -11.9, 11.9, -150, 150, J)
    (price, grad), = engine.swift(E.Params(*p5, r=0.02), 100.0, [(8.0, K)], grad=True, swift_params=[sp], method=method)
    wp, wg = oracle.swift_price(p5, 8.0, 0.02, 100.0, K, np.array(sp, dtype=float), grad=True)
    assert np.isfinite(wp).all() and np.isfinite(wg).all()
    np.testing.assert_allclose(price, wp, rtol=1e-9)
    tol = K.max() * np.exp(11.9) * 2.0 ** -52 * (8 + np.log2(2 * J))   # as below
    np.testing.assert_allclose(grad, wg, rtol=0, atol=100 * tol)


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("tau,far", [(0.8, 0), (0.9, 35), (0.95, 87)])
def test_far_frequencies_are_finite(engine, oracle, tau, far, method):
    p5, sp = [0.04, 0.05, -0.3, 1.5, 0.9], (8, 256, 16.0, -4.0, 4.0, -1000, 1000, 1024)
    u = np.pi * (2 * np.arange(1024) + 1) * 256 / 2048
    d = np.sqrt((p5[3] + 1j * u * p5[4] * p5[2]) ** 2 + p5[4] ** 2 * (u * u - 1j * u))
    assert (d.real * tau >= 600.0).sum() == far and d.real.max() * tau / 2 < 350.0
    (price, grad), = engine.swift(E.Params(*p5, r=0.02), 100.0, [(tau, K)], grad=True, swift_params=[sp], method=method)
    wp, wg = oracle.swift_price(p5, tau, 0.02, 100.0, K, np.array(sp, dtype=float), grad=True)
    assert np.isfinite(wp).all() and np.isfinite(wg).all()
    # the sums' terms are of the order K e^upper and carry a few roundings of every factor and of log2 N passes;
    # the gradient's factors reach a hundred times that
    tol = K.max() * np.exp(4.0) * 2.0 ** -52 * (8 + np.log2(2 * 1024))
    np.testing.assert_allclose(price, wp, rtol=0, atol=tol)
    np.testing.assert_allclose(grad, wg, rtol=0, atol=100 * tol)
