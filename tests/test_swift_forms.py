"""SWIFT transforms and characteristic function at the edges of their forms.

The transforms run as FFTs in one part (below 64 points), eight or sixteen,
or as direct sums; the payoff range k1..k2 starts at any residue and wraps the
FFT's N = 2J points up to twice; the characteristic function has its own form
for stiff expiries (upper above 12) and for frequencies with d tau above 600.
All against the oracle's direct sums.

Tolerance: the sums' terms are of the order K e^upper and each result carries
a few roundings of every factor and of log2 N passes, so prices agree to K
e^upper 2^-52 (8 + log2 N), a gradient component to 100 times that (the
derivatives of the characteristic function reach that size here).
"""
import numpy as np
import pytest

from hestonexotics_gb300 import engine as E

pytestmark = pytest.mark.gpu

P5 = [0.04, 0.05, -0.6, 1.5, 0.5]
K = np.array([70.0, 100.0, 130.0])


def check(engine, oracle, p5, tau, sp, method):
    r = 0.02
    (price, grad), = engine.swift(E.Params(*p5, r=r), 100.0, [(tau, K)], grad=True, swift_params=[sp], method=method)
    only, = engine.swift(E.Params(*p5, r=r), 100.0, [(tau, K)], grad=False, swift_params=[sp], method=method)
    wp, wg = oracle.swift_price(p5, tau, r, 100.0, K, np.array(sp[:8], dtype=float), grad=True)
    tol = K.max() * np.exp(sp[4]) * 2.0 ** -52 * (8 + np.log2(2 * sp[7]))
    np.testing.assert_allclose(price, wp, rtol=0, atol=tol)
    np.testing.assert_allclose(grad, wg, rtol=0, atol=100 * tol)
    np.testing.assert_allclose(only, price, rtol=0, atol=tol)


@pytest.mark.parametrize("method", [0, 1, 2])
@pytest.mark.parametrize("J,k1,k2", [(1, 0, 3), (2, -1, 2), (8, -5, 9), (16, -17, 14), (32, -31, 33), (64, -255, 0),
                                     (128, 7, 40), (256, -300, 301), (1024, -2047, 2048)])
def test_transforms(engine, oracle, J, k1, k2, method):
    check(engine, oracle, P5, 0.5, (4, 16, 4.0, -3.0, 3.0, k1, k2, J), method)


@pytest.mark.parametrize("method", [0, 2])
@pytest.mark.parametrize("upper", [11.9, 12.1])
@pytest.mark.parametrize("J", [256, 1024])
def test_stiff_expiries(engine, oracle, J, upper, method):
    check(engine, oracle, P5, 3.0, (4, 16, 4.0, -upper, upper, -150, 150, J), method)


def test_far_frequencies(engine, oracle):
    # u up to 2^9 pi: d tau / 2 passes 300 (phi is below e^-300 there)
    p5 = [0.04, 0.05, -0.3, 1.5, 0.9]
    check(engine, oracle, p5, 4.0, (8, 256, 16.0, -4.0, 4.0, -1000, 1000, 1024), 0)


@pytest.mark.parametrize("J", [256, 512, 2048, 4096])   # below the folds; segments of 16 and 32, one to four rounds
@pytest.mark.parametrize("method", [1, 2])
def test_folded_segments(engine, oracle, J, method):
    check(engine, oracle, P5, 0.3, (6, 64, 8.0, -3.0, 3.0, -192, 191, J), method)


def test_many_parts(engine):
    # enough parts for the narrow FFT blocks (8 an expiry, 4 a multiprocessor): the same operations
    # in the same order as in an expiry's call of its own, so the same bits
    sps = [(4, 16, 4.0, -3.0, 3.0, -int(1.1 * J) - 1, int(1.7 * J) + 1, J) for J in (2, 16, 32, 64, 256, 1024, 4096)]
    chains = [(0.5, K)] * (16 * len(sps))
    many = engine.swift(E.Params(*P5, r=0.02), 100.0, chains, grad=True, swift_params=sps * 16, method=2)
    for (price, grad), sp in zip(many, sps * 16):
        (p1, g1), = engine.swift(E.Params(*P5, r=0.02), 100.0, chains[:1], grad=True, swift_params=[sp], method=2)
        np.testing.assert_array_equal(price, p1)
        np.testing.assert_array_equal(grad, g1)
