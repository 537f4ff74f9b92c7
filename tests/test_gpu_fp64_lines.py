"""The FP64 form on both sides of the lines where the step changes its functions.

The step takes its own roots and quotients while the mean m of the next
variance lies in [2^-30, 2^30), s^2 in [2^-60, 2^60) and s^2 / m^2 above 2^-40,
plain double operations outside; the spot's exponential is tabulated for log
spots below 512 in size.  Each pair of sets lies on either side of one of those
lines (asserted from m and s^2 at the set's own variances), and the oracle
prices the same streams.

Tolerance: 1e-10 relative as everywhere in the FP64 form, and what a last bit
of the variance does to the log-spot: rho / sigma magnifies it, so each step
moves the spot by up to |rho| / sigma max(v0, theta) 2^-53 times the few
roundings (8) of v on both sides.
"""
import numpy as np
import pytest

from hestonexotics_gb300 import engine as E

pytestmark = pytest.mark.gpu

#                          v0, theta, rho, kappa, sigma, r, q; T, steps; line: log2 of what, below or above
SETS = {
    "ratio below 2^-40": ((0.04, 0.05, -0.5, 1.5, 4e-7, 0.02, 0.0), 1.0, 50, ("ratio", -40, -1)),
    "ratio above 2^-40": ((0.04, 0.05, -0.5, 1.5, 4e-6, 0.02, 0.0), 1.0, 50, ("ratio", -40, 1)),
    "mean below 2^30": ((0.8e9, 0.8e9, 0.3, 1e7, 1e9, 0.0, 0.0), 1e-9, 10, ("m", 30, -1)),
    "mean above 2^30": ((1.4e9, 1.4e9, 0.3, 1e7, 1e9, 0.0, 0.0), 1e-9, 10, ("m", 30, 1)),
    "s^2 below 2^60": ((0.9e9, 0.9e9, 0.3, 1e7, 1.5e9, 0.0, 0.0), 1e-9, 10, ("s2", 60, -1)),
    "s^2 above 2^60": ((0.9e9, 0.9e9, 0.3, 1e7, 8e9, 0.0, 0.0), 1e-9, 10, ("s2", 60, 1)),
    "mean below 2^-30": ((2e-10, 2e-10, -0.5, 2.0, 3e-3, 0.01, 0.0), 1.0, 20, ("m", -30, -1)),
    "mean above 2^-30": ((4e-9, 4e-9, -0.5, 2.0, 3e-3, 0.01, 0.0), 1.0, 20, ("m", -30, 1)),
    "s^2 below 2^-60": ((4e-9, 4e-9, -0.5, 2.0, 2e-5, 0.01, 0.0), 1.0, 40, ("s2", -60, -1)),
    "s^2 above 2^-60": ((4e-9, 4e-9, -0.5, 2.0, 2e-3, 0.01, 0.0), 1.0, 40, ("s2", -60, 1)),
    "log spot to -500": ((90.0, 90.0, -0.5, 1.0, 2.0, 0.0, 0.0), 9.0, 60, None),
    "log spot past -512": ((180.0, 180.0, -0.5, 1.0, 2.0, 0.0, 0.0), 9.0, 60, None),
}


@pytest.mark.parametrize("name", SETS)
def test_prices_on_either_side(engine, oracle, name):
    p, T, steps, line = SETS[name]
    v0, theta, rho, kappa, sigma, r, q = p
    if line is not None:
        om = -np.expm1(-kappa * T / steps)
        m = np.array([v0, theta])
        s2 = sigma ** 2 * om / kappa * ((1 - om) * m + theta * om / 2)
        x = np.log2({"m": m, "s2": s2, "ratio": s2 / m ** 2}[line[0]])
        assert (np.sign(x - line[1]) == line[2]).all(), x
    n, S0 = 1500, 100.0
    K = np.array([0.0, 60.0, 95.0, 100.0, 110.0, 180.0] * 2)
    kind = np.repeat([E.ASIAN, E.EUROPEAN], 6).astype(np.uint32)
    opts = E.Options(K, T, kind)
    price, _ = engine.price(E.Params(*p), S0, opts, E.Config(n_paths=n, steps=steps, seed=21))
    want, _, _ = oracle.price_paths(np.array(p), S0, K, opts.T, kind.astype(np.uint8), n_default=n, steps=steps, seed=21)
    assert np.isfinite(want).all()
    magnified = steps * abs(rho) / sigma * max(v0, theta) * 8 * 2.0 ** -53
    np.testing.assert_allclose(price, want, rtol=1e-10, atol=S0 * (1e-12 + magnified))


@pytest.mark.parametrize("steps,T", [(1, 0.5), (30, 0.001)])
@pytest.mark.parametrize("v0,theta,kappa", [(1e-20, 0.04, 1e-17), (1e-30, 50.0, 1e-18), (1e-12, 1e6, 1e-17)])
def test_reversion_below_a_last_bit(engine, oracle, v0, theta, kappa, steps, T):
    # exp(-kappa dt) is 1: the reference's theta + (v - theta) disc loses v0 beside theta, the mean and s^2 are 0, and
    # the variance stays 0.  Outside its own functions' range the step has to branch on that mean, not on v0's.
    p = (v0, theta, -0.5, kappa, 0.3, 0.01, 0.0)
    assert np.exp(-kappa * T / steps) == 1.0 and (v0 - theta) + theta == 0.0
    K = np.array([0.0, 60.0, 95.0, 100.0] * 2)
    kind = np.repeat([E.ASIAN, E.EUROPEAN], 4).astype(np.uint32)
    opts = E.Options(K, T, kind)
    price, _ = engine.price(E.Params(*p), 100.0, opts, E.Config(n_paths=200, steps=steps, seed=3))
    want, _, _ = oracle.price_paths(np.array(p), 100.0, K, opts.T, kind.astype(np.uint8), n_default=200, steps=steps, seed=3)
    assert want[4] > 99.0   # a European call struck at 0 is the spot
    np.testing.assert_allclose(price, want, rtol=1e-10, atol=1e-10)
