"""The FP64 form's roots, quotients, log and exp at the ends of their ranges.

The step takes them from double-single seeds corrected with integer
remainders while the mean m of the next variance lies in [2^-30, 2^30) and
s^2 in [2^-60, 2^60) and above 2^-40 m^2, and from the plain double operations
outside; the
log-spot's root is clamped at 2^-120 and its exponential tabulated below 512.
The parameter sets here put paths on both sides of each of those lines.  The
oracle prices the same streams; the tolerance is the one the FP64 form is held
to everywhere, 1e-10 relative (1e-12 S0 for prices that are essentially zero).
"""
import numpy as np
import pytest

from hestonexotics_gb300 import engine as E

pytestmark = pytest.mark.gpu

#        v0, theta, rho, kappa, sigma, r, q
SETS = {
    "variance starts at zero": (0.0, 0.04, -0.7, 1.5, 0.5, 0.02, 0.0),
    "mean below 2^-30": (1e-12, 1e-12, -0.5, 2.0, 1e-3, 0.01, 0.0),
    "mean around 2^-30, s2 below 2^-60": (1e-9, 1e-9, -0.5, 2.0, 1e-4, 0.01, 0.0),
    "rho = -1, no noise of its own in the spot": (0.04, 0.05, -1.0, 1.2, 0.4, 0.02, 0.01),
    "rho = 1": (0.02, 0.03, 1.0, 2.0, 0.3, 0.0, 0.0),
    "vol-of-vol far beyond Feller": (0.04, 0.02, -0.9, 0.3, 4.0, 0.03, 0.0),
    "fast reversion": (0.5, 0.09, -0.2, 60.0, 1.5, 0.05, 0.02),
    "variance of order one": (2.0, 1.5, -0.6, 0.8, 1.0, 0.0, 0.0),
}


@pytest.mark.parametrize("steps,T", [(1, 0.1), (5, 4.0), (63, 0.25), (500, 2.0)])
@pytest.mark.parametrize("name", SETS)
def test_fp64_prices_at_the_ends_of_the_ranges(engine, oracle, name, steps, T):
    n, S0 = 1500, 100.0
    K = np.array([0.0, 60.0, 95.0, 100.0, 110.0, 180.0] * 2)
    kind = np.repeat([E.ASIAN, E.EUROPEAN], 6).astype(np.uint32)
    opts = E.Options(K, T, kind)
    cfg = E.Config(n_paths=n, steps=steps, seed=77)
    p, se = engine.price(E.Params(*SETS[name]), S0, opts, cfg)
    op, ose, _ = oracle.price_paths(np.array(SETS[name]), S0, K, opts.T, kind.astype(np.uint8), n_default=n, steps=steps,
                                    seed=77)
    np.testing.assert_allclose(p, op, rtol=1e-10, atol=1e-12 * S0)


@pytest.mark.parametrize("S0", [2.0 ** -60, 1e-3, 1e8, 2.0 ** 59])
@pytest.mark.parametrize("cv", [0, 1])
def test_fp64_prices_at_the_ends_of_the_spots(engine, oracle, S0, cv):
    n = 1000
    prm = (0.04, 0.04, -0.7, 1.5, 0.5, 0.02, 0.0)
    K = S0 * np.array([0.5, 0.9, 1.0, 1.1, 2.0])
    T = np.array([0.3, 0.3, 1.0, 1.0, 1.0])
    opts = E.Options(K, T, E.ASIAN)
    cfg = E.Config(n_paths=n, steps=40, seed=5, control_variate=cv)
    p, se = engine.price(E.Params(*prm), S0, opts, cfg)
    if cv:
        plain, pse = engine.price(E.Params(*prm), S0, opts, E.Config(n_paths=n, steps=40, seed=5))
        assert np.all(np.isfinite(p)) and np.all(np.abs(p - plain) <= 5 * pse + 1e-12 * S0)
        return
    op, _, _ = oracle.price_paths(np.array(prm), S0, K, T, np.zeros(5, dtype=np.uint8), n_default=n, steps=40, seed=5)
    np.testing.assert_allclose(p, op, rtol=1e-10, atol=1e-12 * S0)
