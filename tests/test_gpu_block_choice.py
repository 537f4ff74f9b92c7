"""The CTA width chosen for one uniform set changes no result.

Path counts around a scheduler's first warp, the SMs' first round of CTAs and
the next one, where the engine takes 96 to 256 threads: the prices and
standard errors are those of 256-thread CTAs bit for bit, and the batch's
tiles cover every path once (a set's nominal path-steps are the same).
"""
import numpy as np
import pytest

from hestonexotics_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [E.FP64, E.FP32])
@pytest.mark.parametrize("n", [1, 31, 129, 19457, 38913, 50000, 77825, 80000, 131073, 200001])
def test_width_changes_nothing(engine, n, precision):
    prm = E.Params(0.04, 0.04, -0.7, 1.5, 0.5, 0.02)
    opts = E.Options(np.array([90.0, 100.0, 110.0]), np.array([0.5, 1.0, 1.0]), E.ASIAN)
    got = []
    for block in (0, 256):
        cfg = E.Config(n_paths=n, steps=12, seed=9, precision=precision, block=block)
        b = engine.prepare_batch([E.Request(prm, 100.0, opts, seed=9)], cfg)
        b.launch()
        (p, se), = b.collect()
        got.append((p.copy(), se.copy(), b.info()["nominal_path_steps"], b.info()["n_paths"]))
        b.close()
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)
