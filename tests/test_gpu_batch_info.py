"""hexo_batch_info counts the bytes that a run copies back.

One copy brings the control block and the outputs as they lie on the device:
the status, the prices and the standard errors, each from a 256-byte boundary.
"""
import numpy as np
import pytest

from hestonexotics_gb300 import engine as E

pytestmark = pytest.mark.gpu


def up256(n):
    return (n + 255) // 256 * 256


@pytest.mark.parametrize("cv", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 200])
def test_bytes_copied_back(engine, n, cv):
    opts = E.Options(np.linspace(80.0, 120.0, n), 1.0, E.ASIAN)
    cfg = E.Config(n_paths=64, steps=5, control_variate=cv)
    b = engine.prepare_batch([E.Request(E.Params(0.04, 0.04, -0.7, 1.5, 0.5, 0.02), 100.0, opts)], cfg)
    slots = n * (3 if cv else 1)   # the control variate's two sums per option have slots of their own
    assert b.info()["d2h_bytes"] == 256 + up256(8 * slots) + 8 * slots
    b.close()
