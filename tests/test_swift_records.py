"""What Engine.swift_batch hands to the C ABI (CPU: the library call is recorded).

A chain record's fields take the same values, and refuse the same ones, as a
ctypes record does: a truncation precision is a real number (no text, None or
array), a method is any integer modulo 2^32, for the library to refuse.
"""
import ctypes as C

import numpy as np
import pytest

from hestonexotics_gb300 import _lib as L
from hestonexotics_gb300.engine import Engine, Params

P = Params(0.04, 0.05, -0.6, 1.5, 0.5, 0.02)
K = [90.0, 100.0, 110.0]


class Recorder:
    def __init__(self):
        self.chains = []

    def hexo_swift_price(self, ctx, reqs, n):
        for q in range(n):
            for c in range(reqs[q].n_chains):
                ch = reqs[q].chains[c]
                self.chains.append({"tau": ch.tau, "method": ch.method, "trunc": ch.trunc_precision,
                                    "strikes": [ch.strikes[i] for i in range(ch.n)],
                                    "params": ch.params.contents.J if ch.params else None, "grad": bool(ch.grad_out)})
                for i in range(ch.n):
                    ch.price_out[i] = 10.0 * len(self.chains) + i
        return 0


@pytest.fixture
def eng():
    e = object.__new__(Engine)
    e._lib, e._ctx = Recorder(), None   # no context: nothing to close
    e._check = lambda status: None
    return e


def test_records(eng):
    sp = [None, (4, 16, 4.0, -3.0, 3.0, -48, 47, 32)]
    out = eng.swift_batch([(P, 100.0, [(0.5, K), (1.0, K[:1])]), (P, 90.0, []), (P, 80.0, [(2.0, [])])], True,
                          [sp, None, None], 1e-9, 2)
    assert eng._lib.chains == [
        {"tau": 0.5, "method": 2, "trunc": 1e-9, "strikes": K, "params": None, "grad": True},
        {"tau": 1.0, "method": 2, "trunc": 1e-9, "strikes": K[:1], "params": 32, "grad": True},
        {"tau": 2.0, "method": 2, "trunc": 1e-9, "strikes": [], "params": None, "grad": True}]
    assert [[(p.tolist(), g.shape) for p, g in res] for res in out] == [
        [([10.0, 11.0, 12.0], (3, 5)), ([20.0], (1, 5))], [], [([], (0, 5))]]


@pytest.mark.parametrize("bad", [None, "1e-7", np.array([1e-7, 1e-3]), [1e-7]])
def test_truncation_precision_is_a_number(eng, bad):
    with pytest.raises(TypeError):
        eng.swift_batch([(P, 100.0, [(0.5, K), (1.0, K)])], trunc_precision=bad)
    assert eng._lib.chains == []


@pytest.mark.parametrize("ok,value", [(0, 0.0), (1e-7, 1e-7), (np.float32(0.5), 0.5), (True, 1.0)])
def test_truncation_precision_of_any_number_type(eng, ok, value):
    eng.swift_batch([(P, 100.0, [(0.5, K)])], trunc_precision=ok)
    assert eng._lib.chains[0]["trunc"] == value


@pytest.mark.parametrize("method,field", [(0, 0), (7, 7), (-1, 0xFFFFFFFF), (1 << 33, 0), (1.9, 1)])
def test_method_reaches_the_library(eng, method, field):
    eng.swift_batch([(P, 100.0, [(0.5, K)])], method=method)
    assert eng._lib.chains[0]["method"] == field


def test_pairs_are_read_once(eng):
    # a chain given as a one-shot iterator, as unpacking a pair accepts
    (price,), = eng.swift_batch([(P, 100.0, [iter((0.5, K))])])
    assert price.tolist() == [10.0, 11.0, 12.0]
