"""The two forms of the FP64 contraction on one input: TINCR_GB300_CONTRACTION=fp64 selects the FP64 tiles for all
work, and the switch of the Davidson's subspace products leaves the contraction alone."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import tda as T
from test_gpu_product_sizes import _chain, _system

N, O, V, K = 128, 64, 64, 24   # 252e6 multiply-adds with exchange, 50e6 without: digit GEMMs


def _products(monkeypatch, lc, x, **env):
    for name in ("TINCR_GB300_CONTRACTION", "TINCR_GB300_SUBSPACE_GEMM"):
        monkeypatch.delenv(name, raising=False)
    for name, value in env.items():
        monkeypatch.setenv(name, value)
    q = _system(N, O, V, lc, 7)
    ctx = _lib.Context(0)
    try:
        return T.ExcitedStateSystem(ctx, q["opa"], q["c"], q["s"], q["orbe"], O, V, q["gamma"], q["glr"],
                                    q["xyz"]).compute_products(x)
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("lc", [True, False])
def test_contraction_switch(monkeypatch, lc):
    x = np.random.default_rng(3).normal(size=(O * V, K))
    digits = _products(monkeypatch, lc, x)
    assert np.array_equal(digits, _products(monkeypatch, lc, x, TINCR_GB300_SUBSPACE_GEMM="fp64"))
    tiles = _products(monkeypatch, lc, x, TINCR_GB300_CONTRACTION="fp64")
    assert not np.array_equal(digits, tiles)
    # each form is within (total length of the sums) eps of the chain on absolute values
    q = _system(N, O, V, lc, 7)
    terms = 6 * N + O + V + 2 * len(q["opa"]) + 20
    tol = terms * np.finfo(float).eps * _chain(q, N, O, V, x, True)
    assert np.all(np.abs(digits - tiles) <= 2.0 * tol)
    assert np.all(np.abs(tiles - _chain(q, N, O, V, x, False)) <= tol)
