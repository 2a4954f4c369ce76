"""The FP64 contraction far from 1: results in the last binade, beyond it, and subnormal ones, on both sides of
the number of multiply-adds from which it runs on digits."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import tda as T
from test_gpu_product_sizes import _chain, _system

SIZES = [(33, 16, 17, 2), (96, 31, 65, 20), (128, 64, 64, 24)]   # FP64 tiles, digit GEMMs twice


def _solver(n, o, v, lc, occupied=1.0):
    q = _system(n, o, v, lc, n)
    q["c"][:, :o] *= occupied
    ctx = _lib.Context(0)
    return q, T.ExcitedStateSystem(ctx, q["opa"], q["c"], q["s"], q["orbe"], o, v, q["gamma"], q["glr"], q["xyz"])


def _largest_exponents(q, n, o, v, x):
    """Largest binary exponents of A.X and of all values formed on the way."""
    c = q["c"]
    sc = q["s"] @ c
    at = np.repeat(np.arange(len(q["opa"])), q["opa"])
    seen = np.abs(x).max()
    for j in range(x.shape[1]):
        h = np.vstack([c[:, :o], sc[:, :o]]) @ x[:, j].reshape(o, v)
        m = h @ np.vstack([c[:, o:o + v], sc[:, o:o + v]]).T
        i = np.arange(n)
        y = np.bincount(at, np.abs(m[i, n + i]) + np.abs(m[n + i, i]), len(q["opa"]))
        f = np.abs(m) + (np.abs(q["gamma"]) @ y).max()
        g = np.abs(f) @ np.abs(np.vstack([sc[:, o:o + v], c[:, o:o + v]]))
        seen = max(seen, np.abs(h).max(), f.max(), g.max())
    return int(np.frexp(np.abs(_chain(q, n, o, v, x, False)).max())[1]), int(np.frexp(seen)[1])


@pytest.mark.gpu
@pytest.mark.parametrize("lc", [True, False])
@pytest.mark.parametrize("n,o,v,k", SIZES)
def test_products_up_to_the_largest_double(n, o, v, k, lc):
    q, es = _solver(n, o, v, lc, 2.0 ** 12)   # the last product, with the occupied orbitals again, is the largest
    x = np.random.default_rng(5).normal(size=(o * v, k))
    x[:, 1] *= 2.0 ** -30   # stays in range when the others leave it
    y = es.compute_products(x)
    top, way = _largest_exponents(q, n, o, v, x)
    assert top > way
    # a power of two times X: exactly that multiple, up to the last binade
    p = 1024 - top
    assert np.array_equal(es.compute_products(np.ldexp(x, p)), np.ldexp(y, p))
    assert np.frexp(np.abs(np.ldexp(y, p)).max())[1] == 1024
    for p in range(1025 - top, 1025 - top + 40, 3):
        got = es.compute_products(np.ldexp(x, min(p, 1020)))
        with np.errstate(over="ignore"):
            want = np.ldexp(y, min(p, 1020))
        # what is out of range is not finite, what is finite is right
        assert not np.any(np.isfinite(got) & ~np.isfinite(want))
        fine = np.isfinite(got)
        assert np.array_equal(got[fine], want[fine])
        # the column far below is not touched by the others
        if np.all(np.isfinite(want[:, 1])) and p < 1024 - top + 28:
            assert np.array_equal(got[:, 1], want[:, 1])


@pytest.mark.gpu
@pytest.mark.parametrize("lc", [True, False])
@pytest.mark.parametrize("n,o,v,k", SIZES)
def test_subnormal_products(n, o, v, k, lc):
    q, es = _solver(n, o, v, lc)
    x0 = np.random.default_rng(6).normal(size=(o * v, k))
    terms = 6 * n + o + v + 2 * len(q["opa"]) + 20
    # a unit in the last subnormal place at every value on the way, through the rest of the chain
    unit = _chain(q, n, o, v, np.ones((o * v, 1)), True).max()
    for p in (-1010, -1030, -1045, -1060, -1070):
        x = np.ldexp(x0, p)
        want = np.ldexp(_chain(q, n, o, v, np.ldexp(x, 600), False), -600)
        tol = terms * np.finfo(float).eps * np.ldexp(_chain(q, n, o, v, np.ldexp(x, 600), True), -600) + 4.0 * np.ldexp(unit, -1074)
        got = es.compute_products(x)
        assert np.all(np.abs(got - want) <= tol), p
        assert np.abs(got).max() > 0.5 * np.abs(want).max() > 0.0
