"""A.X products of synthetic systems at the sizes where the GEMM tiles end, against numpy in 64 bits.

The orbitals are random matrices (the product's formula does not need orthonormal ones).  Each result
is a chain of four matrix products; its rounding error is bounded element by element by
(total length of the sums) * eps * the same chain on absolute values, which is the tolerance."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import tda as T

# (orbitals, occupied, virtual, vectors): one tile and less, tile edges and one past them, odd sizes,
# few vectors (small FP64 tiles) and many; the last rows have enough work for the digit GEMMs (also in
# more than one chunk of vectors)
SIZES = [(4, 1, 3, 1), (16, 8, 8, 1), (17, 8, 9, 2), (33, 16, 17, 1), (48, 24, 24, 1), (65, 32, 33, 20), (96, 64, 32, 3),
         (102, 51, 51, 5), (129, 64, 65, 2), (200, 99, 101, 7), (261, 130, 131, 1), (330, 200, 130, 11),
         (17, 8, 9, 2200), (65, 32, 33, 70), (128, 64, 64, 12), (129, 64, 65, 12), (96, 31, 65, 20)]


def _system(n, o, v, lc, seed):
    rng = np.random.default_rng(seed)
    opa = []
    while sum(opa) < n:
        opa.append(min(int(rng.integers(1, 5)), n - sum(opa)))
    na = len(opa)
    sym = lambda m: (m + m.T) / 2
    return dict(opa=np.array(opa, np.int32), c=rng.normal(size=(n, n)) * np.exp(rng.normal(size=(n, 1))),
                s=np.eye(n) + 0.1 * sym(rng.normal(size=(n, n))), orbe=np.sort(rng.normal(size=n)),
                gamma=sym(rng.random((na, na))), glr=sym(rng.random((na, na))) if lc else None,
                xyz=rng.normal(size=(na, 3)))


def _chain(q, n, o, v, x, absolute):
    """A.X for the columns of x, or the same chain with absolute values."""
    f = np.abs if absolute else (lambda m: m)
    c, om = f(q["c"]), f((q["orbe"][None, o:o + v] - q["orbe"][:o, None]))
    sc = f(q["s"]) @ c
    at = np.repeat(np.arange(len(q["opa"])), q["opa"])
    out = np.empty_like(x)
    for j in range(x.shape[1]):
        xj = f(x[:, j].reshape(o, v))
        m = np.vstack([c[:, :o], sc[:, :o]]) @ xj @ np.vstack([c[:, o:o + v], sc[:, o:o + v]]).T
        i = np.arange(n)
        z = (f(q["gamma"]) @ np.bincount(at, 0.5 * (m[i, n + i] + m[n + i, i]), len(q["opa"])))[at]
        g = np.zeros((2 * n, 2 * n))
        if q["glr"] is not None:
            g = (0.25 if absolute else -0.25) * np.tile(f(q["glr"])[np.ix_(at, at)], (2, 2)) * m
        g[i, n + i] += z
        g[n + i, i] += z
        out[:, j] = (om * xj + np.vstack([sc[:, :o], c[:, :o]]).T @ g @ np.vstack([sc[:, o:o + v], c[:, o:o + v]])).ravel()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("lc", [True, False])
@pytest.mark.parametrize("n,o,v,k", SIZES)
def test_products_at_tile_edges(n, o, v, k, lc):
    q = _system(n, o, v, lc, 1000 * n + k)
    x = np.random.default_rng(k).normal(size=(o * v, k))
    ctx = _lib.Context(0)
    es = T.ExcitedStateSystem(ctx, q["opa"], q["c"], q["s"], q["orbe"], o, v, q["gamma"], q["glr"], q["xyz"])
    got = es.compute_products(x)
    # S C, C X, M, gamma y (and its sums over AOs), F C, out
    terms = 2 * n + o + v + 2 * n + 2 * n + 2 * len(q["opa"]) + 20
    tol = terms * np.finfo(float).eps * _chain(q, n, o, v, x, True)
    assert np.all(np.abs(got - _chain(q, n, o, v, x, False)) <= tol)


@pytest.mark.gpu
@pytest.mark.parametrize("n,o,v,k", [(33, 16, 17, 2), (129, 64, 65, 12)])
def test_products_scale_exactly(n, o, v, k):
    """A power of two times X gives exactly that multiple of A.X, far from 1 too; zero gives zero."""
    q = _system(n, o, v, True, n)
    ctx = _lib.Context(0)
    es = T.ExcitedStateSystem(ctx, q["opa"], q["c"], q["s"], q["orbe"], o, v, q["gamma"], q["glr"], q["xyz"])
    x = np.random.default_rng(k).normal(size=(o * v, k))
    x[:, 1] = 0.0
    got = es.compute_products(x)
    assert np.all(got[:, 1] == 0.0) and np.all(np.isfinite(got))
    for p in (-400, 300):
        assert np.array_equal(es.compute_products(np.ldexp(x, p)), np.ldexp(got, p))
