"""The batched SCC at every number of CTAs per system: batches from one system (16 CTAs) to more
systems than CTAs fit (2 CTAs), of molecules from 2 to 66 orbitals, against the host SCC; the products
and densities of the larger ones run on digits and by purification."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import geometry as G
from tincr_gb300 import groundstate as gs
from tincr_gb300 import scc as gscc

_HOST = {}


def _molecules(lc):
    """(System, host ground state) of H2, H2O, a stretched H2O pair, benzene-like and three-ring acenes."""
    if lc not in _HOST:
        z1, x1 = G.water_cluster(1, 1, 1)
        z2, x2 = G.water_cluster(2, 1, 1, seed=3)
        mols = [(np.array([1, 1]), np.array([[0.0, 0, 0], [0.74, 0, 0]])), (z1, x1), (z2, x2), G.acene(1), G.acene(3)]
        rng = np.random.default_rng(5)
        out = []
        for z, x in mols:
            sy = gs.build_system(z, G.to_bohr(x + rng.uniform(-0.02, 0.02, size=x.shape)), lc=lc)
            out.append((sy, gs.run_scc(sy, tol=1e-11)))
        _HOST[lc] = out
    return _HOST[lc]


@pytest.mark.gpu
@pytest.mark.parametrize("lc", [True, False])
@pytest.mark.parametrize("count", [1, 20, 40, 80, 160, 330])
def test_scc_of_batches_of_every_size(count, lc):
    mols = _molecules(lc)
    pick = [(4 - i) % 5 for i in range(count)]
    got, rc = gscc.scc_batch(_lib.Context(0), [mols[k][0] for k in pick], tol=1e-11)
    assert rc == _lib.OK
    for k, g in zip(pick, got):
        h = mols[k][1]
        # both stop at a commutator below 1e-11, which leaves ~1e-11 / gap in the density
        assert abs(g.energy - h.energy) < 1e-11
        assert np.max(np.abs(g.orbe - h.orbe)) < 1e-9
        assert np.max(np.abs(g.p - h.p)) < 1e-9
        assert np.max(np.abs(g.h_coul_x - h.h_coul_x)) < 1e-9
        assert np.max(np.abs(g.orbs.T @ h.s @ g.orbs - np.eye(len(h.orbe)))) < 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("rings", [4, 5, 7, 10])
def test_scc_of_larger_systems(rings):
    """84, 102, 138 and 192 orbitals: one and two chunks of 128 k, ragged 16 x 8 tiles."""
    z, x = G.acene(rings)
    sy = gs.build_system(z, G.to_bohr(x + np.random.default_rng(rings).uniform(-0.03, 0.03, size=x.shape)))
    h = gs.run_scc(sy, tol=1e-11)
    got, rc = gscc.scc_batch(_lib.Context(0), [sy], tol=1e-11)
    assert rc == _lib.OK
    assert abs(got[0].energy - h.energy) < 1e-10
    assert np.max(np.abs(got[0].orbe - h.orbe)) < 1e-9
    assert np.max(np.abs(got[0].p - h.p)) < 1e-9
    assert np.max(np.abs(got[0].orbs.T @ h.s @ got[0].orbs - np.eye(len(h.orbe)))) < 1e-11


@pytest.mark.gpu
def test_scc_without_a_gap():
    """Two H atoms beyond the range of the integrals: occupied and virtual level coincide, so there is no
    density to purify to; the iterations fall back on the eigenpairs and end in a finite result."""
    sy = gs.build_system(np.array([1, 1]), np.array([[0.0, 0, 0], [15.0, 0, 0]]))
    got, rc = gscc.scc_batch(_lib.Context(0), [sy], tol=1e-10, max_iter=30)
    assert rc in (_lib.OK, _lib.NOT_CONVERGED)
    assert np.isfinite(got[0].energy) and np.all(np.isfinite(got[0].orbe))
