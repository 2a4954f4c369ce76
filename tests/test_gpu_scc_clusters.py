"""The batched SCC at every number of CTAs per system: batches from one system (16 CTAs) to more
systems than CTAs fit (1 CTA), of molecules from 2 to 66 orbitals, against the host SCC."""

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
