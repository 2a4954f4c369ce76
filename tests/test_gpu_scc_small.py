"""Batches of small systems in the batched SCC at every number of CTAs per system, one included: against the
host SCC, and as fast in a batch that fills the GPU once as alone."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import geometry as G
from tincr_gb300 import groundstate as gs
from tincr_gb300 import scc as gscc

# 2, 6, 12, 18, 24, 30, 48, 66 and 84 orbitals
MOLECULES = {"h2": lambda: (np.array([1, 1]), np.array([[0.0, 0, 0], [0.74, 0, 0]])),
             "water1": lambda: G.water_cluster(1, 1, 1), "water2": lambda: G.water_cluster(2, 1, 1),
             "water3": lambda: G.water_cluster(3, 1, 1), "water4": lambda: G.water_cluster(2, 2, 1),
             "acene1": lambda: G.acene(1), "acene2": lambda: G.acene(2), "acene3": lambda: G.acene(3),
             "acene4": lambda: G.acene(4)}
_HOST = {}


def _systems(name, lc):
    """Four geometries of a molecule and their host ground states."""
    if (name, lc) not in _HOST:
        z, x = MOLECULES[name]()
        rng = np.random.default_rng(len(z))
        sys_ = [gs.build_system(z, G.to_bohr(x + rng.uniform(-0.02, 0.02, size=x.shape)), lc=lc) for _ in range(4)]
        _HOST[name, lc] = [(sy, gs.run_scc(sy, tol=1e-11)) for sy in sys_]
    return _HOST[name, lc]


@pytest.mark.gpu
@pytest.mark.parametrize("lc", [True, False])
@pytest.mark.parametrize("count", [1, 5, 20, 40, 77, 153, 310])
@pytest.mark.parametrize("name", sorted(MOLECULES))
def test_scc_of_equal_small_systems(gpu_ctx, name, count, lc):
    ref = _systems(name, lc)
    got, rc = gscc.scc_batch(gpu_ctx, [ref[i % 4][0] for i in range(count)], tol=1e-11)
    assert rc == _lib.OK
    for i, g in enumerate(got):
        h = ref[i % 4][1]
        # both stop at a commutator below 1e-11, which leaves ~1e-11 / gap in the density
        assert abs(g.energy - h.energy) < 1e-11
        assert np.max(np.abs(g.orbe - h.orbe)) < 1e-9
        assert np.max(np.abs(g.p - h.p)) < 1e-9
        assert np.max(np.abs(g.orbs.T @ h.s @ g.orbs - np.eye(len(h.orbe)))) < 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["water1", "water2"])
def test_a_full_gpu_of_small_systems_takes_about_the_time_of_one(gpu_ctx, name):
    """Two CTAs of each of 152 SMs take a system each, so 304 of them are one wave."""
    z, x = MOLECULES[name]()
    sy = gs.build_system(z, G.to_bohr(x))
    ms = {}
    for count in (1, 304):
        t = []
        for _ in range(7):
            gscc.scc_batch(gpu_ctx, [sy] * count, tol=1e-10, full=False)
            t.append(gscc.last_ms(gpu_ctx))
        ms[count] = min(t)
    assert ms[304] < 1.8 * ms[1], ms


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 40, 310])
@pytest.mark.parametrize("name", ["h2", "water2", "acene1", "acene3"])
def test_scc_fp32_start_of_small_systems(gpu_ctx, name, count):
    ref = _systems(name, True)
    got, rc = gscc.scc_batch(gpu_ctx, [ref[i % 4][0] for i in range(count)], tol=1e-11, fp32_start=True)
    assert rc == _lib.OK
    for i, g in enumerate(got):
        h = ref[i % 4][1]
        assert abs(g.energy - h.energy) < 1e-11
        assert np.max(np.abs(g.p - h.p)) < 1e-9
