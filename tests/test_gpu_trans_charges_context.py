"""Transition charges of another molecule leave the system that a context was set up with as it is: its products,
roots and gradients come out as before."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import geometry as G
from tincr_gb300 import gradients as GR
from tincr_gb300 import groundstate as gs
from tincr_gb300 import tda as T

_GROUND = {}


def _molecule(rings, seed):
    if (rings, seed) not in _GROUND:
        z, x = G.acene(rings)
        x = x + np.random.default_rng(seed).uniform(-0.03, 0.03, size=x.shape)
        sy = gs.build_system(z, G.to_bohr(x))
        _GROUND[rings, seed] = (sy, gs.run_scc(sy, tol=1e-10))
    return _GROUND[rings, seed]


@pytest.mark.gpu
@pytest.mark.parametrize("rings", [2, 1, 3])   # as many orbitals as the system, fewer, more
def test_charges_of_another_molecule(gpu_ctx, rings):
    sy, g = _molecule(2, 1)
    other, go = _molecule(rings, 2)
    es = T.ExcitedStateSystem.from_ground_state(gpu_ctx, sy, g)
    x = np.random.default_rng(3).normal(size=(sy.n_occ * sy.n_virt, 3))

    def results():
        r = es.run_tda(3, 200, 1e-8)
        grads = GR.GradientSystem(es, sy, g).both(0)
        return [es.compute_products(x), r["ci_eigenvalues"].copy(), r["ci_coefficients"].copy()] + [q.copy() for q in grads]

    def after():   # without a solve in between: what the context holds
        return [es.compute_products(x)] + [q.copy() for q in GR.GradientSystem(es, sy, g).both(0)]

    first = results()
    q = T.trans_charges(gpu_ctx, other.orbs_per_atom, go.orbs, go.s, np.arange(other.n_occ),
                        np.arange(other.n_occ, other.n_orbs))
    again = after()
    for a, b in zip([first[0]] + first[3:], again):
        assert np.array_equal(a, b)
    for a, b in zip(first, results()):
        assert np.array_equal(a, b)
    # and the charges themselves do not depend on the context's system
    ctx = _lib.Context(0)
    try:
        for a, b in zip(q, T.trans_charges(ctx, other.orbs_per_atom, go.orbs, go.s, np.arange(other.n_occ),
                                           np.arange(other.n_occ, other.n_orbs))):
            assert np.array_equal(a, b)
    finally:
        ctx.close()
