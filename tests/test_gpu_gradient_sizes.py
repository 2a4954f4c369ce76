"""Gradients at the smallest sizes (one single excitation, one atom pair, kinds with and without p
orbitals) and around the blocks of the Z-vector's reductions, against the oracle."""

import numpy as np
import pytest

import cases as TC
from tincr_gb300 import _lib
from tincr_gb300 import geometry as G
from tincr_gb300 import gradients as GR
from tincr_gb300 import groundstate as gs
from tincr_gb300 import tda as T

# H2 has one single excitation; NH3 + H2O mixes H, N and O; the acenes have 225 (one reduction block of
# 256), 576 and 1089 single excitations
MOLECULES = {
    "h2": lambda: (np.array([1, 1]), np.array([[0.0, 0, 0], [0.1, 0.2, 0.71]])),
    "nh3-h2o": lambda: (np.array([7, 1, 1, 1, 8, 1, 1]),
                        np.array([[0, 0, 0], [0.94, 0, 0.38], [-0.47, 0.81, 0.38], [-0.47, -0.81, 0.38],
                                  [0.1, 0.2, -2.8], [0.8, 0.3, -3.4], [-0.6, 0.3, -3.4]])),
    "acene1": lambda: G.acene(1), "acene2": lambda: G.acene(2), "acene3": lambda: G.acene(3),
}


@pytest.mark.gpu
@pytest.mark.parametrize("lc", [True, False])
@pytest.mark.parametrize("name", sorted(MOLECULES))
def test_gradients_of_small_systems(name, lc):
    from oracle import gradients as OG
    z, x = MOLECULES[name]()
    sy = gs.build_system(z, G.to_bohr(x + np.random.default_rng(3).uniform(-0.02, 0.02, size=x.shape)), lc=lc)
    g = gs.run_scc(sy, tol=1e-11)
    om = (g.orbe[sy.n_occ:][None, :] - g.orbe[:sy.n_occ, None]).ravel()
    v = np.exp(-3.0 * (om - om.min())) * np.cos(np.arange(om.size))
    e, v = np.array([0.8 * om.min()]), (v / np.linalg.norm(v)).reshape(-1, 1)
    es = T.ExcitedStateSystem.from_ground_state(_lib.Context(0), sy, g)
    es.set_states(e, v)
    got = GR.GradientSystem(es, sy, g).both(0)
    inp = TC.oracle_gradient_inputs(sy, g, lc, e, v)
    inp["gamma_ao"] = gs.atom_to_ao(sy, g.gamma)
    der = OG.derivative_tensors(sy.numbers, sy.xyz, sy.ao_offset, sy.ao_atom, sy.hubbard, sy.r_lr, sy.params)
    ref_gs, flr = OG.ground_state_gradient(inp, der, lc)
    ref_ex = OG.tda_gradient(inp, der, 0, lc, flr)
    # the Z-vector stops at r.r <= 1e-19 in both, which leaves about 3e-10 / gap in Z
    assert np.max(np.abs(got[0] - ref_gs)) < 1e-11
    assert np.max(np.abs(got[1] - ref_ex)) < 1e-8
