"""The Davidson's Gram-Schmidt of new vectors, at correction counts on both sides of each group of eight rows
up to the 32 of the cooperative kernel, against the oracle."""

import numpy as np
import pytest

from cases import oracle_inputs, synthetic_case
from oracle import tda as OT
from tincr_gb300 import tda as T


@pytest.mark.gpu
@pytest.mark.parametrize("n_roots", [1, 7, 8, 9, 16, 17, 25, 32, 33])
def test_davidson_at_every_correction_count(gpu_ctx, n_roots):
    c = synthetic_case("water8", True)
    o = oracle_inputs(c)
    ref = OT.run_tda(o["omega"], o["q_ov"], o["gamma"], c["xyz"], n_roots, 200, 1e-8, o["q_oo"], o["q_vv"],
                     o["gamma_lr"], o["n_occ"], o["n_virt"])
    es = T.ExcitedStateSystem(gpu_ctx, c["opa"], c["orbs"], c["s"], c["orbe"], c["n_occ"], c["n_virt"], c["gamma"],
                              c["gamma_lr"], c["xyz"])
    got = es.run_tda(n_roots, 200, 1e-8)
    # residuals below 1e-8 leave (1e-8)^2 / gap in the energies; 1e-10 is the bar of the solver
    assert np.abs(got["ci_eigenvalues"] - ref["energies"]).max() < 1e-10
    x = got["ci_coefficients"]
    # the basis is orthonormal to rounding over at most 15 n_roots vectors
    assert np.abs(x.T @ x - np.eye(n_roots)).max() < 1e-11
