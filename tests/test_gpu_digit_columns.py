"""Digits of new basis vectors at odd lengths, odd column starts and every fill of a pair: the mixed Davidson,
whose subspace products read both layouts, against the FP64 form."""

import numpy as np
import pytest

from cases import fixture_case, synthetic_case
from tincr_gb300 import _lib
from tincr_gb300 import tda as T


@pytest.mark.gpu
@pytest.mark.parametrize("n_roots", [1, 2, 3, 7, 20])
@pytest.mark.parametrize("name", ["uracil", "water8"])   # o v odd / even
def test_mixed_davidson_at_every_column_start(gpu_ctx, name, n_roots):
    c = fixture_case(name, True) if name == "uracil" else synthetic_case(name, True)
    es = T.ExcitedStateSystem(gpu_ctx, c["opa"], c["orbs"], c["s"], c["orbe"], c["n_occ"], c["n_virt"], c["gamma"],
                              c["gamma_lr"], c["xyz"])
    a = es.run_tda(n_roots, 200, 1e-6)
    b = es.run_tda(n_roots, 200, 1e-6, precision=_lib.PREC_BF16X3)
    # the bar of the mixed form; a digit in a wrong place is an error of the order of the energies
    assert np.abs(a["ci_eigenvalues"] - b["ci_eigenvalues"]).max() < 1e-6
    x = b["ci_coefficients"]
    # the subspace arithmetic keeps FP64 accuracy, so the roots stay orthonormal to rounding
    assert np.abs(x.T @ x - np.eye(n_roots)).max() < 1e-10
