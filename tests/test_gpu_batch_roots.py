"""The batched Davidson at every number of roots (subspaces from 15 to 90 vectors, one CTA or a cluster per
instance), against the oracle engine instance by instance."""

import numpy as np
import pytest

from cases import fmo_case, fmo_oracle_engine
from oracle import tda as OT
from tincr_gb300 import _lib
from tincr_gb300 import fmo


@pytest.mark.gpu
@pytest.mark.parametrize("nr", [1, 2, 3, 4, 5, 6])
def test_batch_at_every_root_count(gpu_ctx, nr):
    case = fmo_case(2, 1, 1)
    inst = [dict(q, n_roots=nr) for q in case["instances"]]
    rc, res = fmo.solve_batch(gpu_ctx, inst, max_iter=150, tol=1e-8)
    assert rc == _lib.OK
    for k, r in enumerate(res):
        eng, xyz = fmo_oracle_engine(case, k)
        ref = OT.run_tda_engine(eng, xyz, nr, 150, 1e-8)
        assert r["status"] == _lib.OK
        # a residual below 1e-8 leaves (1e-8)^2 / gap in an energy; 1e-10 is the bar of the batch
        assert np.abs(r["energies"] - ref["energies"]).max() < 1e-10, case["labels"][k]
        ov = np.abs(np.einsum("xr,xr->r", r["coefficients"], ref["coefficients"]))
        assert np.abs(ov - 1.0).max() < 1e-7, case["labels"][k]
