"""An exciton call that fails on its host data while its exchange kernels are queued leaves the context usable:
the call reports the status, and the next one gives the matrix of the one before."""

import numpy as np
import pytest

from cases import fmo_case
from tincr_gb300 import _lib
from tincr_gb300 import fmo


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_BF16X3])
def test_exciton_call_after_a_failed_one(gpu_ctx, prec):
    c = fmo_case(3, 1, 1)
    setup = fmo.ExcitonSetup(c["monomers"], c["pairs"])
    rc, res = fmo.solve_batch(gpu_ctx, c["instances"], 150, 1e-8, _lib.PREC_FP64)
    assert rc == _lib.OK

    def call():
        return fmo.exciton_states(gpu_ctx, setup, res, c["labels"], 4, 1, n_roots=5, tol=1e-8, max_iter=200,
                                  precision=prec, want_matrix=True)

    first = call()
    pair = next(p for p in setup.pair_scc if setup.real.get(p))
    orbs, orbe = setup.pair_scc[pair]
    for _ in range(3):
        bad = np.array(orbs)
        bad[-1, -1] = np.nan
        setup.pair_scc[pair] = (bad, orbe)
        with pytest.raises(_lib.TincrError) as e:
            call()
        assert e.value.status == _lib.NONFINITE
        setup.pair_scc[pair] = (orbs, orbe)
        again = call()
        # the tiles of an element are added by FP64 atomics in any order: a few dozen terms below one
        assert np.max(np.abs(first["matrix"] - again["matrix"])) < 1e-14
        assert np.max(np.abs(first["energies"] - again["energies"])) < 1e-12
