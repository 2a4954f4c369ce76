"""The same FP64 solve twice gives the same bits, at lengths from one column block of the subspace products to
many: their partial sums are added in a fixed order."""

import numpy as np
import pytest

from tincr_gb300 import geometry as G
from tincr_gb300 import groundstate as gs
from tincr_gb300 import tda as T

# o v = 32, 225, 576, 2601, 4489
MOLECULES = {"water2": lambda: G.water_cluster(2, 1, 1), "acene1": lambda: G.acene(1), "acene2": lambda: G.acene(2),
             "acene5": lambda: G.acene(5), "acene7": lambda: G.acene(7)}


@pytest.mark.gpu
@pytest.mark.parametrize("n_roots", [1, 6, 20])
@pytest.mark.parametrize("name", sorted(MOLECULES))
def test_solve_repeats_bit_for_bit(gpu_ctx, name, n_roots):
    z, x = MOLECULES[name]()
    sy = gs.build_system(z, G.to_bohr(x))
    es = T.ExcitedStateSystem.from_ground_state(gpu_ctx, sy, gs.run_scc(sy, tol=1e-10))
    runs = []
    for _ in range(5):
        r = es.run_tda(n_roots, 200, 1e-8)   # (the same dict each time)
        runs.append((r["ci_eigenvalues"].copy(), r["ci_coefficients"].copy()))
    for e, x in runs[1:]:
        assert np.array_equal(runs[0][0], e)
        assert np.array_equal(runs[0][1], x)
