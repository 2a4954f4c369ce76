"""Device memory that a context keeps after a call: large input buffers go back, workspaces stay within their
budget, and the next call is right again."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import tda as T
from test_gpu_product_sizes import _system


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_BF16X3])
def test_products_of_many_vectors_keep_little(precision):
    torch = pytest.importorskip("torch")
    n, o, v, k = 128, 64, 64, 3000   # X, its transpose and A.X: 295 MB
    q = _system(n, o, v, True, 11)
    torch.cuda.synchronize()

    def free():
        return torch.cuda.mem_get_info(0)[0]

    ctx = _lib.Context(0)
    try:
        es = T.ExcitedStateSystem(ctx, q["opa"], q["c"], q["s"], q["orbe"], o, v, q["gamma"], q["glr"], q["xyz"])
        small = np.random.default_rng(1).normal(size=(o * v, 30))
        ref = es.compute_products(small, precision)
        before = free()
        x = np.tile(small, (1, k // 30))
        big = es.compute_products(x, precision)
        # the workspace of 64 vectors: 1.7 MB each in the larger form
        assert before - free() < 200 << 20
        for j in range(0, k, 30):
            assert np.array_equal(big[:, j:j + 30], ref)
        assert np.array_equal(es.compute_products(small, precision), ref)
    finally:
        ctx.close()
