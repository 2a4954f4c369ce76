"""A.X of an X that is not finite: refused with the status, A.X left as it was, and the context right afterwards,
in both precisions, on both sides of the number of multiply-adds from which FP64 runs on digits and of the 8192
values from which the device checks X."""

import numpy as np
import pytest

from tincr_gb300 import _lib
from tincr_gb300 import tda as T
from tincr_gb300._lib import dptr
from test_gpu_product_sizes import _system

SIZES = [(33, 16, 17, 1), (33, 16, 17, 3), (128, 64, 64, 2), (128, 64, 64, 3), (128, 64, 64, 24)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_BF16X3])
@pytest.mark.parametrize("lc", [True, False])
@pytest.mark.parametrize("n,o,v,k", SIZES)
def test_non_finite_x_is_refused(gpu_ctx, n, o, v, k, lc, precision):
    q = _system(n, o, v, lc, n)
    es = T.ExcitedStateSystem(gpu_ctx, q["opa"], q["c"], q["s"], q["orbe"], o, v, q["gamma"], q["glr"], q["xyz"])
    x = np.random.default_rng(n).normal(size=(o * v, k))
    ref = es.compute_products(x, precision)
    for value in (np.nan, np.inf, -np.inf):
        for at in ((0, 0), (o * v - 1, k - 1), (o * v // 2, k // 2)):
            bad = x.copy()
            bad[at] = value
            out = np.full_like(x, 7.0)
            rc = gpu_ctx.lib.tincr_tda_products(gpu_ctx.h, k, dptr(bad), dptr(out), precision)
            assert rc == _lib.NONFINITE
            assert np.all(out == 7.0)
    assert np.array_equal(es.compute_products(x, precision), ref)
    # the largest and smallest finite values are not refused
    edge = x.copy()
    edge[0, 0], edge[-1, -1] = np.finfo(float).max, 5e-324
    out = np.empty_like(x)
    assert gpu_ctx.lib.tincr_tda_products(gpu_ctx.h, k, dptr(edge), dptr(out), precision) == _lib.OK
