"""Mixed products with atoms without elements beside full clusters: rows that
fill a cluster's 128 exactly leave no row number for the empty atom after them,
whose C blocks have norm 0 and leave with the result filter."""
import numpy as np
import pytest

import oracle
from lamb_b200 import gpu
from tests.helpers import assert_same_pattern, rel_frobenius_error
from tests.test_gpu_panel import _matrix

pytestmark = pytest.mark.gpu

# six digits of A and B carry 47 bits each, as for the other mixed products of normal values
TOL_MIXED = 1e-11


@pytest.mark.parametrize("sizes", [[64, 64, 0], [0, 64, 64], [32, 32, 32, 32, 0], [64, 0, 64, 0], [0, 0, 64, 64]])
@pytest.mark.parametrize("positions", [False, True])
@pytest.mark.parametrize("eps", [0.0, 1e-6])
def test_pattern_is_the_oracles(gpu_ctx, sizes, positions, eps):
    rng = np.random.default_rng(5)
    k = len(sizes)
    n = 6 * k
    bs = np.resize(np.array(sizes), n)
    p = np.kron(np.eye(6, dtype=bool) | np.eye(6, k=1, dtype=bool), np.ones((k, k), bool))
    a, b = _matrix(rng, bs, bs, p), _matrix(rng, bs, bs, p.T)
    ref, _ = oracle.multiply(a, b, eps, oracle.NO_PRODUCT_FILTER)
    da, db = gpu_ctx.upload(a), gpu_ctx.upload(b)
    if positions:
        da.set_positions(np.stack([np.arange(n) * 0.7, np.zeros(n), np.zeros(n)], 1).astype(np.float32),
                         np.array([50.0, 9.0, 9.0], np.float32))
    dc = gpu_ctx.create_like(da)
    gpu_ctx.multiply(da, db, dc, eps, gpu.MIXED | gpu.NO_PRODUCT_FILTER)
    c = dc.download()
    assert_same_pattern(c, ref)
    assert rel_frobenius_error(c, ref) <= TOL_MIXED
    for m in (dc, db, da):
        m.destroy()
