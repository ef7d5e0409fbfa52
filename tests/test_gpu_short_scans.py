"""Layout and result filter of matrices whose scans change from the one-launch
to the library form (8,192 values), and at the edges of its rounds of 1,024."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_same_pattern, rel_frobenius_error
from tests.test_gpu_panel import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.0, 0.5])
@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 8191, 8192, 8193])
def test_band_product(gpu_ctx, n, eps):
    rng = np.random.default_rng(n)
    p = np.zeros((n, n), bool)
    i = np.arange(n)
    p[i, i] = True
    p[i[1:], i[:-1]] = rng.random(n - 1) < 0.5
    sizes = rng.integers(1, 3, n)
    a, b = _matrix(rng, sizes, sizes, p), _matrix(rng, sizes, sizes, p)
    ref, _ = oracle.multiply(a, b, eps, 0)
    da, db = gpu_ctx.upload(a), gpu_ctx.upload(b)
    dc = gpu_ctx.create_like(da)
    gpu_ctx.multiply(da, db, dc, eps, 0)
    c = dc.download()
    for m in (dc, db, da):
        m.destroy()
    assert_same_pattern(c, ref)
    # at most two products of inner size 2 a value
    assert rel_frobenius_error(c, ref) <= 1e-14
