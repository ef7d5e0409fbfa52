"""Row orders from one-directional patterns (no coordinates): every row has its
place, on each of the multiply's paths."""
import numpy as np
import pytest

import oracle
from lamb_b200 import gpu
from tests.helpers import assert_same_pattern, rel_frobenius_error
from tests.test_gpu_panel import _matrix

pytestmark = pytest.mark.gpu


def _patterns():
    rng = np.random.default_rng(0)
    i = np.arange(90)
    chain = np.zeros((90, 90), bool)
    chain[i[:-1], i[1:]] = True
    upper = np.triu(rng.random((90, 90)) < 0.3)
    star = np.zeros((90, 90), bool)
    star[rng.integers(0, 90, 3)] = True
    parts = np.kron(np.eye(3, dtype=bool), chain[:30, :30])
    return {"chain": chain, "upper": upper, "star": star, "parts": parts, "full_upper": np.triu(np.ones((90, 90), bool))}


PATTERNS = _patterns()


@pytest.mark.parametrize("flags", [0, gpu.ASYNC, gpu.MIXED])
@pytest.mark.parametrize("sync_kernel", [False, True])
@pytest.mark.parametrize("name", sorted(PATTERNS))
def test_multiply(gpu_ctx, monkeypatch, name, sync_kernel, flags):
    if sync_kernel:
        monkeypatch.setenv("LAMB_GPU_MIXED_MMA_SYNC", "1")
    rng = np.random.default_rng(1)
    bs = np.resize(np.array([13, 5, 5]), 90)
    a, b = _matrix(rng, bs, bs, PATTERNS[name]), _matrix(rng, bs, bs, rng.random((90, 90)) < 0.4)
    ref, _ = oracle.multiply(a, b, 0.0, 0)
    da, db = gpu_ctx.upload(a), gpu_ctx.upload(b)
    dc = gpu_ctx.create_like(db)
    gpu_ctx.multiply(da, db, dc, 0.0, flags)
    c = dc.download()
    for m in (dc, db, da):
        m.destroy()
    assert_same_pattern(c, ref)
    # the orders of the FP64 sums and the digits are those of the other products
    assert rel_frobenius_error(c, ref) <= (1e-11 if flags & gpu.MIXED else 1e-12)
