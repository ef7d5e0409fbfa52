"""Digits of a mixed product whose tiles have long inner lists: beyond 1,024
separate runs of inner rows it has the digits of the mma.sync kernel, seven or
as many as the caller asks for."""
import numpy as np
import pytest

from lamb_b200 import gpu
from tests.test_gpu_panel import _matrix

pytestmark = pytest.mark.gpu


def _product(ctx, runs):
    rng = np.random.default_rng(runs)
    n = 2 * runs
    rows, inner, cols = np.array([13, 5, 5]), np.resize([13, 5, 5], n), np.array([7, 9])
    pa = np.zeros((3, n), bool)
    pa[:, ::2] = True  # no two runs follow on
    a, b = _matrix(rng, rows, inner, pa), _matrix(rng, inner, cols, np.ones((n, 2), bool))
    da, db = ctx.upload(a), ctx.upload(b)
    dc = ctx.create_like(db)
    st = ctx.multiply(da, db, dc, 0.0, gpu.MIXED)
    c, ref = dc.download().to_dense(), a.to_dense().astype(np.longdouble) @ b.to_dense().astype(np.longdouble)
    for m in (dc, db, da):
        m.destroy()
    return st["mixed_slices"], float(np.linalg.norm((c - ref).astype(float)) / np.linalg.norm(ref.astype(float)))


@pytest.mark.parametrize("runs", [1023, 1024, 1025, 1500])
def test_long_lists_have_seven_digits(gpu_ctx, runs):
    digits, error = _product(gpu_ctx, runs)
    assert digits == (6 if runs <= 1024 else 7)
    assert error <= 1e-11  # the bound of the mixed multiply


@pytest.mark.parametrize("slices", [5, 8])
def test_the_caller_s_digit_count_holds(gpu_ctx, monkeypatch, slices):
    monkeypatch.setenv("LAMB_GPU_MIXED_SLICES", str(slices))
    assert _product(gpu_ctx, 1100)[0] == slices
