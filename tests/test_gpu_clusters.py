"""Mixed multiply on clusters of nearby atoms: pools smaller and larger than
the register pool, several ranges of the order, atoms without elements, blocks
as wide as a tile, coincident and wrapped coordinates, rectangular operands."""
import numpy as np
import pytest

import oracle
from lamb_b200 import gpu
from tests.helpers import assert_same_pattern, rel_frobenius_error
from tests.test_gpu_panel import _matrix

pytestmark = pytest.mark.gpu

# six digits of A and B carry 47 bits each: a product is off by less than 2^-46
# of its row and column maxima, which random normal values stay within a factor
# of five of (the bound stated for the mixed multiply)
TOL_MIXED = 1e-11

SIZES = {"water": [13, 5, 5], "ones": [1], "empty": [0, 7, 0, 1], "wide": [64, 3, 40], "odd": [9, 11, 2]}


def _band(rng, n, m, sizes, csizes):
    p = np.zeros((n, m), bool)
    i = np.arange(max(n, m))
    for d in (-3, -1, 0, 2):
        k = (i + d >= 0) & (i + d < m) & (i < n)
        p[i[k], i[k] + d] = True
    return _matrix(rng, np.resize(sizes, n), np.resize(csizes, m), p, cut=(n // 2, m // 2) if n > 2 and m > 2 else None)


def _positions(rng, n, how):
    if how == "line":
        return np.stack([np.arange(n) * 0.7, np.zeros(n), np.zeros(n)], 1)
    if how == "same":
        return np.zeros((n, 3))
    return rng.random((n, 3)) * 60.0 - 30.0  # outside the box on purpose: wrapped


def _check(ctx, a, b, pos):
    ref, _ = oracle.multiply(a, b, 0.0, 0)
    da, db = ctx.upload(a), ctx.upload(b)
    if pos is not None:
        da.set_positions(pos.astype(np.float32), np.array([20.0, 30.0, 25.0], np.float32))
    dc = ctx.create_like(db)
    for _ in range(2):  # the second multiply finds the clusters made
        ctx.multiply(da, db, dc, 0.0, gpu.MIXED)
        c = dc.download()
        assert_same_pattern(c, ref)
        assert rel_frobenius_error(c, ref) <= TOL_MIXED
    for m in (dc, db, da):
        m.destroy()


@pytest.mark.parametrize("how", ["line", "same", "random", None])
@pytest.mark.parametrize("sizes", sorted(SIZES))
@pytest.mark.parametrize("n", [1, 2, 31, 255, 256, 257])
def test_clusters(gpu_ctx, n, sizes, how):
    rng = np.random.default_rng(n)
    s = np.array(SIZES[sizes])
    if np.resize(s, n).sum() == 0:
        s = s[::-1]
    a, b = _band(rng, n, n, s, s), _band(rng, n, n, s, s)
    _check(gpu_ctx, a, b, None if how is None else _positions(rng, n, how))


@pytest.mark.parametrize("n", [2047, 2048, 3100])
def test_cluster_ranges(gpu_ctx, n):
    rng = np.random.default_rng(n)
    s = np.array([2, 1, 3])
    a, b = _band(rng, n, n, s, s), _band(rng, n, n, s, s)
    _check(gpu_ctx, a, b, _positions(rng, n, "random"))


@pytest.mark.parametrize("m", [3, 90, 300])
def test_rectangular_clusters(gpu_ctx, m):
    rng = np.random.default_rng(m)
    r, k, c = np.array([100, 13, 5]), np.array([13, 5, 5]), np.array([7, 0, 30])
    a, b = _band(rng, 120, 150, r, k), _band(rng, 150, m, k, c)
    _check(gpu_ctx, a, b, _positions(rng, 120, "random"))


@pytest.mark.parametrize("sizes", [[1], [3, 1, 2], [33, 31]])
@pytest.mark.parametrize("runs", [1, 31, 32, 33, 63, 64, 65, 97, 1100])
def test_inner_runs(gpu_ctx, runs, sizes):
    """Tiles whose inner list has `runs` runs of panel rows: A couples to every
    other inner atom, B to all of them, so that no two runs follow on."""
    rng = np.random.default_rng(runs)
    n = 2 * runs
    rows, inner, cols = np.array([13, 5, 5]), np.resize(sizes, n), np.array([7, 9])
    pa = np.zeros((3, n), bool)
    pa[:, ::2] = True
    a = _matrix(rng, rows, inner, pa)
    b = _matrix(rng, inner, cols, np.ones((n, 2), bool))
    _check(gpu_ctx, a, b, None)


@pytest.mark.parametrize("ea,eb", [(600, -600), (-1005, 1000), (-1005, 5)])
def test_wide_exponents(gpu_ctx, ea, eb):
    """Row and column scales beyond what a single exact factor covers."""
    rng = np.random.default_rng(7)
    s = np.array([13, 5, 5])
    a, b = _band(rng, 60, 60, s, s), _band(rng, 60, 60, s, s)
    for m, e in ((a, ea), (b, eb)):
        for sec in m.sectors:
            sec.data[:] = np.ldexp(sec.data, e)
    _check(gpu_ctx, a, b, _positions(rng, 60, "line"))
