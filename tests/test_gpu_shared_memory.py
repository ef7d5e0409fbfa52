"""Sizes at which a kernel's dynamic and static shared memory together pass the
48 KB that need no asking while the dynamic part alone does not."""
import numpy as np
import pytest

import oracle
from lamb_b200 import gpu
from lamb_b200.matrix import LambMatrix, Sector
from tests.helpers import assert_same_pattern, rel_frobenius_error
from tests.test_gpu_panel import _matrix

pytestmark = pytest.mark.gpu

# sums of up to 1,540 normally distributed products in another order than the oracle's at most
TOL = 1e-12


def _sectors(rng, row_sizes, col_sizes, r, c, rcut, ccut):
    """Host matrix of the blocks (r, c), with the rows and columns cut into subsets."""
    secs = []
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    for m in range(len(rcut) - 1):
        for n in range(len(ccut) - 1):
            k = (r >= rcut[m]) & (r < rcut[m + 1]) & (c >= ccut[n]) & (c < ccut[n + 1])
            rr, cc = r[k] - rcut[m], c[k] - ccut[n]
            rb, cb = row_sizes[rcut[m]:rcut[m + 1]], col_sizes[ccut[n]:ccut[n + 1]]
            sz = rb[rr].astype(np.int64) * cb[cc]
            end = np.cumsum(sz)
            row_p = np.concatenate([[0], np.cumsum(np.bincount(rr, minlength=len(rb)))]).astype(np.int64)
            secs.append(Sector(m + 1, n + 1, rb.astype(np.int8), cb.astype(np.int8), row_p, (cc + 1).astype(np.int16),
                               np.stack([end - sz + 1, end], 1).astype(np.int64),
                               rng.standard_normal(int(end[-1]) if len(end) else 0)))
    return LambMatrix(secs)


def _check(ctx, a, b, flags=0, tol=TOL):
    da = ctx.upload(a)
    db = da if b is a else ctx.upload(b)
    dc = ctx.create_like(db)
    ctx.multiply(da, db, dc, 0.0, flags)
    c, ref = dc.download(), oracle.multiply(a, b, 0.0, 0)[0]
    for m in {dc, db, da}:
        m.destroy()
    assert_same_pattern(c, ref)
    assert rel_frobenius_error(c, ref) <= tol


@pytest.mark.parametrize("groups", [12256, 12258, 12288, 12290])
def test_tile_masks(gpu_ctx, groups):
    """Runs of four atoms that share nothing with their neighbours: a group each,
    and 8 bytes of masks for two of them."""
    rng = np.random.default_rng(groups)
    run = np.arange(groups)
    other = rng.permutation(groups)
    pairs = np.unique(np.concatenate([np.stack([run, run], 1), np.stack([run, other], 1)]), axis=0)
    i, j = np.meshgrid(np.arange(4), np.arange(4), indexing="ij")
    r = (4 * pairs[:, 0, None] + i.reshape(1, -1)).reshape(-1)
    c = (4 * pairs[:, 1, None] + j.reshape(1, -1)).reshape(-1)
    ones, cut = np.ones(4 * groups, int), [0, 2 * groups, 4 * groups]
    _check(gpu_ctx, _sectors(rng, ones, ones, r, c, cut, cut), _sectors(rng, ones, ones, r, c, cut, cut))


@pytest.mark.parametrize("flags", [0, gpu.MIXED])
@pytest.mark.parametrize("blocks", [1497, 1500, 1534, 1540])
def test_stack_fill(gpu_ctx, monkeypatch, blocks, flags):
    """Rows of A with `blocks` blocks, 32 bytes each in the fill's table."""
    monkeypatch.setenv("LAMB_GPU_MIXED_MMA_SYNC", "1")  # the mixed path that builds stacks
    rng = np.random.default_rng(blocks)
    rows, inner, cols = np.array([3, 2]), np.resize([2, 1], blocks), np.array([2, 4])
    a, b = _matrix(rng, rows, inner, np.ones((2, blocks), bool)), _matrix(rng, inner, cols, np.ones((blocks, 2), bool))
    _check(gpu_ctx, a, b, flags, 1e-11 if flags else TOL)


@pytest.mark.parametrize("n", [388480, 389000, 393216, 393300])
def test_count_bitmap(gpu_ctx, n):
    """C rows of n columns, a bit each in the count's bitmap."""
    rng = np.random.default_rng(n)
    cut = list(range(0, n, 30000)) + [n]
    ones = np.ones(n, int)
    c = np.sort(rng.choice(n, 5000, replace=False))
    a = _matrix(rng, np.array([2, 1, 3]), np.array([1, 2, 3, 4, 5]), np.ones((3, 5), bool))
    b = _sectors(rng, np.array([1, 2, 3, 4, 5]), ones, rng.integers(0, 5, 5000), c, [0, 5], cut)
    _check(gpu_ctx, a, b)
