"""Adjoint products whose rows, inner atoms and columns differ in number and
size, on group tiles and beyond what those can hold, with both outputs or one."""
import numpy as np
import pytest

from tests.test_gpu_panel import _matrix

pytestmark = pytest.mark.gpu

# sums of up to a few thousand normally distributed products, added in another order by
# the dense reference: a relative error of 1e-13 is some thousand roundings
TOL = 1e-13


def _check(ctx, a, b, dc, want_a=True, want_b=True):
    da, db, ddc = (ctx.upload(x) for x in (a, b, dc))
    ga = ctx.create_like(da) if want_a else None
    gb = ctx.create_like(db) if want_b else None
    ctx.adjoint(da, db, ddc, ga, gb)
    A, B, D = a.to_dense(), b.to_dense(), dc.to_dense()
    for g, like, dense in ((ga, a, lambda: D @ B.T), (gb, b, lambda: A.T @ D)):
        if g is None:
            continue
        got, ref = g.download(), dense()
        assert [s.n_blks for s in got.sectors] == [s.n_blks for s in like.sectors]
        for s, t in zip(got.sectors, like.sectors):
            assert np.array_equal(s.row_p, t.row_p) and np.array_equal(s.col_i, t.col_i)
        x = got.to_dense()
        mask = _mask(like)
        assert np.linalg.norm((x - ref)[mask]) <= TOL * np.linalg.norm(ref[mask])
        assert not x[~mask].any()
    for m in (ga, gb, ddc, db, da):
        if m is not None:
            m.destroy()


def _mask(m):
    """Elements of the blocks that m holds."""
    rb, cb = np.concatenate(m.subset_blk_sizes(0)), np.concatenate(m.subset_blk_sizes(1))
    rs = np.cumsum([0] + [len(x) for x in m.subset_blk_sizes(0)])
    cs = np.cumsum([0] + [len(x) for x in m.subset_blk_sizes(1)])
    p = np.zeros((len(rb), len(cb)), bool)
    for s in m.sectors:
        p[rs[s.subset_row - 1] + s.block_rows(), cs[s.subset_col - 1] + s.col_i.astype(int) - 1] = True
    return np.repeat(np.repeat(p, rb.astype(int), 0), cb.astype(int), 1)


@pytest.mark.parametrize("which", ["both", "a", "b"])
@pytest.mark.parametrize("shape", [(24, 200, 150), (150, 60, 300), (300, 150, 24), (90, 90, 260)])
def test_rectangular(gpu_ctx, shape, which):
    rng = np.random.default_rng(shape[0])
    m, k, n = shape
    rb, kb, cb = (rng.integers(0, 14, x) for x in (m, k, n))
    a = _matrix(rng, rb, kb, rng.random((m, k)) < 0.8)
    b = _matrix(rng, kb, cb, rng.random((k, n)) < 0.8)
    dc = _matrix(rng, rb, cb, rng.random((m, n)) < 0.8)
    _check(gpu_ctx, a, b, dc, which != "b", which != "a")


@pytest.mark.parametrize("which", ["both", "a", "b"])
@pytest.mark.parametrize("inner", [51200, 51202, 60000])
def test_inner_atoms_that_form_no_groups(gpu_ctx, inner, which):
    """dA has a column group for every inner atom: above 51,200 of them its tiles
    do not fit and it runs on stacks, while dB stays on the tiles."""
    rng = np.random.default_rng(inner)
    rows, cols, half = np.ones(8, int), np.ones(8, int), inner // 2
    kb = np.ones(inner, int)
    p = np.zeros((8, inner), bool)
    p[:4, ::2] = p[4:, 1::2] = True  # neighbouring inner atoms share no row
    a = _matrix(rng, rows, kb, p, cut=(4, half))
    b = _matrix(rng, kb, cols, np.ones((inner, 8), bool), cut=(half, 4))
    dc = _matrix(rng, rows, cols, np.ones((8, 8), bool), cut=(4, 4))
    _check(gpu_ctx, a, b, dc, which != "b", which != "a")
