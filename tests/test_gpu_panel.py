"""FP64 multiply on group tiles (panel products) against the oracle at the
edges of its shapes: group and slab boundaries, zero-size blocks, blocks at and
beyond the 24-row limit, atom orders without groups, rectangular structures,
filters that split superblock pairs, and non-finite operands.  Every product
is large enough (half a million block products) for the panels to be taken."""
import numpy as np
import pytest

import oracle
from lamb_b200 import gpu
from lamb_b200.gen import WaterGeometry
from lamb_b200.matrix import LambMatrix, Sector
from tests.helpers import assert_same_pattern, block_values, rel_frobenius_error

pytestmark = pytest.mark.gpu

# both sides add a C element's products in the same order (k ascending): only the fused
# multiply-adds of the oracle's compiler could differ, a few ulp of the partial sums
TOL = 1e-12


def _matrix(rng, row_sizes, col_sizes, present, cut=None):
    """Host matrix with the block pattern `present` [rows, cols]; `cut` splits rows and columns into two subsets."""
    rs = [0, len(row_sizes)] if cut is None else [0, cut[0], len(row_sizes)]
    cs = [0, len(col_sizes)] if cut is None else [0, cut[1], len(col_sizes)]
    secs = []
    for m in range(len(rs) - 1):
        for n in range(len(cs) - 1):
            r, c = np.nonzero(present[rs[m]:rs[m + 1], cs[n]:cs[n + 1]])
            rb, cb = row_sizes[rs[m]:rs[m + 1]], col_sizes[cs[n]:cs[n + 1]]
            sz = rb[r].astype(np.int64) * cb[c]
            end = np.cumsum(sz)
            row_p = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=len(rb)))]).astype(np.int64)
            secs.append(Sector(m + 1, n + 1, rb.astype(np.int8), cb.astype(np.int8), row_p, (c + 1).astype(np.int16),
                               np.stack([end - sz + 1, end], 1).astype(np.int64),
                               rng.standard_normal(int(end[-1]) if len(end) else 0)))
    return LambMatrix(secs)


def _check(ctx, a, b, eps=0.0, flags=0, same=False):
    ref, st_ref = oracle.multiply(a, b, eps, flags)
    da = ctx.upload(a)
    db = da if same else ctx.upload(b)
    dc = ctx.create_like(da) if same else ctx.create_like(db)
    st = ctx.multiply(da, db, dc, eps, flags)
    c = dc.download()
    for m in {dc, db, da}:
        m.destroy()
    assert_same_pattern(c, ref)
    assert st["n_products"] == st_ref["n_products"]
    assert st["n_products_skipped"] == st_ref["n_products_skipped"]
    return c, ref


# sizes: runs that fill a group exactly (24 = 8 + 8 + 8 = 13 + 5 + 5 + 1), slab edges, singles, empty atoms
SIZES = {"ones": [1], "slabs": [8], "edge": [7, 8, 9, 16, 17], "full": [24], "molecule": [13, 5, 5], "big": [23, 5, 5],
         "empty": [0, 3, 0, 5, 24, 1], "mixed24": [24, 1, 12, 12, 2], "beyond": [25, 5, 13]}


@pytest.mark.parametrize("sizes", sorted(SIZES))
@pytest.mark.parametrize("fill", [0.6, 1.0])
def test_block_sizes(gpu_ctx, sizes, fill):
    rng = np.random.default_rng([len(sizes), int(10 * fill)])
    n = 151
    bs = np.resize(np.array(SIZES[sizes]), n)
    # neighbouring atoms share most of their pattern, so that groups form
    base = rng.random((n // 3 + 1, n // 3 + 1)) < fill
    p = np.kron(base, np.ones((3, 3), bool))[:n, :n] & (rng.random((n, n)) < 0.9)
    a = _matrix(rng, bs, bs, p, cut=(61, 61))
    b = _matrix(rng, bs, bs, p.T, cut=(61, 61))
    c, ref = _check(gpu_ctx, a, b)
    assert rel_frobenius_error(c, ref) <= TOL


@pytest.mark.parametrize("shape", [(3, 900, 600), (60, 500, 70), (150, 90, 400), (600, 1000, 3)])
def test_rectangular(gpu_ctx, shape):
    """Rows, inner atoms and columns with their own sizes and counts."""
    rng = np.random.default_rng(shape[0])
    m, k, n = shape
    rb, kb, cb = (rng.integers(0, 14, x) for x in (m, k, n))
    a = _matrix(rng, rb, kb, rng.random((m, k)) < 0.8)
    b = _matrix(rng, kb, cb, rng.random((k, n)) < 0.8)
    ref, _ = oracle.multiply(a, b, 0.0)
    da, db = gpu_ctx.upload(a), gpu_ctx.upload(b)
    dc = gpu_ctx.create_like(da)
    gpu_ctx.multiply(da, db, dc, 0.0)
    c = dc.download()
    assert_same_pattern(c, ref)
    assert rel_frobenius_error(c, ref) <= TOL
    for x in (dc, db, da):
        x.destroy()


@pytest.mark.parametrize("eps", [1e-4, 3e-3, 3e-2, 0.5])
@pytest.mark.parametrize("shuffled", [False, True])
def test_filters(gpu_ctx, eps, shuffled):
    """Superblock pairs with all, some and none of their products above eps;
    `shuffled`: neighbouring atoms are unrelated, groups of single atoms."""
    g = WaterGeometry(50, None, 6.5, seed=4)
    a, b = g.matrix(1), g.matrix(2)
    if shuffled:
        perm = np.random.default_rng(0).permutation(g.n_atoms)
        size = np.concatenate(a.subset_blk_sizes(0)).astype(np.int64)
        off = np.concatenate([[0], np.cumsum(size)])
        out = []
        for m in (a, b):
            d = m.to_dense()
            p = np.zeros((g.n_atoms, g.n_atoms), bool)
            base = np.cumsum([0] + [len(x) for x in m.subset_blk_sizes(0)])
            for s in m.sectors:
                p[base[s.subset_row - 1] + s.block_rows(), base[s.subset_col - 1] + s.col_i.astype(int) - 1] = True
            x = _matrix(np.random.default_rng(1), size[perm], size[perm], p[np.ix_(perm, perm)])
            sec = x.sectors[0]
            rows = sec.block_rows()
            for k in range(sec.n_blks):
                r, c = perm[rows[k]], perm[sec.col_i[k] - 1]
                f, l = sec.extents[k]
                sec.data[f - 1:l] = d[off[r]:off[r + 1], off[c]:off[c + 1]].T.reshape(-1)
            out.append(x)
        a, b = out
    c, ref = _check(gpu_ctx, a, b, eps, oracle.NO_RESULT_FILTER)
    assert rel_frobenius_error(c, ref) <= TOL


def test_zero_norm_blocks_leave_with_the_result_filter(gpu_ctx):
    """C blocks without elements have norm 0: the result filter drops them."""
    rng = np.random.default_rng(3)
    bs = np.resize(np.array([0, 4, 0, 6, 2]), 90)
    a = _matrix(rng, bs, bs, np.ones((90, 90), bool))
    ref, _ = oracle.multiply(a, a, 1e-6, oracle.NO_PRODUCT_FILTER)
    da = gpu_ctx.upload(a)
    dc = gpu_ctx.create_like(da)
    gpu_ctx.multiply(da, da, dc, 1e-6, gpu.NO_PRODUCT_FILTER)
    assert_same_pattern(dc.download(), ref)
    for x in (dc, da):
        x.destroy()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e200])
def test_non_finite_operands_stay_in_their_products(gpu_ctx, bad):
    """An infinity, a NaN or a value whose norm overflows reaches exactly the C
    blocks that have a product with its block."""
    g = WaterGeometry(64, None, 6.0, seed=2)
    a, b = g.matrix(1), g.matrix(2)
    b.sectors[0].data[7] = bad
    ref, _ = oracle.multiply(a, b, 0.0)
    da, db = gpu_ctx.upload(a), gpu_ctx.upload(b)
    dc = gpu_ctx.create_like(da)
    gpu_ctx.multiply(da, db, dc, 0.0)
    got, want = block_values(dc.download()), block_values(ref)
    assert set(got) == set(want)
    for k in want:
        fin = np.isfinite(want[k])
        assert np.array_equal(fin, np.isfinite(got[k])), k
        assert np.allclose(got[k][fin], want[k][fin], rtol=1e-11, atol=1e-12 * max(1.0, np.abs(want[k][fin]).max(initial=0)))
    for x in (dc, db, da):
        x.destroy()


def test_chunked_download_after_async(gpu_ctx):
    """An asynchronous multiply runs in several launches, the download copies
    each launch's rows: same C as the synchronous call, block for block."""
    g = WaterGeometry(150, None, 6.0, seed=6)
    a, b = g.matrix(1), g.matrix(2)
    da, db = gpu_ctx.upload(a), gpu_ctx.upload(b)
    da.set_positions(g.sector_positions(), g.box)
    outs = []
    for flags in (gpu.ASYNC, 0):
        dc = gpu_ctx.create_like(da)
        gpu_ctx.multiply(da, db, dc, 1e-10, flags)
        outs.append(dc.download())
        dc.destroy()
    for s1, s2 in zip(outs[0].sectors, outs[1].sectors):
        assert np.array_equal(s1.extents, s2.extents) and np.array_equal(s1.data, s2.data)
    for x in (db, da):
        x.destroy()


@pytest.mark.parametrize("sizes", ["molecule", "edge", "empty", "full", "beyond"])
@pytest.mark.parametrize("bad", [None, np.inf])
def test_adjoint(gpu_ctx, sizes, bad):
    """Both masked products over group tiles; a dC on a pattern that is not
    A.B's, and with an infinity (then only its own products see it)."""
    rng = np.random.default_rng(len(sizes))
    n = 110
    bs = np.resize(np.array(SIZES[sizes]), n)
    base = rng.random((3, n // 3 + 1, n // 3 + 1)) < 0.7
    pa, pb, pc = (np.kron(x, np.ones((3, 3), bool))[:n, :n] & (rng.random((n, n)) < 0.95) for x in base)
    a, b, dc = (_matrix(rng, bs, bs, p, cut=(40, 40)) for p in (pa, pb, pc))
    if bad is not None:
        dc.sectors[1].data[0] = bad
    da, db, ddc = (gpu_ctx.upload(x) for x in (a, b, dc))
    ga, gb = gpu_ctx.create_like(da), gpu_ctx.create_like(db)
    gpu_ctx.adjoint(da, db, ddc, ga, gb)
    A, B, D = a.to_dense(), b.to_dense(), dc.to_dense()
    with np.errstate(invalid="ignore"):
        if bad is None:
            want = {"a": D @ B.T, "b": A.T @ D}
        else:  # block by block, so that 0 * inf does not spread
            off = np.concatenate([[0], np.cumsum(bs)])
            want = {"a": np.zeros_like(A), "b": np.zeros_like(B)}
            for i in range(n):
                for k in range(n):
                    I, K = slice(off[i], off[i + 1]), slice(off[k], off[k + 1])
                    for j in np.nonzero(pc[i] & pb[k])[0]:
                        J = slice(off[j], off[j + 1])
                        want["a"][I, K] += D[I, J] @ B[K, J].T
                    for j in np.nonzero(pa[:, i] & pc[:, k])[0]:
                        J = slice(off[j], off[j + 1])
                        want["b"][I, K] += A[J, I].T @ D[J, K]
    for got, ref, p in ((ga.download(), want["a"], pa), (gb.download(), want["b"], pb)):
        mask = np.repeat(np.repeat(p, bs, 0), bs, 1)
        g = got.to_dense()
        assert [s.n_blks for s in got.sectors] == [int(p[r, c].sum()) for r in (slice(0, 40), slice(40, n))
                                                  for c in (slice(0, 40), slice(40, n))]
        fin = np.isfinite(ref) & mask
        assert np.array_equal(np.isfinite(g) & mask, fin)
        assert np.linalg.norm(g[fin] - ref[fin]) <= 1e-13 * np.linalg.norm(ref[fin])
    for x in (gb, ga, ddc, db, da):
        x.destroy()


@pytest.mark.parametrize("n", [40, 700])
@pytest.mark.parametrize("top", [3, 6, 24])
def test_norms_decide_the_filter(gpu_ctx, n, top):
    """Block norms over element counts around the 32 that are summed at a time,
    on few rows and on many (1,024 or 256 threads a row): the product filter at
    the median of the norm products must skip exactly what the oracle skips."""
    rng = np.random.default_rng([n, top])
    bs = rng.integers(0, top + 1, n)
    p = rng.random((n, n)) < (1.0 if n < 100 else 0.05)
    a, b = _matrix(rng, bs, bs, p), _matrix(rng, bs, bs, p)
    norms = np.array([np.linalg.norm(v) for v in block_values(a).values()])
    norms = norms[norms > 0]
    eps = float(np.median(rng.choice(norms, 1000) * rng.choice(norms, 1000)))
    c, ref = _check(gpu_ctx, a, b, eps, oracle.NO_RESULT_FILTER)
    assert rel_frobenius_error(c, ref) <= TOL
