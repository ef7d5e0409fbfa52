"""Which kernel computes an FP64 product: the context's trace names it.  The
shapes are those of the group tile tests, which compare the results; here the
tiles must be the ones that ran, and the stacks where the rules say so."""
import numpy as np
import pytest

import oracle
from lamb_b200 import gpu
from lamb_b200.gen import WaterGeometry
from tests.helpers import assert_same_pattern, rel_frobenius_error
from tests.test_gpu_panel import SIZES, _matrix

pytestmark = pytest.mark.gpu

# as for the group tile tests: the same sums in the same order
TOL = 1e-12


class Traced:
    def __init__(self, ctx, capfd):
        self.ctx, self.capfd = ctx, capfd

    def routes(self, names=("numeric",)):
        """Kernels named since the last call, in order."""
        lines = self.capfd.readouterr().err.splitlines()
        return [x.split("(")[1].split(")")[0] for x in lines
                if "[lamb trace]" in x and x.split("[lamb trace] ")[1].split(" (")[0] in names]


@pytest.fixture
def traced(monkeypatch, capfd):
    monkeypatch.setenv("LAMB_GPU_TRACE", "2")
    ctx = gpu.Context(0)
    monkeypatch.delenv("LAMB_GPU_TRACE")
    yield Traced(ctx, capfd)
    ctx.close()


def _product(t, a, b, eps=0.0, flags=0):
    da, db = t.ctx.upload(a), t.ctx.upload(b)
    dc = t.ctx.create_like(da)
    t.routes()
    t.ctx.multiply(da, db, dc, eps, flags)
    (route,) = t.routes()
    c = dc.download()
    ref, _ = oracle.multiply(a, b, eps, flags)
    assert_same_pattern(c, ref)
    assert rel_frobenius_error(c, ref) <= TOL
    for m in (dc, db, da):
        m.destroy()
    return route


def _grouped(rng, n, fill):
    """A pattern in which runs of three atoms couple to nearly the same atoms."""
    base = rng.random((n // 3 + 1, n // 3 + 1)) < fill
    return np.kron(base, np.ones((3, 3), bool))[:n, :n] & (rng.random((n, n)) < 0.9)


@pytest.mark.parametrize("sizes", sorted(SIZES))
@pytest.mark.parametrize("fill", [0.6, 1.0])
def test_block_sizes(traced, sizes, fill):
    rng = np.random.default_rng([len(sizes), int(10 * fill)])
    bs = np.resize(np.array(SIZES[sizes]), 151)
    p = _grouped(rng, 151, fill)
    a, b = _matrix(rng, bs, bs, p, cut=(61, 61)), _matrix(rng, bs, bs, p.T, cut=(61, 61))
    assert _product(traced, a, b) == ("stacks" if sizes == "beyond" else "group tiles")


# norms of the 17 to 24 rows' blocks are about 14 and 20: below 200 few products fall, and what the
# tiles gain is counted in products that pass
@pytest.mark.parametrize("eps", [0.0, 120.0, 200.0])
def test_groups_of_one_atom(traced, eps):
    """Unrelated neighbours: blocks of 17 rows and more still take the tiles
    (their products fill two 16-row slabs a side), also where the filter splits them;
    blocks of 9 rows do not."""
    rng = np.random.default_rng(8)
    n = 120
    p = rng.random((n, n)) < 0.45
    for lo, hi, want in ((17, 25, "group tiles"), (9, 10, "stacks")):
        bs = rng.integers(lo, hi, n)
        bs[::7] = lo
        a, b = _matrix(rng, bs, bs, p), _matrix(rng, bs, bs, p.T)
        a.sectors[0].data *= rng.choice([0.2, 1.0], a.sectors[0].data.size)
        big = np.concatenate([p, p]), np.concatenate([bs, bs])  # twice the rows: half a million products
        a = _matrix(rng, big[1], bs, big[0])
        b = _matrix(rng, bs, big[1], big[0].T)
        assert len(a.sectors[0].col_i) * len(b.sectors[0].col_i) >= n << 19
        assert _product(traced, a, b, eps, oracle.NO_RESULT_FILTER) == want


def test_water_boxes_and_small_or_non_finite_operands(traced):
    g = WaterGeometry(72, None, 6.0, seed=3)
    a, b = g.matrix(1), g.matrix(2)
    assert _product(traced, a, b) == "group tiles"
    assert _product(traced, a, b, 1e-6) == "group tiles"
    s = WaterGeometry(12, None, 6.0, seed=3)
    assert _product(traced, s.matrix(1), s.matrix(2)) == "stacks"
    b.sectors[0].data[7] = np.inf
    da, db = traced.ctx.upload(a), traced.ctx.upload(b)
    dc = traced.ctx.create_like(da)
    traced.routes()
    traced.ctx.multiply(da, db, dc, 0.0)
    assert traced.routes() == ["stacks"]


def test_adjoint(traced):
    rng = np.random.default_rng(2)
    for sizes, want in (("molecule", "group tiles"), ("beyond", "stacks")):
        bs = np.resize(np.array(SIZES[sizes]), 110)
        a, b, d = (_matrix(rng, bs, bs, _grouped(rng, 110, 0.8)) for _ in range(3))
        da, db, dd = (traced.ctx.upload(x) for x in (a, b, d))
        ga, gb = traced.ctx.create_like(da), traced.ctx.create_like(db)
        traced.routes()
        traced.ctx.adjoint(da, db, dd, ga, gb)
        assert traced.routes(("dA", "dB")) == [want, want]
        d.sectors[0].data[0] = np.nan  # met while packing: both products again, on stacks
        dn = traced.ctx.upload(d)
        traced.ctx.adjoint(da, db, dn, ga, gb)
        assert traced.routes(("dA", "dB")) == ["stacks", "stacks"]


@pytest.mark.parametrize("positions", [False, True])
def test_groups_inherited_from_another_pattern(traced, positions):
    """A result keeps the groups of its factors, whatever its own pattern: of a
    sparser matrix, of one atom each (from a factor whose neighbours are
    unrelated), through copies and sums."""
    ctx = traced.ctx
    g = WaterGeometry(72, None, 6.0, seed=3)
    a, b = g.matrix(1), g.matrix(2)
    sizes = np.concatenate(a.subset_blk_sizes(0)).astype(int)
    half = len(a.subset_blk_sizes(0)[0])
    rng = np.random.default_rng(4)
    one = _matrix(rng, sizes, sizes, rng.random((len(sizes),) * 2) < 0.4, cut=(half, half))

    def up(m):
        d = ctx.upload(m)
        if positions:
            d.set_positions(g.sector_positions(), g.box)
        return d

    def check(dx, dy, x, y):
        dz = ctx.create_like(dx)
        ctx.multiply(dx, dy, dz, 0.0)
        z, ref = dz.download(), oracle.multiply(x, y, 0.0)[0]
        assert_same_pattern(z, ref)
        assert rel_frobenius_error(z, ref) <= TOL
        return dz, z

    da, db, d1 = up(a), up(b), up(one)
    dc, c = check(da, db, a, b)            # groups of the box
    dd, d = check(dc, db, c, b)            # on a denser matrix
    check(dd, dc, d, c)
    de, e = check(d1, db, one, b)          # groups of one atom
    check(de, db, e, b)
    df = ctx.create_like(da)
    ctx.copy(de, df)
    ctx.axpby(1.0, dc, 2.0, df)
    check(df, db, df.download(), b)
    ctx.copy(dc, df)
    ctx.axpby(0.5, de, 1.0, df)
    traced.routes()
    check(df, db, df.download(), b)
    assert traced.routes() == ["group tiles"]
