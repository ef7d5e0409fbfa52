"""FP64 products whose bounded waits run out.  A context whose limit is 0 counts
every wait of the group tile kernel as run out: its warps record that, let their
copies land and end, so the calls return an error status and the context stays
usable."""
import pytest

import oracle
from lamb_b200 import gpu
from lamb_b200.gen import WaterGeometry
from tests.helpers import assert_same_pattern, rel_frobenius_error

pytestmark = pytest.mark.gpu


@pytest.fixture
def stopping(monkeypatch):
    """A context in which every product on group tiles stops."""
    monkeypatch.setenv("LAMB_GPU_WAIT_MS", "0")
    ctx = gpu.Context(0)
    monkeypatch.delenv("LAMB_GPU_WAIT_MS")
    yield ctx
    ctx.close()


def _box(n=72, seed=3):
    g = WaterGeometry(n, None, 6.0, seed=seed)
    return g, g.matrix(1), g.matrix(2)


@pytest.mark.parametrize("n", [72, 260])
@pytest.mark.parametrize("eps", [0.0, 1e-8])
def test_multiply_reports_and_the_context_stays_usable(stopping, n, eps):
    g, a, b = _box(n)
    da, db = stopping.upload(a), stopping.upload(b)
    da.set_positions(g.sector_positions(), g.box)
    dc = stopping.create_like(da)
    for _ in range(2):
        with pytest.raises(gpu.LambError, match="a wait ran out"):
            stopping.multiply(da, db, dc, eps)
    stopping.synchronize()  # told once a product, not again
    # other products of the same context: digits on the tensor cores, and stacks (few block products)
    stopping.multiply(da, db, dc, 0.0, gpu.MIXED)
    ref, _ = oracle.multiply(a, b, 0.0)
    c = dc.download()
    assert_same_pattern(c, ref)
    assert rel_frobenius_error(c, ref) <= 1e-11
    gs, sa, sb = _box(12)
    ea, eb = stopping.upload(sa), stopping.upload(sb)
    ec = stopping.create_like(ea)
    stopping.multiply(ea, eb, ec, 0.0)
    assert rel_frobenius_error(ec.download(), oracle.multiply(sa, sb, 0.0)[0]) <= 1e-12


def test_adjoint_reports(stopping):
    _, a, b = _box()
    da, db, dc = stopping.upload(a), stopping.upload(b), stopping.upload(a)
    ga, gb = stopping.create_like(da), stopping.create_like(db)
    with pytest.raises(gpu.LambError, match="a wait ran out"):
        stopping.adjoint(da, db, dc, ga, gb)
    stopping.synchronize()


def _tell_goods(ctx, c):
    c.goods(0)


def _tell_goods_device(ctx, c):
    c.goods(3, device=True)


def _tell_download(ctx, c):
    c.download()


def _tell_multiply(ctx, c):
    ctx.multiply(c, c, ctx.create_like(c), 0.0, gpu.ASYNC)


def _tell_mixed(ctx, c):
    ctx.multiply(c, c, ctx.create_like(c), 0.0, gpu.MIXED)


def _tell_axpby(ctx, c):
    ctx.axpby(1.0, c, 1.0, ctx.create_like(c))


def _tell_copy(ctx, c):
    ctx.copy(c, ctx.create_like(c))


def _tell_scale(ctx, c):
    ctx.scale_shift(c, 2.0, 0.0)


def _tell_norm(ctx, c):
    ctx.frobenius(c)


def _tell_synchronize(ctx, c):
    ctx.synchronize()


TELLERS = {f.__name__[6:]: f for f in (_tell_goods, _tell_goods_device, _tell_download, _tell_multiply, _tell_mixed,
                                       _tell_axpby, _tell_copy, _tell_scale, _tell_norm, _tell_synchronize)}


@pytest.mark.parametrize("eps", [0.0, 1e-8])
@pytest.mark.parametrize("who", sorted(TELLERS) + ["trace", "trace_product", "diff_frobenius"])
def test_asynchronous_product_is_told_once(stopping, who, eps):
    """With eps > 0 a result filter is pending: the calls in between complete it,
    and leave the error to the call that returns data."""
    tell = TELLERS.get(who)
    if tell is None:
        tell = lambda ctx, c: getattr(ctx, who)(*([c] if who == "trace" else [c, c]))  # noqa: E731
    g, a, b = _box()
    da, db = stopping.upload(a), stopping.upload(b)
    dc = stopping.create_like(da)
    stopping.multiply(da, db, dc, eps, gpu.ASYNC)
    stopping.create_like(dc).destroy()
    dc.sizes()
    db.destroy()
    with pytest.raises(gpu.LambError, match="a wait ran out"):
        tell(stopping, dc)
    stopping.synchronize()


@pytest.mark.parametrize("eps", [0.0, 1e-8])
def test_destroyed_context_tells(monkeypatch, eps):
    monkeypatch.setenv("LAMB_GPU_WAIT_MS", "0")
    ctx = gpu.Context(0)
    g, a, b = _box()
    da, db = ctx.upload(a), ctx.upload(b)
    dc = ctx.create_like(da)
    ctx.multiply(da, db, dc, eps, gpu.ASYNC)
    status = gpu.lib().lamb_gpu_ctx_destroy(ctx._h)
    ctx._h = type(ctx._h)()
    assert gpu.lib().lamb_gpu_status_level(status) == 3 and gpu.lib().lamb_gpu_status_type(status) == -1
