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
