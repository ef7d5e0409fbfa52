"""Products on a GPU that is nearly full.  A library loaded ahead of the CUDA
runtime (tests/low_memory.cpp) refuses allocations beyond a limit.  Group tiles
need panels and tables that the stacks do without: with room for the stacks
only, a product must still come, with the same bits (both add a C element's
products in the same order)."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MB = 1 << 20


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("low_memory") / "low_memory.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror",
                           os.path.join(REPO, "tests", "low_memory.cpp"), "-o", out, "-ldl"])
    return out


def _run(shim, case):
    env = dict(os.environ, LD_PRELOAD=shim, PYTHONPATH=REPO)
    r = subprocess.run([sys.executable, os.path.abspath(__file__), shim, case], env=env, cwd=REPO, text=True,
                       capture_output=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["panels", "panels_filtered", "tables", "adjoint"])
def test_stacks_where_panels_do_not_fit(shim, case):
    _run(shim, case)


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["upload", "copy", "adjoint_stacks"])
def test_idle_scratch_is_given_back(shim, how):
    """The panels of a finished product stay with the context, but not when
    something else needs the memory."""
    _run(shim, "idle_" + how)


# ---- the child process ------------------------------------------------------------------
def _band(rng, n, sizes, width):
    """Atoms in runs of len(sizes) that couple to the same atoms, `width` runs to either side."""
    from lamb_b200.matrix import LambMatrix, Sector
    k = len(sizes)
    bs = np.resize(np.array(sizes), n * k)
    run = np.arange(n * k) // k
    lo, hi = np.maximum(run - width, 0) * k, np.minimum(run + width + 1, n) * k
    cnt = hi - lo
    r = np.repeat(np.arange(n * k), cnt)
    row_p = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    c = np.arange(row_p[-1]) - np.repeat(row_p[:-1], cnt) + np.repeat(lo, cnt)
    end = np.cumsum(bs[r].astype(np.int64) * bs[c])
    first = np.concatenate([[0], end[:-1]])
    return LambMatrix([Sector(1, 1, bs.astype(np.int8), bs.astype(np.int8), row_p, (c + 1).astype(np.int16),
                              np.stack([first + 1, end], 1), rng.standard_normal(int(end[-1])))])


def _bytes_of(sizes):
    """Device bytes of a result: row_p, col, off and data."""
    return sum(8 * (s.n_rows + 1) + 12 * s.n_blks + 8 * s.data_len for s in sizes)


def _idle(gpu, mem, case):
    rng = np.random.default_rng(1)
    a, b = _band(rng, 1300, [13, 5, 5], 10), _band(rng, 1300, [13, 5, 5], 10)
    ctx = gpu.Context(0)
    da, db = ctx.upload(a), ctx.upload(b)
    dc = ctx.create_like(da)
    ctx.synchronize()
    held = mem.low_memory_live()
    ctx.multiply(da, db, dc, 0.0)
    c_bytes = _bytes_of(dc.sizes())
    kept = mem.low_memory_live() - held - c_bytes
    assert kept > 200 * MB  # the panels
    want = dc.download()
    # room for less than a second C beside the panels, and for more than one without them
    mem.low_memory_limit(held + c_bytes + kept + c_bytes // 2)
    if case == "idle_upload":
        m = ctx.upload(want)
    elif case == "idle_copy":
        m = ctx.create_like(dc)
        ctx.copy(dc, m)
    else:  # blocks of 25 rows take no panels: results of 2 x 100 MB, stacks of 40 MB
        mem.low_memory_limit(1 << 62)
        x = [ctx.upload(_band(rng, 700, [25, 5], 10)) for _ in range(3)]
        ga, gb = ctx.create_like(x[0]), ctx.create_like(x[1])
        mem.low_memory_limit(mem.low_memory_live() + 100 * MB)
        ctx.adjoint(*x, ga, gb)
        m = dc
    got = m.download()
    for s, t in zip(got.sectors, want.sectors):
        assert np.array_equal(s.data, t.data) and np.array_equal(s.col_i, t.col_i)
    # and the next product makes its panels again
    mem.low_memory_limit(ctypes.c_size_t(-1).value)
    ctx.multiply(da, db, dc, 0.0)
    for s, t in zip(dc.download().sectors, want.sectors):
        assert np.array_equal(s.data, t.data)
    ctx.close()


def _child(path, case):
    from lamb_b200 import gpu
    mem = ctypes.CDLL(path)
    for f in ("low_memory_live", "low_memory_peak"):
        getattr(mem, f).restype = ctypes.c_size_t
    mem.low_memory_limit.argtypes = [ctypes.c_size_t]
    if case.startswith("idle"):
        return _idle(gpu, mem, case)
    none = ctypes.c_size_t(-1).value
    rng = np.random.default_rng(1)
    # `stacks`: what the stack kernel's entries, work items and tables take, generously
    if case == "tables":  # many atoms of one row: bitmaps of 2 x 122 MB, a result of 25 MB
        shape, eps, stacks = (4000, [1] * 8, 1), 0.0, 120 * MB
    elif case == "adjoint":  # stacks of 4 million products, panels of 2 x 132 MB
        shape, eps, stacks = (6000, [13, 5, 5], 2), 0.0, 120 * MB
    else:
        # panels of 2 x 120 MB, with norms 2 x 15 MB more; the stacks run in three chunks of 5.1 million
        # products, 16 bytes each: 87 MB of entries, 20 MB of work items, offsets and norms
        shape, eps, stacks = (1300, [13, 5, 5], 10), (40.0 if case == "panels_filtered" else 0.0), 120 * MB
    a, b, d = (_band(rng, *shape) for _ in range(3))
    ctx = gpu.Context(0)
    da, db, dd = (ctx.upload(x) for x in (a, b, d))

    def product():
        if case == "adjoint":
            ga, gb = ctx.create_like(da), ctx.create_like(db)
            ctx.adjoint(da, db, dd, ga, gb)
            return [ga, gb]
        dc = ctx.create_like(da)
        ctx.multiply(da, db, dc, eps, gpu.NO_RESULT_FILTER)
        return [dc]

    ctx.synchronize()
    held = mem.low_memory_live()
    mem.low_memory_peak(1)
    out = product()
    used = mem.low_memory_peak(0) - held
    want = [m.download() for m in out]
    need = sum(_bytes_of(m.sizes()) for m in out) + stacks
    for m in out:
        m.destroy()
    assert used > need + 60 * MB, (used, need)  # the panels are what the limit takes away
    ctx.close()
    # every limit from what the tiles took down to what the stacks need, on a new context each
    for limit in np.linspace(used + MB, need, 9):
        mem.low_memory_limit(none)
        ctx = gpu.Context(0)
        da, db, dd = (ctx.upload(x) for x in (a, b, d))
        ctx.synchronize()
        held = mem.low_memory_live()
        for _ in range(2):
            mem.low_memory_limit(held + int(limit))
            out = product()
            mem.low_memory_limit(none)
            for m, w in zip(out, want):
                for s, t in zip(m.download().sectors, w.sectors):
                    assert np.array_equal(s.row_p, t.row_p) and np.array_equal(s.col_i, t.col_i)
                    assert np.array_equal(s.extents, t.extents) and np.array_equal(s.data, t.data)
                m.destroy()
        ctx.close()
    # too little for anything: an error status, and the context goes on
    mem.low_memory_limit(none)
    ctx = gpu.Context(0)
    da, db, dd = (ctx.upload(x) for x in (a, b, d))
    ctx.synchronize()
    mem.low_memory_limit(mem.low_memory_live() + 4 * MB)
    try:
        product()
        raise SystemExit("a product fitted into 4 MB")
    except gpu.LambError as e:
        assert e.level == 4, e
    mem.low_memory_limit(none)
    for m, w in zip(product(), want):
        assert all(np.array_equal(s.data, t.data) for s, t in zip(m.download().sectors, w.sectors))
    ctx.close()


if __name__ == "__main__":
    _child(sys.argv[1], sys.argv[2])
