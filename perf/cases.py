"""What a program that uses lamb_b200 has it do, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes what the program has in
hand, ``run`` is one pass through the public entry points (lamb_b200.gpu),
``work`` the bytes and flops the pass cannot do without and ``exact`` the
same outputs from dense 64-bit torch.

The matrices are those of the package's own workloads: water boxes (blocks of
O and H atoms, a distance cutoff, two x subsets) and the random-fill fixture.
A case fixes the geometry, so the block patterns; the seed gives the values.

Results of device-resident passes are taken as goods messages in device
memory (``DeviceMatrix.goods(sector, device=True)``): index and block data of
every sector, the form in which a result goes to torch or to another rank.
Passes on host data return the downloaded sectors.
"""
import functools
import math

import numpy as np
import torch

from lamb_b200 import gen, gpu
from lamb_b200.matrix import LambMatrix, Sector


# ---- the cases --------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: the reference's random-fill fixture (blocks of 0 to
        # 3 rows, fill 0.7) through the drop-in path, host sectors to host sectors.
        {"name": "host_fixture48", "kind": "host", "matrix": "fill", "n": 48, "geom": 3, "eps": 0.0},
        # A small box through the same path: upload, coordinates, multiply, download.
        {"name": "host_water64", "kind": "host", "matrix": "water", "n": 64, "cutoff": 6.0, "blk_o": 13, "geom": 0,
         "eps": 1e-8},
        # One multiply on resident matrices, the package's smallest named box.
        {"name": "fp64_water192", "kind": "multiply", "mixed": False, "n": 192, "cutoff": 6.0, "blk_o": 13, "geom": 0,
         "eps": 1e-8},
        # A larger O basis (23 functions) and an odd molecule count.
        {"name": "fp64_o23_water389", "kind": "multiply", "mixed": False, "n": 389, "cutoff": 7.3, "blk_o": 23,
         "geom": 5, "eps": 1e-10},
        # The benchmark's multiply: 18,432 atoms, cutoff 8, matrix dimension 141,312.
        {"name": "fp64_water6144", "kind": "multiply", "mixed": False, "n": 6144, "cutoff": 8.0, "blk_o": 13,
         "geom": 1, "eps": 1e-10},
        # The int8-digit product on the tensor cores: a small and a large box.
        {"name": "mixed_water200", "kind": "multiply", "mixed": True, "n": 200, "cutoff": 8.0, "blk_o": 13, "geom": 21,
         "eps": 1e-10},
        {"name": "mixed_water1536", "kind": "multiply", "mixed": True, "n": 1536, "cutoff": 7.0, "blk_o": 13,
         "geom": 4, "eps": 1e-10},
        # Backward of a multiply: both masked products on fixed patterns.
        {"name": "adjoint_water384", "kind": "adjoint", "n": 384, "cutoff": 6.0, "blk_o": 13, "geom": 9},
        # Purification, most steps on the mixed path and an FP64 tail.  No filter:
        # with one, the blocks next to it would come and go with the last bits.
        {"name": "purify_mixed_water96", "kind": "purify", "n": 96, "cutoff": 6.0, "blk_o": 13, "geom": 4,
         "steps": 30, "tail": 5, "eps": 0.0},
        # Purification in FP64 throughout, filtered as the benchmark's.
        {"name": "purify_fp64_water48", "kind": "purify", "n": 48, "cutoff": 5.5, "blk_o": 13, "geom": 6,
         "steps": 30, "tail": 30, "eps": 1e-10},
        # Uneven boxes in one batch: the whole multiply of every instance, and
        # the replayed numeric launch alone.
        {"name": "batch_full6", "kind": "batch", "full": True, "count": 6, "low": 96, "high": 384, "geom": 3,
         "eps": 1e-10},
        {"name": "batch_replay6", "kind": "batch", "full": False, "count": 6, "low": 96, "high": 384, "geom": 7,
         "eps": 1e-10},
    ]


def draw(rng):
    """One more case of the ranges above: sizes over their logarithm, cutoffs,
    O blocks of 13 or 23 functions; the work stays below the largest listed."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def cut(lo, hi):
        return round(rng.uniform(lo, hi), 2)

    geom = rng.randrange(1000)
    kind = rng.choice(["host", "multiply", "multiply", "multiply", "adjoint", "purify", "batch"])
    blk_o = rng.choice([13, 13, 23])
    if kind == "host":
        if rng.random() < 0.4:
            return {"kind": "host", "matrix": "fill", "n": size(12, 100), "geom": geom, "eps": 0.0}
        return {"kind": "host", "matrix": "water", "n": size(24, 200), "cutoff": cut(5.0, 7.0), "blk_o": blk_o,
                "geom": geom, "eps": rng.choice([0.0, 1e-10])}
    if kind == "multiply":
        return {"kind": "multiply", "mixed": rng.random() < 0.4, "n": size(48, 1200), "cutoff": cut(5.0, 7.5),
                "blk_o": blk_o, "geom": geom, "eps": rng.choice([0.0, 1e-10, 1e-8])}
    if kind == "adjoint":
        return {"kind": "adjoint", "n": size(24, 450), "cutoff": cut(5.0, 6.5), "blk_o": blk_o, "geom": geom}
    if kind == "purify":
        steps = rng.randint(8, 30)
        tail = rng.choice([5, steps])
        return {"kind": "purify", "n": size(16, 110), "cutoff": cut(4.5, 6.0), "blk_o": 13, "geom": geom,
                "steps": steps, "tail": tail, "eps": 0.0}
    return {"kind": "batch", "full": rng.random() < 0.6, "count": rng.randint(2, 7), "low": size(24, 96),
            "high": size(120, 400), "geom": geom, "eps": 1e-10}


# ---- inputs -----------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _geometry(n, cutoff, blk_o, geom):
    return gen.WaterGeometry(n, None, cutoff, blk_o=blk_o, seed=geom)


def _box(case):
    return _geometry(case["n"], case["cutoff"], case["blk_o"], case["geom"])


def _pair(g, seed):
    return g.matrix(2 * seed + 1), g.matrix(2 * seed + 2)


def _fill_pair(case, seed):
    """The fixture's pattern with values of the seed, and coordinates for its atoms."""
    pat = gen.random_fill_matrix(case["geom"], n_atoms=case["n"])
    rng = np.random.default_rng([case["geom"], seed])

    def values():
        return LambMatrix([Sector(s.subset_row, s.subset_col, s.row_blk_sizes, s.col_blk_sizes, s.row_p, s.col_i,
                                  s.extents, rng.random(s.data.shape[0])) for s in pat.sectors])
    xyz = np.random.default_rng(case["geom"]).random((case["n"], 3)).astype(np.float32)
    return values(), values(), xyz, 1.0


def _host_inputs(case, seed):
    if case["matrix"] == "fill":
        return _fill_pair(case, seed)
    g = _box(case)
    return (*_pair(g, seed), g.sector_positions(), g.box)


@functools.lru_cache(maxsize=64)
def _boxes(count, low, high, geom):
    """Uneven boxes as the benchmark's batch has them: sizes log-uniform, cutoffs uniform, O blocks of 13 and 23."""
    return tuple(_geometry(w.n_mol, w.cutoff, w.blk_o, w.geom_seed)
                 for w in gen.batch_instances(count, geom, (low, high), (5.0, 7.0)))


def _case_boxes(case):
    return _boxes(case["count"], case["low"], case["high"], case["geom"])


def _product_pattern(a, b, seed):
    """A matrix on the block pattern of A.B with normally distributed values (host sectors)."""
    p = (_pattern(a).float() @ _pattern(b).float() > 0).cpu().numpy()
    rb, cb = _sizes(a, 0), _sizes(b, 1)
    rs, cs = _starts(a.subset_blk_sizes(0)), _starts(b.subset_blk_sizes(1))
    rng = np.random.default_rng(seed)
    out = []
    for m in range(len(rs) - 1):
        for n in range(len(cs) - 1):
            r, c = np.nonzero(p[rs[m]:rs[m + 1], cs[n]:cs[n + 1]])
            sz = rb[rs[m] + r] * cb[cs[n] + c]
            end = np.cumsum(sz)
            row_p = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=rs[m + 1] - rs[m]))]).astype(np.int64)
            out.append(Sector(m + 1, n + 1, rb[rs[m]:rs[m + 1]].astype(np.int8), cb[cs[n]:cs[n + 1]].astype(np.int8),
                              row_p, (c + 1).astype(np.int16), np.stack([end - sz + 1, end], 1).astype(np.int64),
                              rng.standard_normal(int(end[-1]) if len(end) else 0)))
    return LambMatrix(out)


class _State:
    """What a program holds: device matrices (and a batch), given back with the object."""

    def __init__(self, case):
        self.case, self.ctx, self.mats, self.batch = case, gpu.default_context(), [], None

    def keep(self, m):
        self.mats.append(m)
        return m

    def __del__(self):
        if self.batch is not None:
            self.batch.destroy()
        for m in self.mats:
            m.destroy()


def prepare(case, seed):
    s = _State(case)
    ctx = s.ctx
    if case["kind"] == "host":
        s.a, s.b, s.xyz, s.box = _host_inputs(case, seed)
    elif case["kind"] == "multiply":
        g = _box(case)
        a, b = _pair(g, seed)
        s.a, s.b = s.keep(ctx.upload(a)), s.keep(ctx.upload(b))
        s.a.set_positions(g.sector_positions(), g.box)
        s.c = s.keep(ctx.create_like(s.a))
    elif case["kind"] == "adjoint":
        a, b = _pair(_box(case), seed)
        s.a, s.b = s.keep(ctx.upload(a)), s.keep(ctx.upload(b))
        s.dc = s.keep(ctx.upload(_product_pattern(a, b, seed)))
        s.da, s.db = s.keep(ctx.create_like(s.a)), s.keep(ctx.create_like(s.b))
    elif case["kind"] == "purify":
        s.h = s.keep(ctx.upload(gen.gapped_hamiltonian(_box(case), seed)))
        s.p = s.keep(ctx.create_like(s.h))
    else:
        s.cs, trip = [], []
        for i, g in enumerate(_case_boxes(case)):
            a, b = _pair(g, 100 * seed + i)
            da, db = s.keep(ctx.upload(a)), s.keep(ctx.upload(b))
            da.set_positions(g.sector_positions(), g.box)
            s.cs.append(s.keep(ctx.create_like(da)))
            trip.append((da, db, s.cs[-1]))
        s.batch = ctx.batch(*zip(*trip), eps=case["eps"])
    return s


# ---- the passes -------------------------------------------------------------------------
def _goods(m):
    return [m.goods(k, device=True) for k in range(4)]


def run(s):
    case, ctx = s.case, s.ctx
    if case["kind"] == "host":
        a, b = ctx.upload(s.a), ctx.upload(s.b)
        a.set_positions(s.xyz, s.box)
        c = ctx.create_like(a)
        ctx.multiply(a, b, c, case["eps"], gpu.ASYNC)
        out = c.download()
        for m in (c, b, a):
            m.destroy()
        return [{"row_p": x.row_p, "col_i": x.col_i, "extents": x.extents, "data": x.data} for x in out.sectors]
    if case["kind"] == "multiply":
        ctx.multiply(s.a, s.b, s.c, case["eps"], gpu.MIXED if case["mixed"] else gpu.FP64)
        return _goods(s.c)
    if case["kind"] == "adjoint":
        ctx.adjoint(s.a, s.b, s.dc, s.da, s.db)
        return {"da": _goods(s.da), "db": _goods(s.db)}
    if case["kind"] == "purify":
        rep = ctx.purify(s.h, s.p, mu=0.0, steps=case["steps"], fp64_tail=case["tail"], eps=case["eps"])
        return {"p": _goods(s.p), "trace": rep["trace"]}
    if case["full"]:
        s.batch.run_full()
    else:
        s.batch.execute()
    return [_goods(c) for c in s.cs]


# ---- dense 64-bit restatement -------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _starts(parts):
    return np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.int64)


def _sizes(m, axis):
    return np.concatenate(m.subset_blk_sizes(axis)).astype(np.int64)


def _pattern(m):
    """Block pattern over atoms in sector order (a boolean matrix)."""
    rs, cs = _starts(m.subset_blk_sizes(0)), _starts(m.subset_blk_sizes(1))
    p = np.zeros((rs[-1], cs[-1]), bool)
    for s in m.sectors:
        p[rs[s.subset_row - 1] + s.block_rows(), cs[s.subset_col - 1] + s.col_i.astype(np.int64) - 1] = True
    return torch.from_numpy(p).to(_dev())


def _positions(pattern, rb, cb, rs, cs, order=None):
    """Per sector, the place in the dense matrix of every value of its data
    store: rows in `order` (default: as they are), a row's blocks by column,
    a block's elements by column."""
    dev = pattern.device
    rbt, cbt = torch.from_numpy(rb).to(dev), torch.from_numpy(cb).to(dev)
    ro, co = torch.cumsum(rbt, 0) - rbt, torch.cumsum(cbt, 0) - cbt
    width = int(cb.sum())
    order = np.arange(len(rb)) if order is None else order
    out = []
    for m in range(len(rs) - 1):
        rows = torch.from_numpy(order[(order >= rs[m]) & (order < rs[m + 1])]).to(dev)
        for n in range(len(cs) - 1):
            r, c = torch.nonzero(pattern[rows][:, cs[n]:cs[n + 1]], as_tuple=True)
            r, c = rows[r], c + int(cs[n])
            sz = rbt[r] * cbt[c]
            first = torch.repeat_interleave(torch.cumsum(sz, 0) - sz, sz)
            e = torch.arange(first.shape[0], device=dev) - first
            blk = torch.repeat_interleave(torch.arange(r.shape[0], device=dev), sz)
            h = torch.clamp(rbt[r][blk], min=1)
            out.append((ro[r][blk] + e % h) * width + co[c][blk] + e // h)
    return out


def _structure(m):
    return (_sizes(m, 0), _sizes(m, 1), _starts(m.subset_blk_sizes(0)), _starts(m.subset_blk_sizes(1)))


def _dense(m):
    """Dense matrix of host sectors whose blocks are stored one after another in row order."""
    rb, cb, rs, cs = _structure(m)
    d = torch.zeros(int(rb.sum()) * int(cb.sum()), dtype=torch.float64, device=_dev())
    for s, pos in zip(m.sectors, _positions(_pattern(m), rb, cb, rs, cs)):
        d[pos] = torch.from_numpy(s.data).to(d.device)
    return d.view(int(rb.sum()), int(cb.sum()))


def _morton(xyz, box):
    """Atoms along the Z curve of their cells (1,024 a side), ties by index: the order of a result's rows."""
    b = np.broadcast_to(np.asarray(box, np.float32), (3,))
    f = np.asarray(xyz, np.float32) / b
    q = np.clip(((f - np.floor(f)) * np.float32(1024)).astype(np.int64), 0, 1023)
    key = np.zeros(len(q), np.int64)
    for bit in range(10):
        for d in range(3):
            key |= ((q[:, d] >> bit) & 1) << (3 * bit + d)
    return np.argsort(key, kind="stable")


def _exact_product(a, b, xyz, box):
    rb, cb = _sizes(a, 0), _sizes(b, 1)
    rs, cs = _starts(a.subset_blk_sizes(0)), _starts(b.subset_blk_sizes(1))
    p = _pattern(a).float() @ _pattern(b).float() > 0
    d = (_dense(a) @ _dense(b)).view(-1)
    return [d[x] for x in _positions(p, rb, cb, rs, cs, _morton(xyz, box))]


def exact(case, seed):
    if case["kind"] == "host":
        return [{"row_p": None, "col_i": None, "extents": None, "data": x.cpu().numpy()}
                for x in _exact_product(*_host_inputs(case, seed))]
    if case["kind"] == "multiply":
        if case["n"] > 1600:
            return None  # a dense product of dimension 141,312
        g = _box(case)
        return [(None, x) for x in _exact_product(*_pair(g, seed), g.sector_positions(), g.box)]
    if case["kind"] == "adjoint":
        a, b = _pair(_box(case), seed)
        da, db, dc = _dense(a), _dense(b), _dense(_product_pattern(a, b, seed))
        ga, gb = (dc @ db.T).view(-1), (da.T @ dc).view(-1)
        return {"da": [(None, ga[x]) for x in _positions(_pattern(a), *_structure(a))],
                "db": [(None, gb[x]) for x in _positions(_pattern(b), *_structure(b))]}
    if case["kind"] == "purify":
        hm = gen.gapped_hamiltonian(_box(case), seed)
        h = _dense(hm)
        d = torch.diagonal(h)
        rad = h.abs().sum(1) - d.abs()
        lam = min(1.0 / float((d + rad).max()), -1.0 / float((d - rad).min()))
        p = 0.5 * torch.eye(h.shape[0], dtype=torch.float64, device=h.device) - 0.5 * lam * h
        for _ in range(case["steps"]):
            p2 = p @ p
            p = 3 * p2 - 2 * p2 @ p
        rb, cb, rs, cs = _structure(hm)
        full = torch.ones(len(rb), len(cb), dtype=torch.bool, device=h.device)
        return {"p": [(None, p.reshape(-1)[x]) for x in _positions(full, rb, cb, rs, cs)],
                "trace": float(torch.trace(p))}
    return [[(None, x) for x in _exact_product(*_pair(g, 100 * seed + i), g.sector_positions(), g.box)]
            for i, g in enumerate(_case_boxes(case))]


# ---- what a pass cannot do without ----------------------------------------------------------
def _box_work(g):
    """Bytes of A, B and C (values and index) and flops of one product on a box."""
    n, b = g.n_atoms, torch.from_numpy(g.blk.astype(np.float64))
    x = torch.from_numpy(g.positions)
    p = torch.zeros(n, n, dtype=torch.bool)
    for lo in range(0, n, 1024):
        d = x[lo:lo + 1024, None, :] - x[None]
        d -= g.box * torch.round(d / g.box)
        p[lo:lo + 1024] = (d * d).sum(-1) < g.cutoff ** 2
    pf = p.float().to(_dev())
    pc = (pf @ pf > 0).double().cpu()
    pd = p.double()
    flops = 2.0 * float(((pd.T @ b) * b * (pd @ b)).sum())
    val = lambda q: 8.0 * float(b @ q @ b) + 18.0 * float(q.sum()) + 8.0 * n  # noqa: E731
    return {"a": val(pd), "c": val(pc), "flops": flops}


@functools.lru_cache(maxsize=64)
def _work_of(n, cutoff, blk_o, geom):
    return _box_work(_geometry(n, cutoff, blk_o, geom))


def work(case):
    if case["kind"] == "batch":
        w = [_work_of(g.n_mol, g.cutoff, int(g.blk.max()), g.seed) for g in _case_boxes(case)]
        return {"bytes": sum(2 * x["a"] + x["c"] for x in w), "flops": sum(x["flops"] for x in w)}
    if case["kind"] == "host" and case["matrix"] == "fill":
        m = gen.random_fill_matrix(case["geom"], n_atoms=case["n"])
        p, rb = _pattern(m).double().cpu(), torch.from_numpy(_sizes(m, 0)).double()
        val = lambda q: 8.0 * float(rb @ q @ rb) + 18.0 * float(q.sum())  # noqa: E731
        return {"bytes": 2 * val(p) + val((p @ p > 0).double()), "flops": 2.0 * float(((p.T @ rb) * rb * (p @ rb)).sum())}
    w = _work_of(case["n"], case["cutoff"], case["blk_o"], case["geom"])
    if case["kind"] == "adjoint":  # A, B and dC read, dA and dB written; each masked product has the forward's flops
        return {"bytes": 4 * w["a"] + w["c"], "flops": 2 * w["flops"]}
    if case["kind"] == "purify":  # P is dense after the first steps; two products a step and the idempotency check
        dim = float(_box(case).blk.astype(np.int64).sum())
        return {"bytes": w["a"] + 8.0 * dim * dim, "flops": (2 * case["steps"] + 1) * 2.0 * dim ** 3}
    return {"bytes": 2 * w["a"] + w["c"], "flops": w["flops"]}
