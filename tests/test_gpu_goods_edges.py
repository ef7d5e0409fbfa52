"""Goods messages written on the device, at the edges of their sections: empty
sectors, block counts that do not fill the last column word, blocks without
elements, rows without blocks, host and device destinations."""
import numpy as np
import pytest
import torch

from oracle import goods as og
from lamb_b200.gen import random_fill_matrix
from lamb_b200.matrix import LambMatrix, Sector

pytestmark = pytest.mark.gpu


def _one(n_rows, n_cols, present):
    r, c = np.nonzero(present)
    row_p = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n_rows))]).astype(np.int64)
    sz = np.full(len(r), 6)
    end = np.cumsum(sz)
    return LambMatrix([Sector(1, 1, np.full(n_rows, 2, np.int8), np.full(n_cols, 3, np.int8), row_p,
                              (c + 1).astype(np.int16), np.stack([end - sz + 1, end], 1).astype(np.int64).reshape(-1, 2),
                              np.arange(6.0 * len(r)))])


def _cases():
    rng = np.random.default_rng(0)
    yield "none", _one(3, 4, np.zeros((3, 4), bool))
    for n in (1, 2, 3, 4, 5):
        p = np.zeros((4, 9), bool)
        p.flat[rng.choice(36, n, replace=False)] = True
        yield f"blocks{n}", _one(4, 9, p)
    yield "rows1025", _one(1025, 2, rng.random((1025, 2)) < 0.4)
    yield "row_major", _one(2, 1200, np.ones((2, 1200), bool))
    for s in (0, 4, 9):
        yield f"fill{s}", random_fill_matrix(s, n_atoms=30 + s)


@pytest.mark.parametrize("name,m", list(_cases()), ids=[n for n, _ in _cases()])
def test_message_bytes(gpu_ctx, name, m):
    d = gpu_ctx.upload(m)
    for k, s in enumerate(d.download().sectors):
        ref_idx, ref_data = og.pack(s)
        idx, data = d.goods(k)
        assert np.array_equal(idx, ref_idx) and np.array_equal(data, ref_data)
        tidx, tdat = d.goods(k, device=True)
        assert torch.equal(tidx.cpu(), torch.from_numpy(ref_idx)) and torch.equal(tdat.cpu(), torch.from_numpy(ref_data))
    d.destroy()
