"""Column split at the borders of the tiles it moves entries by, with lines of empty rows, and columns out of order
at any place of a tile."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(lens, n, chunks, seed):
    from scorch_b200 import kernels as K
    rng = np.random.default_rng(seed)
    pos = np.zeros(len(lens) + 1, np.int32)
    np.cumsum(lens, out=pos[1:])
    crd = np.concatenate([np.sort(rng.integers(0, n, x)) for x in lens]).astype(np.int32)
    val = rng.standard_normal(len(crd)).astype(np.float32)
    d = lambda a: torch.from_numpy(a).cuda()
    s = K.ColumnSplit(d(pos), d(crd), d(val), n, chunks)
    width, row = -(-n // chunks), np.repeat(np.arange(len(lens)), lens)
    for c in range(chunks):
        here = crd // width == c
        first, count = s.first[c], s.counts[c]
        assert count == here.sum()
        assert np.array_equal(np.diff(s.pos[c].cpu().numpy()), np.bincount(row[here], minlength=len(lens)))
        assert np.array_equal(s.crd[first:first + count].cpu().numpy(), crd[here])
        assert np.array_equal(s.val[first:first + count].cpu().numpy(), val[here])


@pytest.mark.parametrize("total", [1, 31, 1023, 1024, 1025, 8191, 8192, 8193, 16385])
@pytest.mark.parametrize("chunks", [1, 3, 64])
def test_tile_borders(total, chunks):
    rng = np.random.default_rng(total)
    cuts = np.sort(rng.integers(0, total + 1, 40))
    _check([int(x) for x in np.diff(np.concatenate([[0], cuts, [total]]))], 1000, chunks, total)


def test_lines_of_empty_rows():
    _check([0] * 1500 + [3] + [0] * 1024 + [1] * 2100 + [0] * 700 + [9000, 0, 2] + [0] * 40, 5000, 5, 0)


@pytest.mark.parametrize("at", [1, 31, 32, 255, 256, 1024, 8191, 8192, 8200, 9999])
def test_columns_out_of_order_are_seen(at):
    from scorch_b200 import _lib, kernels as K
    crd = np.arange(10000, dtype=np.int32)
    crd[at] = crd[at - 1] - 1 if at > 1 else 0
    crd[at - 1] += 1
    pos = np.array([0, 0, 10000, 10000], np.int32)
    d = lambda a: torch.from_numpy(a).cuda()
    with pytest.raises(_lib.ScorchB200Error):
        K.ColumnSplit(d(pos), d(crd), torch.ones(10000, device="cuda"), 10001, 4)
    # the same between two rows is no disorder
    K.ColumnSplit(d(np.array([0, at, 10000], np.int32)), d(np.concatenate([np.arange(at), np.arange(10000 - at)]).astype(np.int32)),
                  torch.ones(10000, device="cuda"), 10001, 4)
