"""Per-row top-k at the edges of its two selections (bound + ranking, radix passes)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rows(kind, m, n, rng):
    x = rng.standard_normal((m, n)).astype(np.float32)
    if kind == "ties":                      # far more equal values than candidates are kept for
        x = np.round(x * 2) / 2 + 0.0          # (no -0: the oracle does not order it below +0)
    elif kind == "zeros":                   # fewer positives than k
        x = np.maximum(x - 3.2, 0).astype(np.float32)
    elif kind == "sorted":
        x = np.sort(x, 1)
    elif kind == "special":
        x[:, ::7], x[:, 3::11], x[:, 5::13] = np.inf, -np.inf, 0.0
    return x


@pytest.mark.parametrize("kind", ["normal", "ties", "zeros", "sorted", "special"])
@pytest.mark.parametrize("n,k", [(1, 1), (31, 31), (513, 256), (1000, 257), (4096, 32), (5003, 64), (32768, 33)])
def test_topk_selection(kind, n, k):
    from scorch_b200 import kernels as K
    x = _rows(kind, 5, n, np.random.default_rng(n + k))
    pos, crd, val = K.topk_rows_to_csr(torch.from_numpy(x).cuda(), k)
    wpos, wcrd, wval = O.topk_rows_to_csr(x, k, False)
    assert np.array_equal(pos.cpu().numpy(), wpos) and np.array_equal(val.cpu().numpy(), wval)
    assert np.array_equal(crd.cpu().numpy(), wcrd)


def test_topk_rows_of_a_wider_buffer():
    from scorch_b200 import kernels as K
    wide = np.random.default_rng(3).standard_normal((9, 2051)).astype(np.float32)
    got = K.topk_rows_to_csr(torch.from_numpy(wide).cuda()[:, 1:2000], 17, relu=True)
    want = O.topk_rows_to_csr(np.ascontiguousarray(wide[:, 1:2000]), 17, True)
    assert all(np.array_equal(g.cpu().numpy(), w) for g, w in zip(got, want))
