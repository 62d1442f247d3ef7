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


@pytest.mark.parametrize("n,k", [(33, 32), (512, 8), (1000, 256), (1000, 300), (3000, 2), (4096, 32), (32768, 64)])
@pytest.mark.parametrize("numbers", [0, 1, 5, 400])
def test_topk_rows_of_nans(n, k, numbers):
    # Rows of few numbers, many of them fewer than k.  A NaN with the sign bit set (0xffc00000, what x86 arithmetic
    # yields) orders below -inf, one without above +inf; equal bits go to the lower column.
    from scorch_b200 import kernels as K
    rng = np.random.default_rng(n + k + numbers)
    bits = np.full((4, n), 0xFFC00000, np.uint32)
    bits[1] = np.where(rng.random(n) < 0.5, 0xFFC00000, 0xFFFFFFFF)
    bits[2, rng.choice(n, 3, replace=False)] = 0x7FC00000
    bits[3, rng.choice(n, 3, replace=False)] = 0xFF800000              # -inf
    for row in bits:
        at = rng.choice(np.flatnonzero(row >= 0xFFC00000), min(numbers, n // 2), replace=False)
        row[at] = rng.standard_normal(at.size).astype(np.float32).view(np.uint32)
    pos, crd, val = K.topk_rows_to_csr(torch.from_numpy(bits.view(np.float32)).cuda(), k)
    key = np.where(bits >> 31, ~bits, bits | np.uint32(0x80000000)).astype(np.int64)
    want = np.sort(np.argsort(-key, axis=1, kind="stable")[:, :k], axis=1)
    assert np.array_equal(pos.cpu().numpy(), np.arange(5) * k)
    assert np.array_equal(crd.cpu().numpy().reshape(4, k), want)
    assert np.array_equal(val.cpu().numpy().view(np.uint32).reshape(4, k), np.take_along_axis(bits, want, 1))
    relu = K.topk_rows_to_csr(torch.from_numpy(bits.view(np.float32)).cuda(), k, relu=True)
    assert torch.equal(relu[1], crd) and torch.equal(relu[2], torch.where(val > 0, val, torch.zeros_like(val)))
