"""SpMM over entry tiles: rows at the borders of the length classes and of who takes a row, more rows of one
class than a turn holds, and the same bits for a block of rows as for the whole matrix."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

BORDERS = [1, 7, 8, 9, 10, 11, 16, 17, 20, 21, 24, 25, 30, 31, 32, 33, 40, 41, 64, 65, 191, 192, 193, 512, 513, 0]


@pytest.mark.parametrize("lens", [BORDERS * 40, [1, 0] * 1100, [8] * 1023 + [33] + [9] * 1025, [3] * 700 + [600] + [25] * 400],
                         ids=["borders", "ones", "two_turns", "around_a_long_row"])
@pytest.mark.parametrize("dtype,k", [("f32", 8), ("f32", 40), ("f32", 77), ("f32", 128), ("f64", 3), ("f64", 16), ("f64", 24)])
def test_rows_by_length(lens, dtype, k):
    from scorch_b200 import kernels as K
    t = np.float32 if dtype == "f32" else np.float64
    n, rng = 600, np.random.default_rng(len(lens) + k)
    pos = np.zeros(len(lens) + 1, np.int32)
    np.cumsum(lens, out=pos[1:])
    crd = rng.integers(0, n, pos[-1]).astype(np.int32)
    val, B = rng.standard_normal(pos[-1]).astype(t), rng.standard_normal((n, k)).astype(t)
    d = lambda a: torch.from_numpy(a).cuda()
    dpos, dcrd, dval, dB = d(pos), d(crd), d(val), d(B)
    got = K.spmm_csr(dpos, dcrd, dval, dB)
    rows = np.repeat(np.arange(len(lens)), lens)
    want, size = np.zeros((len(lens), k)), np.zeros((len(lens), k))
    np.add.at(want, rows, val[:, None].astype(np.float64) * B[crd])
    np.add.at(size, rows, np.abs(val[:, None].astype(np.float64) * B[crd]))
    # a sum of n terms in any order errs by at most n u sum |a b|; rows add slices of at most 32 terms and a few more
    eps = 2.0 ** -24 if dtype == "f32" else 2.0 ** -53
    assert np.all(np.abs(got.cpu().numpy() - want) <= 64 * eps * size + 1e-300)
    r0, r1 = len(lens) // 3, len(lens) - 5
    part = K.spmm_csr(d(pos[r0:r1 + 1] - pos[r0]), dcrd[pos[r0]:pos[r1]].clone(), dval[pos[r0]:pos[r1]].clone(), dB)
    assert torch.equal(part, got[r0:r1])


@pytest.mark.parametrize("units", [1, 2, 7, 8, 9, 16, 17, 200])
@pytest.mark.parametrize("dtype,k", [("f32", 8), ("f32", 77), ("f64", 40)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_rows_of_several_units(units, dtype, k, accumulate):
    # alone (few entries) and among more than 2^17 entries, where the CTA adds the unit sums: the same bits
    from scorch_b200 import kernels as K
    t = np.float32 if dtype == "f32" else np.float64
    if accumulate and dtype == "f64":
        pytest.skip("accumulation is float32")
    n, rng = 3000, np.random.default_rng(units)
    lens = [3, 512 * units - 511, 0, 512 * units] + [40] * 3300
    pos = np.zeros(len(lens) + 1, np.int32)
    np.cumsum(lens, out=pos[1:])
    assert pos[-1] > 1 << 17
    crd = rng.integers(0, n, pos[-1]).astype(np.int32)
    val, B = rng.standard_normal(pos[-1]).astype(t), rng.standard_normal((n, k)).astype(t)
    d = lambda a: torch.from_numpy(a).cuda()
    dB, base = d(B), torch.full((len(lens), k), 2.0, device="cuda")
    run = (lambda p, c, v, out: K.spmm_csr(p, c, v, dB, accumulate=True, out=out)) if accumulate else (
        lambda p, c, v, out: K.spmm_csr(p, c, v, dB))
    got = run(d(pos), d(crd), d(val), base.clone())
    e = pos[4]
    part = run(d(pos[:5]), d(crd[:e]), d(val[:e]), base[:4].clone())
    assert torch.equal(part, got[:4])
    rows = np.repeat(np.arange(4), lens[:4])
    term = val[:e, None].astype(np.float64) * B[crd[:e]]
    want, size = np.full((4, k), 2.0 * accumulate), np.full((4, k), 2.0 * accumulate)
    np.add.at(want, rows, term)
    np.add.at(size, rows, np.abs(term))
    eps = 2.0 ** -24 if dtype == "f32" else 2.0 ** -53
    assert np.all(np.abs(part.cpu().numpy() - want) <= 128 * eps * size)     # (at most some 100 additions one after another)
