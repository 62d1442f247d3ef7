"""SpMM over entry tiles (sb_spmm_csr_once) at the edges of its tiles and slices, for every load width."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(lens, n, seed, dtype=np.float32):
    rng = np.random.default_rng(seed)
    pos = np.zeros(len(lens) + 1, np.int32)
    np.cumsum(lens, out=pos[1:])
    crd = np.concatenate([np.sort(rng.integers(0, n, x)) for x in lens] or [np.zeros(0)]).astype(np.int32)
    return pos, crd, rng.standard_normal(int(pos[-1])).astype(dtype)


PATTERNS = {
    "one_entry": [1],
    "empty_rows_around": [0] * 700 + [5, 0, 0, 3] + [0] * 2500,      # more empty rows than a tile keeps pointers of
    "rows_of_one": [1] * 2049,                                       # one row more than a tile has entries
    "hub_over_tiles": [3, 9000, 1, 0, 40, 2],
    "row_ends_on_slices": [8] * 300 + [64] * 40 + [128] * 8,
    "mixed": [int(x) for x in np.random.default_rng(0).zipf(1.6, 3000).clip(0, 4000) - 1],
}


@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("k", [1, 3, 6, 16, 33, 64, 77, 130, 256, 301])
def test_tiles_f32(pattern, k):
    from scorch_b200 import kernels as K
    lens = PATTERNS[pattern]
    n = 500
    pos, crd, val = _csr(lens, n, seed=k)
    rng = np.random.default_rng(k + 1)
    B, bias = rng.standard_normal((n, k)).astype(np.float32), rng.standard_normal(k).astype(np.float32)
    d = lambda a: torch.from_numpy(a).cuda()
    want = O.spmm_csr_acc64(pos, crd, val, B)
    got = K.spmm_csr(d(pos), d(crd), d(val), d(B))
    assert O.allclose_report(got.cpu().numpy(), want, 1e-4, 1e-5 * max(1.0, max(lens) ** 0.5))[0]
    # bias and ReLU reach empty rows too; accumulation; a second run gives the same bits
    got2 = K.spmm_csr(d(pos), d(crd), d(val), d(B), bias=d(bias), relu=True)
    assert O.allclose_report(got2.cpu().numpy(), np.maximum(want + bias, 0), 1e-4, 1e-5 * max(1.0, max(lens) ** 0.5))[0]
    assert torch.equal(got, K.spmm_csr(d(pos), d(crd), d(val), d(B)))
    base = torch.ones((len(lens), k), device="cuda")
    got3 = K.spmm_csr(d(pos), d(crd), d(val), d(B), accumulate=True, out=base)
    assert O.allclose_report(got3.cpu().numpy(), want + 1, 1e-4, 1e-5 * max(1.0, max(lens) ** 0.5))[0]


@pytest.mark.parametrize("k", [1, 2, 7, 16, 20, 65, 132])
@pytest.mark.parametrize("dtype", [np.float64, np.int32, np.int64])
def test_tiles_other_dtypes(k, dtype):
    from scorch_b200 import kernels as K
    pos, crd, val = _csr(PATTERNS["mixed"], 400, seed=k, dtype=np.float64)
    B = np.random.default_rng(k).standard_normal((400, k))
    if dtype != np.float64:
        val, B = (val * 100).astype(dtype), (B * 100).astype(dtype)
    d = lambda a: torch.from_numpy(a).cuda()
    got = K.spmm_csr(d(pos), d(crd), d(val), d(B)).cpu().numpy()
    dense = np.zeros((len(pos) - 1, 400), val.dtype)
    np.add.at(dense, (np.repeat(np.arange(len(pos) - 1), np.diff(pos)), crd), val)
    want = dense @ B
    assert np.allclose(got, want, 1e-12, 1e-10) if dtype == np.float64 else np.array_equal(got, want)


def test_column_slices_of_wider_buffers():
    from scorch_b200 import kernels as K
    pos, crd, val = _csr(PATTERNS["mixed"], 500, seed=5)
    wide = np.random.default_rng(6).standard_normal((500, 101)).astype(np.float32)
    out = torch.zeros((len(pos) - 1, 90), device="cuda")
    d = lambda a: torch.from_numpy(a).cuda()
    K.spmm_csr(d(pos), d(crd), d(val), d(wide)[:, 3:40], out=out[:, 7:44])
    want = O.spmm_csr_acc64(pos, crd, val, np.ascontiguousarray(wide[:, 3:40]))
    assert O.allclose_report(out[:, 7:44].cpu().numpy(), want, 1e-4, 1e-3)[0]
    assert not out[:, :7].any() and not out[:, 44:].any()
