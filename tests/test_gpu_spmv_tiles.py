"""SpMV over entry tiles: rows that end, begin or are empty at tile borders, for every dtype."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

T = 2048
PATTERNS = {
    "one": [1],
    "empty_everywhere": [0, 0, T, 0, 0, T - 1, 0, 1, 0, 0, 5, 0],
    "exact_tiles": [T] * 3,
    "hub": [7, 5 * T + 3, 0, 2],
    "short": [3] * 3000 + [0] * 500,
    "mixed": [int(x) for x in np.random.default_rng(0).zipf(1.5, 4000).clip(0, 9000) - 1],
}


@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.int64])
def test_spmv_tiles(pattern, dtype):
    from scorch_b200 import kernels as K
    lens, rng, n = PATTERNS[pattern], np.random.default_rng(5), 700
    pos = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    crd = rng.integers(0, n, pos[-1]).astype(np.int32)
    val, x = rng.standard_normal(pos[-1]), rng.standard_normal(n)
    if not np.issubdtype(dtype, np.floating):
        val, x = val * 100, x * 100
    val, x = val.astype(dtype), x.astype(dtype)
    acc = np.float64 if np.issubdtype(dtype, np.floating) else dtype
    want = np.zeros(len(lens), acc)
    np.add.at(want, np.repeat(np.arange(len(lens)), lens), val.astype(acc) * x[crd].astype(acc))
    d = lambda a: torch.from_numpy(a).cuda()
    got = K.spmv_csr(d(pos), d(crd), d(val), d(x)).cpu().numpy()
    if acc is np.float64:
        assert np.allclose(got, want, rtol=1e-4 if dtype == np.float32 else 1e-12, atol=1e-3 if dtype == np.float32 else 1e-11)
    else:
        assert np.array_equal(got, want)
    assert np.array_equal(got, K.spmv_csr(d(pos), d(crd), d(val), d(x)).cpu().numpy())
