"""SpGEMM at the borders of its bins (sorting networks, CTA rows, buckets, windows, dense rows), one
pass and two phases."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(lens, n, rng, dtype, cols=None):
    pos = np.zeros(len(lens) + 1, np.int32)
    np.cumsum(lens, out=pos[1:])
    pick = (lambda x: np.sort(rng.choice(n if cols is None else cols, size=x, replace=False)))
    crd = np.concatenate([pick(x) for x in lens] or [np.zeros(0)]).astype(np.int32)
    val = rng.standard_normal(int(pos[-1]))
    return pos, crd, (val.astype(dtype) if np.issubdtype(dtype, np.floating) else (val * 50).astype(dtype))


def _check(A, B, n, dtype):
    from scorch_b200 import kernels as K
    d = lambda t: tuple(torch.from_numpy(x).cuda() for x in t)
    a, b = d(A), d(B)
    wpos, wcrd, wval = O.spgemm(*A, *B, n)
    first = None
    for timings in (None, {}):                    # one pass, then symbolic + numeric
        cpos, ccrd, cval = K.spgemm_csr(*a, *b, n, timings=timings)
        assert np.array_equal(cpos.cpu().numpy(), wpos) and np.array_equal(ccrd.cpu().numpy(), wcrd)
        got = cval.cpu().numpy()
        if np.issubdtype(dtype, np.floating):
            want = O.spgemm_values_acc64(*A, *B, n, wpos, wcrd) if dtype == np.float32 else wval
            tol = dict(rtol=1e-4, atol=1e-5) if dtype == np.float32 else dict(rtol=1e-11, atol=1e-11)
            assert np.allclose(got, want, **tol)
        else:
            assert np.array_equal(got, wval)
        assert first is None or np.array_equal(first, got)      # the same bits either way
        first = got


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.int64])
@pytest.mark.parametrize("n", [300, 5000, 1 << 20])
def test_bin_borders(n, dtype):
    rng = np.random.default_rng(n)
    blen = [0, 1, 7, 8, 128] * 60
    B = _csr(blen, n, rng, dtype)
    # rows of A by number of products: around 32, 64, 128, 256, 512, 2048, 8192 and beyond
    lens = [0, 1, 1, 4, 5, 11, 20, 33, 40, 64, 65, 100, 200, 290, 300]
    _check(_csr(lens, 300, rng, dtype), B, n, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.int64])
def test_exact_bin_sizes(dtype):
    rng = np.random.default_rng(1)
    n, sizes = 1 << 16, [32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097, 8192, 8193]
    B = _csr(sizes + [1, 2], n, rng, dtype)
    A = (np.arange(len(sizes) + 1, dtype=np.int32), np.arange(len(sizes), dtype=np.int32),
         np.ones(len(sizes), dtype))
    _check(A, B, n, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32])
def test_buckets_with_many_equal_columns(dtype):
    # 2000 B rows of 40 entries in the same 60 columns: every bucket of the long row is over-full
    rng = np.random.default_rng(2)
    n = 1 << 18
    B = _csr([40] * 2000, n, rng, dtype, cols=np.arange(131000, 131060))
    _check(_csr([2000, 3, 1500], 2000, rng, dtype), B, n, dtype)


def test_row_beyond_the_area():
    # more products in one row than the area of a wider matrix holds (1 M): summed in shared memory here
    rng = np.random.default_rng(3)
    B = _csr([900] * 1300, 1000, rng, np.float32)
    _check(_csr([1300, 2, 700], 1300, rng, np.float32), B, 1000, np.float32)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32])
@pytest.mark.parametrize("rows,n", [(1, 24576), (18, 45), (19, 5000), (38, 24575), (75, 1000)])
def test_long_rows_shared_by_clusters(rows, n, dtype):
    # over 8192 products a row: 8, 8, 4, 2 and 1 CTAs per row on 148 SMs; 45 columns leave most CTAs none
    rng = np.random.default_rng(rows)
    B = _csr([40] * 299 + [min(n, 3000)], n, rng, dtype)
    _check(_csr([250] * rows + [0, 7], 300, rng, dtype), B, n, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32])
def test_row_beyond_the_area_of_a_wide_matrix(dtype):
    # as test_row_beyond_the_area, with more columns than shared memory holds sums of: there the rows of more
    # products than the workspace's area takes (64 (m + n) here) go to the dense kernel one by one
    rng = np.random.default_rng(4)
    n = 30000
    B = _csr([1500] * 1400, n, rng, dtype)
    assert 1400 * 1500 > 64 * (3 + n) > 700 * 1500 > 8192
    _check(_csr([1400, 2, 700], 1400, rng, dtype), B, n, dtype)
