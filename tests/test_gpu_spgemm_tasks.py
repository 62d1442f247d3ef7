"""SpGEMM: how the work of long rows is dealt out (by entries, by products, what is left over), rows of a CTA with 16
and 32 warps, the scan and the move of results of few and many rows."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_spgemm_bins import _check, _csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int64])
@pytest.mark.parametrize("n", [20000, 60000])
def test_entries_with_most_of_the_products(n, dtype):
    # B row 0 has 30,000 (or all) entries, the others 9: rows of A that bring it alone, among few entries, and among
    # more entries than a task takes (512) or the parts of a cluster share (2048), first, in the middle and last
    rng = np.random.default_rng(n)
    big = min(n, 30000)
    B = _csr([big] + [9] * 5998 + [big // 2], n, rng, dtype)
    rows = [[0], [0, 5, 7, 5999], list(range(1, 1500)), list(range(0, 1600)), list(range(1, 513)), list(range(5000, 6000)),
            list(range(0, 6000)), [3], list(range(0, 4200, 2))]
    pos = np.zeros(len(rows) + 1, np.int32)
    np.cumsum([len(r) for r in rows], out=pos[1:])
    val = rng.standard_normal(int(pos[-1])) * 3
    _check((pos, np.concatenate(rows).astype(np.int32), val.astype(dtype)), B, n, dtype)


@pytest.mark.parametrize("dtype", [np.float32])
def test_row_of_more_buckets_than_are_counted_together(dtype):
    # 2.2 M products in 4096 buckets: a place per product
    rng = np.random.default_rng(8)
    n = 100000
    B = _csr([22000] * 100, n, rng, dtype)
    _check(_csr([100, 3], 100, rng, dtype), B, n, dtype)


@pytest.mark.parametrize("beyond", [0, 1])
@pytest.mark.parametrize("n", [64, 65, 3000, 1 << 21])
def test_cta_rows_of_both_sizes(beyond, n):
    # 2049 to 8192 products; as many rows as SMs, which a CTA of 1024 threads takes each, and one more, where CTAs have
    # 512.  64 and 65 columns: segments of one and two columns
    rows = torch.cuda.get_device_properties(0).multi_processor_count + beyond
    rng = np.random.default_rng(rows)
    B = _csr([min(n, 50)] * 150, n, rng, np.float32)
    _check(_csr([int(x) for x in rng.integers(45, 140, rows)], 150, rng, np.float32), B, n, np.float32)


@pytest.mark.parametrize("m", [1, 1023, 1024, 1025, 8191, 32768, 32769])
def test_results_of_many_rows(m):
    # scans of up to 32 parts and beyond, moves of tiles with thousands of empty rows in a line
    rng = np.random.default_rng(m)
    lens = np.where(rng.random(m) < 0.5, 0, rng.integers(0, 4, m))
    lens[m // 3: m // 3 + 2500] = 0
    lens[-1] = 3
    B = _csr([2, 5, 0, 9], 40, rng, np.float32)
    _check(_csr([int(x) for x in lens], 4, rng, np.float32), B, 40, np.float32)
