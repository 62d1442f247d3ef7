"""The benchmark's own count of kernel launches per step follows the rules that choose the kernels."""
from __future__ import annotations

from types import SimpleNamespace

import pytest


# Row chunks, and how many of the transforms with 256 and with 64 result columns the tensor cores compute.
@pytest.mark.parametrize("rows,offsets,wide,narrow", [
    (500_000, [0, 500_000], 1, 1),
    (48_000, [0, 6_000, 24_000, 48_000], 3, 0),               # from 350 M multiplications on, for wide results
    (40_000, [0, 4_095, 9_435, 40_000], 1, 0),                # too few rows, too few multiplications
    (90_000, [0, 5_400, 50_000, 100_000], 3, 2),              # the last chunk ends with the rows
])
def test_transforms_of_row_chunks(rows, offsets, wide, narrow):
    import bench
    work = bench.GcnSharded(n=rows)
    blocks = [SimpleNamespace(columns=None)] * (len(offsets) - 1)
    work.shard = SimpleNamespace(rows=rows, splits=[SimpleNamespace(blocks=blocks, offsets=offsets)])
    assert work.launches_per_step == 2 * 2 * len(blocks) + 2 * (wide + narrow)


def test_sizes_that_the_tensor_cores_take():
    from scorch_b200 import kernels as K
    took = lambda *mkn: K.dense_on_tensor_cores(*mkn)
    assert took(32768, 4, 8) and took(32768, 256, 64) and not took(32767, 256, 64)
    assert took(5342, 256, 256) and not took(5340, 256, 256) and not took(4095, 256, 512)
    for m, k, n in ((40000, 260, 64), (40000, 102, 64), (40000, 0, 64), (40000, 64, 0), (40000, 64, 12), (21363, 16, 1024)):
        assert not took(m, k, n)
