"""How many column chunks the products of a large graph are cut into (``kernels.split_chunks``)."""
from __future__ import annotations

import pytest

from scorch_b200 import kernels as K


# Rows, entries per row, columns, and the counts (0: one pass) whose products with 256 and 64 columns, with the cut,
# took at most 4 % more than the best count's on a B200.
@pytest.mark.parametrize("n,d,best", [
    (400_000, 101, {2, 3}), (500_000, 51, {2}), (500_000, 101, {2, 3, 4}), (700_000, 25, {0}), (700_000, 51, {2, 3}),
    (700_000, 101, {3, 4, 5}), (850_000, 101, {3, 4, 5, 6}), (1_000_000, 25, {0, 2}), (1_000_000, 51, {2, 3}),
    (1_000_000, 71, {3, 4}), (1_000_000, 101, {3, 4, 5, 6, 7}), (1_200_000, 101, {4, 5, 6, 7}), (1_400_000, 25, {0}),
    (1_400_000, 51, {2, 3}), (1_400_000, 101, {4, 5, 6, 7}), (1_700_000, 101, {4, 5, 6, 7, 8}), (2_000_000, 25, {0}),
    (2_000_000, 51, {0, 2, 3, 4}), (2_000_000, 71, {3, 4, 5, 6}), (2_000_000, 101, {4, 5, 6, 7, 8}),
    (2_020_000, 101, {4, 5, 6, 7, 8}), (2_500_000, 101, {5, 6, 7, 8}), (3_000_000, 25, {0}), (3_000_000, 51, {0}),
    (3_000_000, 101, {6, 7, 8, 9}), (4_000_000, 51, {0}), (4_000_000, 101, {0, 2, 8, 9, 10}),
])
def test_counts_that_were_measured_best(n, d, best):
    assert K.split_chunks(n, n, n * d, 256) in best


@pytest.mark.parametrize("d", [30, 101, 400])
@pytest.mark.parametrize("k", [40, 64, 256])
def test_neighbouring_sizes_differ_by_one_chunk(d, k):
    # 2.02 M rows are multiplied like 2 M
    n, counts = 800_000, []
    while n < 20_000_000:
        counts.append(K.split_chunks(n, n, n * d, k))
        n = int(n * 1.01)
    split = [c for c in counts if c]
    first = counts.index(split[0])
    assert counts[first:first + len(split)] == split                 # one range of sizes
    assert all(a <= b <= a + 1 for a, b in zip(split, split[1:]))


@pytest.mark.parametrize("n,k", [(0, 64), (1000, 256), (300_000, 64), (600_000, 40), (1_700_000, 16),
                                 (400_000, 64), (430_000, 64), (690_000, 40)])
def test_operands_that_l2_holds_are_not_split(n, k):
    assert K.split_chunks(n, n, n * 400, k) == 0


def test_blocks_of_rows():
    # entries per row decide, not the number of rows; none where a block has none
    assert K.split_chunks(500_000, 2_000_000, 50_500_000, 256) == K.split_chunks(2_000_000, 2_000_000, 202_000_000, 256) == 6
    assert K.split_chunks(0, 2_000_000, 0, 256) == 0
