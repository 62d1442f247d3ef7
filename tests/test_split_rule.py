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


# Forwards that cut their matrix on every call: rows, entries per row, hidden and result columns, and the counts that
# took at most 9 % more than the best (0: one pass) for graphs with or without hubs among their columns.
@pytest.mark.parametrize("n,d,hidden,width,best", [
    (340_000, 13, 256, 64, {0}), (400_000, 19, 256, 64, {0}), (400_000, 31, 256, 64, {2}), (480_000, 31, 256, 64, {2}),
    (480_000, 41, 256, 64, {2}), (480_000, 71, 256, 64, {2, 3}), (600_000, 31, 256, 64, {0, 2}),
    (800_000, 51, 256, 64, {2, 3, 4}), (1_200_000, 31, 256, 64, {0, 2}), (2_000_000, 41, 256, 64, {0, 2, 3}),
    (2_000_000, 101, 256, 64, {4, 5, 6, 7, 8}), (340_000, 51, 128, 40, {0}), (480_000, 41, 128, 40, {0}),
    (600_000, 100, 128, 40, {3, 4}), (1_200_000, 101, 128, 40, {3, 4, 5, 6}), (480_000, 31, 64, 64, {0}),
    (560_000, 49, 64, 64, {0, 2}), (800_000, 51, 64, 64, {0, 2, 3}), (1_200_000, 51, 64, 64, {0, 3}),
    (800_000, 101, 64, 64, {3, 4}), (480_000, 71, 64, 16, {0}), (700_000, 50, 64, 16, {0}),
    (1_200_000, 71, 64, 16, {0, 3, 4}),
])
def test_forwards_that_cut_on_every_call(n, d, hidden, width, best):
    panels = sum(-(-k // K.SPLIT_PANEL) for k in (hidden, width) if K.split_pays(n, k))
    assert K.split_chunks(n, n, n * d, max(hidden, width), panels) in best
