"""SpGEMM where entries are numbered up to 2^31 - 2, the last number that int32 row pointers leave room for."""
from __future__ import annotations

import gc

import pytest
import torch

pytestmark = pytest.mark.gpu

MOST = 2**31 - 1


@pytest.fixture
def room():
    gc.collect()
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of GPU memory")
    yield
    gc.collect()
    torch.cuda.empty_cache()


@pytest.mark.parametrize("nnz", [MOST - 1024, MOST - 700, MOST - 1, MOST])
def test_move_of_the_largest_results(room, nnz):
    # two long rows and short ones at the end, the last ones' entries MOST - nnz places behind their product offsets
    from scorch_b200 import _lib
    gap = MOST - nnz
    pos = torch.tensor([0, 1 << 30, nnz - 40, nnz - 40, nnz - 33, nnz - 1, nnz], dtype=torch.int32, device="cuda")
    off = pos.clone()
    off[2:] += gap
    t = torch.arange(MOST, dtype=torch.int32, device="cuda")      # (columns and values alike: what went where)
    crd, val = torch.full((nnz,), -1, dtype=torch.int32, device="cuda"), torch.full((nnz,), -1, dtype=torch.int32, device="cuda")
    code = 2                                                      # SB_I32
    _lib.check(_lib.lib().sb_spgemm_finish(code, 6, nnz, off.data_ptr(), t.data_ptr(), t.data_ptr(), pos.data_ptr(),
                                           crd.data_ptr(), val.data_ptr(), torch.cuda.current_stream().cuda_stream))
    for got in (crd, val):
        assert torch.equal(got[:nnz - 40], t[:nnz - 40])
        assert torch.equal(got[nnz - 40:], t[nnz - 40 + gap:])


# Rows of A at the very end of 2^31 - 1 entries, one kind for every kernel: (entries, columns of C, which rows of B)
ENDS = {
    "warp": (30, 20000, "short"), "cta_64": (100, 20000, "short"), "cta_128": (400, 20000, "short"),
    "split": (1500, 20000, "short"), "shared_by_entries": (5000, 20000, "short"), "shared_by_products": (30, 20000, "long"),
    "buckets_by_entries": (5000, 30000, "short"), "buckets_by_products": (30, 30000, "long"),
    "buckets_left_over": (1000, 30000, "short and long"), "beyond_the_area": (5500, 30000, "medium"),
}


@pytest.fixture(scope="module")
def largest():
    """Columns and values of A; all but the last 16,384 entries lie in B's empty row 0."""
    gc.collect()
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of GPU memory")
    a = {"crd": torch.zeros(MOST, dtype=torch.int32, device="cuda"), "val": torch.ones(MOST, device="cuda")}
    yield a
    a.clear()
    gc.collect()
    torch.cuda.empty_cache()


def _right_operand(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    lens = torch.tensor([0] + [4] * 6000 + [1500] * 40 + [500] * 6000, device="cuda")
    pos = torch.zeros(lens.numel() + 1, dtype=torch.int64, device="cuda")
    pos[1:] = lens.cumsum(0)
    row = torch.repeat_interleave(torch.arange(lens.numel(), device="cuda"), lens)
    # distinct ascending columns: a start and steps that stay below n
    step = torch.clamp(n // torch.clamp(lens, min=1) - 1, min=1)[row]
    k = torch.arange(row.numel(), device="cuda") - pos[row]
    start = (torch.rand(lens.numel(), generator=g, device="cuda") * (n // torch.clamp(lens, min=1))).long()[row]
    return pos.int(), (start + k * step).int(), torch.randn(row.numel(), generator=g, device="cuda")


@pytest.mark.parametrize("kind", ENDS)
def test_last_rows_of_the_largest_matrix(largest, kind):
    from scorch_b200 import kernels as K
    entries, n, which = ENDS[kind]
    g = torch.Generator(device="cuda").manual_seed(entries)
    pick = lambda lo, count, of: lo + torch.randperm(of, generator=g, device="cuda")[:count]
    row = {"short": lambda: pick(1, entries, 6000), "long": lambda: pick(6001, entries, 40),
           "medium": lambda: pick(6041, entries, 6000),
           "short and long": lambda: torch.cat([pick(1, entries - 40, 6000), pick(6001, 40, 40)])}[which]().sort()[0].int()
    val = torch.randn(entries, generator=g, device="cuda")
    B = _right_operand(n)
    small = (torch.tensor([0, entries], dtype=torch.int32, device="cuda"), row, val)
    largest["crd"][-16384:], largest["val"][-16384:] = 0, 1
    largest["crd"][-entries:], largest["val"][-entries:] = row, val
    # 4096 rows of B's empty row, then the one that ends at entry 2^31 - 2
    pos = torch.linspace(0, MOST - entries, 4097, dtype=torch.float64, device="cuda").long()
    pos[-1] = MOST - entries
    pos = torch.cat([pos, torch.tensor([MOST], device="cuda")]).int()
    for timings in (None, {}):                    # one pass, then symbolic + numeric
        want = K.spgemm_csr(*small, *B, n, timings=timings)
        got = K.spgemm_csr(pos, largest["crd"], largest["val"], *B, n, timings=timings)
        assert torch.equal(got[0][4096:], want[0]) and not got[0][:4096].any()
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])     # the same bits


def test_check_of_the_largest_matrix(largest):
    # what SCORCH_B200_VALIDATE=1 runs on the operands: the last row ends at entry 2^31 - 2
    from scorch_b200 import kernels as K
    pos = torch.linspace(0, MOST, 8193, dtype=torch.float64, device="cuda").long()
    pos[-1] = MOST
    largest["crd"][-16384:] = 0
    assert K.csr_validate(pos.int(), largest["crd"], 6001, sorted_unique=False) is None
    largest["crd"][-1] = 6001
    try:
        assert K.csr_validate(pos.int(), largest["crd"], 6001, sorted_unique=False) == (
            "column index out of range", 8191, MOST - 1, 6001)
    finally:
        largest["crd"][-1] = 0
