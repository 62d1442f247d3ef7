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
