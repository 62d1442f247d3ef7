"""Device-side CSR validation: the first violation of what the kernels assume about their inputs
is named (smallest row, then entry), reading nothing outside pos[0..m] and crd[0..nnz); with
SCORCH_B200_VALIDATE=1 the front end refuses an invalid operand before any kernel reads it."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a, dt=np.int32):
    return torch.from_numpy(np.asarray(a, dt)).cuda()


POS = [0, 2, 2, 5, 6]
CRD = [1, 4, 0, 2, 3, 4]


def test_valid_matrices_pass():
    from scorch_b200 import kernels as K, workloads as W
    assert K.csr_validate(dev(POS), dev(CRD), 5) is None
    assert K.csr_validate(dev([0]), dev([]), 3) is None                       # no rows
    assert K.csr_validate(dev([0, 0, 0]), dev([]), 3) is None                 # no entries
    A = W.powerlaw_square(20000, mean_nnz=8.0, seed=2)
    assert K.csr_validate(A.pos.cuda(), A.crd.cuda(), 20000) is None


@pytest.mark.parametrize("pos,crd,n,sorted_unique,want", [
    ([1, 2, 2, 5, 6], CRD, 5, True, ("pos[0] is not 0", 0, 0, 1)),
    ([0, 2, 2, 5, 5], CRD, 5, True, ("pos[m] is not nnz", 4, 0, 5)),
    ([0, 2, 9, 5, 6], CRD, 5, True, ("row pointer out of [0, nnz]", 2, 0, 9)),
    ([0, 2, 1, 5, 6], CRD, 5, True, ("row pointers decrease", 1, 0, 1)),
    ([0, 3, 2, 5, 6], CRD, 5, True, ("row pointers decrease", 1, 0, 2)),
    (POS, [1, 4, 0, 2, 5, 4], 5, True, ("column index out of range", 2, 4, 5)),
    (POS, [1, -4, 0, 2, 3, 4], 5, True, ("column index out of range", 0, 1, -4)),
    (POS, [1, 4, 0, 3, 3, 4], 5, True, ("columns of a row not strictly ascending", 2, 4, 3)),
    (POS, [4, 1, 0, 2, 3, 9], 5, True, ("columns of a row not strictly ascending", 0, 1, 1)),   # the first of two
])
def test_first_violation_is_named(pos, crd, n, sorted_unique, want):
    from scorch_b200 import kernels as K
    assert K.csr_validate(dev(pos), dev(crd), n, sorted_unique) == want


def test_unsorted_rows_are_accepted_when_order_is_not_required():
    from scorch_b200 import kernels as K
    assert K.csr_validate(dev(POS), dev([4, 1, 0, 3, 3, 2]), 5, sorted_unique=False) is None
    assert K.csr_validate(dev(POS), dev([4, 1, 0, 3, 3, 7]), 5, sorted_unique=False) == (
        "column index out of range", 3, 5, 7)


def test_front_end_refuses_invalid_operands_when_asked(monkeypatch):
    from scorch_b200 import kernels as K
    B = torch.ones((5, 8), device="cuda")
    val = torch.ones(6, device="cuda")
    good = K.spmm_csr(dev(POS), dev(CRD), val, B)
    monkeypatch.setenv("SCORCH_B200_VALIDATE", "1")
    assert torch.equal(K.spmm_csr(dev(POS), dev(CRD), val, B), good)
    with pytest.raises(ValueError, match="column index out of range"):
        K.spmm_csr(dev(POS), dev([1, 4, 0, 2, 3, 5]), val, B)            # never reaches the kernel
    with pytest.raises(ValueError, match="row pointers decrease"):
        K.spmv_csr(dev([0, 3, 2, 5, 6]), dev(CRD), val, torch.ones(5, device="cuda"))
    with pytest.raises(ValueError, match="not strictly ascending"):
        K.spgemm_csr(dev(POS), dev([4, 1, 0, 2, 3, 4]), val, dev([0, 1, 2, 3, 4, 5]), dev([0, 1, 2, 3, 4]),
                     torch.ones(5, device="cuda"), 5)


def test_column_split_refuses_invalid_operands_when_asked(monkeypatch):
    # the products of large graphs go through the column split, not through spmm_csr
    from scorch_b200 import kernels as K, pipelines as P, sharded as S
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 2e5)
    n, per = 2000, 40
    pos = np.arange(n + 1, dtype=np.int32) * per
    crd = np.tile(np.arange(per, dtype=np.int32) * 50, n)
    val = torch.ones(n * per, device="cuda")
    X, W1, W2 = (torch.ones(s, device="cuda") for s in ((n, 64), (64, 64), (64, 40)))
    monkeypatch.setenv("SCORCH_B200_VALIDATE", "1")
    good = P.gcn_forward(dev(pos), dev(crd), val, X, W1, W2)
    assert K.ColumnSplit.of(dev(pos), dev(crd), val, n, 64) is not None and torch.isfinite(good).all()
    far = crd.copy()
    far[-1] = n
    down = pos.copy()
    down[7] = down[9]
    for p, c, message in ((pos, far, "column index out of range"), (down, crd, "row pointers decrease")):
        with pytest.raises(ValueError, match=message):
            P.gcn_forward(dev(p), dev(c), val, X, W1, W2)                 # never reaches the kernels
        block = S.CsrBlock(dev(p), dev(c), val)
        with pytest.raises(ValueError, match=message):
            S._default_spmm(block, X, torch.empty((n, 64), device="cuda"), False)
    split = K.ColumnSplit(dev(pos), dev(crd), val, n, 4)
    split.crd[3] = n + 5                                                  # a split is an operand of its own
    with pytest.raises(ValueError, match="column index out of range"):
        split.matmul(X)


def test_column_split_leaves_host_tensors_to_spmm(monkeypatch):
    from scorch_b200 import kernels as K, pipelines as P
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 2e5)
    n, per = 2000, 40
    pos, crd = dev(np.arange(n + 1) * per), dev(np.tile(np.arange(per) * 50, n))
    val, X, W1, W2 = (torch.ones(s, device="cuda") for s in ((n * per,), (n, 64), (64, 64), (64, 40)))
    for args in ((pos.cpu(), crd, val), (pos, crd.cpu(), val), (pos, crd, val.cpu())):
        with pytest.raises(TypeError, match="CUDA tensor"):
            P.gcn_forward(*args, X, W1, W2)
