"""Results written through raw pointers count as in-place writes of their tensors."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_out_tensors_count_the_write():
    from scorch_b200 import kernels as K, workloads as W
    A = W.csr_uniform(300, 400, 0.05, seed=0).to("cuda")
    B = torch.randn((400, 16), device="cuda")
    split = K.ColumnSplit(A.pos, A.crd, A.val, 400, 3)
    X, Wt = torch.randn((K.DENSE_MATMUL_MIN_ROWS, 64), device="cuda"), torch.randn((64, 16), device="cuda")
    for write, shape in ((lambda out: K.spmm_csr(A.pos, A.crd, A.val, B, out=out), (300, 16)),
                         (lambda out: split.matmul(B, out=out), (300, 16)),
                         (lambda out: split.matmul(B, out=out, accumulate=True), (300, 16)),
                         (lambda out: K.dense_matmul(X, Wt, out=out), (X.shape[0], 16)),
                         (lambda out: K.dense_matmul(X[:100], Wt, out=out), (100, 16))):
        out = torch.zeros(shape, device="cuda")
        view, before = out[1:], out._version
        assert write(out) is out and out._version > before and view._version == out._version


def test_out_of_inference_mode_is_written():
    from scorch_b200 import kernels as K
    with torch.inference_mode():
        X, Wt = torch.randn((K.DENSE_MATMUL_MIN_ROWS, 64), device="cuda"), torch.randn((64, 16), device="cuda")
        out = torch.zeros((X.shape[0], 16), device="cuda")
        assert torch.equal(K.dense_matmul(X, Wt, out=out), K.dense_matmul(X, Wt))
