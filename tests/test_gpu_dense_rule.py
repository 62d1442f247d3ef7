"""Which products of two dense matrices run on the tensor cores below 32,768 rows, and that they are as close to
float64 there as a chain of fp32 operations."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(4096, 256, 336), (5341, 256, 256), (11000, 256, 128), (21363, 128, 128), (32767, 100, 112),
                                   (4095, 256, 512), (5340, 256, 256), (30000, 64, 64)])
def test_products_by_work(m, k, n):
    from scorch_b200 import kernels as K
    own = m >= 4096 and m * k * n >= K.DENSE_MATMUL_MIN_WORK
    g = torch.Generator(device="cuda").manual_seed(m)
    X, W = torch.randn((m, k), generator=g, device="cuda"), torch.randn((k, n), generator=g, device="cuda")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        got = K.dense_matmul(X, W)
        torch.cuda.synchronize()
    assert any("gemm_f32_kernel" in e.key for e in p.key_averages()) == own
    # a chain of k fused multiply-adds errs by at most k u sum |a b|, some sqrt(k) u in the mean
    size = X.abs().double() @ W.abs().double()
    err = (got.double() - X.double() @ W.double()).abs() / size
    assert err.max().item() <= 2 * k ** 0.5 * 2.0 ** -24
