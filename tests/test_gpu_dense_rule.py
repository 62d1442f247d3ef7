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


@pytest.mark.parametrize("m,k,n", [(30000, 256, 64), (32767, 200, 56), (21364, 256, 64), (28485, 24, 512),
                                   (21363, 16, 1024)])
def test_narrow_products_stay_with_the_library(m, k, n):
    from scorch_b200 import kernels as K
    assert 4096 <= m < K.DENSE_MATMUL_MIN_ROWS and m * k * n >= K.DENSE_MATMUL_MIN_WORK
    X, W = torch.randn((m, k), device="cuda"), torch.randn((k, n), device="cuda")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        got = K.dense_matmul(X, W)
        torch.cuda.synchronize()
    assert not any("gemm_f32_kernel" in e.key for e in p.key_averages())
    assert torch.equal(got, X @ W)


@pytest.mark.parametrize("m,k,n", [(4096, 256, 336), (12000, 256, 256), (11000, 128, 256), (27000, 100, 136),
                                   (32767, 64, 256), (12300, 28, 1024)])
def test_no_further_from_float64_than_the_products_before(m, k, n):
    # two-norm of the error; measured 0.5 to 0.8 of the FMA chain's
    from scorch_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(k)
    X, W = torch.randn((m, k), generator=g, device="cuda"), torch.randn((k, n), generator=g, device="cuda")
    want = X.double() @ W.double()
    error = lambda got: (got.double() - want).norm().item()
    assert error(K.dense_matmul(X, W)) <= error(torch.matmul(X, W))
