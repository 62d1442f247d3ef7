"""The row kernels behind the entry points that take a plan or no scratch (``sb_spmm_csr_f32``,
``sb_spmm_csr_acc_f32``, ``sb_spmm_csr_typed``, ``sb_spmv_csr_typed``) on one matrix.  ``kernels.spmm_csr`` and
``spmv_csr`` reach them for batches only, so they are called here through the C ABI."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_parity import assert_close, dev, random_csr

pytestmark = pytest.mark.gpu

CODE = {np.float32: 0, np.float64: 1, np.int32: 2, np.int64: 3}


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _spmm(pos, crd, val, B, C, bias=None, relu=False, plan=None, accumulate=False):
    from scorch_b200 import _lib
    L = _lib.lib()
    m, nnz, (n, k) = pos.numel() - 1, crd.numel(), B.shape
    segments = plan.segments if plan else 0
    need = L.sb_spmm_csr_scratch_bytes(segments, k, 1)
    scratch = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
    fn = L.sb_spmm_csr_acc_f32 if accumulate else L.sb_spmm_csr_f32
    rc = fn(m, n, k, nnz, pos.data_ptr(), crd.data_ptr(), val.data_ptr(), B.data_ptr(), B.stride(0),
            bias.data_ptr() if bias is not None else None, int(relu), C.data_ptr(), C.stride(0), 1, 0, 0, 0,
            plan.buf.data_ptr() if plan else None, segments, scratch.data_ptr(), need, _stream())
    torch.cuda.synchronize()
    return rc


@pytest.mark.parametrize("k", [64, 70, 256, 520])
def test_heavy_rows(oracle, k):
    # rows around and far above the threshold: the segment kernels, added in the order of the segments
    from scorch_b200 import kernels as K
    from scorch_b200._lib import HEAVY_ROW_NNZ as T
    m, n = 40, 6000
    lens = np.full(m, 9)
    lens[[1, 7, 8, 20, 39]] = [T, T + 1, 2 * T, 5 * T + 17, 3 * T - 1]
    lens[3] = 0
    pos, crd, val = random_csr(m, n, lens, seed=11)
    val = (val / np.sqrt(np.repeat(np.maximum(lens, 1), lens))).astype(np.float32)
    rng = np.random.default_rng(12)
    B, bias = rng.standard_normal((n, k)).astype(np.float32), rng.standard_normal(k).astype(np.float32)
    d = [dev(x) for x in (pos, crd, val, B, bias)]
    plan = K.CsrPlan(d[0], len(crd))
    assert plan.heavy_rows == 4 and plan.segments == 2 + 2 + 6 + 3
    want = oracle.spmm_csr_acc64(pos, crd, val, B, bias, False)
    first = None
    for p in (plan, plan, None):
        C = torch.full((m, k), 7.0, device="cuda")
        assert _spmm(*d[:4], C, bias=d[4], plan=p) == 0
        assert_close(oracle, C, want, f"k={k} plan={p is not None}")
        assert p is None or first is None or torch.equal(first, C)        # bitwise reproducible
        first = C


@pytest.mark.parametrize("k", [8, 16, 20, 32, 64, 72, 77, 128, 256, 300])
def test_many_short_rows(oracle, k):
    # mean length below the short-row threshold: a row per lane group or several per warp, with rows too long
    # for a lane group, empty and heavy rows among them
    from scorch_b200 import kernels as K
    from scorch_b200._lib import HEAVY_ROW_NNZ as T
    rng = np.random.default_rng(100 + k)
    m, n = 1003, 4000
    lens = rng.poisson(9, size=m)
    lens[rng.integers(0, m, 25)] = 0
    lens[[3, 40, 41, 500, 1002]] = [65, 300, 64, 1024, 97]
    lens[[7, 600]] = [T + 9, 2 * T + 100]
    pos, crd, val = random_csr(m, n, lens, seed=200 + k)
    assert len(crd) < 24 * m
    val = (val / np.sqrt(np.repeat(np.maximum(lens, 1), lens))).astype(np.float32)
    B, C0 = (rng.standard_normal(s).astype(np.float32) for s in ((n, k), (m, k)))
    bias = rng.standard_normal(k).astype(np.float32)
    want = oracle.spmm_csr_acc64(pos, crd, val, B)
    d = [dev(x) for x in (pos, crd, val, B)]
    for plan in (None, K.CsrPlan(d[0], len(crd))):
        C = torch.full((m, k), 7.0, device="cuda")
        assert _spmm(*d, C, plan=plan) == 0
        assert_close(oracle, C, want, f"k={k}")
        C = dev(C0.copy())
        rc = _spmm(*d, C, bias=dev(bias), relu=True, plan=plan, accumulate=True)
        assert rc == (0 if k % 4 == 0 else 5)                             # the accumulating form needs vector loads
        if rc == 0:
            assert_close(oracle, C, np.maximum(want + C0.astype(np.float64) + bias, 0), f"k={k} accumulating")


@pytest.mark.parametrize("k", [64, 256])
@pytest.mark.parametrize("relu", [False, True])
def test_accumulating_form_of_long_rows(oracle, k, relu):
    from scorch_b200 import kernels as K
    from scorch_b200._lib import HEAVY_ROW_NNZ as T
    m, n = 50, 5000
    lens = np.full(m, 41)
    lens[[2, 9, 30]] = [T + 5, 3 * T + 1, 0]
    pos, crd, val = random_csr(m, n, lens, seed=21)
    val = (val / np.sqrt(np.repeat(np.maximum(lens, 1), lens))).astype(np.float32)
    rng = np.random.default_rng(22)
    B, C0, bias = (rng.standard_normal(s).astype(np.float32) for s in ((n, k), (m, k), (k,)))
    want = oracle.spmm_csr_acc64(pos, crd, val, B) + C0.astype(np.float64) + bias
    wide = torch.full((m, k + 8), 7.0, device="cuda")                     # rows of a wider buffer
    C = wide[:, :k]
    C.copy_(dev(C0))
    plan = K.CsrPlan(dev(pos), len(crd))
    assert _spmm(dev(pos), dev(crd), dev(val), dev(B), C, bias=dev(bias), relu=relu, plan=plan, accumulate=True) == 0
    assert_close(oracle, C.contiguous(), np.maximum(want, 0) if relu else want, f"accumulate relu={relu}")
    assert (wide[:, k:] == 7.0).all()


def _typed(rng, size, dtype):
    return rng.standard_normal(size).astype(dtype) if np.issubdtype(dtype, np.floating) else \
        rng.integers(-9, 10, size).astype(dtype)


def _check_typed(got, want, dtype):
    if np.issubdtype(dtype, np.floating):
        np.testing.assert_allclose(got, want, **(dict(rtol=1e-4, atol=1e-4) if dtype == np.float32 else
                                                 dict(rtol=1e-12, atol=1e-12)))
    else:
        assert np.array_equal(got, want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.int64])
@pytest.mark.parametrize("k", [1, 5, 16, 33, 100])
def test_typed_spmm_without_scratch(dtype, k):
    from scorch_b200 import _lib
    rng = np.random.default_rng(k)
    m, n = 203, 900
    lens = rng.integers(0, 40, size=m)
    lens[[0, 7, 202]] = [0, 800, 0]
    pos, crd, _ = random_csr(m, n, lens, seed=k)
    val, B = _typed(rng, len(crd), dtype), _typed(rng, (n, k), dtype)
    d = [dev(x) for x in (pos, crd, val, B)]
    C = dev(np.full((m, k), 7, dtype))
    _lib.check(_lib.lib().sb_spmm_csr_typed(CODE[dtype], m, n, k, len(crd), *(x.data_ptr() for x in d), k, C.data_ptr(),
                                            k, _stream()))
    A = np.zeros((m, n), np.float64 if np.issubdtype(dtype, np.floating) else dtype)
    A[np.repeat(np.arange(m), lens), crd] = val
    _check_typed(C.cpu().numpy(), A @ B.astype(A.dtype), dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.int64])
@pytest.mark.parametrize("mean", [1, 5, 9, 30, 100])
def test_typed_spmv_without_scratch(dtype, mean):
    from scorch_b200 import _lib
    rng = np.random.default_rng(mean)
    m, n = 1501, 9000
    lens = rng.poisson(mean, size=m)
    lens[[2, 700, 1500]] = [1027, 4096, 0]
    pos, crd, _ = random_csr(m, n, lens, seed=mean)
    val, x = _typed(rng, len(crd), dtype), _typed(rng, n, dtype)
    d = [dev(a) for a in (pos, crd, val, x)]
    y = dev(np.full(m, 7, dtype))
    _lib.check(_lib.lib().sb_spmv_csr_typed(CODE[dtype], m, n, len(crd), *(a.data_ptr() for a in d), y.data_ptr(),
                                            _stream()))
    wide = np.float64 if np.issubdtype(dtype, np.floating) else dtype
    want = np.zeros(m, wide)
    np.add.at(want, np.repeat(np.arange(m), lens), val.astype(wide) * x[crd].astype(wide))
    _check_typed(y.cpu().numpy(), want, dtype)
