"""Dense transform on the tensor cores: edges of its tiles, chunks and panels, and values it cannot split."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(X, W):
    from scorch_b200 import _lib
    L, (m, k), n = _lib.lib(), X.shape, W.shape[1]
    out = torch.full((m + 1, n), 7.0, device="cuda")          # a guard row behind the result
    ws = torch.empty(L.sb_dense_matmul_workspace_bytes(n, k), dtype=torch.uint8, device="cuda")
    _lib.check(L.sb_dense_matmul_f32(m, n, k, X.data_ptr(), k, W.data_ptr(), n, out.data_ptr(), n, ws.data_ptr(),
                                     ws.numel(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert L.sb_dense_matmul_status() == 0
    assert (out[m] == 7.0).all()
    return out[:m]


@pytest.mark.parametrize("m", [1, 127, 128, 129, 148 * 128 + 5, 60000])
@pytest.mark.parametrize("n,k", [(8, 4), (16, 32), (40, 36), (64, 256), (72, 100), (128, 64), (136, 128), (256, 260)])
def test_dense_matmul(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    X = torch.randn((m, k), generator=g, device="cuda")
    W = torch.randn((k, n), generator=g, device="cuda") * k ** -0.5
    want = X.double() @ W.double()
    err = lambda c: ((c.double() - want).norm() / want.norm()).item()
    # no further from float64 than a chain of fp32 FMAs is (2.9e-7 at k = 256)
    assert err(_run(X, W)) <= 1.2e-7 + 1.7e-7 * (k / 256) ** 0.5
    assert torch.equal(_run(X, W), _run(X, W))


def test_values_beyond_the_split():
    X = torch.randn((1000, 64), device="cuda")
    W = torch.randn((64, 64), device="cuda") * 0.125
    X[130, 3], X[131, 5], X[700, 0] = float("inf"), float("nan"), 3.0e38
    got, want = _run(X, W), X.double() @ W.double()
    assert torch.isinf(got[130]).all() and torch.isnan(got[131]).all()
    fine = torch.isfinite(want.float())
    assert torch.equal(fine, torch.isfinite(got))
    assert torch.allclose(got[fine].double(), want[fine], rtol=1e-4, atol=1e-5)
    W[3, 7] = float("nan")
    got = _run(X, W)
    assert torch.isnan(got[:, 7]).all() and torch.isfinite(got[0, :7]).all()


@pytest.mark.parametrize("m,n,k,stop", [(128, 64, 64, 0), (5000, 72, 100, 0), (60000, 128, 64, 1), (60000, 64, 256, 11),
                                        (60000, 136, 128, 10 ** 6)])
def test_result_is_whole_behind_a_wait_that_ran_out(m, n, k, stop):
    # the issuing thread of every CTA stops: the other waits run out after a second, the rest of the rows is
    # done without the tensor cores
    import ctypes as C
    from scorch_b200 import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    X = torch.randn((m, k), generator=g, device="cuda")
    W = torch.randn((k, n), generator=g, device="cuda") * k ** -0.5
    out = torch.full((m + 1, n), 7.0, device="cuda")
    ws = torch.empty(L.sb_dense_matmul_workspace_bytes(n, k), dtype=torch.uint8, device="cuda")
    status = C.c_int(-1)
    _lib.check(L.sb_dense_matmul_probe(m, n, k, X.data_ptr(), k, W.data_ptr(), n, out.data_ptr(), n, ws.data_ptr(),
                                       ws.numel(), stop, C.byref(status), torch.cuda.current_stream().cuda_stream))
    assert status.value == (1 if stop < 10 ** 6 else 0)
    assert L.sb_dense_matmul_status() == 0 and (out[m] == 7.0).all()
    want = X.double() @ W.double()
    assert ((out[:m].double() - want).norm() / want.norm()).item() <= 1.2e-7 + 1.7e-7 * (k / 256) ** 0.5
    assert torch.equal(_run(X, W), _run(X, W))


def test_values_beyond_the_split_take_no_longer_than_other_kernels_do():
    # one NaN in W sends every tile to the FMA form: 4 times the library product at this size (measured);
    # a thread per row, walking K for every column, took 100 times the library's
    X = torch.randn((200_000, 256), device="cuda")
    W = torch.randn((256, 256), device="cuda")

    def ms(f):
        f()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            f()
        b.record()
        b.synchronize()
        return a.elapsed_time(b) / 5
    from scorch_b200 import kernels as K
    library = ms(lambda: torch.matmul(X, W))
    W[5, 7] = float("nan")
    mine = ms(lambda: K.dense_matmul(X, W))
    print(f"library {library:.3f} ms, FMA form {mine:.3f} ms")
    assert mine < 8 * library


def test_results_that_overflow():
    # the library's answer to sums beyond the largest float: infinities, not what the parts of the split add up to
    g = torch.Generator(device="cuda").manual_seed(0)
    X, W = torch.randn((40000, 64), generator=g, device="cuda"), torch.randn((64, 72), generator=g, device="cuda")
    X[5], X[6, 0], X[39999, 3] = 1.6e38, 1.6e38, -1.6e38
    W[0], W[3] = 1414.2135, 141.42135
    got, want = _run(X, W), X.double() @ W.double()
    for row, sign in ((6, 1), (39999, -1)):
        assert (got[row] == sign * float("inf")).all()
    assert not torch.isnan(got[torch.arange(40000, device="cuda") != 5]).any()
    fine = want.abs().amax(1) < 1e30
    assert fine.sum() == 40000 - 3
    assert ((got[fine].double() - want[fine]).norm() / want[fine].norm()).item() < 2e-7


@pytest.mark.parametrize("scale", [1e-38, 1e-36, 1e-33, 1e-30, 1e30, 1e36])
@pytest.mark.parametrize("of", ["X", "W", "one row", "one column"])
def test_results_far_from_one(scale, of):
    g = torch.Generator(device="cuda").manual_seed(1)
    X, W = torch.randn((40000, 64), generator=g, device="cuda"), torch.randn((64, 72), generator=g, device="cuda")
    rows, cols = slice(None), slice(None)
    if of == "X":
        X *= scale
    elif of == "W":
        W *= scale
    elif of == "one row":
        rows = slice(777, 778)
        X[rows] *= scale
    else:
        cols = slice(70, 71)
        W[:, cols] *= scale
    got, want, library = (c[rows, cols].double() for c in (_run(X, W), X.double() @ W.double(), torch.matmul(X, W)))
    err = lambda c: ((c - want).norm() / want.norm()).item()
    # (one denormal step of 2^-149 per product where operands of 1e-38 lose bits of their own)
    assert err(got) <= max(2e-7, 1.5 * err(library))


@pytest.mark.parametrize("n", [8, 16, 40, 72, 136])
def test_bits_do_not_depend_on_what_ran_before(n):
    # tensor-memory columns behind the last one of C hold what an earlier product left: NaNs here
    g = torch.Generator(device="cuda").manual_seed(n)
    X, W = torch.randn((40000, 64), generator=g, device="cuda"), torch.randn((64, n), generator=g, device="cuda")
    wide = torch.randn((64, 64 if n <= 64 else 128), generator=g, device="cuda")
    bad = X.clone()
    bad[:, 5] = float("nan")
    results = []
    for before in (bad, X, X * 1e-36):
        _run(before, wide)
        results.append(_run(X, W))
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])
