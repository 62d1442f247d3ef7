"""Calls that wait for the device leave the interpreter to other threads."""
from __future__ import annotations

import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_other_threads_run_while_a_product_is_computed():
    from scorch_b200 import kernels as K, workloads as W
    n = 1_000_000
    A = W.powerlaw_square(n, mean_nnz=12.0, seed=0, device="cuda")
    product = lambda: K.spgemm_csr(A.pos, A.crd, A.val, A.pos, A.crd, A.val, n)
    first = product()
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(1e-4)
    thread = threading.Thread(target=tick)
    thread.start()
    calls = []
    try:
        for _ in range(8):
            begin = time.perf_counter()
            again = product()
            calls.append((begin, time.perf_counter()))
            del again
            torch.cuda.synchronize()
    finally:
        stop.set()
        thread.join()
    # several milliseconds a call, of which a thread that ticks every 0.1 ms sees more than its edges
    longest = max(calls, key=lambda c: c[1] - c[0])
    assert longest[1] - longest[0] > 2e-3
    assert all(sum(b < t < e for t in ticks) >= 5 for b, e in calls if e - b > 2e-3), calls
    again = product()
    assert all(torch.equal(a, b) for a, b in zip(first, again))


def test_products_of_several_threads_at_a_time():
    # the same product on streams of their own: every thread gets the bits of a call alone
    from scorch_b200 import kernels as K, workloads as W
    n = 20011
    A = [W.powerlaw_square(n, mean_nnz=8.0, seed=s, device="cuda") for s in range(4)]
    product = lambda a: K.spgemm_csr(a.pos, a.crd, a.val, a.pos, a.crd, a.val, n)
    want = [product(a) for a in A]
    torch.cuda.synchronize()
    got, errors = [[] for _ in A], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    got[i].append(product(A[i]))
                torch.cuda.current_stream().synchronize()
        except Exception as e:   # noqa: BLE001 - reported below
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(A))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for i, results in enumerate(got):
        assert len(results) == 5 and all(torch.equal(a, b) for r in results for a, b in zip(r, want[i]))
