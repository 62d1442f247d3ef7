"""Column split of a CSR matrix and the chunked product."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(lens, n, seed):
    rng = np.random.default_rng(seed)
    pos = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    crd = np.concatenate([np.sort(rng.choice(n, size=x, replace=False)) for x in lens]).astype(np.int32)
    return pos, crd, rng.standard_normal(crd.size).astype(np.float32)


@pytest.mark.parametrize("chunks", [1, 2, 5, 64])
@pytest.mark.parametrize("k", [1, 40, 64, 200])
def test_split_and_product(chunks, k):
    from scorch_b200 import kernels as K
    n = 3001
    lens = [0, 0, 3000, 1, 0, 33, 700] + [int(x) for x in np.random.default_rng(1).integers(0, 40, 900)] + [0, 0]
    pos, crd, val = _csr(lens, n, seed=chunks)
    d = lambda a: torch.from_numpy(a).cuda()
    split = K.ColumnSplit(d(pos), d(crd), d(val), n, chunks)
    width, first = -(-n // chunks), 0
    rows = np.repeat(np.arange(len(lens)), lens)
    for c in range(chunks):
        keep = crd // width == c
        p = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=len(lens)))])
        assert split.counts[c] == keep.sum() and np.array_equal(split.pos[c].cpu().numpy(), p)
        part = slice(first, first + split.counts[c])
        assert np.array_equal(split.crd[part].cpu().numpy(), crd[keep])
        assert np.array_equal(split.val[part].cpu().numpy(), val[keep])
        first += split.counts[c]
    B = np.random.default_rng(k).standard_normal((n, k)).astype(np.float32)
    want = O.spmm_csr_acc64(pos, crd, val, B)
    for relu in (False, True):
        got = split.matmul(d(B), relu=relu).cpu().numpy()
        assert O.allclose_report(got, np.maximum(want, 0) if relu else want, 1e-4, 1e-4)[0]


def test_columns_that_do_not_ascend_are_not_split(monkeypatch):
    from scorch_b200 import kernels as K, pipelines as P
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 2e5)
    pos, crd, val = _csr([40] * 2000, 2000, seed=3)
    g = torch.Generator().manual_seed(0)
    X, W1, W2 = (torch.randn(s, generator=g).cuda() for s in ((2000, 64), (64, 64), (64, 40)))
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    assert K.ColumnSplit.of(d(pos), d(crd), d(val), 2000, 64) is not None
    out = P.gcn_forward(d(pos), d(crd), d(val), X, W1, W2)
    flip = lambda a: a.reshape(2000, 40)[:, ::-1].reshape(-1)
    assert K.ColumnSplit.of(d(pos), d(flip(crd)), d(flip(val)), 2000, 64) is None
    back = P.gcn_forward(d(pos), d(flip(crd)), d(flip(val)), X, W1, W2)
    A = torch.sparse_csr_tensor(d(pos), d(crd), d(val), size=(2000, 2000)).to_dense().double()
    want = A @ (torch.relu(A @ (X.double() @ W1.double())) @ W2.double())
    for got in (out, back):
        assert ((got.double() - want).norm() / want.norm()).item() < 1e-6


@pytest.mark.parametrize("chunks", [1, 2])
def test_sharded_forward_by_column_chunks(monkeypatch, chunks):
    # one rank; row chunks of the operand accumulate, each cut by columns on its own
    from scorch_b200 import kernels as K, sharded as S
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 1e5)
    pos, crd, val = _csr([60] * 2000, 2000, seed=4)
    g = torch.Generator().manual_seed(1)
    X, W1, W2 = (torch.randn(s, generator=g).cuda() for s in ((2000, 64), (64, 72), (72, 40)))
    p, c, v = (torch.from_numpy(a).cuda() for a in (pos, crd, val))
    shard = S.ShardedCsr.from_global(p, c, v, 0, 1, chunks=chunks)
    A = torch.sparse_csr_tensor(p, c, v, size=(2000, 2000)).to_dense().double()
    want = A @ (torch.relu(A @ (X.double() @ W1.double())) @ W2.double())
    for _ in range(2):
        got = S.gcn_forward_sharded(shard, X, W1, W2)
        assert ((got.double() - want).norm() / want.norm()).item() < 1e-6
    assert all(b.columns[1] is not None for b in shard.blocks)


@pytest.mark.parametrize("chunks", [1, 2])
def test_sharded_forward_sees_values_written_in_place(monkeypatch, chunks):
    # with one row chunk the block's arrays are the caller's own: the kept split has to follow them
    from scorch_b200 import kernels as K, sharded as S
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 1e5)
    pos, crd, val = _csr([60] * 2000, 2000, seed=5)
    g = torch.Generator().manual_seed(2)
    X, W1, W2 = (torch.randn(s, generator=g).cuda() for s in ((2000, 64), (64, 72), (72, 64)))
    p, c, v = (torch.from_numpy(a).cuda() for a in (pos, crd, val))
    shard = S.ShardedCsr.from_global(p, c, v, 0, 1, chunks=chunks)
    blocks = shard.blocks

    def check():
        # (the pieces' columns are numbered from 0)
        A = torch.cat([torch.sparse_csr_tensor(b.pos, b.crd, b.val, size=(2000, 2000 // chunks)).to_dense()
                       for b in blocks], 1).double()
        want = A @ (torch.relu(A @ (X.double() @ W1.double())) @ W2.double())
        got = S.gcn_forward_sharded(shard, X, W1, W2)
        assert ((got.double() - want).norm() / want.norm()).item() < 1e-6

    check()
    assert all(b.columns[1] is not None for b in blocks)
    kept = [b.columns[1] for b in blocks]
    check()
    assert all(b.columns[1] is k for b, k in zip(blocks, kept))          # nothing was written: cut once
    for b in blocks:
        b.val.mul_(torch.linspace(0.5, 2.0, b.nnz, device="cuda"))
    check()
    if chunks == 1:
        v[::3] = 0.25                                                    # through the caller's tensor
        check()
    for b in blocks:
        last = torch.full_like(b.crd, 2000 // chunks - 1)
        b.crd.copy_(last - torch.flip(b.crd, (0,)))                      # other columns, ascending in a row again
        b.pos.copy_(b.nnz - torch.flip(b.pos, (0,)))
    check()
    for b in blocks:
        b.val = torch.ones_like(b.val)                                   # another tensor
    check()


def test_sharded_forward_in_inference_mode(monkeypatch):
    # tensors made there count no writes
    from scorch_b200 import kernels as K, sharded as S
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 1e5)
    pos, crd, val = _csr([60] * 2000, 2000, seed=6)
    with torch.inference_mode():
        g = torch.Generator().manual_seed(3)
        X, W1, W2 = (torch.randn(s, generator=g).cuda() for s in ((2000, 64), (64, 72), (72, 64)))
        p, c, v = (torch.from_numpy(a).cuda() for a in (pos, crd, val))
        shard = S.ShardedCsr.from_global(p, c, v, 0, 1)
        for _ in range(2):
            A = torch.sparse_csr_tensor(p, c, v, size=(2000, 2000)).to_dense().double()
            want = A @ (torch.relu(A @ (X.double() @ W1.double())) @ W2.double())
            got = S.gcn_forward_sharded(shard, X, W1, W2)
            assert ((got.double() - want).norm() / want.norm()).item() < 1e-6
            v.mul_(-0.5)


def test_split_product_refuses_what_spmm_refuses():
    from scorch_b200 import kernels as K
    pos, crd, val = (torch.from_numpy(a).cuda() for a in _csr([5] * 30, 40, seed=7))
    split = K.ColumnSplit(pos, crd, val, 40, 3)
    B = torch.randn((40, 12), device="cuda")
    want = K.spmm_csr(pos, crd, val, B)
    got = split.matmul(B.t().contiguous().t())
    assert torch.allclose(got, want, rtol=1e-4, atol=1e-5)               # other strides: copied, as there
    for bad in (B.double(), B.cpu()):
        with pytest.raises(TypeError):
            split.matmul(bad)
    for bad in (B[:39], B[:, 0]):
        with pytest.raises(ValueError):
            split.matmul(bad)
    for out in (torch.empty((30, 11), device="cuda"), torch.empty((30, 12), device="cuda").double(),
                torch.empty((12, 30), device="cuda").t()):
        with pytest.raises(ValueError):
            split.matmul(B, out=out)
    with pytest.raises(ValueError):
        split.matmul(B, accumulate=True)


def test_graph_without_rows_is_not_split():
    from scorch_b200 import kernels as K
    assert K.split_chunks(0, 1_000_000, 0, 64) == 0
    none = torch.empty(0, dtype=torch.int32, device="cuda")
    A = torch.zeros(1, dtype=torch.int32, device="cuda"), none, none.float()
    assert K.ColumnSplit.of(*A, 1_000_000, 64) is None


@pytest.mark.parametrize("sharded", [False, True])
def test_captured_forward_reads_the_matrix_itself(monkeypatch, sharded):
    # no wait for the device while a graph is captured, and a replay sees values written since
    from scorch_b200 import kernels as K, pipelines as P, sharded as S
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 1e5)
    pos, crd, val = _csr([60] * 2000, 2000, seed=8)
    g = torch.Generator().manual_seed(4)
    X, W1, W2 = (torch.randn(s, generator=g).cuda() for s in ((2000, 64), (64, 72), (72, 64)))
    p, c, v = (torch.from_numpy(a).cuda() for a in (pos, crd, val))
    shard = S.ShardedCsr.from_global(p, c, v, 0, 1)
    forward = (lambda: S.gcn_forward_sharded(shard, X, W1, W2)) if sharded else (lambda: P.gcn_forward(p, c, v, X, W1, W2))
    forward()                                    # buffers, kept split
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        forward()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = forward()
    for _ in range(2):
        v.mul_(-0.5)
        forward()                                # another split takes the kept one's place
        junk = [torch.full((1 << 20,), 1 << 30, dtype=torch.int32, device="cuda") for _ in range(4)]
        graph.replay()
        del junk
        A = torch.sparse_csr_tensor(p, c, v, size=(2000, 2000)).to_dense().double()
        want = A @ (torch.relu(A @ (X.double() @ W1.double())) @ W2.double())
        assert ((out.double() - want).norm() / want.norm()).item() < 1e-6


@pytest.mark.parametrize("sharded", [False, True])
def test_forward_without_memory_for_the_copy(monkeypatch, sharded):
    # the products of the matrix itself need none
    from scorch_b200 import kernels as K, pipelines as P, sharded as S
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 1e5)
    pos, crd, val = _csr([60] * 2000, 2000, seed=9)
    g = torch.Generator().manual_seed(5)
    X, W1, W2 = (torch.randn(s, generator=g).cuda() for s in ((2000, 64), (64, 72), (72, 64)))
    p, c, v = (torch.from_numpy(a).cuda() for a in (pos, crd, val))
    tried = []

    def no_memory(self, *args):
        tried.append(args)
        raise torch.OutOfMemoryError("no memory")
    monkeypatch.setattr(K.ColumnSplit, "__init__", no_memory)
    got = (S.gcn_forward_sharded(S.ShardedCsr.from_global(p, c, v, 0, 1), X, W1, W2) if sharded
           else P.gcn_forward(p, c, v, X, W1, W2))
    A = torch.sparse_csr_tensor(p, c, v, size=(2000, 2000)).to_dense().double()
    want = A @ (torch.relu(A @ (X.double() @ W1.double())) @ W2.double())
    assert tried and ((got.double() - want).norm() / want.norm()).item() < 1e-6


def test_split_dropped_while_another_stream_multiplies_it():
    from scorch_b200 import kernels as K
    pos, crd, val = (torch.from_numpy(a).cuda() for a in _csr([60] * 20000, 20000, seed=10))
    B = torch.randn((20000, 64), device="cuda")
    want = K.spmm_csr(pos, crd, val, B)
    out = torch.empty_like(want)
    split, side = K.ColumnSplit(pos, crd, val, 20000, 5), torch.cuda.Stream()
    sizes = [(t.numel(), t.dtype) for t in (split.pos, split.crd, split.val)]
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)           # a tenth of a second: the product is still to come
        split.matmul(B, out=out)
    del split
    fresh = [torch.zeros(n, dtype=t, device="cuda") for n, t in sizes]      # would take the split's memory
    torch.cuda.synchronize()
    assert all((t == 0).all() for t in fresh)
    assert torch.allclose(out, want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("hidden,width", [(64, 40), (64, 64), (256, 64)])
def test_forward_that_cuts_on_every_call(monkeypatch, hidden, width):
    from scorch_b200 import kernels as K, pipelines as P
    monkeypatch.setattr(K, "SPLIT_CHUNK_BYTES", 1e5)
    products, matmul = [], K.ColumnSplit.matmul
    monkeypatch.setattr(K.ColumnSplit, "matmul",
                        lambda self, B, *a, **kw: products.append(B.shape[1]) or matmul(self, B, *a, **kw))
    pos, crd, val = _csr([100] * 2000, 2000, seed=10)
    g = torch.Generator().manual_seed(6)
    X, W1, W2 = (torch.randn(s, generator=g).cuda() for s in ((2000, 32), (32, hidden), (hidden, width)))
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = torch.sparse_csr_tensor(d(pos), d(crd), d(val), size=(2000, 2000)).to_dense().double()
    want = A @ (torch.relu(A @ (X.double() @ W1.double())) @ W2.double())
    got = P.gcn_forward(d(pos), d(crd), d(val), X, W1, W2)
    assert products == [hidden, width] and ((got.double() - want).norm() / want.norm()).item() < 1e-6
    flip = lambda a: a.reshape(2000, 100)[:, ::-1].reshape(-1)           # columns that do not ascend: one pass
    got = P.gcn_forward(d(pos), d(flip(crd)), d(flip(val)), X, W1, W2)
    assert len(products) == 2 and ((got.double() - want).norm() / want.norm()).item() < 1e-6
    crd[-1] = 2000
    monkeypatch.setenv("SCORCH_B200_VALIDATE", "1")
    with pytest.raises(ValueError, match="column index out of range"):
        P.gcn_forward(d(pos), d(crd), d(val), X, W1, W2)
