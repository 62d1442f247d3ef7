"""One-call sparse attention with rows of many scattered entries (global tokens), around the length
from which the whole CTA takes a row."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [32, 64])
@pytest.mark.parametrize("seq,tokens", [(80, 1), (300, 1), (1000, 3), (2100, 1)])
@pytest.mark.parametrize("with_values", [False, True])
def test_global_tokens(d, seq, tokens, with_values):
    from scorch_b200 import kernels as K
    rng = np.random.default_rng(seq + d)
    i = np.arange(seq)
    mask = np.abs(i[:, None] - i[None, :]) <= 20
    mask[:tokens] = mask[:, -tokens:] = True
    # rows of 63, 64, 65, 66 scattered entries far from the band
    for r, extra in enumerate((63, 64, 65, 66)):
        far = np.flatnonzero(~mask[seq // 2 + r] & (np.abs(i - seq // 2 - r) > 40))
        mask[seq // 2 + r, rng.permutation(far)[:extra]] = True
    pos = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    crd = np.nonzero(mask)[1].astype(np.int32)
    val = rng.uniform(0.5, 1.5, crd.size).astype(np.float32) if with_values else np.ones(crd.size, np.float32)
    Q, Km, V = ((rng.standard_normal((3, seq, d)) * 0.4).astype(np.float32) for _ in range(3))
    c = lambda a: torch.from_numpy(a).cuda()
    got = K.sparse_attention_csr(c(pos), c(crd), c(val), c(Q), c(Km), c(V), scale=0.2).cpu().numpy()
    dense = np.zeros((seq, seq))
    dense[mask] = val
    for u in range(3):
        s = 0.2 * dense * (Q[u].astype(np.float64) @ Km[u].T.astype(np.float64))
        s[~mask] = -np.inf
        p = np.exp(s - s.max(1, keepdims=True))
        want = (p / p.sum(1, keepdims=True)) @ V[u]
        assert np.allclose(got[u], want, rtol=1e-4, atol=1e-5)
    again = K.sparse_attention_csr(c(pos), c(crd), c(val), c(Q), c(Km), c(V), scale=0.2).cpu().numpy()
    assert np.array_equal(got, again)
