"""Performance cases of the sparse hot path: what a program that uses this package has it compute, through the
entry points such a program calls (``matmul``, ``einsum``, ``spmm_bias_act``, ``pipelines``, ``kernels``), on
operands that stay on the GPU.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges; ``prepare`` makes a case's inputs,
``run`` is one pass, ``work`` the bytes and operations a pass cannot do without, ``tolerance`` how far two correct
implementations may differ.  Patterns and values follow ``scorch_b200/workloads.py``.
"""
import math

import numpy as np
import torch

import scorch_b200 as scorch
from scorch_b200 import kernels as K
from scorch_b200 import pipelines as P
from scorch_b200 import workloads as W

DTYPES = {"f32": torch.float32, "f64": torch.float64}
SIZEOF = {"f32": 4, "f64": 8}


def listed():
    return [
        # One layer act(A X + b) of a graph network on a citation-sized graph: a few microseconds of GPU work,
        # so launches and the host path are what a training loop over small graphs pays for.
        {"name": "layer_small", "kind": "layer", "n": 2500, "mean": 5.0, "k": 16, "relu": True},
        # Configuration 1: uniform 1 % matrix times a 64-column operand, as torch CSR tensor through matmul.
        {"name": "spmm_uniform", "kind": "spmm", "dtype": "f32", "pattern": "uniform", "m": 4096, "n": 4096, "mean": 41.0, "k": 64},
        # The same call on a power-law matrix of no convenient size, with an operand width that is no multiple of
        # a vector load (class scores, concatenated features).
        {"name": "spmm_ragged", "kind": "spmm", "dtype": "f32", "pattern": "powerlaw", "m": 70001, "n": 70001, "mean": 20.0, "k": 77},
        # Double precision block of vectors, as iterative solvers and eigensolvers multiply it.
        {"name": "spmm_f64", "kind": "spmm", "dtype": "f64", "pattern": "uniform", "m": 120000, "n": 120000, "mean": 27.0, "k": 16},
        # Configuration 3: top-k sparse autoencoder, encode (per-row top-k of the pre-activations to CSR) and decode.
        {"name": "sae_topk_decode", "kind": "sae", "batch": 8192, "latent": 32768, "topk": 32, "width": 4096},
        # Configuration 2: sparse attention of 4 x 8 heads over a band with random pairs.
        {"name": "attention_band", "kind": "attention", "units": 32, "seq": 4096, "d": 64, "window": 128, "density": 0.01, "global": 0},
        # A short ragged sequence, narrow heads, a sliding window with one global token.
        {"name": "attention_short", "kind": "attention", "units": 12, "seq": 1000, "d": 32, "window": 32, "density": 0.0, "global": 1},
        # Scores alone, one head per einsum call, with the mask in coordinate form.
        {"name": "sddmm_coo", "kind": "sddmm", "format": "coo", "seq": 4096, "d": 64, "window": 128, "density": 0.01, "global": 0},
        # Configuration 4: two-layer GCN forward on a two-million-node power-law graph.
        {"name": "gcn_large", "kind": "gcn", "n": 2000000, "mean": 50.0, "k_in": 256, "k_hidden": 256, "k_out": 64},
        # Configuration 5: matrix-vector product of a power-law matrix.
        {"name": "spmv_large", "kind": "spmv", "dtype": "f32", "n": 2000000, "mean": 12.0},
        # Sparse products: A A of a small matrix (two-hop neighbourhoods, coarse-grid operators) ...
        {"name": "spgemm_small", "kind": "spgemm", "dtype": "f32", "n": 20011, "mean": 8.0},
        # ... and configuration 5's.
        {"name": "spgemm_large", "kind": "spgemm", "dtype": "f32", "n": 2000000, "mean": 12.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["layer", "spmm", "spmm", "sae", "attention", "attention", "sddmm", "gcn", "spmv", "spgemm", "spgemm"])
    if kind == "layer":
        return {"kind": kind, "n": int(_log(rng, 500, 50000)), "mean": round(_log(rng, 3, 40), 1), "k": int(_log(rng, 3, 256)), "relu": rng.random() < 0.5}
    if kind == "spmm":
        pattern = rng.choice(["uniform", "powerlaw"])
        m = int(_log(rng, 1000, 200000))
        n = m if pattern == "powerlaw" else int(_log(rng, 1000, 200000))
        f64 = rng.random() < 0.3
        k = int(_log(rng, 1, 32 if f64 else 512))
        if not f64 and rng.random() < 0.5:
            k = max(16, k // 16 * 16)
        return {"kind": kind, "dtype": "f64" if f64 else "f32", "pattern": pattern, "m": m, "n": n, "mean": round(_log(rng, 4, 64), 1), "k": k}
    if kind == "sae":
        return {"kind": kind, "batch": int(_log(rng, 200, 8192)), "latent": int(_log(rng, 4096, 32768)), "topk": int(_log(rng, 8, 64)),
                "width": rng.choice([256, 384, 768, 1000, 1024, 2048, 4096])}
    if kind in ("attention", "sddmm"):
        c = {"kind": kind, "seq": int(_log(rng, 300, 4096)), "d": rng.choice([32, 64]), "window": int(_log(rng, 16, 160)),
             "density": rng.choice([0.0, round(_log(rng, 0.001, 0.02), 4)]), "global": rng.choice([0, 1])}
        if kind == "attention":
            return dict(c, units=rng.choice([2, 8, 12, 16, 32]))
        return dict(c, format=rng.choice(["coo", "csr"]))
    if kind == "gcn":
        return {"kind": kind, "n": int(_log(rng, 3000, 2000000)), "mean": round(_log(rng, 4, 50), 1), "k_in": rng.choice([64, 100, 128, 256]),
                "k_hidden": rng.choice([64, 128, 256]), "k_out": rng.choice([16, 40, 64])}
    if kind == "spmv":
        return {"kind": kind, "dtype": rng.choice(["f32", "f32", "f64"]), "n": int(_log(rng, 5000, 2000000)), "mean": round(_log(rng, 3, 24), 1)}
    return {"kind": kind, "dtype": rng.choice(["f32", "f32", "f64"]), "n": int(_log(rng, 3000, 2000000)), "mean": round(_log(rng, 3, 12), 1)}


# ---- inputs --------------------------------------------------------------------------------------------------------
def _uniform(m, n, mean, seed):
    """Columns uniform, about ``mean`` entries per row (duplicates dropped)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    row = torch.randint(0, m, (int(m * mean),), generator=g, device="cuda")
    key = torch.unique(row * n + torch.randint(0, n, (row.numel(),), generator=g, device="cuda"))
    pos = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    pos[1:] = torch.bincount(torch.div(key, n, rounding_mode="floor"), minlength=m).cumsum(0)
    return W.Csr((m, n), pos.int(), (key % n).int(), torch.randn(key.numel(), generator=g, device="cuda"))


def _fixed(case):
    """Entries of a mask's band and global rows and columns."""
    s, w, g = case["seq"], min(case["window"], case["seq"] - 1), case["global"]
    return s * (2 * w + 1) - w * (w + 1) + 2 * g * (s - w - 1)


def _pairs(case):
    return int((case["seq"] ** 2 - _fixed(case)) * case["density"])


def _powerlaw(case, seed):
    """One pattern per case, its rows and columns relabelled at random by the seed: as many entries and products
    with every seed."""
    n = case["n"]
    a = W.powerlaw_square(n, mean_nnz=case["mean"], seed=n, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    label = torch.randperm(n, generator=g, device="cuda")
    row = torch.repeat_interleave(label, (a.pos[1:] - a.pos[:-1]).long())
    key = torch.sort(row * n + label[a.crd.long()])[0]
    pos = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    pos[1:] = torch.bincount(row, minlength=n).cumsum(0)
    return W.Csr(a.shape, pos.int(), (key % n).int(), _normal(key.numel(), seed + 1, case["dtype"]))


def _mask(case, seed):
    """Band, a set number of random pairs beside it, global tokens; values 1."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = case["seq"]
    i = torch.arange(s, device="cuda")
    d = (i[:, None] - i[None, :]).abs() <= case["window"]
    d[:case["global"]] = True
    d[:, :case["global"]] = True
    pairs = _pairs(case)
    if pairs:
        u = torch.rand((s, s), generator=g, device="cuda").masked_fill_(d, 2.0).flatten()
        d.view(-1)[torch.topk(u, pairs, largest=False)[1]] = True
    pos = torch.zeros(s + 1, dtype=torch.int64, device="cuda")
    pos[1:] = d.sum(1).cumsum(0)
    crd = d.nonzero()[:, 1].int().contiguous()
    return W.Csr((s, s), pos.int(), crd, torch.ones(crd.numel(), device="cuda"))


def _values(csr, dtype, seed):
    return csr if dtype == "f32" else W.Csr(csr.shape, csr.pos, csr.crd, _normal(csr.nnz, seed, dtype))


def _normal(shape, seed, dtype="f32"):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda", dtype=DTYPES[dtype])


def _stensor(a):
    return scorch.STensor.from_csr_arrays(a.shape, a.pos, a.crd, a.val)


def prepare(case, seed):
    kind, seed = case["kind"], 16 * seed
    if kind == "layer":
        a = W.gcn_graph(case["n"], mean_deg=case["mean"] / 2, max_deg=max(4, case["n"] // 8), seed=seed, device="cuda")
        return {"case": case, "a": _stensor(a), "x": _normal((case["n"], case["k"]), seed + 1), "bias": _normal(case["k"], seed + 2)}
    if kind == "spmm":
        a = (_uniform(case["m"], case["n"], case["mean"], seed) if case["pattern"] == "uniform"
             else W.powerlaw_square(case["n"], exponent=2.1, mean_nnz=case["mean"], seed=seed, device="cuda"))
        a = _values(a, case["dtype"], seed + 1)
        return {"case": case, "a": a.torch_csr(), "b": _normal((case["n"], case["k"]), seed + 2, case["dtype"])}
    if kind == "sae":
        return {"case": case, "x": _normal((case["batch"], case["latent"]), seed),
                "w": W.sae_decoder(case["latent"], case["width"], seed=seed + 1, device="cuda")}
    if kind == "attention":
        m = _mask(case, seed)
        q, k, v = (_normal((case["units"], case["seq"], case["d"]), seed + i) * 8 ** -0.5 for i in (1, 2, 3))
        return {"case": case, "mask": m, "q": q, "k": k, "v": v}
    if kind == "sddmm":
        m = _mask(case, seed)
        if case["format"] == "csr":
            s = _stensor(m)
        else:
            row = torch.repeat_interleave(torch.arange(case["seq"], device="cuda"), (m.pos[1:] - m.pos[:-1]).long())
            s = scorch.STensor.from_coo(indices=torch.stack([row, m.crd.long()]), values=m.val, shape=m.shape)
        q, k = (_normal((case["seq"], case["d"]), seed + i) * 8 ** -0.5 for i in (1, 2))
        return {"case": case, "s": s, "q": q, "k": k}
    if kind == "gcn":
        a = W.gcn_graph(case["n"], mean_deg=case["mean"], max_deg=max(4, case["n"] // 40), seed=seed, device="cuda")
        return {"case": case, "a": a, "x": _normal((case["n"], case["k_in"]), seed + 1),
                "w1": W.glorot(case["k_in"], case["k_hidden"], seed + 2, "cuda"), "w2": W.glorot(case["k_hidden"], case["k_out"], seed + 3, "cuda")}
    a = _powerlaw(case, seed)
    if kind == "spmv":
        return {"case": case, "a": _stensor(a), "x": _normal(case["n"], seed + 2, case["dtype"])}
    return {"case": case, "a": _stensor(a)}


# ---- one pass ------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["case"]["kind"]
    if kind == "layer":
        return scorch.spmm_bias_act(state["a"], state["x"], state["bias"], state["case"]["relu"])
    if kind == "spmm":
        return scorch.matmul(state["a"], state["b"])
    if kind == "sae":
        pos, crd, val = K.topk_rows_to_csr(state["x"], state["case"]["topk"], relu=True)
        return pos, crd, val, K.spmm_csr(pos, crd, val, state["w"])
    if kind == "attention":
        m = state["mask"]
        return P.sparse_attention(m.pos, m.crd, m.val, state["q"], state["k"], state["v"], scale=state["case"]["d"] ** -0.5)
    if kind == "sddmm":
        r = scorch.einsum("ij,ik,jk->ij", state["s"], state["q"], state["k"])
        return r.index.mode_indices[0][0], r.index.mode_indices[1][0], r.values
    if kind == "gcn":
        a = state["a"]
        return P.gcn_forward(a.pos, a.crd, a.val, state["x"], state["w1"], state["w2"])
    if kind == "spmv":
        return scorch.matmul(state["a"], state["x"])
    r = scorch.matmul(state["a"], state["a"])
    return r.index.mode_indices[1][0], r.index.mode_indices[1][1], r.values


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _degrees(n, exponent, mean):
    """Quantiles of the power-law row lengths of ``workloads.powerlaw_square``."""
    u = (np.arange(min(n, 20000)) + 0.5) / min(n, 20000)
    base = (1 - u) ** (-1 / (exponent - 1))
    lo, hi = 1e-3, 4 * mean + 4
    for _ in range(50):
        mid = (lo + hi) / 2
        lo, hi = (mid, hi) if np.maximum(np.floor(base * mid), 1).mean() < mean else (lo, mid)
    return np.minimum(np.maximum(np.floor(base * hi), 1), n)


def _mask_nnz(case):
    return _fixed(case) + _pairs(case)


def work(case):
    kind = case["kind"]
    if kind == "layer":
        n, k, nnz = case["n"], case["k"], case["n"] * (case["mean"] + 1)
        return {"bytes": 4 * (n + 1) + 8 * nnz + 8 * n * k + 4 * k, "flops": 2 * nnz * k}
    if kind == "spmm":
        m, n, k, b = case["m"], case["n"], case["k"], SIZEOF[case["dtype"]]
        nnz = m * case["mean"] if case["pattern"] == "uniform" else m * _degrees(n, 2.1, case["mean"]).mean()
        return {"bytes": 4 * (m + 1) + (4 + b) * nnz + b * (m + n) * k, "flops": 2 * nnz * k}
    if kind == "sae":
        r, n, t, k = case["batch"], case["latent"], case["topk"], case["width"]
        used = n * (1 - math.exp(-r * t / n))  # rows of the decoder that some activation takes
        return {"bytes": 4 * r * n + 4 * (r + 1) + 8 * r * t + 4 * used * k + 4 * r * k, "flops": 2 * r * t * k}
    if kind == "attention":
        u, s, d, nnz = case["units"], case["seq"], case["d"], _mask_nnz(case)
        return {"bytes": 4 * (s + 1) + 8 * nnz + 16 * u * s * d, "flops": 4 * u * nnz * d}
    if kind == "sddmm":
        s, d, nnz = case["seq"], case["d"], _mask_nnz(case)
        return {"bytes": (4 * nnz if case["format"] == "coo" else 4 * (s + 1)) + 8 * nnz + 8 * s * d + (4 if case["format"] == "coo" else 12) * nnz,
                "flops": 2 * nnz * d}
    if kind == "gcn":
        n, i, h, o, nnz = case["n"], case["k_in"], case["k_hidden"], case["k_out"], case["n"] * (2 * case["mean"] + 1)
        return {"bytes": 4 * (n + 1) + 8 * nnz + 4 * n * (i + o) + 4 * h * (i + o), "flops": 2 * nnz * (h + o) + 2 * n * h * (i + o)}
    n, b = case["n"], SIZEOF[case["dtype"]]
    d = _degrees(n, 2.3, case["mean"])
    nnz = n * d.mean()
    if kind == "spmv":
        return {"bytes": 4 * (n + 1) + (4 + b) * nnz + 2 * b * n, "flops": 2 * nnz}
    products = nnz * d.mean()
    out = n * float(np.mean(n * (1 - np.exp(-d * d.mean() / n))))
    return {"bytes": 4 * (n + 1) + (4 + b) * nnz + 4 * (n + 1) + (4 + b) * out, "flops": 2 * products}


def tolerance(case):
    # sums of a row in another order; indices and row pointers are whole numbers and stay the same
    return {"rel": 1e-13 if case.get("dtype") == "f64" else 1e-5}
