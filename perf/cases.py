"""The work this framework is timed on: products, gradients and attention over
sparse patterns, through the public operators.

Every case names a family of patterns (stile_gb300.synthetic), its size, the
dense width and what is done with it.  A program plans an operator once per
pattern and then calls it on new operands, so the operator of a case is kept
here and shared by every state of that case; the operands, and in the
training steps the matrix values too, come from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import stile_gb300.device as D
from stile_gb300 import synthetic as syn
from stile_gb300.api import HybridSpMMFunction, PlanConfig, SddmmOperator, SparseAttention, SpmmOperator
from stile_gb300.gcn import TwoLayerGCN

FEATURES = 602      # input features of the two-layer GCN


def listed():
    return [
        # a small general sparse matrix in fp32 (split tensor tiles): one product, where launches count
        {"name": "plain_14k_forward", "do": "forward", "pattern": "plain", "m": 4096, "k": 4096, "nnz": 14_700,
         "width": 64, "fp32": True, "operand": "fp32"},
        # the same with longer rows, in training: product, transposed product and value gradients
        {"name": "plain_160k_step", "do": "step", "pattern": "plain", "m": 4096, "k": 4096, "nnz": 160_000,
         "width": 64, "fp32": True, "operand": "fp32"},
        # inference of a graph layer on a citation-sized graph
        {"name": "graph_forward", "do": "forward", "pattern": "graph", "m": 169_343, "k": 169_343, "nnz": 1_170_000,
         "width": 128, "fp32": False, "operand": "fp32"},
        # the same graph with bf16 node features and a wider layer
        {"name": "graph_forward_bf16", "do": "forward", "pattern": "graph", "m": 169_343, "k": 169_343,
         "nnz": 1_170_000, "width": 256, "fp32": False, "operand": "bf16"},
        # training the classifier layer of that graph: an odd class count, rows packed without padding
        {"name": "graph_step_41", "do": "step", "pattern": "graph", "m": 169_343, "k": 169_343, "nnz": 1_170_000,
         "width": 41, "fp32": False, "operand": "fp32"},
        # the whole two-layer GCN (602 -> 128 -> 41) on a mid-sized dense social graph: logits and all gradients
        {"name": "gcn_two_layer_step", "do": "gcn", "pattern": "social", "m": 50_000, "k": 50_000, "nnz": 2_500_000,
         "width": 128, "fp32": False, "operand": "fp32"},
        # training the hidden layer on the large social graph
        {"name": "social_step", "do": "step", "pattern": "social", "m": 232_965, "k": 232_965, "nnz": 11_600_000,
         "width": 128, "fp32": False, "operand": "fp32"},
        # inference through a pruned transformer weight, bf16 activations of 4096 tokens
        {"name": "pruned_forward_bf16", "do": "forward", "pattern": "pruned", "m": 3072, "k": 768, "nnz": 235_930,
         "width": 4096, "fp32": False, "operand": "bf16"},
        # fine-tuning the transposed weight with fp32 activations
        {"name": "pruned_step", "do": "step", "pattern": "pruned", "m": 768, "k": 3072, "nnz": 235_930,
         "width": 4096, "fp32": False, "operand": "fp32"},
        # scores on a large sparse mask
        {"name": "mask_scores", "do": "sddmm", "pattern": "mask", "m": 100_000, "k": 100_000, "nnz": 2_000_000,
         "width": 64, "fp32": True, "operand": "fp32"},
        # scores on a smaller mask, bf16 operands of a feature count that fills no vector
        {"name": "mask_scores_bf16", "do": "sddmm", "pattern": "mask", "m": 20_000, "k": 20_000, "nnz": 400_000,
         "width": 100, "fp32": True, "operand": "bf16"},
        # multi-head attention on the strided pattern of a sparse transformer
        {"name": "attention_strided", "do": "attention", "pattern": "strided", "m": 4096, "k": 4096, "nnz": 766_144,
         "width": 64, "fp32": True, "operand": "fp32", "heads": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "graph", "graph", "social", "pruned", "mask", "attention"])
    if kind == "plain":
        m = _log(rng, 1000, 8000)
        return {"do": rng.choice(["forward", "step"]), "pattern": "plain", "m": m, "k": _log(rng, 1000, 8000),
                "nnz": int(m * rng.uniform(3.6, 40)), "width": _log(rng, 16, 256), "fp32": True, "operand": "fp32"}
    if kind in ("graph", "social"):
        n = _log(rng, 8000, 170_000) if kind == "graph" else _log(rng, 8000, 60_000)
        case = {"do": rng.choice(["forward", "step"]), "pattern": kind, "m": n, "k": n,
                "nnz": int(n * (rng.uniform(5, 12) if kind == "graph" else rng.uniform(30, 50))),
                "width": _log(rng, 16, 256), "fp32": False, "operand": "fp32"}
        if case["do"] == "forward":
            case["operand"] = rng.choice(["fp32", "bf16"])
        elif kind == "social":
            case["do"] = rng.choice(["step", "gcn"])
        return case
    if kind == "pruned":
        m, k = rng.choice([(768, 768), (3072, 768), (768, 3072), (1024, 1024)])
        case = {"do": rng.choice(["forward", "step"]), "pattern": "pruned", "m": m, "k": k,
                "nnz": int(m * k * rng.uniform(0.05, 0.2)), "width": _log(rng, 128, 4096), "fp32": False,
                "operand": "fp32"}
        if case["do"] == "forward":
            case["operand"] = rng.choice(["fp32", "bf16"])
        return case
    if kind == "mask":
        n = _log(rng, 5000, 100_000)
        return {"do": "sddmm", "pattern": "mask", "m": n, "k": n, "nnz": int(n * rng.uniform(10, 25)),
                "width": _log(rng, 16, 128), "fp32": True, "operand": rng.choice(["fp32", "bf16"])}
    n = _log(rng, 512, 4096)
    return {"do": "attention", "pattern": rng.choice(["strided", "logsparse"]), "m": n, "k": n, "nnz": 0,
            "width": rng.choice([32, 64, 80, 128]), "fp32": True, "operand": "fp32", "heads": rng.randint(1, 12)}


def _size(case):
    return case["pattern"], case["m"], case["k"], case["nnz"]


@functools.lru_cache(maxsize=8)
def _pattern(pattern, m, k, nnz):
    """The matrix a program holds: scipy CSR with its initial values."""
    if pattern == "plain":
        mean = nnz / m
        # the shortest row length whose power law has about that mean
        lens = np.arange(1, 1025, dtype=np.float64)
        for shortest in range(1, 64):
            p = lens[shortest - 1:] ** -2.1
            if (lens[shortest - 1:] * p).sum() / p.sum() >= 0.95 * mean:
                break
        return syn.power_law_rows(m, k, exponent=2.1, min_len=shortest, max_len=1024, seed=0)
    if pattern == "graph":
        return syn.community_graph(n=m, target_nnz=nnz, exponent=2.0, block_frac=0.30, seed=0)
    if pattern == "social":
        return syn.gcn_graph(n=m, target_nnz=nnz, exponent=1.9, block_frac=0.10, seed=0)
    if pattern == "pruned":
        return syn.pruned_weight(m, k, sparsity=1.0 - nnz / (m * k), block_frac=0.5, std=0.02, seed=0)
    if pattern == "mask":
        return syn.sddmm_mask(n=m, target_nnz=nnz, exponent=2.1, block_frac=0.10, seed=0)
    return syn.strided_pattern(m) if pattern == "strided" else syn.logsparse_pattern(m)


@functools.lru_cache(maxsize=32)
def _operator(do, pattern, m, k, nnz, width, fp32):
    A = _pattern(pattern, m, k, nnz)
    if do == "sddmm":
        return SddmmOperator(A, width)
    if do == "attention":
        return SparseAttention(A, width)
    cfg = PlanConfig(tc_mode=D.TC_SPLIT_BF16 if fp32 else D.TC_BF16)
    if do == "gcn":
        return SpmmOperator(A, width, cfg), SpmmOperator(A, 41, cfg)
    op = SpmmOperator(A, width, cfg)
    if do == "step":
        op.transposed       # the backward's plan, made with the operator
    return op


def _inputs(case, seed):
    """The operands of one state, on the GPU, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    A = _pattern(*_size(case))
    m, k, width, do = case["m"], case["k"], case["width"], case["do"]

    def normal(*shape):
        x = torch.randn(*shape, generator=gen, device="cuda")
        return x.to(torch.bfloat16) if case["operand"] == "bf16" else x

    def values():
        v = torch.as_tensor(A.data.astype(np.float32), device="cuda")
        return v * (1.0 + 0.1 * torch.randn(len(v), generator=gen, device="cuda"))

    if do == "forward":
        return {"B": normal(k, width)}
    if do == "step":
        return {"vals": values(), "B": normal(k, width), "dC": normal(m, width)}
    if do == "gcn":
        return {"vals": values(), "X": normal(m, FEATURES), "W1": normal(FEATURES, width) / math.sqrt(FEATURES),
                "W2": normal(width, 41) / math.sqrt(width), "dC": normal(m, 41)}
    if do == "sddmm":
        return {"X": normal(m, width), "Y": normal(k, width)}
    h = case["heads"]
    return {"Q": normal(h, m, width), "K": normal(h, k, width), "V": normal(h, k, width)}


def prepare(case, seed):
    state = _inputs(case, seed)
    state["do"] = case["do"]
    op = _operator(case["do"], *_size(case), case["width"], case["fp32"])
    if case["do"] == "gcn":
        A = _pattern(*_size(case))
        model = TwoLayerGCN(A, state.pop("W1"), state.pop("W2"), ops=op)
        with torch.no_grad():
            model.vals.copy_(state.pop("vals"))
        state["model"] = model
        return state
    if case["do"] == "step":
        for name in ("vals", "B"):
            state[name].requires_grad_(True)
    state["op"] = op
    return state


def run(state):
    do = state["do"]
    if do == "forward":
        return {"C": state["op"](state["B"])}
    if do == "step":
        C = HybridSpMMFunction.apply(state["vals"], state["B"], state["op"])
        dvals, dB = torch.autograd.grad(C, (state["vals"], state["B"]), state["dC"])
        return {"C": C.detach(), "dvals": dvals, "dB": dB}
    if do == "gcn":
        model = state["model"]
        logits = model(state["X"])
        params = (model.vals, model.lin1.weight, model.lin2.weight)
        dvals, dW1, dW2 = torch.autograd.grad(logits, params, state["dC"])
        return {"logits": logits.detach(), "dvals": dvals, "dW1": dW1, "dW2": dW2}
    if do == "sddmm":
        return {"scores": state["op"](state["X"], state["Y"])}
    return {"out": state["op"](state["Q"], state["K"], state["V"])}


def work(case):
    A = _pattern(*_size(case))
    m, k, n, nnz, do = case["m"], case["k"], case["width"], A.nnz, case["do"]
    index = 4 * (m + 1) + 4 * nnz
    size = 2 if case["operand"] == "bf16" else 4
    if do == "forward":
        return {"bytes": index + 4 * nnz + size * k * n + 4 * m * n, "flops": 2.0 * nnz * n}
    if do == "step":    # A, vals, B, dC in; C, dB, dvals out
        return {"bytes": index + 8 * nnz + 8 * k * n + 8 * m * n, "flops": 6.0 * nnz * n}
    if do == "gcn":     # A, vals, X, weights, dC in; logits and gradients out; the hidden layer out and in again
        hidden = n
        dense = 4 * m * FEATURES + 8 * (FEATURES * hidden + hidden * 41) + 8 * m * 41 + 8 * m * hidden
        return {"bytes": index + 8 * nnz + dense,
                "flops": 6.0 * nnz * (hidden + 41) + 4.0 * m * FEATURES * hidden + 6.0 * m * hidden * 41}
    if do == "sddmm":
        return {"bytes": index + 4 * nnz + size * (m + k) * n, "flops": 2.0 * nnz * n}
    h = case["heads"]
    return {"bytes": index + 16 * h * m * n, "flops": 4.0 * h * nnz * n}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _csr64(A, vals=None):
    v = torch.as_tensor(A.data, dtype=torch.float64, device="cuda") if vals is None else vals.double()
    return torch.sparse_csr_tensor(torch.as_tensor(A.indptr.astype(np.int64), device="cuda"),
                                   torch.as_tensor(A.indices.astype(np.int64), device="cuda"), v, size=A.shape)


def _entries(A):
    rows = np.repeat(np.arange(A.shape[0], dtype=np.int64), np.diff(A.indptr))
    return torch.as_tensor(rows, device="cuda"), torch.as_tensor(A.indices.astype(np.int64), device="cuda")


def _dots(rows, cols, X, Y):
    """<X[rows[t]], Y[cols[t]]> for every t, some entries at a time."""
    out = torch.empty(len(rows), dtype=torch.float64, device="cuda")
    for a in range(0, len(rows), 1 << 20):
        r, c = rows[a:a + (1 << 20)], cols[a:a + (1 << 20)]
        out[a:a + (1 << 20)] = (X[r] * Y[c]).sum(1)
    return out


def _transposed_product(A, rows, cols, vals, dC):
    out = torch.zeros(A.shape[1], dC.shape[1], dtype=torch.float64, device="cuda")
    for a in range(0, len(rows), 1 << 20):
        r, c = rows[a:a + (1 << 20)], cols[a:a + (1 << 20)]
        out.index_add_(0, c, vals[a:a + (1 << 20), None] * dC[r])
    return out


def exact(case, seed):
    A, do = _pattern(*_size(case)), case["do"]
    x = {name: t.double() for name, t in _inputs(case, seed).items()}
    if do == "forward":
        # the operator holds the matrix values as fp32
        vals = torch.as_tensor(A.data.astype(np.float32), device="cuda")
        return {"C": _csr64(A, vals) @ x["B"]}
    rows, cols = _entries(A)
    if do == "step":
        return {"C": _csr64(A, x["vals"]) @ x["B"], "dvals": _dots(rows, cols, x["dC"], x["B"]),
                "dB": _transposed_product(A, rows, cols, x["vals"], x["dC"])}
    if do == "gcn":
        S = _csr64(A, x["vals"])
        P1 = x["X"] @ x["W1"]
        H1 = S @ P1
        Z1 = torch.relu(H1)
        P2 = Z1 @ x["W2"]
        dP2 = _transposed_product(A, rows, cols, x["vals"], x["dC"])
        dH1 = (dP2 @ x["W2"].T) * (H1 > 0)
        dP1 = _transposed_product(A, rows, cols, x["vals"], dH1)
        return {"logits": S @ P2, "dvals": _dots(rows, cols, x["dC"], P2) + _dots(rows, cols, dH1, P1),
                "dW1": x["X"].T @ dP1, "dW2": Z1.T @ dP2}
    if do == "sddmm":
        return {"scores": _dots(rows, cols, x["X"], x["Y"])}
    out = torch.zeros_like(x["V"])
    for h in range(case["heads"]):
        s = _dots(rows, cols, x["Q"][h], x["K"][h]) / math.sqrt(case["width"])
        top = torch.full((A.shape[0],), -math.inf, dtype=torch.float64, device="cuda")
        top.scatter_reduce_(0, rows, s, "amax")
        e = torch.exp(s - top[rows])
        p = e / torch.zeros_like(top).index_add_(0, rows, e)[rows]
        out[h] = _csr64(A, p) @ x["V"][h]
    return {"out": out}
