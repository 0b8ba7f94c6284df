"""Workloads of the sparse operators and layers, as a user's program runs them, for measuring.

Each case is a dict of plain values; ``prepare`` makes the inputs and the objects such a program
keeps (patterns, layers, plans), ``run`` is one pass through the public entry points.  Shapes and
distributions are those of the benchmark's five workloads plus the sizes around them: pruned
weights with uneven rows, Bernoulli masks, magnitude-pruned projections of a LLaMA-7B-shaped
layer, ReLU activations.
"""
from __future__ import annotations

import math

import torch

from intrasm_engine_b200.pytorch.attention import SparseAttentionChain
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.sputnik import MySpMM
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.torch import MyLinear
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.utils import default_fwd_kwargs
from intrasm_engine_b200.pytorch.ffn import ReluSparseDownProj, relu_down_proj
from intrasm_engine_b200.pytorch.horizontal_rewriter import SparseDenseLayer
from intrasm_engine_b200.pytorch.huggingface_rewriter import SparseLinear
from intrasm_engine_b200.pytorch.utils import dense_to_sparse_cuda, get_transpose_info

DEVICE = "cuda"
DTYPES = {"f16": torch.float16, "f32": torch.float32}
INDEX = {16: torch.int16, 32: torch.int32}

# the largest listed attention and pruned-product cases; drawn ones stay below
ATTENTION_WORK = 24 * 4096 * 4096 * 0.05 * 64
SPMM_WORK = 2048 * 2048 * 0.5 * 256


def listed():
    return [
        # one fp32 product with a 90 % sparse matrix: the plain operator call
        dict(name="spmm-f32", kind="spmm", dtype="f32", m=1024, k=1024, n=256, sparsity=0.9, batch=1, index_bits=32),
        # the smallest pruned-transformer weight: latency and launches are what counts
        dict(name="spmm-f16-small", kind="spmm", dtype="f16", m=512, k=512, n=128, sparsity=0.95, batch=1,
             index_bits=16),
        # forward and backward of a pruned weight in fine-tuning, fp16
        dict(name="spmm-train-f16", kind="spmm_train", dtype="f16", m=2048, k=512, n=256, sparsity=0.8,
             index_bits=16),
        # the same in fp32 at sizes that divide by nothing
        dict(name="spmm-train-f32-odd", kind="spmm_train", dtype="f32", m=1531, k=1177, n=100, sparsity=0.85,
             index_bits=32),
        # masked attention over the heads of a layer, long sequence
        dict(name="attention", kind="attention", heads=24, m=4096, n=4096, d=64, sparsity=0.95),
        # the same for a short, ragged sequence and a denser mask
        dict(name="attention-short", kind="attention", heads=6, m=1003, n=1003, d=80, sparsity=0.9),
        # pruned up projection beside the dense qkv projection on the same 64 activations
        dict(name="sparse-dense-layer", kind="sparse_dense", m_sparse=11008, m_dense=12288, k=4096, tokens=64,
             sparsity=0.5, index_bits=16),
        # a pruned projection swapped into a model: one token of decoding ...
        dict(name="sparse-linear-decode", kind="sparse_linear", out=11008, inp=4096, tokens=1, sparsity=0.5),
        # ... and the prefill of a prompt
        dict(name="sparse-linear-prefill", kind="sparse_linear", out=11008, inp=4096, tokens=500, sparsity=0.5),
        # forward and backward of the dense branch over a training batch
        dict(name="linear-train", kind="linear", tokens=2048, inp=4096, out=12288, train=True),
        # ReLU-sparse down projection, activations already in CSR
        dict(name="ffn-down", kind="ffn", tokens=256, k=11008, n=4096, density=0.1, from_dense=False),
        # the same from the dense hidden activations of a smaller batch, conversion included
        dict(name="ffn-down-hidden", kind="ffn", tokens=96, k=11008, n=4096, density=0.1, from_dense=True),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["spmm", "spmm", "spmm_train", "spmm_train", "attention", "attention", "sparse_dense",
                       "sparse_linear", "sparse_linear", "linear", "linear", "ffn"])
    if kind in ("spmm", "spmm_train"):
        dtype = rng.choice(["f16", "f32"])
        case = dict(kind=kind, dtype=dtype)
        while True:
            case.update(m=_log_int(rng, 256, 2048), k=_log_int(rng, 256, 2048),
                        n=_log_int(rng, 16, 512, rng.choice([1, 8, 64])), sparsity=round(rng.uniform(0.5, 0.98), 3))
            batch = rng.choice([1, 1, 2, 4, 8]) if kind == "spmm" and dtype == "f32" else 1
            if batch * case["m"] * case["k"] * (1 - case["sparsity"]) * case["n"] <= SPMM_WORK:
                break
        if kind == "spmm":
            case["batch"] = batch
        case["index_bits"] = rng.choice([16, 32]) if dtype == "f16" else 32
        return case
    if kind == "attention":
        while True:
            m, d, sparsity = _log_int(rng, 256, 4096), rng.choice([32, 64, 80, 128]), round(rng.uniform(0.8, 0.98), 3)
            n = m if rng.random() < 0.5 else _log_int(rng, 256, 4096)
            heads = rng.randint(1, 24)
            if heads * m * n * (1 - sparsity) * d <= ATTENTION_WORK:
                return dict(kind=kind, heads=heads, m=m, n=n, d=d, sparsity=sparsity)
    if kind == "sparse_dense":
        tokens = rng.choice([64, 128, 192, 256])  # what the layer takes
        return dict(kind=kind, m_sparse=_log_int(rng, 1024, 11008, 8), m_dense=_log_int(rng, 1024, 12288, 8),
                    k=_log_int(rng, 1024, 4096, 64), tokens=tokens, sparsity=round(rng.uniform(0.5, 0.9), 3),
                    index_bits=rng.choice([16, 32]))
    if kind == "sparse_linear":
        return dict(kind=kind, out=_log_int(rng, 1024, 11008, rng.choice([8, 64])),
                    inp=_log_int(rng, 1024, 4096, rng.choice([8, 64])), tokens=_log_int(rng, 1, 500),
                    sparsity=round(rng.uniform(0.5, 0.9), 3))
    if kind == "linear":
        return dict(kind=kind, tokens=_log_int(rng, 1, 2048), inp=_log_int(rng, 512, 4096, rng.choice([8, 128])),
                    out=_log_int(rng, 512, 12288, rng.choice([8, 128])), train=rng.random() < 0.5)
    return dict(kind="ffn", tokens=_log_int(rng, 32, 256, 32), k=_log_int(rng, 2048, 11008, 8),
                n=_log_int(rng, 1024, 4096, 8), density=round(rng.uniform(0.05, 0.3), 3),
                from_dense=rng.random() < 0.5)


def _randn(shape, gen, dtype=torch.float16, std=1.0):
    return (torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float32) * std).to(dtype)


def _nnz(m, k, sparsity):
    """Stored positions: a multiple of four, as the batched operator wants."""
    return max(4, int(round(m * k * (1.0 - sparsity))) // 4 * 4)


def _pruned(m, k, sparsity, gen, dtype, std):
    """Pruned weight as a dense matrix: the density of a row varies (lognormal, CV 0.3)."""
    sigma = math.sqrt(math.log(1.09))
    row = torch.randn((m, 1), generator=gen, device=DEVICE) * sigma - 0.5 * sigma * sigma
    score = torch.rand((m, k), generator=gen, device=DEVICE) / row.exp()
    kept = score.flatten().argsort()[:_nnz(m, k, sparsity)]
    values = _randn(kept.shape, gen, dtype, std)
    weight = torch.zeros(m * k, dtype=dtype, device=DEVICE)
    weight[kept] = torch.where(values == 0, torch.full_like(values, std), values)
    return weight.view(m, k)


def _magnitude_pruned(m, k, sparsity, gen):
    """N(0, 0.02) weight without its ``sparsity`` share of small values."""
    w = _randn((m, k), gen, torch.float16, 0.02)
    threshold = 0.02 * math.sqrt(2.0) * float(torch.erfinv(torch.tensor(sparsity, dtype=torch.float64)))
    return torch.where(w.abs().float() > threshold, w, torch.zeros((), dtype=w.dtype, device=DEVICE))


def _bernoulli_mask(m, n, density, gen):
    mask = torch.rand((m, n), generator=gen, device=DEVICE) < density
    _values, _ri, row_offsets, cols = dense_to_sparse_cuda(mask.to(torch.float16))
    return row_offsets, cols


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(int(seed))
    kind, s = case["kind"], dict(case)
    if kind in ("spmm", "spmm_train"):
        dtype = DTYPES[case["dtype"]]
        m, k, n = case["m"], case["k"], case["n"]
        weight = _pruned(m, k, case["sparsity"], gen, dtype, 1.0 if dtype == torch.float32 else 0.02)
        values, ri, ro, ci = dense_to_sparse_cuda(weight, index_dtype=INDEX[case["index_bits"]])
        batch = case.get("batch", 1)
        s.update(values=values, ri=ri, ro=ro, ci=ci, transp=())
        if kind == "spmm":
            s["b"] = _randn((batch, k, n) if dtype == torch.float32 else (k, n), gen, dtype)
        else:
            s["transp"] = get_transpose_info(m, k, ri, ro, ci)
            s["values"].requires_grad_(True)
            s["b"] = _randn((k, n), gen, dtype).requires_grad_(True)
            s["grad"] = _randn((m, n), gen, dtype)
    elif kind == "attention":
        m, n, d, heads = case["m"], case["n"], case["d"], case["heads"]
        ro, ci = _bernoulli_mask(m, n, 1.0 - case["sparsity"], gen)
        s["chain"] = SparseAttentionChain(ro, ci, m, n)
        s["q"] = _randn((heads, m, d), gen, torch.float32)
        s["k"] = _randn((heads, n, d), gen, torch.float32)
        s["v"] = _randn((heads, n, d), gen, torch.float32)
    elif kind == "sparse_dense":
        w = _magnitude_pruned(case["m_sparse"], case["k"], case["sparsity"], gen)
        values, ri, ro, ci = dense_to_sparse_cuda(w, index_dtype=INDEX[case["index_bits"]])
        dense = _randn((case["m_dense"], case["k"]), gen, torch.float16, 0.02)
        s["layer"] = SparseDenseLayer(values, ri, ro, ci, case["m_sparse"], dense, mode="fused")
        s["x"] = _randn((case["k"], case["tokens"]), gen)
    elif kind == "sparse_linear":
        s["layer"] = SparseLinear(_magnitude_pruned(case["out"], case["inp"], case["sparsity"], gen))
        s["x"] = _randn((case["tokens"], case["inp"]), gen)
    elif kind == "linear":
        s["x"] = _randn((case["tokens"], case["inp"]), gen).requires_grad_(case["train"])
        s["w"] = _randn((case["out"], case["inp"]), gen, torch.float16, 0.02).requires_grad_(case["train"])
        s["grad"] = _randn((case["tokens"], case["out"]), gen)
    else:
        tokens, k, n = case["tokens"], case["k"], case["n"]
        act = _randn((tokens, k), gen).abs()
        keep = torch.rand((tokens, k), generator=gen, device=DEVICE) < case["density"]
        s["w"] = _randn((n, k), gen, torch.float16, 0.02)
        if case["from_dense"]:  # pre-activations: what the ReLU drops is negative
            s["hidden"] = torch.where(keep, act, -act)
        else:
            act = torch.where(keep, act, torch.zeros((), dtype=act.dtype, device=DEVICE))
            s["values"], _ri, s["ro"], s["ci"] = dense_to_sparse_cuda(act)
            s["layer"] = ReluSparseDownProj(tokens, k, n, device=act.device, gather="none")
    return s


def run(s):
    kind = s["kind"]
    if kind == "spmm":
        if s["dtype"] == "f32":
            return torch.ops.iex_ops.spmm_sputnik_reuse_weight(s["b"], s["ri"], s["values"], s["ro"], s["ci"], s["m"])
        with torch.no_grad():
            return MySpMM.run(s["b"], s["ri"], s["values"], s["ro"], s["ci"], s["m"], s["transp"],
                              fwd_kwargs_1=default_fwd_kwargs(use_tensor_cores="auto"))
    if kind == "spmm_train":
        out = MySpMM.run(s["b"], s["ri"], s["values"], s["ro"], s["ci"], s["m"], s["transp"],
                         fwd_kwargs_1=default_fwd_kwargs(use_tensor_cores="auto"))
        return (out, *torch.autograd.grad(out, (s["b"], s["values"]), s["grad"]))
    if kind == "attention":
        return s["chain"](s["q"], s["k"], s["v"])
    if kind in ("sparse_dense", "sparse_linear"):
        with torch.no_grad():
            return s["layer"](s["x"])
    if kind == "linear":
        out = MyLinear.run(s["x"], s["w"])
        return (out, *torch.autograd.grad(out, (s["x"], s["w"]), s["grad"])) if s["train"] else out
    if s["from_dense"]:
        return relu_down_proj(s["hidden"], s["w"])
    return s["layer"](s["values"], s["ro"], s["ci"], s["w"])


def work(case):
    """Compulsory traffic (each array once) and useful operations (stored positions only)."""
    kind = case["kind"]
    if kind in ("spmm", "spmm_train"):
        m, k, n, batch = case["m"], case["k"], case["n"], case.get("batch", 1)
        e, i = (2 if case["dtype"] == "f16" else 4), case["index_bits"] // 8
        nnz = _nnz(m, k, case["sparsity"])
        nbytes = nnz * (e + i) + 8 * m + batch * e * (k * n + m * n)
        if kind == "spmm":
            return {"bytes": nbytes, "flops": 2 * nnz * n * batch}
        return {"bytes": nbytes + nnz * e + e * (k * n + m * n), "flops": 6 * nnz * n}
    if kind == "attention":
        m, n, d, heads = case["m"], case["n"], case["d"], case["heads"]
        nnz = m * n * (1 - case["sparsity"])
        return {"bytes": 4 * nnz + 4 * m + 4 * heads * d * (2 * m + 2 * n), "flops": 4 * nnz * d * heads}
    if kind == "sparse_dense":
        ms, md, k, t = case["m_sparse"], case["m_dense"], case["k"], case["tokens"]
        nnz = ms * k * (1 - case["sparsity"])
        return {"bytes": nnz * (2 + case["index_bits"] // 8) + 4 * ms + 2 * (md * k + k * t + (ms + md) * t),
                "flops": 2 * t * (nnz + md * k)}
    if kind == "sparse_linear":
        out, inp, t = case["out"], case["inp"], case["tokens"]
        nnz = out * inp * (1 - case["sparsity"])
        return {"bytes": 4 * nnz + 4 * out + 2 * t * (inp + out), "flops": 2 * nnz * t}
    if kind == "linear":
        t, i, o = case["tokens"], case["inp"], case["out"]
        once = 2 * (t * i + i * o + t * o)
        return {"bytes": 2 * once if case["train"] else once, "flops": (6 if case["train"] else 2) * t * i * o}
    t, k, n = case["tokens"], case["k"], case["n"]
    nnz = t * k * case["density"]
    act = 2 * t * k if case["from_dense"] else nnz * 6 + 4 * t
    return {"bytes": act + 2 * (n * k + t * n), "flops": 2 * nnz * n}


def tolerance(case):
    """fp32 operands: fp32 sums in another order.  fp16 operands: one rounding of an fp32 sum."""
    if case["kind"] == "attention" or case.get("dtype") == "f32":
        return {"rel": 1e-5}
    return {"rel": 1e-3, "max": 1e-2}
