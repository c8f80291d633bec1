"""Performance cases of the SVC -> vector-sparse SpMM path, through the package's public Python entry points.

A case is a dict of plain values; its ``kind`` says which part of the path it exercises:

    spmm      one product through the reference-signature call ``ops.sspmm`` (magnitude-pruned weights)
    powerlaw  the same call on a power-law matrix with length-sorted row order (a sweep / graph operand)
    bspmm     ``sptrans.spmm.bspmm``: a batch of products with one structure and values per batch entry
    planned   one product through a plan (``ops.sspmm_planned``)
    group     the pruned conv layers as one ``ops.Group`` (every layer x two sparsities x V = 8 and 16)
    encoder   ``SparseEncoderLayer``, whole layer, per-call or grouped linears
    svc       compression of one pruned weight matrix with its values, and its row order
    svcstack  compression of a stack of power-law matrices in one pass

``listed`` are the fixed cases, ``draw`` gives others over the same ranges, ``prepare`` builds what a program holds
before the call (operands, compressed weights, plans, groups), ``run`` is one pass, ``work`` the bytes and operations
the pass cannot do without, ``tolerance`` how far two correct implementations may be apart."""
from __future__ import annotations

import math
import random

import torch

from sspmm_b200 import ops, synthetic
from sspmm_b200.encoder import SparseEncoderLayer
from sspmm_b200.sptrans.spmm import bspmm

DEVICE = "cuda:0"


def listed():
    return [
        # one small pruned layer on a 256-token batch: launch latency and host work of the plain call
        {"name": "spmm_512_n256", "kind": "spmm", "M": 512, "K": 512, "sparsity": 0.7, "V": 8, "N": 256, "f32": False, "order": False},
        # transformer FFN weight, fp32 results wanted (the driver's output type), rows in length order
        {"name": "spmm_ffn_f32", "kind": "spmm", "M": 2048, "K": 512, "sparsity": 0.9, "V": 16, "N": 256, "f32": True, "order": True},
        # last conv stage at batch 1: a 7 x 7 feature map, a column count that is not a multiple of 8
        {"name": "spmm_conv_n49", "kind": "spmm", "M": 512, "K": 4608, "sparsity": 0.9, "V": 8, "N": 49, "f32": False, "order": False},
        # a matrix of the power-law sweep: scattered columns, rows from 1 to thousands of entries
        {"name": "powerlaw_52k", "kind": "powerlaw", "n": 51970, "V": 8, "N": 128},
        # sparse attention probabilities x values: 8 sequences x 12 heads share one mask, head width 64
        {"name": "bspmm_attention", "kind": "bspmm", "M": 512, "K": 512, "sparsity": 0.9, "V": 8, "N": 64, "batch": 96},
        # FFN weight through a plan, on a token count that fills no tile
        {"name": "planned_ffn_n200", "kind": "planned", "M": 512, "K": 2048, "sparsity": 0.9, "V": 16, "N": 200, "f32": False},
        # all conv layers at one eighth of the batch (one rank of eight)
        {"name": "group_conv_n3136", "kind": "group", "N": 3136},
        # all conv layers at the full batch of eight 56 x 56 maps
        {"name": "group_conv_n25088", "kind": "group", "N": 25088},
        # encoder layer on one short sequence, linears grouped: latency of a serving step
        {"name": "encoder_b1_s128", "kind": "encoder", "hidden": 256, "ffn": 1024, "heads": 4, "batch": 1, "seq": 128, "grouped": True},
        # encoder layer at training / offline-inference size
        {"name": "encoder_b32_s512", "kind": "encoder", "hidden": 768, "ffn": 3072, "heads": 12, "batch": 32, "seq": 512, "grouped": False},
        # compressing one conv weight when a model is loaded
        {"name": "svc_conv_512x4608", "kind": "svc", "M": 512, "K": 4608, "sparsity": 0.9, "V": 8},
        # compressing a stack of the power-law sweep
        {"name": "svcstack_16", "kind": "svcstack", "count": 16, "n_min": 4096, "n_max": 65536, "V": 8, "sizes": 1},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(["spmm", "spmm", "spmm", "powerlaw", "bspmm", "planned", "planned", "group", "group", "encoder", "svc", "svcstack"])
    V = rng.choice([8, 16])
    sparsity = rng.choice([0.5, 0.7, 0.8, 0.9, 0.95, 0.98])
    if kind == "spmm":
        odd = rng.random() < 0.25                     # feature maps and token counts of small batches
        N = _log_int(rng, 1, 1024) if odd else 8 * _log_int(rng, 1, 1024)
        return {"kind": kind, "M": _log_int(rng, 64, 2048), "K": _log_int(rng, 64, 4608), "sparsity": sparsity, "V": V, "N": N,
                "f32": rng.random() < 0.5, "order": rng.random() < 0.5}
    if kind == "powerlaw":
        return {"kind": kind, "n": _log_int(rng, 4096, 65536), "V": V, "N": rng.choice([32, 64, 96, 128, 200, 256])}
    if kind == "bspmm":
        return {"kind": kind, "M": V * _log_int(rng, 8, 128), "K": _log_int(rng, 64, 1024), "sparsity": rng.choice([0.5, 0.8, 0.9, 0.95]),
                "V": V, "N": rng.choice([64, 80, 128, 256]), "batch": _log_int(rng, 2, 96)}
    if kind == "planned":
        return {"kind": kind, "M": _log_int(rng, 64, 2048), "K": _log_int(rng, 64, 4608), "sparsity": rng.choice([0.5, 0.7, 0.8, 0.9]), "V": V,
                "N": 8 * _log_int(rng, 1, 2048), "f32": rng.random() < 0.25}
    if kind == "group":
        return {"kind": kind, "N": 8 * _log_int(rng, 25, 3136)}
    if kind == "encoder":
        heads = rng.choice([4, 8, 12])
        return {"kind": kind, "hidden": 64 * heads, "ffn": 256 * heads, "heads": heads, "batch": _log_int(rng, 1, 16),
                "seq": 8 * _log_int(rng, 8, 64), "grouped": rng.random() < 0.5}
    if kind == "svc":
        return {"kind": kind, "M": _log_int(rng, 64, 2048), "K": _log_int(rng, 64, 4608), "sparsity": sparsity, "V": V}
    return {"kind": kind, "count": rng.randint(2, 20), "n_min": 4096, "n_max": 65536, "V": V, "sizes": rng.randint(2, 10 ** 6)}


# ---- inputs ---------------------------------------------------------------------------------------

def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _normal(g, *shape, std=1.0):
    t = torch.randn(shape, device=DEVICE, dtype=torch.float16, generator=g)
    return t if std == 1.0 else t * std


def _pruned_csr(M, K, sparsity, g):
    """Magnitude-pruned N(0, 0.02) weights (``synthetic.magnitude_pruned``) drawn on the GPU, as CSR."""
    w = _normal(g, M, K, std=0.02)
    keep = max(1, int(round((1.0 - sparsity) * M * K)))
    order = torch.sort(w.float().abs().flatten(), descending=True, stable=True).indices[:keep]
    mask = torch.zeros(M * K, dtype=torch.bool, device=DEVICE)
    mask[order] = True
    mask = mask.view(M, K)
    row_ptr = torch.zeros(M + 1, dtype=torch.int32, device=DEVICE)
    row_ptr[1:] = torch.cumsum(mask.sum(1), 0)
    at = mask.nonzero()
    return row_ptr, at[:, 1].int().contiguous(), w[mask].contiguous()


def _with_columns_permuted(row_ptr, col, K, g):
    """The same matrix with its columns in another order (ids ascending inside a row): other column ids, and as many
    vectors in every vector row, so that results of different seeds have one shape.  Values are drawn anew."""
    rows = torch.repeat_interleave(torch.arange(row_ptr.numel() - 1, device=DEVICE), (row_ptr[1:] - row_ptr[:-1]).long())
    perm = torch.randperm(K, device=DEVICE, generator=g)
    keys, _ = torch.sort(rows * K + perm[col.long()])
    return row_ptr, (keys % K).int()


def _weights(M, K, sparsity, V, g):
    row_ptr, col, val = _pruned_csr(M, K, sparsity, g)
    ptr, vcol, vval, _ = ops.svc(row_ptr, col, val, M, K, V)
    return ptr, vcol, vval


def _stack_sizes(case):
    rng = random.Random(case["sizes"])
    return [_log_int(rng, case["n_min"], case["n_max"]) for _ in range(case["count"])]


def _group_products():
    return [(M, K, s, V) for s in synthetic.CONV_SPARSITIES for V in (8, 16) for (M, K) in synthetic.CONV_LAYERS]


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind in ("spmm", "planned"):
        M, K, V, N = case["M"], case["K"], case["V"], case["N"]
        st["ptr"], st["col"], st["val"] = _weights(M, K, case["sparsity"], V, g)
        st["rhs"] = _normal(g, K, N)
        st["dtype"] = torch.float32 if case["f32"] else torch.float16
        if kind == "planned":
            st["plan"] = ops.Plan(st["ptr"], st["col"], V, K)
        else:
            st["order"] = ops.sorted_row_swizzle(st["ptr"]) if case["order"] else None
    elif kind == "powerlaw":
        n, V = case["n"], case["V"]
        row_ptr, col, val = synthetic.power_law_device(n, seed, torch.device(DEVICE))
        st["ptr"], st["col"], st["val"], _ = ops.svc(row_ptr, col, val, n, n, V)
        st["order"] = ops.sorted_row_swizzle(st["ptr"])
        st["rhs"] = _normal(g, n, case["N"])
        st["dtype"] = torch.float16
    elif kind == "bspmm":
        M, K, V, b = case["M"], case["K"], case["V"], case["batch"]
        mask = torch.rand((M // V, K), device=DEVICE, generator=g) >= case["sparsity"]
        st["ptr"] = torch.zeros(M // V + 1, dtype=torch.int32, device=DEVICE)
        st["ptr"][1:] = torch.cumsum(mask.sum(1), 0)
        st["col"] = mask.nonzero()[:, 1].int().contiguous()
        st["order"] = ops.sorted_row_swizzle(st["ptr"])
        st["val"] = torch.rand((b, st["col"].numel() * V), device=DEVICE, generator=g).half()      # attention probabilities
        st["rhs"] = _normal(g, b, K, case["N"])
    elif kind == "group":
        st["out"], items = [], []
        for (M, K, s, V) in _group_products():
            ptr, col, val = _weights(M, K, s, V, g)
            rhs = _normal(g, K, case["N"])
            out = torch.empty((M, case["N"]), dtype=torch.float16, device=DEVICE)
            items.append((ops.Plan(ptr, col, V, K), val, rhs, out))
            st["out"].append(out)
        st["group"] = ops.Group(items)
    elif kind == "encoder":
        st["layer"] = SparseEncoderLayer(case["hidden"], case["ffn"], case["heads"], 0.9, 16, DEVICE, seed=seed)
        st["x"] = _normal(g, case["hidden"], case["batch"] * case["seq"])
    elif kind == "svc":
        row_ptr, col, _ = _pruned_csr(case["M"], case["K"], case["sparsity"], _generator(case["M"]))
        st["csr"] = _with_columns_permuted(row_ptr, col, case["K"], g) + (_normal(g, col.numel(), std=0.02),)
    elif kind == "svcstack":
        st["mats"] = []
        for i, n in enumerate(_stack_sizes(case)):
            row_ptr, col, _ = synthetic.power_law_device(n, 5000 + i, torch.device(DEVICE))
            val = (torch.rand(col.numel(), device=DEVICE, generator=g) * 2 - 1).half()
            st["mats"].append(_with_columns_permuted(row_ptr, col, n, g) + (val, n, n))
    else:
        raise ValueError(kind)
    return st


# ---- one pass -------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("spmm", "powerlaw"):
        return ops.sspmm(state["ptr"], state["col"], state["val"], state["rhs"], case["V"], row_indices=state["order"],
                         out_dtype=state["dtype"])
    if kind == "bspmm":
        return bspmm(state["order"], state["ptr"], state["col"], state["val"], state["rhs"], case["V"])
    if kind == "planned":
        return ops.sspmm_planned(state["plan"], state["val"], state["rhs"], out_dtype=state["dtype"])
    if kind == "group":
        state["group"].run()
        return state["out"]
    if kind == "encoder":
        forward = state["layer"].forward_grouped if case["grouped"] else state["layer"].forward
        return forward(state["x"], case["batch"], case["seq"])
    if kind == "svc":
        row_ptr, col, val = state["csr"]
        ptr, vcol, vval, _ = ops.svc(row_ptr, col, val, case["M"], case["K"], case["V"])
        return ptr, vcol, vval, ops.sorted_row_swizzle(ptr)
    out, _ = ops.svc_batch(state["mats"], case["V"])
    return out


# ---- what a pass cannot do without ------------------------------------------------------------------

def _product_work(M, K, N, V, nvec, out_bytes, batch=1, structures=1):
    m_vec = -(-M // V)
    return {"bytes": structures * (4 * (m_vec + 1) + 4 * nvec) + batch * (2 * V * nvec + 2 * K * N + out_bytes * m_vec * V * N),
            "flops": batch * 2 * nvec * V * N}


def _expected_vectors(M, K, sparsity, V):
    """Expected vectors of an unstructured matrix: a column of a vector row is empty with probability sparsity^V."""
    full, rest = divmod(M, V)
    return int(K * (full * (1 - sparsity ** V) + (1 - sparsity ** rest if rest else 0)))


def work(case):
    kind = case["kind"]
    if kind in ("spmm", "planned"):
        nvec = _expected_vectors(case["M"], case["K"], case["sparsity"], case["V"])
        return _product_work(case["M"], case["K"], case["N"], case["V"], nvec, 4 if case["f32"] else 2)
    if kind == "powerlaw":
        return _product_work(case["n"], case["n"], case["N"], case["V"], 16 * case["n"], 2)
    if kind == "bspmm":
        nvec = int(case["M"] // case["V"] * case["K"] * (1 - case["sparsity"]))
        return _product_work(case["M"], case["K"], case["N"], case["V"], nvec, 2, batch=case["batch"])
    if kind == "group":
        each = [_product_work(M, K, case["N"], V, _expected_vectors(M, K, s, V), 2) for (M, K, s, V) in _group_products()]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "encoder":
        h, f, T = case["hidden"], case["ffn"], case["batch"] * case["seq"]
        shapes = [(h, h)] * 4 + [(f, h), (h, f)]
        nvec = [_expected_vectors(m, k, 0.9, 16) for m, k in shapes]
        weights = sum(4 * (m // 16 + 1) + (4 + 2 * 16) * n + 2 * m for (m, _), n in zip(shapes, nvec))
        return {"bytes": weights + 8 * h + 2 * 2 * h * T, "flops": sum(2 * n * 16 * T for n in nvec) + 4 * T * case["seq"] * h}
    if kind == "svc":
        M, K, V = case["M"], case["K"], case["V"]
        nnz, nvec, m_vec = round((1 - case["sparsity"]) * M * K), _expected_vectors(M, K, case["sparsity"], V), -(-M // V)
        return {"bytes": 4 * (M + 1) + 6 * nnz + 8 * m_vec + 4 + (4 + 2 * V) * nvec, "flops": 0}
    V, total = case["V"], 0
    for n in _stack_sizes(case):
        total += 4 * (n + 1) + 6 * 16 * n + 4 * (-(-n // V) + 1) + (4 + 2 * V) * 16 * n
    return {"bytes": total, "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("svc", "svcstack"):
        return "exact"                                # integers, and values that are only moved
    # four times the distance from the same product (or layer) computed in 64 bits
    if kind == "encoder":
        return {"rel": 1.3e-3, "max": 6e-3}           # fp16 activations between the layer's parts
    if case.get("f32"):
        return {"rel": 2e-5, "max": 8e-5}             # fp32 sums in another order; the tensor cores truncate when they add
    return {"rel": 8e-4, "max": 2e-3}                 # the fp32 sum rounded once to fp16
