"""The work that is timed: one case is one call (or one training step) that a user's program makes, through the package's
public entry points.

A case is a dict of plain values:

    op      what is called
              spmm       C = A @ B on device tensors                      Plan.spmm
              sddmm      one dot product per stored nonzero of A           Plan.sddmm
              train      C = A @ B and dB = A^T @ dC under autograd        SparseOperator.__call__
              attention  C = A_w @ B, dw and dB under autograd             SparseOperator.weighted
              build      a plan for a new matrix and its first product     Plan.from_device_csr, Plan.spmm
              noalloc    C = A @ B from plain CSR, nothing allocated       spmm_csr_noalloc
              host       C = A @ B, host buffers in and out                Plan.spmm_host
    matrix  the family of A (generators.py): uniform, stencil, elasticity, rmat, with its size parameters
    N       columns of the dense operands

Matrices are made on the GPU from the seed; the stencil's and the elasticity matrix's patterns are fixed by their sizes
(their values change with the seed), the others change entirely.
"""
from __future__ import annotations

import math

import torch

import cutespmm_ae_b200 as cs
from cutespmm_ae_b200 import generators as gen
from cutespmm_ae_b200 import torch_ops


def listed():
    return [
        # a small product inside a larger program: a launch and a few memory latencies
        {"name": "spmm-uniform-4096-n32", "op": "spmm", "matrix": "uniform", "M": 4096, "K": 4096, "per_row": 16, "N": 32},
        # a discretised operator applied to a block of vectors
        {"name": "spmm-stencil-512-n128", "op": "spmm", "matrix": "stencil", "nx": 512, "ny": 512, "N": 128},
        # a finite-element matrix applied to a narrow block of vectors
        {"name": "spmm-elasticity-40-n32", "op": "spmm", "matrix": "elasticity", "n": 40, "N": 32},
        # neighbourhood aggregation over a power-law graph
        {"name": "spmm-rmat-20-n128", "op": "spmm", "matrix": "rmat", "scale": 20, "edge_factor": 8, "N": 128},
        # the same on the largest graph one GPU is asked to hold
        {"name": "spmm-rmat-24-n128", "op": "spmm", "matrix": "rmat", "scale": 24, "edge_factor": 8, "N": 128},
        # a rectangular matrix of odd sizes and a number of columns (classes) that no vector load divides
        {"name": "spmm-uniform-odd-n47", "op": "spmm", "matrix": "uniform", "M": 170003, "K": 99991, "per_row": 7, "N": 47},
        # edge scores of a graph layer
        {"name": "sddmm-rmat-18-n64", "op": "sddmm", "matrix": "rmat", "scale": 18, "edge_factor": 8, "N": 64},
        # one aggregation of a training step, forward and backward
        {"name": "train-rmat-17-n64", "op": "train", "matrix": "rmat", "scale": 17, "edge_factor": 8, "N": 64},
        # one attention aggregation of a training step on a mini-batch graph, forward and backward
        {"name": "attention-rmat-14-n32", "op": "attention", "matrix": "rmat", "scale": 14, "edge_factor": 8, "N": 32},
        # a graph that changes from step to step: a plan is made for each product
        {"name": "build-rmat-17-n64", "op": "build", "matrix": "rmat", "scale": 17, "edge_factor": 8, "N": 64},
        # a host framework that owns all of device memory
        {"name": "noalloc-rmat-18-n64", "op": "noalloc", "matrix": "rmat", "scale": 18, "edge_factor": 8, "N": 64},
        # a solver that keeps its vectors in host memory
        {"name": "host-elasticity-40-n64", "op": "host", "matrix": "elasticity", "n": 40, "N": 64},
    ]


# ---- sizes --------------------------------------------------------------------------------------------------------

_A, _B, _C = 0.57, 0.19, 0.19  # R-MAT quadrant probabilities (generators.rmat's defaults; the fourth is 0.05)


def _rmat_counts(scale, edge_factor):
    """Expected (nonzeros, rows that have any) of a symmetrised, deduplicated R-MAT graph: the cells (and rows) of equal
    probability are counted together."""
    draws, d = edge_factor * 2.0 ** scale, 1.0 - _A - _B - _C
    nnz = 0.0
    for i in range(scale + 1):  # levels in quadrant a
        for m in range(scale + 1 - i):  # levels in quadrants b and c, two choices each
            cells = math.comb(scale, i) * math.comb(scale - i, m) * 2.0 ** m
            p = _A ** i * _B ** m * d ** (scale - i - m)
            nnz -= cells * math.expm1(-draws * p * (1 if m == 0 else 2))  # off the diagonal either direction names the cell
    top = _A + _B
    rows = -sum(math.comb(scale, i) * math.expm1(-2 * draws * top ** (scale - i) * (1 - top) ** i) for i in range(scale + 1))
    return nnz, rows


def _sizes(case):
    """(M, K, nonzeros, columns that a nonzero names)."""
    kind = case["matrix"]
    if kind == "uniform":
        nnz = case["M"] * case["per_row"]
        return case["M"], case["K"], nnz, -case["K"] * math.expm1(-nnz / case["K"])
    if kind == "stencil":
        n = case["nx"] * case["ny"]
        return n, n, (3 * case["nx"] - 2) * (3 * case["ny"] - 2), n
    if kind == "elasticity":
        n = 3 * case["n"] ** 3
        return n, n, 9 * (7 * case["n"] ** 3 - 6 * case["n"] ** 2), n
    n = 1 << case["scale"]
    nnz, rows = _rmat_counts(case["scale"], case["edge_factor"])
    if case["op"] in ("sddmm", "attention"):
        nnz = int(0.98 * nnz)  # results per nonzero: every seed gets the same number of them (_matrix)
    return n, n, nnz, rows


def work(case):
    M, K, nnz, used = _sizes(case)
    N, op = case["N"], case["op"]
    csr = 8 * nnz + 4 * (M + 1)
    if op == "sddmm":  # columns, rows of X and Y, one score per nonzero
        return {"bytes": 8 * nnz + 4 * (M + 1) + 4 * N * (M + used), "flops": 2 * nnz * N}
    if op == "train":  # A once, B and dC in, C and dB out
        return {"bytes": csr + 4 * N * (used + M + M + K), "flops": 4 * nnz * N}
    if op == "attention":  # the pattern with its weights, B and dC in, C, dB and dw out
        return {"bytes": csr + 4 * nnz + 4 * N * (used + M + M + K), "flops": 6 * nnz * N}
    return {"bytes": csr + 4 * N * (used + M), "flops": 2 * nnz * N}


def tolerance(case):
    # the tensor cores' tf32 products (banded and block matrices of 4440 panels of 16 rows or more, 64 columns or more)
    # against fp32 sums
    dense_panels = case["matrix"] in ("stencil", "elasticity") and _sizes(case)[0] >= 16 * 4440
    tf32 = dense_panels and case["N"] >= 64 and case["op"] not in ("sddmm", "attention", "noalloc")
    return {"rel": 1e-3} if tf32 else {"rel": 1e-5}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng, kinds, largest):
    """A family and its sizes, about `largest` nonzeros at most."""
    kind = rng.choice(kinds)
    if kind == "uniform":
        per_row = _log(rng, 2, 64)
        M = _log(rng, 1000, max(2000, min(1 << 20, largest // per_row)))
        return {"matrix": kind, "M": M, "K": _log(rng, max(1000, M // 4), 4 * M), "per_row": per_row}
    if kind == "stencil":
        side = min(1024, math.isqrt(largest // 9))
        return {"matrix": kind, "nx": _log(rng, 40, side), "ny": _log(rng, 40, side)}
    if kind == "elasticity":
        return {"matrix": kind, "n": _log(rng, 9, min(64, round((largest / 63) ** (1 / 3))))}
    edge_factor = rng.randint(4, 16)
    return {"matrix": kind, "scale": rng.randint(11, max(12, int(math.log2(largest / (2 * edge_factor))))), "edge_factor": edge_factor}


def draw(rng):
    op = rng.choice(["spmm"] * 6 + ["sddmm", "train", "attention", "build", "noalloc", "host"])
    every = ["uniform", "stencil", "elasticity", "rmat"]
    graphs = ["uniform", "rmat", "rmat"]
    kinds, largest, n_most = {
        "spmm": (every, 1 << 26, 512),
        "sddmm": (every, 1 << 24, 256),
        "train": (graphs, 1 << 22, 256),
        "attention": (graphs, 1 << 21, 128),
        "build": (every, 1 << 23, 128),
        "noalloc": (every, 1 << 23, 256),
        "host": (["stencil", "elasticity", "uniform"], 1 << 22, 128),
    }[op]
    # half of the time a usual width, half of the time any
    N = rng.choice([n for n in (16, 32, 64, 128, 256, 512) if n <= n_most]) if rng.random() < 0.5 else _log(rng, 3, n_most)
    while True:
        case = {"op": op, **_draw_matrix(rng, kinds, largest), "N": N}
        M, K, nnz, _ = _sizes(case)
        if max(M, K) * N > 1 << 29 or (op == "host" and max(M, K) * N > 1 << 25):
            continue
        if op == "noalloc" and (2 * math.ceil(nnz / 1024) + 2) * (N + 3) * 4 > 16 << 20:  # what its built-in scratch holds
            continue
        return case


# ---- one case -----------------------------------------------------------------------------------------------------

def _matrix(case, seed):
    kind = case["matrix"]
    if kind == "uniform":
        return gen.uniform_random(case["M"], case["K"], case["per_row"], seed, "cuda")
    if kind == "stencil":
        return gen.stencil9(case["nx"], case["ny"], seed, "cuda")
    if kind == "elasticity":
        return gen.elasticity3d(case["n"], 3, seed, "cuda")
    A = gen.rmat(case["scale"], case["edge_factor"], _A, _B, _C, seed, "rownorm" if case["op"] == "train" else "uniform", "cuda")
    if case["op"] in ("sddmm", "attention"):  # the last rows lose the 2 % of the edges that differ in number between seeds
        nnz = _sizes(case)[2]
        A.row_ptr, A.cols, A.vals = A.row_ptr.clamp(max=nnz), A.cols[:nnz].contiguous(), A.vals[:nnz].contiguous()
    return A


def prepare(case, seed):
    op, N = case["op"], case["N"]
    rng = torch.Generator("cuda").manual_seed(seed)

    def dense(rows):
        return torch.randn((rows, N), generator=rng, device="cuda")

    A = _matrix(case, seed)
    row_ptr = A.row_ptr.to(torch.int32)
    if op == "host":
        plan = cs.Plan.from_csr(A)
        return {"op": op, "plan": plan, "B": dense(A.K).cpu().pin_memory(), "C": torch.empty((A.M, N), dtype=torch.float32, pin_memory=True)}
    if op in ("build", "noalloc"):
        state = {"op": op, "M": A.M, "K": A.K, "row_ptr": row_ptr, "cols": A.cols, "vals": A.vals, "B": dense(A.K)}
        if op == "noalloc":
            state["C"] = torch.empty((A.M, N), dtype=torch.float32, device="cuda")
        return state
    # the attention form replaces the values of its plans, which the row kernel's plans allow
    options = {"path": cs.PATH_ROWS} if op == "attention" else {}
    plan = cs.Plan.from_device_csr(A.M, A.K, row_ptr, A.cols, A.vals, **options)
    if op == "spmm":
        return {"op": op, "plan": plan, "B": dense(A.K)}
    if op == "sddmm":
        return {"op": op, "plan": plan, "X": dense(A.M), "Y": dense(A.K)}
    state = {"op": op, "operator": torch_ops.SparseOperator(plan, plan_kwargs=options), "B": dense(A.K).requires_grad_(), "dC": dense(A.M)}
    if op == "attention":
        state["w"] = torch.rand(A.nnz, generator=rng, device="cuda").requires_grad_()
    return state


def run(state):
    op = state["op"]
    if op == "spmm":
        return state["plan"].spmm(state["B"])
    if op == "sddmm":
        return state["plan"].sddmm(state["X"], state["Y"])
    if op == "train":
        C = state["operator"](state["B"])
        (dB,) = torch.autograd.grad(C, state["B"], state["dC"])
        return C.detach(), dB
    if op == "attention":
        C = state["operator"].weighted(state["w"], state["B"])
        dw, dB = torch.autograd.grad(C, (state["w"], state["B"]), state["dC"])
        return C.detach(), dw, dB
    if op == "build":
        plan = cs.Plan.from_device_csr(state["M"], state["K"], state["row_ptr"], state["cols"], state["vals"])
        return plan.spmm(state["B"])
    if op == "noalloc":
        return cs.spmm_csr_noalloc(state["M"], state["K"], state["row_ptr"], state["cols"], state["vals"], state["B"], state["C"])
    return state["plan"].spmm_host(state["B"], state["C"])[0]
