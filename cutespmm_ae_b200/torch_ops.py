"""PyTorch operator over the C ABI: `torch.ops.cutespmm.spmm(plan_id, B)` and `torch.ops.cutespmm.sddmm(...)`.

The reference tree ships its graph-layer operators as a pybind extension of the TC-GNN baseline
(TC-GNN_ATC23/TCGNN_conv/TCGNN.cpp:260-271: forward / backward are the same SpMM on the symmetric
adjacency, forward_ef is SDDMM).  Here the same two operators are `torch.library` custom ops on top of
libcutespmm, registered from native code, so they work under autograd, `torch.compile` (through the registered fake kernels) and on
any stream:

    op = SparseOperator(plan)          # registers the plan, gives it an integer id
    C = op(B)                          # C = A @ B, differentiable with respect to B
    scores = op.sddmm(X, Y)            # one dot product per stored nonzero
    C = op.weighted(w, B)              # C = (pattern of A with values w) @ B, differentiable with respect to w and B

The gradient of C = A @ B with respect to B is A^T @ dC: the transposed plan is built on first use
(from the plan's own decoded CSR) and cached.  In `op(B)` A is constant data of the plan, so no gradient flows
to its values.  `op.weighted(w, B)` is the attention form (TCGNN.cpp:260-264, forward_AGNN): w -- one weight per
stored nonzero in the plan's storage order, typically normalised `op.sddmm` scores -- replaces the plan's values
(Plan.set_values) before the product; its gradients are dB = A_w^T @ dC (the transposed plan receives w through a
permutation computed once) and dw = sddmm(dC, B).
"""
from __future__ import annotations

import itertools
import threading
import weakref

import numpy as np
import torch

from . import PATH_SLAB, CuteSpmmError, Plan
from . import _native as _load_native

_native = _load_native()

__all__ = ["SparseOperator", "register_plan", "unregister_plan", "transpose_csr"]

_plans: dict[int, "SparseOperator"] = {}
_ids = itertools.count(1)


def transpose_csr(M: int, K: int, row_ptr, cols, vals):
    """CSR of A^T (K x M) from CSR of A (M x K); entries of a row of A^T ordered by their row in A."""
    rp = np.asarray(row_ptr, dtype=np.int64)
    cols = np.asarray(cols, dtype=np.int64)
    rows = np.repeat(np.arange(M, dtype=np.int64), np.diff(rp))
    order = np.argsort(cols, kind="stable")
    t_rp = np.zeros(K + 1, dtype=np.uint64)
    np.cumsum(np.bincount(cols, minlength=K), out=t_rp[1:])
    return t_rp, rows[order].astype(np.uint32), np.asarray(vals, dtype=np.float32)[order]


class SparseOperator:
    """A plan registered for use from torch ops.  Keeps the plan (and, once a backward pass has run, the plan of
    A^T) alive until `close()` or garbage collection."""

    def __init__(self, plan: Plan, *, plan_kwargs: dict | None = None):
        self.plan = plan
        self.M, self.K, self.nnz = plan.M, plan.K, plan.nnz
        self._plan_kwargs = plan_kwargs or {}
        self._transposed: Plan | None = None
        self._t_perm: torch.Tensor | None = None  # storage position in A of every stored position of A^T (int32)
        self._t_lock = threading.RLock()  # around the two: backward passes of several threads may ask for them at once
        self.id = next(_ids)
        _plans[self.id] = self
        weakref.finalize(self, _plans.pop, self.id, None)
        _native.register_op(self.id, plan._h.value, self.M, self.K, self.nnz, self._make_transposed)
        plan.__dict__.setdefault("_op_ids", []).append(self.id)

    def transposed(self) -> Plan:
        self._make_transposed(False)
        return self._transposed

    def _make_transposed(self, with_order: bool) -> None:
        """Builds what is missing of the plan of A^T and the order its stored positions have in A, and hands both to the
        native operators.  On the device where the plan's options and layout allow it."""
        with self._t_lock:
            if self._transposed is not None and (self._t_perm is not None or not with_order):
                return
            on_device = self._plan_kwargs.get("path", 0) != PATH_SLAB and not set(self._plan_kwargs) - {"path", "split_nnz", "tile_nnz", "min_brick_panels"}
            csr = None
            if on_device:
                try:
                    csr = self.plan.csr_device()
                except CuteSpmmError:  # rows reordered, or a host-only plan
                    csr = None
            if csr is not None:
                rp, cols, vals = csr
                _, order = torch.sort(cols.to(torch.int64) & 0xFFFFFFFF, stable=True)
                if self._transposed is None:
                    rows = torch.repeat_interleave(torch.arange(self.M, dtype=torch.int32, device=cols.device), (rp[1:] - rp[:-1]).to(torch.int64), output_size=self.nnz)
                    t_rp = torch.zeros(self.K + 1, dtype=torch.int64, device=cols.device)
                    torch.cumsum(torch.bincount(cols.to(torch.int64) & 0xFFFFFFFF, minlength=self.K), 0, out=t_rp[1:])
                    self._transposed = Plan.from_device_csr(self.K, self.M, t_rp.to(torch.int32), rows[order], vals[order], **self._plan_kwargs)
                if with_order and self._t_perm is None:
                    self._t_perm = order.to(torch.int32)
                    if not torch.cuda.is_current_stream_capturing():
                        torch.cuda.current_stream(cols.device).synchronize()  # the next user may be on another stream
            else:
                rp, cols, vals = self.plan.decode_csr()
                if self._transposed is None:
                    t_rp, t_cols, t_vals = transpose_csr(self.M, self.K, rp, cols, vals)
                    self._transposed = Plan(self.K, self.M, t_rp, t_cols, t_vals, **self._plan_kwargs)
                if with_order and self._t_perm is None:
                    self._t_perm = torch.from_numpy(np.argsort(np.asarray(cols, dtype=np.int64), kind="stable").astype(np.uint32).view(np.int32)).cuda()
            _native.set_transposed(self.id, self._transposed._h.value, self._t_perm)

    def __call__(self, B: torch.Tensor) -> torch.Tensor:
        if torch.compiler.is_compiling():
            return torch.ops.cutespmm.spmm(self.id, B)
        return _native.op_spmm(self.id, B)

    def sddmm(self, X: torch.Tensor, Y: torch.Tensor, scale_by_values: bool = False) -> torch.Tensor:
        if torch.compiler.is_compiling():
            return torch.ops.cutespmm.sddmm(self.id, X, Y, scale_by_values)
        return _native.op_sddmm(self.id, X, Y, scale_by_values)

    def weighted(self, w: torch.Tensor, B: torch.Tensor) -> torch.Tensor:
        if torch.compiler.is_compiling():
            return torch.ops.cutespmm.spmm_weighted(self.id, w, B)
        return _native.op_weighted(self.id, w, B)

    def set_values(self, vals: torch.Tensor) -> None:
        """New values for the same pattern (Plan.set_values), e.g. normalised `sddmm` scores as attention weights.  The
        plan of A^T, if a backward pass has built one, is dropped and rebuilt from the new values on next use."""
        self.plan.set_values(vals)
        with self._t_lock:
            if self._transposed is not None:
                _native.set_transposed(self.id, None, self._t_perm)
                self._transposed.close()
                self._transposed = None

    def close(self) -> None:
        _plans.pop(self.id, None)
        _native.unregister_op(self.id)
        for p in (self.plan, self._transposed):
            if p is not None:
                p.close()


def register_plan(plan: Plan, **kw) -> int:
    """Registers `plan` and returns the id the ops take; the registry holds the only strong reference."""
    op = SparseOperator(plan, **kw)
    _keep[op.id] = op
    return op.id


def unregister_plan(plan_id: int) -> None:
    op = _keep.pop(plan_id, None) or _plans.get(plan_id)
    if op is not None:
        op.close()


_keep: dict[int, SparseOperator] = {}


def _get(plan_id: int) -> SparseOperator:
    try:
        return _plans[plan_id]
    except KeyError:
        raise RuntimeError(f"cutespmm: no plan registered under id {plan_id}") from None


# The operators and their gradients are native (csrc/torch_bind.cpp); the fake kernels give shapes to tracing.
@torch.library.register_fake("cutespmm::spmm")
def _(plan_id: int, B: torch.Tensor) -> torch.Tensor:
    return B.new_empty((_get(plan_id).M, B.shape[1]))


@torch.library.register_fake("cutespmm::spmm_transposed")
def _(plan_id: int, G: torch.Tensor) -> torch.Tensor:
    return G.new_empty((_get(plan_id).K, G.shape[1]))


@torch.library.register_fake("cutespmm::spmm_weighted")
def _(plan_id: int, w: torch.Tensor, B: torch.Tensor) -> torch.Tensor:
    return B.new_empty((_get(plan_id).M, B.shape[1]))


@torch.library.register_fake("cutespmm::spmm_weighted_transposed")
def _(plan_id: int, w: torch.Tensor, G: torch.Tensor) -> torch.Tensor:
    return G.new_empty((_get(plan_id).K, G.shape[1]))


@torch.library.register_fake("cutespmm::sddmm")
def _(plan_id: int, X: torch.Tensor, Y: torch.Tensor, scale_by_values: bool) -> torch.Tensor:
    return X.new_empty((_get(plan_id).nnz,))
