"""cutespmm_spmm_csr_noalloc -- the entry point for callers that may not allocate device memory at
call time (their framework owns all of HBM, or they run where allocating calls are forbidden).  It
keeps its partial sums in a scratch array built into the library, so this test checks what such a
caller relies on: the result equals the plan-based entry point's and the CPU oracle's on two calls
in a row (the second call meets the scratch as the first left it), requests beyond the built-in
scratch are refused with an error instead of being attempted, and input that would index outside
the caller's buffers is stopped before or inside the call.  Collected last on purpose (file name)."""
import subprocess
import sys

import numpy as np
import pytest
import torch

import cutespmm_ae_b200 as cs
from cutespmm_ae_b200 import generators as g
from conftest import REL_FRO_TOL_FP32, ROOT

pytestmark = pytest.mark.gpu


def _rel_fro(ref, got):
    return float((got.double() - ref.double()).norm() / ref.double().norm())


def test_noalloc_matches_plan_entry_point_twice_in_a_row(oracle_mod):
    A = g.rmat(15, 8, seed=91, values="uniform")  # hub rows well above the 1024-nonzero chunk length
    assert int((A.row_ptr[1:] - A.row_ptr[:-1]).max()) > 2 * 1024
    plan = cs.Plan.from_csr(A, path=cs.PATH_ROWS)  # the existing entry point, fp32 row kernel
    rp, cols, vals = A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda()
    for call, (N, seed) in enumerate(((128, 92), (200, 93))):  # second call: other width, other B, same scratch
        B = g.dense_operand(A.K, N, seed, device="cuda")
        ref = plan.spmm(B)
        C = torch.full((A.M, N), float("nan"), device="cuda")  # caller-provided output, fully overwritten
        cs.spmm_csr_noalloc(A.M, A.K, rp, cols, vals, B, C)
        torch.cuda.synchronize()
        assert _rel_fro(ref, C) <= REL_FRO_TOL_FP32, f"call {call}"
        # and against the independent checker, not only against another kernel of this library
        want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), A.M, A.K)
        assert oracle_mod.rel_fro(want, C.cpu().numpy()) <= REL_FRO_TOL_FP32, f"call {call} vs oracle"


def test_noalloc_small_and_empty_rows():
    M, K, N = 40, 30, 33
    rp = np.zeros(M + 1, np.int32)
    rp[5:] = 3
    rp[20:] = 4
    cols = torch.tensor([1, 7, 29, 0], dtype=torch.int32, device="cuda")
    vals = torch.tensor([1.0, -2.0, 0.5, 3.0], device="cuda")
    B = g.dense_operand(K, N, 94, device="cuda")
    C = torch.full((M, N), float("nan"), device="cuda")
    cs.spmm_csr_noalloc(M, K, torch.from_numpy(rp).cuda(), cols, vals, B, C)
    torch.cuda.synchronize()
    exp = torch.zeros((M, N), device="cuda")
    exp[4] = B[1] - 2.0 * B[7] + 0.5 * B[29]
    exp[19] = 3.0 * B[0]
    assert torch.allclose(C, exp, rtol=1e-6, atol=1e-6)


def test_noalloc_rejects_what_the_builtin_scratch_cannot_hold():
    d = torch.zeros(8, dtype=torch.int32, device="cuda")
    f = torch.zeros(8, device="cuda")
    # N above the maximum
    st = cs.lib.cutespmm_spmm_csr_noalloc(1, 1, 1, d.data_ptr(), d.data_ptr(), f.data_ptr(), f.data_ptr(), 513,
                                          f.data_ptr(), 513, 513, None)
    assert st == -4 and b"MAX_N" in cs.lib.cutespmm_last_error()
    # more nonzeros than (scratch / N) allows: refused before any pointer is touched
    st = cs.lib.cutespmm_spmm_csr_noalloc(1 << 20, 1 << 20, 1 << 30, d.data_ptr(), d.data_ptr(), f.data_ptr(),
                                          f.data_ptr(), 128, f.data_ptr(), 128, 128, None)
    assert st == -4 and b"scratch" in cs.lib.cutespmm_last_error()
    assert cs.lib.cutespmm_spmm_csr_noalloc(4, 4, 0, None, None, None, None, 8, f.data_ptr(), 8, 8, None) == -1


def test_noalloc_wrapper_refuses_mis_shaped_operands():
    A = g.uniform_random(64, 48, 4, seed=95)
    rp, cols, vals = A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda()
    B = g.dense_operand(A.K, 32, 96, device="cuda")
    good = torch.empty((A.M, 32), device="cuda")
    for kw in (dict(Cout=torch.empty((A.M - 1, 32), device="cuda")),   # too few rows: the kernel would write past the end
               dict(Cout=torch.empty((A.M, 31), device="cuda")),       # too narrow
               dict(B=g.dense_operand(A.K - 1, 32, 96, device="cuda")),  # B shorter than A is wide
               dict(row_ptr=rp[:-1])):
        args = dict(row_ptr=rp, cols=cols, vals=vals, B=B, Cout=good)
        args.update(kw)
        with pytest.raises(ValueError):
            cs.spmm_csr_noalloc(A.M, A.K, args["row_ptr"], args["cols"], args["vals"], args["B"], args["Cout"])


def test_noalloc_survives_row_pointers_and_columns_beyond_the_arrays(oracle_mod):
    """A row pointer array whose last entries exceed the `nnz` the caller states, and a column index that is not below
    K, must not make the kernels index outside the scratch, the CSR arrays or B: positions are clamped to nnz and the
    out-of-range column contributes nothing."""
    A = g.rmat(12, 16, seed=97, values="uniform")  # rows longer than 1024 nonzeros: the chunk and fix-up kernels run
    assert int((A.row_ptr[1:] - A.row_ptr[:-1]).max()) > 1024
    N = 64
    B = g.dense_operand(A.K, N, 98, device="cuda")
    cols = A.cols.clone()
    cols[7] = A.K + 5  # not a row of B
    vals_ok = A.vals.clone()
    vals_ok[7] = 0.0   # what "contributes nothing" means for the checker
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, vals_ok, B.cpu().numpy(), A.M, A.K)
    C = torch.full((A.M, N), float("nan"), device="cuda")
    cs.spmm_csr_noalloc(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), cols.cuda(), A.vals.cuda(), B, C)
    torch.cuda.synchronize()
    assert oracle_mod.rel_fro(want, C.cpu().numpy()) <= REL_FRO_TOL_FP32
    # row pointers that run past the stated nnz: rows are cut off at nnz, nothing beyond the arrays is touched
    rp_bad = A.row_ptr.clone()
    rp_bad[-40:] += 5000
    nnz_kept = A.nnz
    rp_clamped = rp_bad.clamp(max=nnz_kept)
    want2 = oracle_mod.spmm_csr(rp_clamped, A.cols, A.vals, B.cpu().numpy(), A.M, A.K)
    C2 = torch.full((A.M, N), float("nan"), device="cuda")
    cs.spmm_csr_noalloc(A.M, A.K, rp_bad.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), B, C2)
    torch.cuda.synchronize()
    assert oracle_mod.rel_fro(want2, C2.cpu().numpy()) <= REL_FRO_TOL_FP32


@pytest.mark.parametrize("N", [1, 4, 8, 9, 16, 17, 32, 33, 64, 65, 100, 128, 132, 256, 257, 512])
def test_noalloc_at_the_edges_of_every_width(oracle_mod, N):
    """One form of the kernel per range of widths and alignment; rows around the staging buffer (256), the row length the
    groups of a warp share (16), the chunk length (128); a chunk list that a claim of too many nonzeros overflows."""
    rng = np.random.default_rng(N)
    ln = rng.integers(0, 12, 700)
    ln[[0, 5, 6, 7, 300, 301, 699]] = (16, 17, 127, 128, 129, 256, 1500)
    rp = np.concatenate([[0], np.cumsum(ln)])
    A = g.CsrMatrix(700, 400, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, 400, rp[-1]).astype(np.int32)),
                    torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
    B = g.dense_operand(A.K, N, 99, device="cuda")
    args = (A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), B)
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), A.M, A.K)
    C = torch.full((A.M + 1, N), float("nan"), device="cuda")
    for _ in range(2):  # the second call meets the counters as the first left them
        cs.spmm_csr_noalloc(A.M, A.K, *args, C[:A.M])
        assert oracle_mod.rel_fro(want, C[:A.M].cpu().numpy()) <= REL_FRO_TOL_FP32 and torch.isnan(C[A.M]).all()
    bad = A.row_ptr.clone()
    bad[1::2] = 0  # every second row claims all nonzeros up to its end: far more chunks than the nonzeros allow
    cs.spmm_csr_noalloc(A.M, A.K, bad.to(torch.int32).cuda(), *args[1:], C[:A.M])
    torch.cuda.synchronize()
    cs.spmm_csr_noalloc(A.M, A.K, *args, C[:A.M])
    assert oracle_mod.rel_fro(want, C[:A.M].cpu().numpy()) <= REL_FRO_TOL_FP32


@pytest.mark.parametrize("N", [7, 16, 31, 32, 64, 65, 128, 250, 256, 512])
@pytest.mark.parametrize("longest", [40, 400])
def test_noalloc_rows_of_whole_steps_beside_a_column_that_counts_nothing(oracle_mod, N, longest):
    """Rows long enough for whole steps, every remainder of one among them, with and without rows that are cut into chunks (which
    choose the claim); a column that is not below K sends the nonzeros staged with it through the checked steps, and the rows of
    B nobody names hold infinities."""
    rng = np.random.default_rng(N + longest)
    M, K = 3000, 500
    ln = rng.integers(0, 40, M)
    ln[:41] = np.arange(41)
    ln[100:103] = longest
    rp = np.concatenate([[0], np.cumsum(ln)])
    cols, vals = rng.integers(1, K, rp[-1]).astype(np.int32), rng.standard_normal(rp[-1]).astype(np.float32)
    B = g.dense_operand(K, N, 100)
    B[0] = float("inf")
    for unsound in (False, True):
        c, v = cols.copy(), vals.copy()
        if unsound:
            at = rng.choice(rp[-1], 25, replace=False)
            c[at], v[at] = K + 5, 0.0  # for the oracle: nothing times a row that is there
        want = oracle_mod.spmm_csr(rp, np.where(c < K, c, 1), v, B.numpy(), M, K)
        C = torch.full((M, N), float("nan"), device="cuda")
        cs.spmm_csr_noalloc(M, K, torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(c).cuda(), torch.from_numpy(vals).cuda(), B.cuda(), C)
        assert oracle_mod.rel_fro(want, C.cpu().numpy()) <= REL_FRO_TOL_FP32


@pytest.mark.parametrize("N", [1, 16, 33, 64, 128, 132, 256])
def test_noalloc_with_row_pointers_that_go_down(oracle_mod, N):
    """Row ends that decrease among rows that a warp takes together: every row is the sum over its own range, cut to the
    stated nnz and empty where it ends before it begins, and nothing else is read."""
    rng = np.random.default_rng(N + 1)
    M, K, nnz = 500, 300, 4000
    rp = np.sort(rng.integers(0, nnz, M + 1))
    rp[:4] = (0, 100, 10, 20)
    at = rng.choice(np.arange(4, M + 1), 120, replace=False)
    rp[at] = np.clip(rp[at] + rng.integers(-60, 61, 120), 0, nnz + 50)
    cols, vals = rng.integers(0, K, nnz).astype(np.int32), rng.standard_normal(nnz).astype(np.float32)
    begin, end = np.minimum(rp[:-1], nnz), np.minimum(rp[1:], nnz)
    own = [np.arange(b, max(b, e)) for b, e in zip(begin, end)]
    pos = np.concatenate(own)
    want_rp = np.concatenate([[0], np.cumsum([len(o) for o in own])]).astype(np.uint64)
    B = g.dense_operand(K, N, 101, device="cuda")
    want = oracle_mod.spmm_csr(want_rp, cols[pos].astype(np.uint32), vals[pos], B.cpu().numpy(), M, K)
    C = torch.full((M, N), float("nan"), device="cuda")
    cs.spmm_csr_noalloc(M, K, torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(cols).cuda(), torch.from_numpy(vals).cuda(), B, C)
    assert oracle_mod.rel_fro(want, C.cpu().numpy()) <= REL_FRO_TOL_FP32


def test_noalloc_calls_after_overlapping_ones_are_whole(oracle_mod):
    """Calls that overlap on two streams race on the scratch, the list of chunks and the counters: what they write is not
    defined, but they stay inside their own operands, and the ordered calls after them compute every row."""
    A, S = g.rmat(16, 8, seed=103, values="uniform"), g.rmat(11, 8, seed=104, values="uniform")
    dev = [(m.M, m.K, m.row_ptr.to(torch.int32).cuda(), m.cols.cuda(), m.vals.cuda()) for m in (A, S)]
    want, ops = [], []
    for m, N in ((A, 64), (S, 160)):
        B = g.dense_operand(m.K, N, 105, device="cuda")
        ops.append((B, torch.full((m.M + 64, N), float("nan"), device="cuda")))
        want.append(oracle_mod.spmm_csr(m.row_ptr, m.cols, m.vals, B.cpu().numpy(), m.M, m.K))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(20):
        for d, (B, C), s in zip(dev, ops, streams):
            cs.spmm_csr_noalloc(*d, B, C[: d[0]], stream=s)
    torch.cuda.synchronize()
    for d, (B, C), w in zip(dev, ops, want):
        assert torch.isnan(C[d[0]:]).all()  # nothing behind the last row
        C.fill_(float("nan"))
        for _ in range(2):
            cs.spmm_csr_noalloc(*d, B, C[: d[0]])
            assert oracle_mod.rel_fro(w, C[: d[0]].cpu().numpy()) <= REL_FRO_TOL_FP32


def _best_us(call):
    best = float("inf")
    for _ in range(6):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(10):
            call()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end) * 100)
    return best


@pytest.mark.parametrize("N", [16, 32])
def test_noalloc_a_long_row_leaves_the_others_their_time(oracle_mod, N):
    """Rows of four nonzeros, one of them replaced by a long one: the rows are claimed as without it (1.01 to 1.05 times the time;
    1.8 to 2.1 with claims of a quarter of the rows).  Rows of a hundred nonzeros beside long ones take those claims."""
    rng = np.random.default_rng(107)
    M, K = 1_000_000, 50_000
    times = []
    for kind in ("even", "one long", "many of a hundred"):
        ln = np.full(M, 4)
        if kind != "even":
            ln[M // 3] = 3000
        if kind == "many of a hundred":
            ln[rng.choice(M, 10_000, replace=False)] = 100  # a fifth of the nonzeros
        rp = np.concatenate([[0], np.cumsum(ln)])
        cols, vals = rng.integers(0, K, rp[-1]).astype(np.int32), rng.standard_normal(rp[-1]).astype(np.float32)
        dev = torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(cols).cuda(), torch.from_numpy(vals).cuda()
        B = g.dense_operand(K, N, 108, device="cuda")
        C = torch.full((M, N), float("nan"), device="cuda")
        cs.spmm_csr_noalloc(M, K, *dev, B, C)
        want = oracle_mod.spmm_csr(torch.from_numpy(rp), torch.from_numpy(cols), torch.from_numpy(vals), B.cpu().numpy(), M, K)
        assert oracle_mod.rel_fro(want, C.cpu().numpy()) <= REL_FRO_TOL_FP32, kind
        times.append(_best_us(lambda: cs.spmm_csr_noalloc(M, K, *dev, B, C)))
    assert times[1] <= 1.4 * times[0], times


_FIRST_CALLS = """
import statistics, time
import torch
import cutespmm_ae_b200 as cs
from cutespmm_ae_b200 import generators as g

A = g.uniform_random(64, 48, 40, seed=106)
csr = A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda()
ops = {N: (torch.zeros((A.K, N), device="cuda"), torch.empty((A.M, N), device="cuda")) for N in (64, 8, 16, 32, 128, 256, 7, 15, 31, 63, 255)}

def call(N):
    torch.cuda.synchronize()
    t = time.perf_counter()
    cs.spmm_csr_noalloc(A.M, A.K, *csr, *ops[N])
    return time.perf_counter() - t

first = call(64)  # the one call at start-up
once = [call(N) for N in ops if N != 64]
again = [call(N) for N in ops if N != 64]
print(f"{first * 1e6:.0f} {statistics.median(once) * 1e6:.1f} {statistics.median(again) * 1e6:.1f}")
"""


def test_noalloc_one_call_at_startup_loads_every_width():
    """Code is loaded on its first use, which takes device memory and host time (34 us instead of 7.6 for a call that loads its
    kernel): after one call of one width, the first call of every other width and alignment takes as long as its second
    (medians over ten forms, a process of its own)."""
    res = subprocess.run([sys.executable, "-c", _FIRST_CALLS], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr
    startup, once, again = map(float, res.stdout.split())
    assert startup > 10 * again  # where the code is loaded
    assert once <= 2.5 * again, (startup, once, again)
