"""Parity of the CUDA path (called through the C ABI) with the CPU oracle, on a B200."""
import numpy as np
import pytest
import torch

import cutespmm_ae_b200 as cs
from cutespmm_ae_b200 import generators as g
from conftest import GOLDEN_CASES, REL_FRO_TOL, REL_FRO_TOL_FP32, load_golden

pytestmark = pytest.mark.gpu

PATHS = [cs.PATH_ROWS, cs.PATH_BRICK, cs.PATH_AUTO, cs.PATH_SLAB]
PATH_TOL = {cs.PATH_ROWS: REL_FRO_TOL_FP32, cs.PATH_BRICK: REL_FRO_TOL, cs.PATH_AUTO: REL_FRO_TOL, cs.PATH_SLAB: REL_FRO_TOL}


def run(plan, B_np, **kw):
    B = torch.from_numpy(np.ascontiguousarray(B_np)).cuda()
    C = torch.full((plan.M, B.shape[1]), float("nan"), device="cuda")  # every element must be overwritten
    plan.spmm(B, C, **kw)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    return C.cpu().numpy()


@pytest.mark.parametrize("path", PATHS, ids=["rows", "brick", "auto", "slab"])
@pytest.mark.parametrize("name", GOLDEN_CASES)
def test_golden_fixtures(oracle_mod, name, path):
    gd = load_golden(name)
    N = int(gd["N"])
    p = cs.Plan(int(gd["M"]), int(gd["K"]), gd["row_ptr"], gd["cols"], gd["vals"], path=path)
    C = run(p, gd["B"])
    assert oracle_mod.rel_fro(gd["C"], C) <= PATH_TOL[path]


@pytest.mark.parametrize("path", PATHS, ids=["rows", "brick", "auto", "slab"])
@pytest.mark.parametrize("workload,Ns", [("uniform4096", [32]), ("stencil512", [128]),
                                         ("elasticity40", [32, 64, 128, 256]), ("rmat20", [128])])
def test_named_workloads_match_oracle(oracle_mod, workload, Ns, path):
    if path == cs.PATH_SLAB and workload == "rmat20":
        pytest.skip("forcing a power-law graph through the dense 128-row path is covered at 2^11 nodes (test_slab_path_on_a_small_power_law_graph_and_rounding_modes); here it only costs time")
    w = g.WORKLOADS[workload]
    A = w["make"]()
    p = cs.Plan.from_csr(A, path=path)
    for N in Ns:
        B = g.dense_operand(A.K, N, w["b_seed"], w["b_dist"]).numpy()
        ref = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B, A.M, A.K)
        C = run(p, B)
        err = oracle_mod.rel_fro(ref, C)
        assert err <= PATH_TOL[path], (workload, N, err)


@pytest.mark.parametrize("N", [1, 3, 4, 8, 12, 16, 20, 32, 33, 36, 48, 60, 64, 100, 128, 130, 200, 256, 384, 512, 516, 640, 1024])
def test_any_number_of_columns(oracle_mod, N):
    A = g.rmat(9, 8, seed=31, values="uniform")
    B = g.dense_operand(A.K, N, 32).numpy()
    p = cs.Plan.from_csr(A, path=cs.PATH_ROWS, split_nnz=32)
    assert p.info()["num_long_rows"] > 0
    ref = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B, A.M, A.K)
    assert oracle_mod.rel_fro(ref, run(p, B)) <= REL_FRO_TOL_FP32


def test_slab_path_on_a_small_power_law_graph_and_rounding_modes(oracle_mod):
    A = g.rmat(11, 8, seed=33, values="uniform")  # wide 128-row panels, steps split at 256 values
    B = g.dense_operand(A.K, 256, 34).numpy()
    ref = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B, A.M, A.K)
    e_slab = oracle_mod.rel_fro(ref, run(cs.Plan.from_csr(A, path=cs.PATH_SLAB), B))
    e_brick = oracle_mod.rel_fro(ref, run(cs.Plan.from_csr(A, path=cs.PATH_BRICK), B))
    e_round = oracle_mod.rel_fro(ref, run(cs.Plan.from_csr(A, path=cs.PATH_BRICK, round_b_nearest=True), B))
    assert e_round < e_brick <= REL_FRO_TOL and e_slab <= REL_FRO_TOL
    with pytest.raises(cs.CuteSpmmError) as e:  # B never passes a thread on the slab path, so it cannot be re-rounded
        cs.Plan.from_csr(A, path=cs.PATH_SLAB, round_b_nearest=True)
    assert e.value.status == -4


def test_same_sign_operands_keep_the_stated_bound_on_the_tensor_core_paths(oracle_mod):
    """All-positive A and B: the truncation of B to TF32 on the brick and slab paths is one-sided (every product comes
    out low, by up to 2^-10 of its value and 2^-11.5 on average over mantissas), so the errors of a row do not cancel.
    The stated bound (relative Frobenius 1e-3) must hold there too; rounding B to nearest removes the bias."""
    A0 = g.WORKLOADS["elasticity40"]["make"]()
    vals = A0.vals.abs() + 0.25
    B = (g.dense_operand(A0.K, 128, 52).abs() + 0.25).numpy()
    ref = oracle_mod.spmm_csr(A0.row_ptr, A0.cols, vals, B, A0.M, A0.K)
    rp, cols = A0.row_ptr.numpy(), A0.cols.numpy()
    errs = {}
    for name, kw in (("brick", dict(path=cs.PATH_BRICK)), ("slab", dict(path=cs.PATH_SLAB)),
                     ("brick_nearest", dict(path=cs.PATH_BRICK, round_b_nearest=True))):
        errs[name] = oracle_mod.rel_fro(ref, run(cs.Plan(A0.M, A0.K, rp, cols, vals.numpy(), **kw), B))
    print("same-sign operands, relative Frobenius error:", errs)
    assert errs["brick"] <= REL_FRO_TOL and errs["slab"] <= REL_FRO_TOL
    assert 2e-4 <= errs["brick"] <= 6e-4          # the bias itself: about 2^-11.5 = 3.5e-4
    assert errs["brick_nearest"] <= 0.5 * errs["brick"]


@pytest.mark.parametrize("kind", ["rows_with_long_rows", "brick"])
def test_product_captured_in_a_cuda_graph_and_replayed(oracle_mod, kind):
    """cutespmm_spmm allocates nothing and synchronises nothing, so an iterative caller can capture it in a CUDA graph:
    the replays must give the product of whatever B holds at replay time (the long rows' arrival counters are back at
    zero after every launch)."""
    if kind == "brick":
        A = g.stencil9(64, 64)
        plan = cs.Plan.from_csr(A, path=cs.PATH_BRICK)
        tol = REL_FRO_TOL
    else:
        A = g.rmat(11, 8, seed=71, values="uniform")
        plan = cs.Plan.from_csr(A, path=cs.PATH_ROWS)
        assert plan.info()["num_long_rows"] > 0
        tol = REL_FRO_TOL_FP32
    N = 128
    B = g.dense_operand(A.K, N, 72).cuda()
    C = torch.full((A.M, N), float("nan"), device="cuda")
    plan.spmm(B, C)  # first launch outside the capture (kernel attributes, module load)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.spmm(B, C)
    for seed in (73, 74, 75):
        B.copy_(g.dense_operand(A.K, N, seed).cuda())
        C.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        ref = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), A.M, A.K)
        assert oracle_mod.rel_fro(ref, C.cpu().numpy()) <= tol
    assert plan.device_status() == 0


def test_strided_and_misaligned_operands(oracle_mod):
    A = g.uniform_random(300, 200, 5, seed=41)  # M not a multiple of 16
    p = cs.Plan.from_csr(A, path=cs.PATH_ROWS)
    N = 96
    big = g.dense_operand(A.K, N + 7, 42).cuda()
    Bv = big[:, 3 : 3 + N]  # 12-byte offset: not 16-byte aligned, ld = N + 7
    Cbig = torch.full((A.M, N + 5), float("nan"), device="cuda")
    Cv = Cbig[:, 1 : 1 + N]
    p.spmm(Bv, Cv)
    torch.cuda.synchronize()
    ref = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, Bv.cpu().contiguous().numpy(), A.M, A.K)
    assert oracle_mod.rel_fro(ref, Cv.cpu().contiguous().numpy()) <= REL_FRO_TOL_FP32
    assert torch.isnan(Cbig[:, 0]).all() and torch.isnan(Cbig[:, 1 + N :]).all()  # nothing outside the window


def test_empty_rows_panels_and_matrix(oracle_mod):
    # rows 0..63 empty, a dense row, then empties
    M, K, N = 160, 64, 64
    rp = np.zeros(M + 1, np.uint64)
    rp[70:] = 64
    rp[100:] = 65
    cols = np.concatenate([np.arange(64), [5]]).astype(np.uint32)
    vals = np.linspace(-1, 1, 65).astype(np.float32)
    B = g.dense_operand(K, N, 51).numpy()
    ref = oracle_mod.spmm_csr(rp, cols, vals, B, M, K)
    for path in (cs.PATH_ROWS, cs.PATH_AUTO, cs.PATH_BRICK, cs.PATH_SLAB):
        C = run(cs.Plan(M, K, rp, cols, vals, path=path), B)
        assert oracle_mod.rel_fro(ref, C) <= REL_FRO_TOL
        assert not C[:69].any() and not C[100:].any()
    zero = cs.Plan(48, 16, np.zeros(49, np.uint64), np.zeros(0, np.uint32), np.zeros(0, np.float32))
    assert not run(zero, np.ones((16, 32), np.float32)).any()


def test_unsorted_and_duplicate_columns(oracle_mod):
    gd = load_golden("uniform_256_unsorted")
    p = cs.Plan(int(gd["M"]), int(gd["K"]), gd["row_ptr"], gd["cols"], gd["vals"], path=cs.PATH_ROWS)
    assert oracle_mod.rel_fro(gd["C"], run(p, gd["B"])) <= REL_FRO_TOL_FP32
    # duplicates add up, as in spmm_coo
    rp = np.array([0, 3, 3, 4], np.uint64)
    cols = np.array([2, 2, 0, 1], np.uint32)
    vals = np.array([1.0, 2.0, 4.0, 8.0], np.float32)
    B = g.dense_operand(3, 32, 61).numpy()
    ref = oracle_mod.spmm_csr(rp, cols, vals, B, 3, 3)
    for path in (cs.PATH_ROWS, cs.PATH_BRICK, cs.PATH_SLAB):
        assert oracle_mod.rel_fro(ref, run(cs.Plan(3, 3, rp, cols, vals, path=path), B)) <= REL_FRO_TOL


def test_hub_rows_are_deterministic(oracle_mod):
    A = g.rmat(14, 8, seed=71, values="uniform")
    p = cs.Plan.from_csr(A, path=cs.PATH_ROWS, split_nnz=128)
    assert p.info()["num_chunks"] > 100
    B = g.dense_operand(A.K, 128, 72).numpy()
    c1, c2 = run(p, B), run(p, B)
    assert np.array_equal(c1.view(np.uint32), c2.view(np.uint32))  # no atomics: bit-stable run to run
    ref = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B, A.M, A.K)
    assert oracle_mod.rel_fro(ref, c1) <= REL_FRO_TOL_FP32


def test_host_buffer_call(oracle_mod):
    gd = load_golden("elasticity_4")
    p = cs.Plan(int(gd["M"]), int(gd["K"]), gd["row_ptr"], gd["cols"], gd["vals"])
    Bh = torch.from_numpy(gd["B"]).pin_memory()
    C, ms = p.spmm_host(Bh)
    assert ms > 0.0
    assert oracle_mod.rel_fro(gd["C"], C.numpy()) <= REL_FRO_TOL
    C2, _ = p.spmm_host(gd["B"][:, :17].copy())  # narrower N reuses the staging buffers
    assert oracle_mod.rel_fro(gd["C"][:, :17].copy(), C2.numpy()) <= REL_FRO_TOL


@pytest.mark.parametrize("N", [16, 32, 64, 128, 512])
def test_small_job_sizing_cuts_long_rows_finer_and_sums_them_in_the_kernel(oracle_mod, N):
    """A small matrix (a latency-bound job) with a few rows of thousands of nonzeros among short ones: with the sizes
    left to the library the long rows are cut into pieces of about sqrt(length / 2) nonzeros, rows of more than 128
    nonzeros are cut too, and one launch computes everything -- the pieces of a row are added in the kernel by whoever finishes last.
    Repeated launches must give the same bits (the arrival counters return to zero; the sum order is fixed)."""
    rng = np.random.default_rng(5)
    M, K = 3001, 2500
    lens = rng.integers(0, 9, M)
    lens[[7, 1500, 2999]] = [2400, 700, 128]  # 69 / 22 pieces; 128 stays whole
    lens[100:140] = 140                       # just over the cut length: 5 pieces each
    rp = np.zeros(M + 1, np.int64); np.cumsum(lens, out=rp[1:])
    cols = np.concatenate([np.sort(rng.choice(K, int(l), replace=False)) for l in lens]).astype(np.int32)
    vals = rng.standard_normal(cols.size).astype(np.float32)
    p = cs.Plan(M, K, rp, cols, vals, path=cs.PATH_ROWS)
    info = p.info()
    assert info["num_long_rows"] == 42 and info["num_chunks"] == 69 + 22 + 40 * 5
    assert p.launch_count(N) == 1
    B = g.dense_operand(K, N, 77).numpy()
    ref = oracle_mod.spmm_csr(rp, cols, vals, B, M, K)
    C1 = run(p, B)
    assert oracle_mod.rel_fro(ref, C1) <= REL_FRO_TOL_FP32
    for _ in range(3):
        assert np.array_equal(C1, run(p, B))
    # the same matrix with the sizes given: rows up to 256 nonzeros stay whole
    q = cs.Plan(M, K, rp, cols, vals, path=cs.PATH_ROWS, split_nnz=256, tile_nnz=512)
    assert q.info()["num_long_rows"] == 2
    assert oracle_mod.rel_fro(ref, run(q, B)) <= REL_FRO_TOL_FP32


@pytest.mark.parametrize("N,pad,pinned", [(128, 0, True), (256, 0, True), (200, 12, True), (160, 0, False), (40, 8, True)])
def test_host_call_pipelined_in_column_windows(oracle_mod, N, pad, pinned):
    """Operands of 8 MB and more go through the host call in up to four column windows (copy-in,
    product, copy-out overlapped); the result must be the one-piece product for every window
    shape: full windows, a narrow last window, padded leading dimensions, pageable memory."""
    A = g.stencil9(192)  # M = K = 36864: 36864 x 128 x 4 B = 18.9 MB at N = 128 (two windows), 5.9 MB at N = 40 (one piece)
    p = cs.Plan.from_csr(A)
    Bfull = torch.randn(A.K, N + pad)
    Cfull = torch.full((A.M, N + pad), float("nan"))
    if pinned:
        Bfull, Cfull = Bfull.pin_memory(), Cfull.pin_memory()
    Bh, Ch = Bfull[:, :N], Cfull[:, :N]
    _, ms = p.spmm_host(Bh, Ch)
    assert ms > 0.0
    ref = p.spmm(Bh.cuda().contiguous()).cpu()  # device-resident call, one piece (may take another kernel: compare at tolerance)
    assert oracle_mod.rel_fro(ref.numpy(), Ch.contiguous().numpy()) <= REL_FRO_TOL
    if pad:
        assert torch.isnan(Cfull[:, N:]).all()  # nothing written beyond column N
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, Bh.contiguous().numpy(), A.M, A.K)
    assert oracle_mod.rel_fro(want, Ch.contiguous().numpy()) <= REL_FRO_TOL


def test_execution_errors_are_status_codes():
    gd = load_golden("stencil_16x16")
    p = cs.Plan(int(gd["M"]), int(gd["K"]), gd["row_ptr"], gd["cols"], gd["vals"])
    B = torch.zeros(int(gd["K"]), 16, device="cuda")
    assert cs.lib.cutespmm_spmm(p._h, B.data_ptr(), 8, B.data_ptr(), 16, 16, None) == -1  # ldb < N
    assert cs.lib.cutespmm_spmm(p._h, None, 16, B.data_ptr(), 16, 16, None) == -1
    assert cs.lib.cutespmm_spmm(p._h, B.data_ptr() + 2, 16, B.data_ptr(), 16, 16, None) == -1  # misaligned


def test_full_size_properties_without_cpu_product(oracle_mod):
    """At the size where the CPU product takes too long: linearity in B and the column-sum identity
    1^T (A B) = (A^T 1)^T B, both checked on the device in fp64, and a sample of rows (2^16 random rows plus every
    row with more than 4096 nonzeros) against the CPU oracle.  The plan is built from the device-resident CSR."""
    A = g.rmat(22, 8, seed=1005, values="uniform", device="cuda")
    N = 128
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32), A.cols.to(torch.int32), A.vals)
    B1 = g.dense_operand(A.K, N, 81, device="cuda")
    B2 = g.dense_operand(A.K, N, 82, device="cuda")
    C1, C2, C12 = p.spmm(B1), p.spmm(B2), p.spmm(B1 + B2)
    torch.cuda.synchronize()
    num = (C12.double() - C1.double() - C2.double()).norm()
    assert float(num / C12.double().norm()) < 1e-5
    colsum = torch.zeros(A.K, dtype=torch.float64, device="cuda")
    colsum.index_add_(0, A.cols.long(), A.vals.double())
    expect = colsum @ B1.double()
    got = C1.double().sum(0)
    assert float((got - expect).norm() / expect.norm()) < 1e-5
    deg = (A.row_ptr[1:] - A.row_ptr[:-1]).cpu()
    gen = torch.Generator().manual_seed(7)
    which = torch.unique(torch.cat([torch.randint(0, A.M, (1 << 16,), generator=gen), torch.nonzero(deg > 4096).flatten()]))
    want = oracle_mod.spmm_csr_rows(A.row_ptr.cpu(), A.cols.cpu(), A.vals.cpu(), B1.cpu().numpy(), which.numpy())
    assert oracle_mod.rel_fro(want, C1[which.cuda()].cpu().numpy()) <= REL_FRO_TOL_FP32


def test_largest_configuration_at_its_own_size(oracle_mod):
    """The R-MAT graph with 2^24 nodes at N = 128 on one GPU: B and C hold 2^31 elements each, so every element offset
    above 2^31 - 1 needs the kernels' 64-bit address arithmetic (the reference computes these offsets in 32 bits,
    kernel.cu:149,267,281).  Checked: 2^16 random rows plus every row with more than 4096 nonzeros against the CPU
    oracle, and the column-sum identity 1^T (A B) = (A^T 1)^T B in fp64 as the whole-matrix checksum.  The plan is
    built from the device-resident CSR."""
    free, _ = torch.cuda.mem_get_info()
    if free < 60 << 30:
        pytest.skip("needs about 60 GB of free device memory")
    w = g.WORKLOADS["rmat24"]
    A = w["make"](device="cuda")
    N = w["N"]
    assert A.M == 1 << 24 and A.M * N == 1 << 31
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32), A.cols.to(torch.int32), A.vals)
    B = g.dense_operand(A.K, N, w["b_seed"], w["b_dist"], device="cuda")
    C = torch.full((A.M, N), float("nan"), device="cuda")
    p.spmm(B, C)
    torch.cuda.synchronize()
    assert p.device_status() == 0
    # whole-matrix checksum, fp64, in row chunks (no 17 GB temporaries)
    colsum = torch.zeros(A.K, dtype=torch.float64, device="cuda")
    colsum.index_add_(0, A.cols.long(), A.vals.double())
    expect = torch.zeros(N, dtype=torch.float64, device="cuda")
    got = torch.zeros(N, dtype=torch.float64, device="cuda")
    step = 1 << 20
    for r in range(0, A.K, step):
        expect += colsum[r : r + step] @ B[r : r + step].double()
        got += C[r : r + step].sum(0, dtype=torch.float64)
    assert float((got - expect).norm() / expect.norm()) < 1e-5
    # sampled rows against the oracle: random rows over the whole range (high rows: offsets beyond 2^31) + every hub row
    deg = A.row_ptr[1:] - A.row_ptr[:-1]
    gen = torch.Generator().manual_seed(11)
    hubs = torch.nonzero(deg > 4096).flatten().cpu()
    assert hubs.numel() > 100
    rand = torch.unique(torch.cat([torch.randint(0, A.M, (1 << 16,), generator=gen), torch.tensor([A.M - 1])]))
    assert int(rand.max()) * N + N - 1 > 2**31 - 2**20  # the top of the offset range is sampled
    Bh = B.cpu().numpy()
    rp, cols, vals = A.row_ptr.cpu(), A.cols.cpu(), A.vals.cpu()
    for which, tol in ((rand[deg[rand.cuda()].cpu() <= 4096], REL_FRO_TOL_FP32), (hubs, 10 * REL_FRO_TOL_FP32)):
        # hub rows hold up to 3.7e5 nonzeros: the oracle adds them one after the other in fp32, the kernel in chunks of 256,
        # and the two orders differ by the rounding noise of the longer chain -- hence the wider bound for them
        got_rows = C[which.cuda()].cpu().numpy()
        want = oracle_mod.spmm_csr_rows(rp, cols, vals, Bh, which.numpy())
        assert not np.isnan(got_rows).any()
        assert oracle_mod.rel_fro(want, got_rows) <= tol, (which.numel(), tol)


@pytest.mark.parametrize("how", ["cluster", "similar"])
@pytest.mark.parametrize("path", [cs.PATH_ROWS, cs.PATH_BRICK, cs.PATH_AUTO], ids=["rows", "brick", "auto"])
def test_row_clustering_keeps_the_callers_row_order(oracle_mod, path, how):
    """A plan with CUTESPMM_REORDER_CLUSTER_ROWS processes the rows in another order but writes every row of C to its
    own place: the product of a row-shuffled stencil and of a power-law graph (hub rows cut into chunks: the in-launch sum
    writes mapped rows too) must equal the oracle's on the caller's matrix."""
    from test_host import _shuffle_rows

    S, _ = _shuffle_rows(g.stencil9(160))
    for A, N in ((S, 128), (S, 96), (g.rmat(13, 8, seed=5, values="uniform"), 64)):
        p = cs.Plan.from_csr(A, path=path, reorder=how, split_nnz=64)
        B = g.dense_operand(A.K, N, 77).numpy()
        ref = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B, A.M, A.K)
        assert oracle_mod.rel_fro(ref, run(p, B)) <= PATH_TOL[path], (A.name, N)
    if path == cs.PATH_AUTO:  # the point of the option: the shuffled stencil is back on the tensor-core kernel
        assert cs.Plan.from_csr(S, reorder=how).info()["num_bricks"] > 0 and cs.Plan.from_csr(S).info()["num_bricks"] == 0


@pytest.mark.parametrize("N,pad,path", [(128, 0, cs.PATH_AUTO), (200, 8, cs.PATH_AUTO), (64, 0, cs.PATH_ROWS), (256, 0, cs.PATH_BRICK)])
def test_host_call_in_blocks_of_rows_on_banded_matrices(oracle_mod, N, pad, path):
    """On one GPU, operands of many megabytes and a matrix whose rows name an advancing range of columns, the host call
    uploads B in row order, multiplies block of rows by block of rows and returns each block's rows of C while B is
    still arriving.  Every block boundary, both work lists (N = 200 is not a width the brick kernel takes) and padded
    leading dimensions must give the oracle's product; a matrix that does not qualify (a graph whose every block of
    rows names all of B) takes the column-window path and must be right as well."""
    A = g.stencil9(384)  # M = K = 147456: 75 MB at N = 128 -> 9 blocks of rows
    p = cs.Plan.from_csr(A, path=path, split_nnz=256)
    Bfull = g.dense_operand(A.K, N + pad, 91).pin_memory()
    Cfull = torch.full((A.M, N + pad), float("nan")).pin_memory()
    Bh, Ch = Bfull[:, :N], Cfull[:, :N]
    for _ in range(2):  # the second call reuses the cut and the staging
        Ch.fill_(float("nan"))
        _, ms = p.spmm_host(Bh, Ch)
        assert ms > 0.0
        want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, Bh.contiguous().numpy(), A.M, A.K)
        assert oracle_mod.rel_fro(want, Ch.contiguous().numpy()) <= PATH_TOL[path]
    if pad:
        assert torch.isnan(Cfull[:, N:]).all()
    G = g.rmat(16, 16, seed=93, values="uniform")  # hub rows (chunks + fix-up) and no band: column windows
    pg = cs.Plan.from_csr(G)
    Bg = g.dense_operand(G.K, 128, 94).pin_memory()
    Cg, _ = pg.spmm_host(Bg)
    want = oracle_mod.spmm_csr(G.row_ptr, G.cols, G.vals, Bg.numpy(), G.M, G.K)
    assert oracle_mod.rel_fro(want, Cg.numpy()) <= REL_FRO_TOL_FP32 * 5
    # a banded matrix with long rows inside the band: the chunk and fix-up lists are cut by blocks too
    rows, K2 = 1 << 16, 1 << 16
    lens = np.full(rows, 6, dtype=np.int64)
    lens[::997] = 700
    rp = np.zeros(rows + 1, dtype=np.int64)
    np.cumsum(lens, out=rp[1:])
    r_of = np.repeat(np.arange(rows), lens)
    cols = np.clip(r_of + (np.arange(rp[-1]) - rp[r_of]) - 3, 0, K2 - 1)
    vals = np.linspace(-1.0, 1.0, rp[-1]).astype(np.float32)
    pb = cs.Plan(rows, K2, rp, cols.astype(np.uint32), vals)
    assert pb.info()["num_long_rows"] > 0
    Bb = g.dense_operand(K2, 128, 95).pin_memory()
    Cb, _ = pb.spmm_host(Bb)
    want = oracle_mod.spmm_csr(rp.astype(np.uint64), cols.astype(np.uint32), vals, Bb.numpy(), rows, K2)
    assert oracle_mod.rel_fro(want, Cb.numpy()) <= REL_FRO_TOL


@pytest.mark.parametrize("N", [1, 3, 13, 17, 30, 33, 47, 63, 65, 127, 129, 131, 255, 257, 301, 511, 515])
@pytest.mark.parametrize("hub", [0, 3000])
def test_widths_that_no_vector_divides_on_jobs_worth_a_padded_copy(oracle_mod, N, hub):
    """N not a multiple of four columns: small jobs read B column by column, jobs that name a row of B often enough copy it
    into aligned rows first (both sides of the rule here); C is written column by column up to N; hub rows are summed
    from pieces.  Views with a gap between the rows and operands off the 16-byte grid take the same ways."""
    K = 300
    for M, per_row in ((500, 4), (20000, 40)):
        ln = np.full(M, per_row)
        ln[3], ln[4] = max(hub, per_row), 0
        rng = np.random.default_rng(N)
        rp = np.concatenate([[0], np.cumsum(ln)])
        A = g.CsrMatrix(M, K, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, K, rp[-1]).astype(np.int32)),
                        torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
        p = cs.Plan.from_device_csr(M, K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
        B = g.dense_operand(K, N, 71)
        want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), M, K)
        out = torch.full((M + 1, N), float("nan"), device="cuda")
        p.spmm(B.cuda(), out[:M])
        assert oracle_mod.rel_fro(want, out[:M].cpu().numpy()) <= 2e-6
        assert torch.isnan(out[M]).all()  # nothing behind the last row
        big, cbig = torch.zeros((K, N + 3), device="cuda"), torch.full((M, N + 5), 7.0, device="cuda")
        big[:, 1:N + 1] = B.cuda()
        p.spmm(big[:, 1:N + 1], cbig[:, 2:N + 2])
        assert oracle_mod.rel_fro(want, cbig[:, 2:N + 2].cpu().numpy()) <= 2e-6
        assert (cbig[:, :2] == 7).all() and (cbig[:, N + 2:] == 7).all()  # nothing between the rows
        assert p.device_status() == 0


@pytest.mark.parametrize("N", [16, 30, 64, 128, 160])
def test_tiles_dealt_by_a_counter(oracle_mod, N):
    """A matrix with long rows and at least eight tiles per block has its tiles dealt as they are finished; the counters are
    back at zero after every launch, and a plan whose long rows come from few chunks shares them between lane groups."""
    rng = np.random.default_rng(5)
    ln = rng.integers(0, 6, 900_000)
    ln[[0, 400_000, 899_999]] = (5000, 300, 2000)
    rp = np.concatenate([[0], np.cumsum(ln)])
    A = g.CsrMatrix(ln.size, 5000, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, 5000, rp[-1]).astype(np.int32)),
                    torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
    assert p.info()["num_tiles"] >= 8 * 888 and p.info()["num_long_rows"] == 3
    B = g.dense_operand(A.K, N, 6)
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, A.K)
    Bd = B.cuda()
    first = p.spmm(Bd)
    assert oracle_mod.rel_fro(want, first.cpu().numpy()) <= 2e-6
    for _ in range(3):
        assert torch.equal(p.spmm(Bd), first)
    assert p.device_status() == 0


@pytest.mark.parametrize("N", [4, 16, 17, 32, 47, 64, 100, 128, 130, 256, 515])
@pytest.mark.parametrize("run", [2, 3])
def test_rows_in_runs_of_the_same_columns(oracle_mod, run, N):
    """Runs of two and three rows with the same columns share their loads: tiles that cut a run (tile sizes no run divides),
    runs of empty rows, lengths around a step's eight columns; one row that differs sends the matrix back to the row kernel."""
    rng = np.random.default_rng(10 * N + run)
    nodes, K = 10000, 300  # more runs than a block per SM has lane groups at every width
    ln = rng.integers(0, 20, nodes)
    ln[[0, 7, 8, nodes - 1]] = (1, 0, 0, 9)
    rows = [np.sort(rng.choice(K, n, replace=False)) for n in ln]
    rp = np.concatenate([[0], np.cumsum(np.repeat(ln, run))])
    cols = np.concatenate([c for c in rows for _ in range(run)]).astype(np.int32)
    vals = torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32))
    B = g.dense_operand(K, N, 81)
    for cut in (0, 64):
        for differ in (False, True):
            c = cols.copy()
            if differ:  # the last row of a long run names another last column
                at = int(rp[run * int(np.argmax(ln)) + run]) - 1
                c[at] = K - 1 if c[at] < K - 1 else 0
            A = g.CsrMatrix(nodes * run, K, torch.from_numpy(rp), torch.from_numpy(c), vals)
            want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, K)
            for p in (cs.Plan.from_device_csr(A.M, K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS, tile_nnz=cut),
                      cs.Plan.from_csr(A, path=cs.PATH_ROWS, tile_nnz=cut)):
                out = torch.full((A.M + 1, N), float("nan"), device="cuda")
                p.spmm(B.cuda(), out[:A.M])
                assert oracle_mod.rel_fro(want, out[:A.M].cpu().numpy()) <= 2e-6
                assert torch.isnan(out[A.M]).all() and p.device_status() == 0


@pytest.mark.parametrize("shape", ["few", "short", "long", "chunks", "band"])
@pytest.mark.parametrize("N", [1, 8, 9, 16, 17, 24, 31, 32, 33, 34, 63, 64, 65, 127, 129, 250, 257, 509])
def test_operands_off_the_16_byte_grid(oracle_mod, shape, N):
    """One form of the row kernel per width, alignment (4 or 8 bytes) and kind of matrix: few rows, short rows, long rows, rows cut
    into chunks, neighbouring rows with the same columns.  B and C are views into wider arrays, so nothing beside C's columns may
    be written; the aligned form's result is the same sum (chunks: in another order)."""
    rng = np.random.default_rng(N)
    M, K = {"few": (300, 700), "band": (96 * 96, 96 * 96)}.get(shape, (24001, 997))
    if shape == "band":
        A = g.stencil9(96, 96, 5)
    else:
        ln = rng.integers(0, 13, M) if shape != "long" else rng.integers(20, 40, M)
        if shape == "chunks":
            ln[rng.integers(0, M, 40)] = rng.integers(100, 2500, 40)
        rp = np.concatenate([[0], np.cumsum(ln)])
        A = g.CsrMatrix(M, K, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, K, rp[-1]).astype(np.int32)), torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
    plan = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), **({"min_brick_panels": 1} if shape == "band" else {"path": cs.PATH_ROWS}))
    B = g.dense_operand(A.K, N, 6)
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, A.K)
    for shift, wide in ((1, N + 2 + N % 2), (2, N + 4 + N % 2)):  # 4- and 8-byte aligned rows
        Bd = torch.full((A.K, wide), float("nan"), device="cuda")
        Cd = torch.full((A.M, wide), float("nan"), device="cuda")
        Bd[:, shift:shift + N] = B.cuda()
        plan.spmm(Bd[:, shift:shift + N], Cd[:, shift:shift + N])
        got = Cd[:, shift:shift + N].cpu().numpy()
        assert oracle_mod.rel_fro(want, got) <= REL_FRO_TOL_FP32  # two fp32 sums in (almost) the same order
        assert torch.isnan(Cd[:, :shift]).all() and torch.isnan(Cd[:, shift + N:]).all() and plan.device_status() == 0


@pytest.fixture(scope="module")
def many_tiles():
    """Tiles enough to be dealt by a counter, a few rows cut into chunks, and rows of every length around those a warp shares: a fifth
    of the nonzeros in rows of more than twice the mean, a dozen and more per row."""
    rng = np.random.default_rng(17)
    M, K = 330000, 20000
    ln = rng.integers(0, 26, M)
    ln[rng.choice(M, 8000, replace=False)] = rng.integers(33, 257, 8000)
    ln[:9] = (15, 16, 17, 18, 31, 32, 33, 255, 256)
    ln[5000:5003] = (257, 600, 1500)
    assert ln.mean() >= 12 and ln[(ln > max(32, 2 * ln.mean())) & (ln <= 256)].sum() > ln.sum() / 8
    rp = np.concatenate([[0], np.cumsum(ln)])
    A = g.CsrMatrix(M, K, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, K, rp[-1]).astype(np.int32)), torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
    p = cs.Plan.from_device_csr(M, K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
    assert p.info()["num_chunks"] and p.info()["num_tiles"] >= 8 * 6 * torch.cuda.get_device_properties(0).multi_processor_count
    return A, p


@pytest.mark.parametrize("N", [5, 8, 16, 27, 32, 47, 64, 81])
def test_rows_that_the_groups_of_a_warp_share(oracle_mod, many_tiles, N):
    """Long rows of a tile in narrow products of large matrices, aligned, off the 16-byte grid and after a padded copy of B."""
    A, p = many_tiles
    B = g.dense_operand(A.K, N, 8)
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, A.K)
    Bd = B.cuda()
    first = p.spmm(Bd)
    assert oracle_mod.rel_fro(want, first.cpu().numpy()) <= REL_FRO_TOL_FP32
    for _ in range(3):  # whoever takes a row, its sum is the same
        assert torch.equal(p.spmm(Bd), first)
    assert p.device_status() == 0


@pytest.mark.parametrize("shift", [1, 2])  # rows on the 4- and the 8-byte grid
@pytest.mark.parametrize("N", [7, 13, 20, 34, 50, 66, 130, 300, 301])
def test_dealt_tiles_off_the_16_byte_grid(oracle_mod, many_tiles, N, shift):
    """Every form that reads one or two columns per load, with the tiles dealt by a counter; nothing beside the columns is touched."""
    A, p = many_tiles
    wide = N + 4 + N % 2
    B = g.dense_operand(A.K, N, 9)
    Bd, Cd = torch.full((A.K, wide), float("nan"), device="cuda"), torch.full((A.M, wide), float("nan"), device="cuda")
    Bd[:, shift:shift + N] = B.cuda()
    p.spmm(Bd[:, shift:shift + N], Cd[:, shift:shift + N])
    first = Cd[:, shift:shift + N].clone()
    rows = np.concatenate([np.arange(40), np.arange(4990, 5010), np.arange(A.M // 2, A.M // 2 + 2000), np.arange(A.M - 40, A.M)])
    want = oracle_mod.spmm_csr_rows(A.row_ptr, A.cols, A.vals, B.numpy(), rows)
    assert oracle_mod.rel_fro(want, first[torch.from_numpy(rows).cuda()].cpu().numpy()) <= REL_FRO_TOL_FP32
    assert torch.isfinite(first).all() and torch.isnan(Cd[:, :shift]).all() and torch.isnan(Cd[:, shift + N:]).all()
    Cd.fill_(float("nan"))
    p.spmm(Bd[:, shift:shift + N], Cd[:, shift:shift + N])
    assert torch.equal(Cd[:, shift:shift + N], first) and p.device_status() == 0


@pytest.mark.parametrize("N", [13, 32])
def test_rows_that_the_groups_share_of_a_reordered_plan(oracle_mod, many_tiles, N):
    """The sums of shared rows go through the row map to the caller's rows."""
    A, _ = many_tiles
    p = cs.Plan.from_csr(A, path=cs.PATH_ROWS, reorder="similar")
    assert p.info()["num_tiles"] >= 8 * 6 * torch.cuda.get_device_properties(0).multi_processor_count
    B = g.dense_operand(A.K, N, 10)
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, A.K)
    assert oracle_mod.rel_fro(want, p.spmm(B.cuda()).cpu().numpy()) <= REL_FRO_TOL_FP32
    assert p.device_status() == 0


def _rows_of(ln, K, seed):
    """A matrix of given row lengths, and its CSR arrays on the GPU."""
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(ln)])
    A = g.CsrMatrix(len(ln), K, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, K, rp[-1]).astype(np.int32)), torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
    return A, (A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda())


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


@pytest.mark.parametrize("made", ["device", "host", "file"])
@pytest.mark.parametrize("M, per_row, N", [(60_000, 32, 47), (400_000, 4, 63)])
def test_a_long_row_leaves_the_others_their_kernel(oracle_mod, tmp_path, made, M, per_row, N):
    """Rows off the 16-byte grid: one long row among even ones costs its own pieces (1.1 and 1.25 times the time; 1.9 times where it
    decides which kernel all rows take), whoever made the plan."""
    times = []
    for hub in (False, True):
        ln = np.full(M, per_row)
        if hub:
            ln[M // 3] = 1000
        A, csr = _rows_of(ln, M, 21)
        p = cs.Plan.from_device_csr(M, M, *csr) if made == "device" else cs.Plan.from_csr(A)
        if made == "file":
            p.save(str(tmp_path / "plan"))
            p = cs.Plan.load(str(tmp_path / "plan"))
        B, C = g.dense_operand(M, N, 22, device="cuda"), torch.empty((M, N), device="cuda")
        p.spmm(B, C)
        if hub:
            rows = np.concatenate([np.arange(5), np.arange(M // 3 - 2, M // 3 + 3), np.arange(M - 5, M)])
            want = oracle_mod.spmm_csr_rows(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), rows)
            assert oracle_mod.rel_fro(want, C[torch.from_numpy(rows).cuda()].cpu().numpy()) <= REL_FRO_TOL_FP32
        times.append(_best_us(lambda: p.spmm(B, C)))
        assert p.device_status() == 0
    assert times[1] <= 1.5 * times[0], times


@pytest.mark.parametrize("N", [16, 32, 64])
def test_a_long_row_leaves_short_rows_their_claims(oracle_mod, N):
    """Tiles enough to be dealt by a counter: rows of four are claimed as fast with one long row among them (1.0 to 1.14 times the
    time; 1.09 to 1.22 times in the kernels whose groups share rows, which short rows do not use)."""
    M, K, times = 2_000_000, 100_000, []
    for hub in (False, True):
        ln = np.full(M, 4)
        if hub:
            ln[M // 3] = 3000
        A, csr = _rows_of(ln, K, 23)
        p = cs.Plan.from_device_csr(M, K, *csr, path=cs.PATH_ROWS)
        B, C = g.dense_operand(K, N, 24, device="cuda"), torch.empty((M, N), device="cuda")
        p.spmm(B, C)
        rows = np.concatenate([np.arange(5), np.arange(M // 3 - 2, M // 3 + 3), np.arange(M - 5, M)])
        want = oracle_mod.spmm_csr_rows(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), rows)
        assert oracle_mod.rel_fro(want, C[torch.from_numpy(rows).cuda()].cpu().numpy()) <= REL_FRO_TOL_FP32
        times.append(_best_us(lambda: p.spmm(B, C)))
        assert p.device_status() == 0
    assert times[1] <= {16: 1.18, 32: 1.17, 64: 1.04}[N] * times[0], times


@pytest.mark.parametrize("N", [128, 129, 132, 256, 260, 388, 509])
def test_wide_products_of_rows_in_runs_walk_a_tile_once_per_slab(oracle_mod, N):
    """Five waves of tiles: slabs of equal width, one after the other over each tile; the last one may be narrower."""
    A = g.elasticity3d(32, 3, 9)
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
    B = g.dense_operand(A.K, N, 7)
    out = torch.full((A.M + 1, N), float("nan"), device="cuda")
    p.spmm(B.cuda(), out[:A.M])
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, A.K)
    assert oracle_mod.rel_fro(want, out[:A.M].cpu().numpy()) <= REL_FRO_TOL_FP32
    assert torch.isnan(out[A.M]).all() and p.device_status() == 0


@pytest.mark.parametrize("N", [129, 132, 256, 260, 384, 388, 509, 512])
@pytest.mark.parametrize("n", [13, 21])
def test_wide_products_of_rows_in_runs_with_the_slabs_in_the_grid(oracle_mod, n, N):
    """Fewer than four waves of tiles, less than one and one and a half: a block takes every few tiles of one slab."""
    A = g.elasticity3d(n, 3, 9)
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
    B = g.dense_operand(A.K, N, 7)
    out = torch.full((A.M + 1, N), float("nan"), device="cuda")
    p.spmm(B.cuda(), out[:A.M])
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, A.K)
    assert oracle_mod.rel_fro(want, out[:A.M].cpu().numpy()) <= REL_FRO_TOL_FP32
    assert torch.isnan(out[A.M]).all() and p.device_status() == 0


@pytest.mark.parametrize("N", [256, 512])
def test_slabs_of_rows_in_runs_fill_the_machine(N):
    """1.1 and 1.5 waves of tiles: in blocks that walk whole tiles both are two rounds per slab, and the larger matrix takes 1.03 and 1.01
    times as long per row at 256 and 512 columns; with the slabs in the grid 0.85 and 0.93."""
    times = []
    for n in (19, 21):
        A = g.elasticity3d(n, 3, 9)
        p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
        B, C = g.dense_operand(A.K, N, 7, device="cuda"), torch.empty((A.M, N), device="cuda")
        times.append(_best_us(lambda: p.spmm(B, C)) / A.M)
    assert times[1] <= 0.97 * times[0], times


@pytest.mark.parametrize("make, launches", [
    (lambda: g.uniform_random(2000, 340000, 700, seed=3), 4),  # windows of 384 and 25 columns, a padded copy for each
    (lambda: g.elasticity3d(48, 3, 9), 1),                     # rows in runs: read as they are, whole
])
def test_wide_unaligned_products_of_large_matrices(oracle_mod, make, launches):
    """Columns of B that a padded copy of 512 MiB would not hold (543 and 556 MB)."""
    A = make()
    N = 409
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.to(torch.int32).cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
    assert p.launch_count(N) == launches
    B = torch.randn((A.K, N), generator=torch.Generator("cuda").manual_seed(3), device="cuda")
    C = p.spmm(B)
    for cols in (slice(0, 8), slice(380, 388), slice(401, 409)):  # both sides of the window's edge
        want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B[:, cols].contiguous().cpu().numpy(), A.M, A.K)
        assert oracle_mod.rel_fro(want, C[:, cols].cpu().numpy()) <= 2e-6
    assert p.device_status() == 0


@pytest.mark.parametrize("N", [32, 64, 96, 128, 160, 192, 224, 256, 288, 320, 352, 480, 512, 608])
@pytest.mark.parametrize("make", [lambda: g.stencil9(100), lambda: g.elasticity3d(14, 3, 5)])
def test_brick_spans(oracle_mod, make, N):
    """Every composition of 128-, 96- and 64-column spans, on path brick and on path auto (whose widths up to 64 run by rows)."""
    A = make()
    B = g.dense_operand(A.K, N, 91)
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.numpy(), A.M, A.K)
    for kw in (dict(path=cs.PATH_BRICK), dict(round_b_nearest=True)):
        p = cs.Plan.from_csr(A, **kw)
        out = torch.full((A.M + 1, N), float("nan"), device="cuda")
        p.spmm(B.cuda(), out[:A.M])
        assert oracle_mod.rel_fro(want, out[:A.M].cpu().numpy()) <= 1e-3
        assert torch.isnan(out[A.M]).all() and p.device_status() == 0
    assert cs.Plan.from_csr(A, path=cs.PATH_BRICK).launch_count(N) == {160: 2, 224: 2, 288: 2, 320: 2, 352: 2, 480: 2, 608: 2}.get(N, 1)


def test_product_waits_for_nothing_without_memory_for_a_padded_copy(oracle_mod):
    """Rows of B off the 16-byte grid are read through a padded copy where there is memory for it.  Where there is none
    the product reads B as it is; it does not wait for the stream to find some, nor fail."""
    rng = np.random.default_rng(11)
    M, K, N, per_row = 20000, 330000, 301, 160  # a copy of 401 MB
    A = g.CsrMatrix(M, K, torch.arange(0, M * per_row + 1, per_row), torch.from_numpy(rng.integers(0, K, M * per_row).astype(np.int32)),
                    torch.from_numpy(rng.standard_normal(M * per_row).astype(np.float32)))
    csr = A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda()
    p = cs.Plan.from_device_csr(M, K, *csr, path=cs.PATH_ROWS)
    assert p.launch_count(N) == 2  # the copy and the product
    B = torch.randn((K, N), generator=torch.Generator("cuda").manual_seed(12), device="cuda")
    few = cs.Plan.from_device_csr(64, K, csr[0][:65], csr[1][:64 * per_row], csr[2][:64 * per_row], path=cs.PATH_ROWS)
    assert few.launch_count(N) == 1
    few.spmm(B)  # not worth a copy: the kernel that reads B as it is has been loaded
    C, want = torch.full((M, N), float("nan"), device="cuda"), p.spmm(B)
    stalled = torch.cuda.Event()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert cs.lib.cutespmm_release_memory() == 0  # what the pool keeps
    before = torch.cuda.mem_get_info()[0]
    hog = torch.empty(before - (256 << 20), dtype=torch.uint8, device="cuda")
    try:
        torch.cuda._sleep(2_000_000_000)  # a second
        stalled.record()
        p.spmm(B, C)
        assert not stalled.query()  # the call came back while the stream was still busy
        torch.cuda.synchronize()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert oracle_mod.rel_fro(want.cpu().numpy(), C.cpu().numpy()) <= REL_FRO_TOL_FP32
    rows = np.concatenate([np.arange(5), np.arange(M - 5, M)])
    ref = oracle_mod.spmm_csr_rows(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), rows)
    assert oracle_mod.rel_fro(ref, C[torch.from_numpy(rows).cuda()].cpu().numpy()) <= REL_FRO_TOL_FP32
    assert p.device_status() == 0


@pytest.mark.parametrize("kind", ["tiles_dealt", "two_lists"])
def test_products_after_overlapping_ones_are_whole(oracle_mod, kind):
    """Products of a plan with long rows that overlap on two streams are undefined, but what they leave behind is not: the
    counters of arrived chunks and of dealt tiles are back at zero, whatever the widths (grids, column slabs, work lists)."""
    rng = np.random.default_rng(15)
    if kind == "tiles_dealt":
        ln = rng.integers(0, 6, 900_000)
        ln[rng.choice(ln.size, 300, replace=False)] = 900
        rp = np.concatenate([[0], np.cumsum(ln)])
        A = g.CsrMatrix(ln.size, 5000, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, 5000, rp[-1]).astype(np.int32)),
                        torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
        kw, widths, tol = dict(path=cs.PATH_ROWS), (32, 300), REL_FRO_TOL_FP32
    else:  # brick panels beside long rows: N = 128 runs the rows the bricks leave, N = 33 every row
        S = g.stencil9(120)
        rows = [S.cols[S.row_ptr[r] : S.row_ptr[r + 1]].numpy() for r in range(S.M)]
        for r in range(40, S.M, 997):
            rows[r] = np.sort(rng.choice(S.K, 400 + r % 300, replace=False))
        rp = np.concatenate([[0], np.cumsum([len(c) for c in rows])])
        A = g.CsrMatrix(S.M, S.K, torch.from_numpy(rp), torch.from_numpy(np.concatenate(rows).astype(np.int32)),
                        torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
        kw, widths, tol = dict(), (128, 33), REL_FRO_TOL
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), **kw)
    assert p.info()["num_long_rows"] > 0 and (kind == "tiles_dealt") == (p.info()["num_bricks"] == 0)
    Bs = [g.dense_operand(A.K, N, 16, device="cuda") for N in widths]
    Cs = [torch.empty((A.M, N), device="cuda") for N in widths]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(20):
        for B, C, s in zip(Bs, Cs, streams):
            p.spmm(B, C, stream=s)
    torch.cuda.synchronize()
    for B, C in zip(Bs, Cs):
        want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), A.M, A.K)
        for _ in range(2):
            C.fill_(float("nan"))
            p.spmm(B, C)
            assert oracle_mod.rel_fro(want, C.cpu().numpy()) <= tol
    assert p.device_status() == 0


@pytest.mark.parametrize("call", ["spmm", "sddmm", "set_values", "noalloc", "operator"])
def test_calls_leave_the_interpreter_to_other_threads(call):
    """A call whose stream's queue is full waits in the driver until the GPU has made room.  It waits without the interpreter
    lock: another thread goes on all the while."""
    import threading
    import time

    from cutespmm_ae_b200 import torch_ops

    A = g.uniform_random(64, 48, 4, seed=17)
    csr = A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda()
    plan = cs.Plan.from_device_csr(A.M, A.K, *csr, path=cs.PATH_ROWS)
    op = torch_ops.SparseOperator(plan)
    B, C, out = torch.randn(A.K, 32, device="cuda"), torch.randn(A.M, 32, device="cuda"), torch.empty(A.nnz, device="cuda")
    run = {"spmm": lambda: plan.spmm(B, C), "sddmm": lambda: plan.sddmm(C, B, out), "set_values": lambda: plan.set_values(csr[2]),
           "noalloc": lambda: cs.spmm_csr_noalloc(A.M, A.K, *csr, B, C), "operator": lambda: op(B)}[call]
    run()
    torch.cuda.synchronize()
    stream, times = torch.cuda.Stream(), []

    def fill():
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_000_000_000)  # half a second of GPU time
            for _ in range(4000):  # more launches than a queue holds
                t = time.perf_counter()
                run()
                times.append(time.perf_counter() - t)

    worker = threading.Thread(target=fill)
    longest, last = 0.0, time.perf_counter()
    worker.start()
    while worker.is_alive():
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
        time.sleep(0.001)
    torch.cuda.synchronize()
    assert max(times) > 0.2  # the queue did fill up
    assert longest < 0.5 * max(times), (longest, max(times))  # all of it where the lock is held, a few milliseconds where not
    op.close()


def test_first_product_on_another_stream_sees_a_finished_plan(oracle_mod):
    """A plan made on the host is complete when the call returns, for streams too that do not wait for the default one."""
    A = g.rmat(11, 8, seed=18, values="uniform")
    B = g.dense_operand(A.K, 64, 19, device="cuda")
    want = oracle_mod.spmm_csr(A.row_ptr, A.cols, A.vals, B.cpu().numpy(), A.M, A.K)
    side, C = torch.cuda.Stream(), torch.empty((A.M, 64), device="cuda")  # a stream of torch's does not wait for the default stream
    torch.cuda.synchronize()
    for _ in range(10):
        p = cs.Plan.from_csr(A, path=cs.PATH_ROWS)
        p.spmm(B, C, stream=side)
        side.synchronize()
        assert oracle_mod.rel_fro(want, C.cpu().numpy()) <= REL_FRO_TOL_FP32
