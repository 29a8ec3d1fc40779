"""cutespmm_sddmm against the CPU oracle: one dot product of feature rows per stored nonzero, in the plan's
storage order; every plan flavour, any N, strided operands, hub rows, and its use as the gradient of the product
with respect to the values of A."""
import numpy as np
import pytest
import torch

import cutespmm_ae_b200 as cs
from cutespmm_ae_b200 import generators as g

pytestmark = pytest.mark.gpu
TOL = 2e-6  # fp32 dot products, another summation order than the oracle's


def rel(ref, got):
    ref, got = ref.astype(np.float64), got.astype(np.float64)
    return float(np.linalg.norm(got - ref) / max(np.linalg.norm(ref), 1e-30))


@pytest.mark.parametrize("N", [128, 64, 100, 200, 7, 512])
@pytest.mark.parametrize("scale", [False, True])
def test_sddmm_matches_oracle_for_any_width(oracle_mod, N, scale):
    A = g.rmat(11, 8, seed=51, values="uniform")  # hub rows: the chunked part of the work list
    p = cs.Plan.from_csr(A, split_nnz=64)
    assert p.info()["num_long_rows"] > 0
    X = g.dense_operand(A.M, N, 52, device="cuda")
    Y = g.dense_operand(A.K, N, 53, device="cuda")
    out = torch.full((A.nnz,), float("nan"), device="cuda")
    p.sddmm(X, Y, out, scale_by_values=scale)
    torch.cuda.synchronize()
    want = oracle_mod.sddmm_csr(A.row_ptr, A.cols, A.vals if scale else None, X.cpu().numpy(), Y.cpu().numpy())
    assert rel(want, out.cpu().numpy()) <= TOL


@pytest.mark.parametrize("N", [16, 17, 32, 33, 64, 65, 96, 97, 130])
@pytest.mark.parametrize("shift", [0, 1])
def test_sddmm_where_rows_end_inside_a_run_of_nonzeros(oracle_mod, N, shift):
    """A warp takes 32 nonzeros, a group of lanes eight (four) of them: rows that end in front of, on and behind those borders,
    empty rows between them, a tile whose last claim is one nonzero; aligned operands and operands off the 16-byte grid."""
    lengths = [1, 7, 8, 9, 0, 0, 3, 4, 5, 31, 32, 33, 0, 1, 1, 1, 1, 2, 63, 64, 65, 0, 129, 255, 257, 1]
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.int64), torch.cumsum(torch.tensor(lengths * 3), 0)])
    M, nnz, K = len(lengths) * 3, int(row_ptr[-1]), 301
    cols = torch.arange(nnz, dtype=torch.int64).mul(97).remainder(K).to(torch.int32)
    vals = g.dense_operand(nnz, 1, 71).flatten()
    p = cs.Plan.from_device_csr(M, K, row_ptr.to(torch.int32).cuda(), cols.cuda(), vals.cuda(), path=cs.PATH_ROWS)
    X, Y = g.dense_operand(M, N + shift, 72).cuda()[:, shift:], g.dense_operand(K, N + shift, 73).cuda()[:, shift:]
    out = torch.full((nnz + 1,), float("nan"), device="cuda")  # nothing is written behind the last nonzero
    p.sddmm(X, Y, out[:nnz], scale_by_values=True)
    want = oracle_mod.sddmm_csr(row_ptr, cols, vals, X.cpu().contiguous().numpy(), Y.cpu().contiguous().numpy())
    # two fp32 sums of N <= 130 products in different orders
    assert rel(want, out[:nnz].cpu().numpy()) <= TOL and torch.isnan(out[nnz])


@pytest.mark.parametrize("made", ["device", "host", "file"])
@pytest.mark.parametrize("N", [16, 33, 64])
def test_sddmm_of_a_matrix_of_mostly_empty_rows(oracle_mod, tmp_path, made, N):
    """Twelve nonzeros in every fourth row: three per row on the average, but X is kept along a row."""
    M, K = 8000, 500
    ln = np.where(np.arange(M) % 4 == 1, 12, 0)
    rp = torch.from_numpy(np.concatenate([[0], np.cumsum(ln)]))
    rng = np.random.default_rng(N)
    cols = np.sort(np.argsort(rng.random((M // 4, K)), axis=1)[:, :12], axis=1).astype(np.int32).ravel()  # ascending, as a host plan stores them
    A = g.CsrMatrix(M, K, rp, torch.from_numpy(cols), torch.from_numpy(rng.standard_normal(int(rp[-1])).astype(np.float32)))
    p = cs.Plan.from_device_csr(M, K, rp.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS) if made == "device" else cs.Plan.from_csr(A, path=cs.PATH_ROWS)
    if made == "file":
        p.save(str(tmp_path / "plan"))
        p = cs.Plan.load(str(tmp_path / "plan"))
    X, Y = g.dense_operand(M, N, 81, device="cuda"), g.dense_operand(K, N, 82, device="cuda")
    want = oracle_mod.sddmm_csr(A.row_ptr, A.cols, A.vals, X.cpu().numpy(), Y.cpu().numpy())
    assert rel(want, p.sddmm(X, Y, scale_by_values=True).cpu().numpy()) <= TOL


@pytest.mark.parametrize("N", [7, 16, 20, 32, 33, 64, 100])
def test_sddmm_of_rows_of_few_nonzeros(oracle_mod, N):
    """Fewer than four nonzeros per row: a row of X is loaded for each; long rows among them, empty ones and a last claim of one."""
    rng = np.random.default_rng(N)
    ln = rng.integers(0, 5, 4000)
    ln[[3, 700]] = (300, 33)
    rp = np.concatenate([[0], np.cumsum(ln)])
    M, K, nnz = 4000, 900, int(rp[-1])
    cols, vals = torch.from_numpy(rng.integers(0, K, nnz).astype(np.int32)), g.dense_operand(nnz, 1, 74).flatten()
    p = cs.Plan.from_device_csr(M, K, torch.from_numpy(rp.astype(np.int32)).cuda(), cols.cuda(), vals.cuda(), path=cs.PATH_ROWS)
    X, Y = g.dense_operand(M, N, 75), g.dense_operand(K, N, 76)
    out = torch.full((nnz + 1,), float("nan"), device="cuda")
    p.sddmm(X.cuda(), Y.cuda(), out[:nnz], scale_by_values=True)
    want = oracle_mod.sddmm_csr(rp, cols, vals, X.numpy(), Y.numpy())
    assert rel(want, out[:nnz].cpu().numpy()) <= TOL and torch.isnan(out[nnz])


@pytest.mark.parametrize("make,path", [(lambda: g.stencil9(64), cs.PATH_AUTO), (lambda: g.elasticity3d(8, 3, 4), cs.PATH_BRICK),
                                        (lambda: g.uniform_random(300, 200, 5, seed=41), cs.PATH_ROWS)])
def test_sddmm_on_every_plan_flavour_and_strided_operands(oracle_mod, make, path):
    A = make()
    N = 96
    Xbig, Ybig = g.dense_operand(A.M, N + 5, 54).cuda(), g.dense_operand(A.K, N + 3, 55).cuda()
    X, Y = Xbig[:, 1 : 1 + N], Ybig[:, 3 : 3 + N]  # not 16-byte aligned, padded leading dimensions
    want = oracle_mod.sddmm_csr(A.row_ptr, A.cols, A.vals, X.cpu().contiguous().numpy(), Y.cpu().contiguous().numpy())
    host = cs.Plan.from_csr(A, path=path)
    dev = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=path)
    for plan in (host, dev):
        out = plan.sddmm(X, Y, scale_by_values=True)
        torch.cuda.synchronize()
        assert rel(want, out.cpu().numpy()) <= TOL


def test_sddmm_is_the_gradient_of_the_product_with_respect_to_the_values(oracle_mod):
    """C = A B  =>  dL/dA_j = <dL/dC[row of j], B[column of j]>: check against a finite difference of the oracle."""
    A = g.uniform_random(64, 48, 4, seed=61)
    N = 32
    B = g.dense_operand(A.K, N, 62)
    G = g.dense_operand(A.M, N, 63)  # dL/dC for L = sum(G * C)
    p = cs.Plan.from_csr(A)
    grad = p.sddmm(G.cuda(), B.cuda()).cpu().numpy()
    rows = np.repeat(np.arange(A.M), np.diff(A.row_ptr.numpy()))
    expect = (G.numpy()[rows].astype(np.float64) * B.numpy()[A.cols.numpy()].astype(np.float64)).sum(1)
    assert rel(expect, grad) <= TOL
    j = 17  # one entry by finite difference through the oracle's product
    vals = A.vals.numpy().astype(np.float32).copy()
    loss = lambda v: float((G.numpy().astype(np.float64) * oracle_mod.spmm_csr(A.row_ptr, A.cols, v, B.numpy(), A.M, A.K)).sum())  # noqa: E731
    vp, vm = vals.copy(), vals.copy()
    vp[j] += 0.25
    vm[j] -= 0.25
    assert abs((loss(vp) - loss(vm)) / 0.5 - grad[j]) <= 1e-3 * max(1.0, abs(grad[j]))


def test_sddmm_refusals_and_empty_cases():
    A = g.stencil9(16)
    p = cs.Plan.from_csr(A, reorder="cluster", path=cs.PATH_ROWS)
    X = torch.zeros(A.M, 8, device="cuda")
    if p.info()["nnz"]:
        S, _ = __import__("test_host")._shuffle_rows(A)
        ps = cs.Plan.from_csr(S, reorder="cluster")
        with pytest.raises(cs.CuteSpmmError) as e:
            ps.sddmm(X, X)
        assert e.value.status == -4
    with pytest.raises(ValueError):
        cs.Plan.from_csr(A).sddmm(X, torch.zeros(A.K, 9, device="cuda"))
    empty = cs.Plan(32, 16, np.zeros(33, np.uint64), np.zeros(0, np.uint32), np.zeros(0, np.float32))
    assert empty.sddmm(torch.zeros(32, 8, device="cuda"), torch.zeros(16, 8, device="cuda")).numel() == 0


@pytest.mark.parametrize("builder", ["host", "device"])
def test_set_values_makes_edge_scores_the_weights_of_the_next_product(oracle_mod, builder, tmp_path):
    """The attention step of a graph layer: scores = sddmm(X, Y), any elementwise normalisation, set_values(scores), then
    the product aggregates with those weights.  The pattern and the work lists stay; decode and save see the new values."""
    A = g.rmat(11, 8, seed=81, values="uniform")  # hub rows: chunks whose pieces are summed in the launch
    if builder == "host":
        p = cs.Plan.from_csr(A, path=cs.PATH_ROWS)
    else:
        p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.to(torch.int32).cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
    assert p.info()["num_long_rows"] > 0
    X, Y = g.dense_operand(A.M, 64, 82, device="cuda"), g.dense_operand(A.K, 64, 83, device="cuda")
    w = torch.tanh(p.sddmm(X, Y) / 8.0)
    p.set_values(w)
    rp, cc, vv = p.decode_csr()  # the plan's storage order, with the new values
    assert np.array_equal(vv, w.cpu().numpy())
    B = g.dense_operand(A.K, 128, 84)
    C = torch.full((A.M, 128), float("nan"), device="cuda")
    p.spmm(B.cuda(), C)
    torch.cuda.synchronize()
    ref = oracle_mod.spmm_csr(rp, cc, vv, B.numpy(), A.M, A.K)
    assert oracle_mod.rel_fro(ref, C.cpu().numpy()) <= TOL
    # a second replacement, and the saved plan carries what the device holds
    p.set_values(-w)
    f = tmp_path / "weighted.plan"
    p.save(f)
    q = cs.Plan.load(f)
    C2 = torch.empty_like(C)
    q.spmm(B.cuda(), C2)
    torch.cuda.synchronize()
    assert oracle_mod.rel_fro(-ref, C2.cpu().numpy()) <= TOL
    assert np.array_equal(q.decode_csr()[2], -vv)


def test_set_values_is_refused_where_the_values_live_in_tensor_core_records_or_rows_are_reordered():
    S = g.stencil9(64)
    for kw in (dict(path=cs.PATH_BRICK), dict(path=cs.PATH_ROWS, reorder="cluster")):
        p = cs.Plan.from_csr(S, **kw)
        with pytest.raises(cs.CuteSpmmError) as e:
            p.set_values(torch.ones(S.nnz, device="cuda"))
        assert e.value.status == -4
    p = cs.Plan.from_csr(S, path=cs.PATH_ROWS)
    with pytest.raises(ValueError):
        p.set_values(torch.ones(S.nnz + 1, device="cuda"))


@pytest.mark.parametrize("N", [1, 3, 4, 15, 16, 17, 28, 32, 33, 60, 64, 65, 68, 96, 97, 124, 128, 132, 256])
@pytest.mark.parametrize("per_row", [3, 21])
def test_sddmm_at_the_edges_of_every_span(oracle_mod, N, per_row):
    """Spans of 16, 32, 64, 96 and 128 columns, whole and ragged, aligned and not; rows short enough for the flat form and
    long enough for a warp per row; a hub row beside them and tiles whose last claim is a part of 32 nonzeros."""
    ln = np.full(230, per_row)
    ln[7], ln[100:110] = 400, 0
    rng = np.random.default_rng(N)
    rp = np.concatenate([[0], np.cumsum(ln)])
    A = g.CsrMatrix(230, 500, torch.from_numpy(rp), torch.from_numpy(rng.integers(0, 500, rp[-1]).astype(np.int32)),
                    torch.from_numpy(rng.standard_normal(rp[-1]).astype(np.float32)))
    p = cs.Plan.from_device_csr(A.M, A.K, A.row_ptr.to(torch.int32).cuda(), A.cols.cuda(), A.vals.cuda(), path=cs.PATH_ROWS)
    X, Y = g.dense_operand(A.M, N, 62, device="cuda"), g.dense_operand(A.K, N, 63, device="cuda")
    out = torch.full((A.nnz,), float("nan"), device="cuda")
    p.sddmm(X, Y, out, scale_by_values=True)
    want = oracle_mod.sddmm_csr(A.row_ptr, A.cols, A.vals, X.cpu().numpy(), Y.cpu().numpy())
    assert rel(want, out.cpu().numpy()) <= TOL and p.device_status() == 0
