"""Column-per-CTA triangular solves and the data-flow ILU(0) against the CPU oracle, at the sizes
where their layouts change: one row, warp and chunk remainders, long rows that span several parts
of a level, the last row count kept for the column solves and the first one past it, both factor
types, blocks solved in place and blocks that overlap."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O
from conftest import spd_from

pytestmark = pytest.mark.gpu

FP64_ROWS = 24_767   # 227 KB - 1 KB less two 16 KB chunks, 8 bytes a row and 65 more


@pytest.fixture(scope="module")
def bpf():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import blockpowerflow_b200 as bpf

    return bpf


def _random(n, per_row, seed):
    """Diagonally dominant, about per_row off-diagonal entries a row."""
    rng = np.random.default_rng(seed)
    k = per_row * n
    A = sp.coo_matrix((rng.standard_normal(k), (rng.integers(0, n, k), rng.integers(0, n, k))), shape=(n, n)).tocsr()
    A = A - sp.diags(A.diagonal())
    return (A + sp.diags(1.0 + np.asarray(abs(A).sum(axis=1)).ravel())).tocsr()


def _arrow(n):
    """Dense first and last rows and columns: rows of n entries, single-row levels."""
    A = sp.lil_matrix((n, n))
    A.setdiag(4.0 * n)
    A[0, :] = A[n - 1, :] = 1.0
    A[:, 0] = A[:, n - 1] = 1.0
    A.setdiag(4.0 * n)
    return A.tocsr()


def _block(X):
    import torch

    return torch.as_tensor(np.asfortranarray(X), device="cuda").t().contiguous().t()


@pytest.mark.parametrize("dtype,rtol", [("float64", 1e-12), ("float32", 1e-4)])
@pytest.mark.parametrize("n,per_row,p", [(1, 0, 1), (2, 1, 3), (31, 3, 2), (32, 3, 1), (33, 3, 5), (700, 40, 3),
                                         (5000, 4, 17)])
def test_ilu0_column_solve_sizes(bpf, n, per_row, p, dtype, rtol):
    A = _random(n, per_row, n)
    P = bpf.ilu0(bpf.CuSparseMatrixCSR.from_scipy(A), p, dtype)
    F = O.ilu0(A)
    np.testing.assert_allclose(P.P.nzVal.cpu().numpy(), F.data, rtol=1e-11, atol=1e-11 * np.abs(F.data).max())
    X = np.random.default_rng(1).standard_normal((n, p))
    Y = P.ldiv(_block(X)).cpu().numpy()
    ref = O.prec_apply(1, F, X)
    assert np.linalg.norm(Y - ref) <= rtol * np.linalg.norm(ref)


@pytest.mark.parametrize("dtype,rtol", [("float64", 1e-12), ("float32", 1e-4)])
@pytest.mark.parametrize("n", [200, 1500])
def test_long_rows_span_several_parts(bpf, n, dtype, rtol):
    A = _arrow(n)
    P = bpf.ilu0(bpf.CuSparseMatrixCSR.from_scipy(A), 2, dtype)
    X = np.random.default_rng(2).standard_normal((n, 2))
    ref = O.prec_apply(1, O.ilu0(A), X)
    Y = P.ldiv(_block(X)).cpu().numpy()
    assert np.linalg.norm(Y - ref) <= rtol * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [FP64_ROWS, FP64_ROWS + 1])
def test_last_row_count_of_the_column_solve(bpf, n):
    A = _random(n, 3, 7)
    for p in (1, 20):
        P = bpf.ilu0(bpf.CuSparseMatrixCSR.from_scipy(A), p)
        X = np.random.default_rng(3).standard_normal((n, p))
        ref = O.prec_apply(1, O.ilu0(A), X)
        Y = P.ldiv(_block(X)).cpu().numpy()
        assert np.linalg.norm(Y - ref) <= 1e-12 * np.linalg.norm(ref)


def test_ic0_column_solve(bpf, case300):
    A, _ = case300
    S = spd_from(A)
    for dtype, rtol in (("float64", 1e-12), ("float32", 1e-4)):
        P = bpf.ic0(bpf.CuSparseMatrixCSR.from_scipy(S), 6, dtype)
        X = np.random.default_rng(4).standard_normal((S.shape[0], 6))
        ref = O.prec_apply(2, O.ic0(S), X)
        Y = P.ldiv(_block(X)).cpu().numpy()
        assert np.linalg.norm(Y - ref) <= rtol * np.linalg.norm(ref)


@pytest.mark.parametrize("ordering", ["natural", "AMD", "RCM"])
def test_in_place_and_overlapping_blocks(bpf, ordering):
    A = bpf.grid.synthetic_jacobian(200)
    n = A.shape[0]
    P = bpf.ilu0(bpf.CuSparseMatrixCSR.from_scipy(A), 4, ordering=ordering)
    X = np.random.default_rng(5).standard_normal((n, 5))
    ref = P.ldiv(_block(X)).cpu().numpy()
    W = _block(X)
    bpf.ldiv_(W, P, W)
    np.testing.assert_array_equal(W.cpu().numpy(), ref)
    W = _block(X)
    bpf.ldiv_(W[:, 1:], P, W[:, :4])   # the output is the input shifted by a column
    np.testing.assert_array_equal(W[:, 1:].cpu().numpy(), ref[:, :4])
    W = _block(np.vstack([X, X]))
    bpf.ldiv_(W[3:n + 3, :], P, W[:n, :])   # and by three rows
    np.testing.assert_array_equal(W[3:n + 3, :].cpu().numpy(), ref)


def test_zero_pivot_is_reported_and_the_next_factorization_runs(bpf):
    pat = _random(300, 3, 9)
    Ad = bpf.CuSparseMatrixCSR.from_scipy(pat)
    P = bpf.ilu0(Ad, 1)
    vals = Ad.nzVal.clone()
    vals[pat.indptr[17]:pat.indptr[18]] = 0.0   # a zero row keeps its pivot zero
    with pytest.raises(bpf.SingularException):
        P.refactor(vals)
    P.refactor(Ad.nzVal)
    np.testing.assert_allclose(P.P.nzVal.cpu().numpy(), O.ilu0(pat).data, rtol=1e-11)


@pytest.mark.parametrize("n", [500, 3072, 3073])
@pytest.mark.parametrize("p", [2, 17])
@pytest.mark.parametrize("f32", [False, True])
def test_row_major_blocks(bpf, n, p, f32):
    """Inside a solver the blocks are row-major: in place up to 3,072 rows, through copies beyond.  A solve whose
    blocks came back wrong could not reach the bound: 1.01 covers the estimate's rounding."""
    import torch

    A = _random(n, 3, n + p)
    B = np.random.default_rng(p).standard_normal((n, p))
    Ad = bpf.CuSparseMatrixCSR.from_scipy(A)
    N = bpf.ilu0(Ad, p, factor_dtype="float32") if f32 else bpf.ilu0(Ad, p)
    X, st = bpf.block_gmres(Ad, torch.as_tensor(B, device="cuda"), N=N, ldiv=True, memory=40, atol=0.0, rtol=1e-8)
    assert st.solved
    assert np.linalg.norm(B - A @ X.cpu().numpy()) <= 1.01e-8 * np.linalg.norm(B)


def test_long_rows_in_levels_of_their_own(bpf):
    """Levels of one row of 160 entries: over the lanes of a warp they take 15 MB (in slabs of 32 rows 307), the lists
    of the factorization 618."""
    import torch

    n, w, p = 6000, 160, 3
    A = sp.csr_matrix(sp.diags([np.full(n - d, 0.5 / w) for d in range(w + 1)], [-d for d in range(w + 1)]) + 2.0 * sp.eye(n))
    Ad = bpf.CuSparseMatrixCSR.from_scipy(A)
    X = np.random.default_rng(6).standard_normal((n, p))
    B = _block(X)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    P = bpf.ilu0(Ad, p)
    used = free - torch.cuda.mem_get_info()[0]
    ref = O.prec_apply(1, O.ilu0(A), X)
    Y = P.ldiv(B).cpu().numpy()
    assert np.linalg.norm(Y - ref) <= 1e-12 * np.linalg.norm(ref)
    assert used < 700 << 20


def test_a_stream_past_its_limit_is_not_kept(bpf):
    """A dense lower triangle of 7,600 rows: 292 MB."""
    n, p = 7600, 3
    ptr = np.concatenate([[0], np.cumsum(np.arange(1, n + 1))])
    col = np.concatenate([np.arange(i + 1) for i in range(n)])
    val = np.full(len(col), 0.5 / n)
    val[ptr[1:] - 1] = 2.0
    A = sp.csr_matrix((val, col, ptr), shape=(n, n))
    P = bpf.ilu0(bpf.CuSparseMatrixCSR.from_scipy(A), p)
    X = np.random.default_rng(6).standard_normal((n, p))
    ref = O.prec_apply(1, O.ilu0(A), X)
    Y = P.ldiv(_block(X)).cpu().numpy()
    assert np.linalg.norm(Y - ref) <= 1e-12 * np.linalg.norm(ref)


# rows over the lanes of a warp: in one part, in several (more than 1,536 entries of FP64, 2,688 of FP32), several rows in
# a level, and levels with too many long rows for it; the bound is test_both_ways_of_one_factor's
@pytest.mark.parametrize("dtype,eps", [("float64", 2.0**-52), ("float32", 2.0**-23)])
@pytest.mark.parametrize("kind", ["arrow", "few", "many"])
def test_rows_over_a_warp(bpf, kind, dtype, eps):
    if kind == "arrow":
        A = _arrow(4000)
    else:
        A = sp.csr_matrix(_random(1200, 3, 11))
        rows = np.arange(600, 600 + (7 if kind == "few" else 90))
        extra = sp.coo_matrix((np.full(len(rows) * 200, 1e-2), (np.repeat(rows, 200), np.tile(np.arange(0, 400, 2), len(rows)))),
                              shape=A.shape)
        A = sp.csr_matrix(A + extra + extra.T + 20.0 * sp.eye(1200))
    A.sort_indices()
    n = A.shape[0]
    P = bpf.ilu0(bpf.CuSparseMatrixCSR.from_scipy(A), 4, dtype)
    F = sp.csr_matrix((P.P.nzVal.cpu().numpy(), A.indices, A.indptr), shape=A.shape)
    L, U = sp.tril(F, -1, format="csr") + sp.eye(n, format="csr"), sp.triu(F, format="csr")
    c = 4 * (np.diff(A.indptr).max() + 4) * eps
    X = np.random.default_rng(4).standard_normal((n, 4))
    for p in (1, 4):
        Y = P.ldiv(_block(X[:, :p])).cpu().numpy()
        assert np.all(np.abs(X[:, :p] - L @ (U @ Y)) <= c * (abs(L) @ (abs(U) @ np.abs(Y))))


def test_update_lists_past_their_limit(bpf):
    """Rows of 162 entries with 159 updates each: lists would take 622 MB, pairs 8."""
    import torch

    n, w = 6000, 160
    A = sp.csr_matrix(sp.diags([np.full(n - d, 0.5 / w) for d in range(w + 1)] + [np.full(n - 1, 0.1)],
                               [-d for d in range(w + 1)] + [1]) + 2.0 * sp.eye(n))
    Ad = bpf.CuSparseMatrixCSR.from_scipy(A)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    P = bpf.ilu0(Ad, 1)
    used = free - torch.cuda.mem_get_info()[0]
    F = O.ilu0(A)
    np.testing.assert_allclose(P.P.nzVal.cpu().numpy(), F.data, rtol=1e-12)
    P.refactor(2.0 * Ad.nzVal)
    at = np.flatnonzero(A.indices == np.repeat(np.arange(n), np.diff(A.indptr)))   # the diagonal
    np.testing.assert_allclose(P.P.nzVal.cpu().numpy()[at], 2.0 * F.data[at], rtol=1e-12)
    assert used < 200 << 20


def test_factors_by_lists_and_by_pairs_agree(bpf):
    """Short rows beside one of 300 entries (which takes all update pairs along), and rows of up to 64 by lists alone."""
    for per_row, long in ((4, 300), (20, 0)):
        A = _random(2000, per_row, per_row).tolil()
        if long:
            A[1500, :long] = 1e-3
        A = A.tocsr()
        A.sort_indices()
        P = bpf.ilu0(bpf.CuSparseMatrixCSR.from_scipy(A), 1)
        F = O.ilu0(A)
        np.testing.assert_allclose(P.P.nzVal.cpu().numpy(), F.data, rtol=1e-11, atol=1e-11 * np.abs(F.data).max())


def test_too_many_update_pairs_are_refused(bpf):
    """387 dense blocks of 256 rows: 387 x 5,559,680 pairs exceed 2^31 - 1."""
    import torch

    m, nb = 256, 387
    n = m * nb
    ptr = torch.arange(0, n * m + 1, m, dtype=torch.int32, device="cuda")
    col = (torch.arange(m, dtype=torch.int32, device="cuda").repeat(n).view(nb, m * m)
           + m * torch.arange(nb, dtype=torch.int32, device="cuda")[:, None]).reshape(-1)
    A = bpf.CuSparseMatrixCSR(ptr, col, torch.ones(n * m, dtype=torch.float64, device="cuda"), n)
    with pytest.raises(bpf.BPFError, match="2\\^31"):
        bpf.ilu0(A, 1)


def _wide_levels(n, per_row):
    """Four levels of n / 4 rows, each reading (and read by) random rows of its neighbours."""
    rng = np.random.default_rng(n)
    h = n // 4
    r = np.repeat(np.arange(h, 4 * h), per_row)
    c = rng.integers(0, h, len(r)) + (r // h - 1) * h
    A = sp.coo_matrix((rng.standard_normal(2 * len(r)), (np.concatenate([r, c]), np.concatenate([c, r]))), shape=(n, n)).tocsr()
    return (A + sp.diags(1.0 + np.asarray(abs(A).sum(axis=1)).ravel())).tocsr()


# one factor whose solves take either way by their number of columns: both kinds of storage, before and after new
# values, in place, overlapping, and inside a solver.  A substitution's computed y solves a system whose entries are
# off by at most k eps each (k: the longest row, a reciprocal and the roundings of values and results come on top), so
# |X - L U Y| <= 2 (k + 4) eps |L| |U| |Y|; the residual's own rounding is another 2 k eps of the same.
@pytest.mark.parametrize("dtype,eps", [("float64", 2.0**-52), ("float32", 2.0**-23)])
@pytest.mark.parametrize("case", ["grid natural", "grid AMD", "wide natural", "wide RCM"])
def test_both_ways_of_one_factor(bpf, case, dtype, eps):
    import torch

    kind, ordering = case.split()
    A = bpf.grid.synthetic_jacobian(12500) if kind == "grid" else _wide_levels(8000, 40)
    n = A.shape[0]
    Ad = bpf.CuSparseMatrixCSR.from_scipy(A)
    P = bpf.ilu0(Ad, 200, dtype, ordering=ordering)
    perm = P.perm
    S = sp.csr_matrix(A[perm][:, perm])
    S.sort_indices()

    def check(X, Y):
        F = sp.csr_matrix((P.P.nzVal.cpu().numpy(), S.indices, S.indptr), shape=S.shape)
        L, U = sp.tril(F, -1, format="csr") + sp.eye(n, format="csr"), sp.triu(F, format="csr")
        c = 4 * (np.diff(S.indptr).max() + 4) * eps
        Y = Y.cpu().numpy()[perm]
        assert np.all(np.abs(X[perm] - L @ (U @ Y)) <= c * (abs(L) @ (abs(U) @ np.abs(Y))))

    X = np.random.default_rng(7).standard_normal((n, 200))
    for scale in (1.0, 4.0):
        P.refactor(scale * Ad.nzVal)
        for p in (1, 5, 16, 17, 64, 65, 128, 129, 200):
            check(X[:, :p], P.ldiv(_block(X[:, :p])))
    P.refactor(Ad.nzVal)
    for p in (3, 40):
        W = _block(X[:, :p])
        bpf.ldiv_(W, P, W)
        check(X[:, :p], W)
        W = _block(X[:, :p + 1])
        bpf.ldiv_(W[:, 1:], P, W[:, :p])
        check(X[:, :p], W[:, 1:])
    B = np.random.default_rng(8).standard_normal((n, 20))
    for p in (3, 20):
        Z, st = bpf.block_gmres(Ad, torch.as_tensor(B[:, :p], device="cuda"), N=P, ldiv=True, memory=250, atol=0.0, rtol=1e-8)
        assert st.solved and np.linalg.norm(B[:, :p] - A @ Z.cpu().numpy()) <= 1.01e-8 * np.linalg.norm(B[:, :p])
