"""The RF refactorization's sparse front and dense tail against SciPy's sparse LU: all-dense patterns
around the 64-column tile, fronts of every row length, the last system the column solves take and the
first that goes by row sweeps (each width class of those), distinct replicas, pivots that vanish in
the front and in the tail, and a right-hand side with a NaN column beside finite ones."""
import contextlib

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bpf():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import blockpowerflow_b200 as bpf

    return bpf


def _block(X):
    """X as a column-major device block (strides 1 and n for one row as well)."""
    import torch

    out = torch.empty((X.shape[1], X.shape[0]), dtype=torch.float64, device="cuda").t()
    out.copy_(torch.as_tensor(np.ascontiguousarray(X), device="cuda"))
    return out


def _dominant(n, per_row, seed):
    rng = np.random.default_rng(seed)
    k = per_row * n
    A = sp.coo_matrix((rng.standard_normal(k), (rng.integers(0, n, k), rng.integers(0, n, k))), shape=(n, n)).tocsr()
    A = A - sp.diags(A.diagonal())
    return (A + sp.diags(1.0 + np.asarray(abs(A).sum(axis=1)).ravel())).tocsr()


def _check(bpf, A, widths, ordering="AMD", tol=1e-10):
    """Analyse A, refactor with other values on its pattern, solve blocks of the given widths."""
    import torch

    RF = bpf.CUSOLVERRF
    rng = np.random.default_rng(A.shape[0])
    gA = bpf.CuSparseMatrixCSR.from_scipy(A)
    rf = RF.CusolverRfLU(gA, ordering=ordering)
    A2 = A.copy()
    A2.data = A.data * (1.0 + 0.05 * rng.standard_normal(A.nnz))
    gA.nzVal.copy_(torch.as_tensor(A2.data, device="cuda"))
    RF.update_(rf, gA)
    lu = spl.splu(A2.tocsc())
    for p in widths:
        B = rng.standard_normal((A.shape[0], p))
        X = _block(B)
        RF.ldiv_(rf, X)
        Xd = lu.solve(B)
        assert np.linalg.norm(X.cpu().numpy() - Xd) <= tol * np.linalg.norm(Xd), p
    return rf, gA


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 128, 200])
def test_dense_patterns_around_the_tile(bpf, n):
    A = sp.csr_matrix(np.random.default_rng(n).standard_normal((n, n)) + 2.0 * n * np.eye(n))
    _check(bpf, A, (1, 3), "NATURAL")


@pytest.mark.parametrize("n,per_row", [(700, 1), (700, 3), (1500, 6), (3000, 2)])
def test_fronts_of_short_and_long_rows(bpf, n, per_row):
    _check(bpf, _dominant(n, per_row, n + per_row), (1, 33))


@pytest.mark.parametrize("n", [24_767, 24_768])
def test_last_system_of_the_column_solves(bpf, n):
    """A chain of meshes: short levels at any size."""
    rng = np.random.default_rng(5)
    i = np.arange(n - 1)
    far = rng.integers(0, n - 40, 600)
    r = np.concatenate([i, i + 1, far, far + 37])
    c = np.concatenate([i + 1, i, far + 37, far])
    A = sp.coo_matrix((rng.standard_normal(len(r)), (r, c)), shape=(n, n)).tocsr()
    A = (A + sp.diags(1.0 + np.asarray(abs(A).sum(axis=1)).ravel())).tocsr()
    _check(bpf, A, (1, 5))


def test_row_sweeps_of_every_width(bpf):
    _check(bpf, bpf.grid.synthetic_jacobian(14000), (1, 2, 4, 8, 9, 32, 33, 64, 65, 200, 300))


@pytest.mark.parametrize("buses", [300, 14000])
def test_distinct_replicas(bpf, buses):
    import torch

    RF = bpf.CUSOLVERRF
    A = bpf.grid.synthetic_jacobian(buses)
    gA = bpf.CuSparseMatrixCSR.from_scipy(A)
    rf = RF.CusolverRfLUBatch(gA, 3)
    RF.rf_batch_refactor_(rf, torch.stack([s * gA.nzVal for s in (1.0, 2.0, -4.0)], dim=1))
    b = np.random.default_rng(0).standard_normal(A.shape[0])
    X = _block(np.stack([b] * 3, axis=1))
    RF.ldiv_(rf, X)
    x = spl.splu(A.tocsc()).solve(b)
    for r, s in enumerate((1.0, 2.0, -4.0)):
        assert np.linalg.norm(X[:, r].cpu().numpy() * s - x) <= 1e-9 * np.linalg.norm(x)


@pytest.mark.parametrize("row", [0, 599])
def test_vanishing_pivot_is_singular_and_the_next_refactor_runs(bpf, row):
    """Row 0 is eliminated in the front, row 599 in the tail (natural order)."""
    A = _dominant(600, 2, 3)
    A = sp.csr_matrix(A + sp.eye(600))
    rf, gA = _check(bpf, A, (1,), "NATURAL")
    good = gA.nzVal.clone()
    gA.nzVal[int(A.indptr[row]):int(A.indptr[row + 1])] = 0.0
    with pytest.raises(bpf.SingularException):
        bpf.CUSOLVERRF.update_(rf, gA)
    gA.nzVal.copy_(good)
    bpf.CUSOLVERRF.update_(rf, gA)


@pytest.mark.parametrize("buses", [300, 14000])
def test_nan_column_leaves_the_others_alone(bpf, buses):
    A = bpf.grid.synthetic_jacobian(buses)
    RF = bpf.CUSOLVERRF
    rf = RF.CusolverRfLU(bpf.CuSparseMatrixCSR.from_scipy(A))
    B = np.random.default_rng(1).standard_normal((A.shape[0], 40))
    ref = _block(B)
    RF.ldiv_(rf, ref)
    B[7, 3] = np.nan
    X = _block(B)
    RF.ldiv_(rf, X)
    keep = [c for c in range(40) if c != 3]
    np.testing.assert_array_equal(X[:, keep].cpu().numpy(), ref[:, keep].cpu().numpy())
    assert np.isnan(X[:, 3].cpu().numpy()).any()


# tails of two to nine tiles: the last one partly, or wholly, rows of the matrix
@pytest.mark.parametrize("n", [65, 100, 128, 180, 240, 500])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("at", [0, -1])
def test_a_refactorization_with_a_nan_leaves_the_next_one_alone(bpf, n, bad, at):
    A = sp.csr_matrix(np.random.default_rng(n).standard_normal((n, n)) + 2.0 * n * np.eye(n))
    rf, gA = _check(bpf, A, (1,), "NATURAL")
    good = gA.nzVal.clone()
    B = np.random.default_rng(1).standard_normal((n, 3))
    before = _block(B)
    bpf.CUSOLVERRF.ldiv_(rf, before)
    gA.nzVal[at] = bad
    with contextlib.suppress(bpf.SingularException):
        bpf.CUSOLVERRF.update_(rf, gA)
    gA.nzVal.copy_(good)
    bpf.CUSOLVERRF.update_(rf, gA)
    X = _block(B)
    bpf.CUSOLVERRF.ldiv_(rf, X)
    np.testing.assert_array_equal(X.cpu().numpy(), before.cpu().numpy())


def _growing(kind, n):
    """(L, U) of triangles whose inverses grow like 1.4^n within a tile: ones on the diagonal, -0.4 beside it."""
    K = np.eye(n)
    for b in range(0, n, 64):
        e = min(n, b + 64)
        K[b:e, b:e] -= 0.4 * np.triu(np.ones((e - b, e - b)), 1)
    if kind == "upper":
        return np.eye(n), K
    if kind == "lower":
        return K.T.copy(), np.eye(n)
    C = np.random.default_rng(n).standard_normal((n, n)) / n   # tiles below the diagonal ones
    for b in range(0, n, 64):
        C[b:b + 64, b:] = 0.0
    if kind == "rows":        # U grows: the panels of L
        return np.eye(n) + C, K
    return K.T.copy(), np.eye(n) + C.T   # L grows: the panels of U


# Substitution computes factors and solutions with |A - L U| <= n eps |L| |U| and |B - L U X| <= 2 n eps |L| |U| |X|,
# whatever the condition; the factors of A differ from L and U by at most 64 eps 1.4^64 < 1e-4; another n eps for
# the residual and n eps for A's rounding.  Products with inverted triangles miss it by 1.4^64.
@pytest.mark.parametrize("kind", ["upper", "lower", "rows", "columns"])
@pytest.mark.parametrize("n,before", [(64, 0), (65, 0), (130, 0), (200, 0), (200, 25_000)])
def test_tails_that_grow(bpf, kind, n, before):
    """before: rows of a diagonal ahead of the dense block (so many that the solves go by rows)."""
    import torch

    RF = bpf.CUSOLVERRF
    L, U = _growing(kind, n)
    safe = np.random.default_rng(1).standard_normal((n, n)) + 2.0 * n * np.eye(n)   # the analysis keeps the order
    D = sp.identity(before, format="csr")
    gA = bpf.CuSparseMatrixCSR.from_scipy(sp.csr_matrix(sp.block_diag([D, sp.csr_matrix(safe)])))
    rf = RF.CusolverRfLU(gA, ordering="NATURAL")
    A = L @ U
    gA.nzVal[before:] = torch.as_tensor(A.reshape(-1), device="cuda")
    RF.update_(rf, gA)
    rng = np.random.default_rng(n)
    for p in (1, 5, 17):
        Xt = rng.standard_normal((n, p))
        B = A @ Xt
        X = _block(np.vstack([np.ones((before, p)), B]))
        RF.ldiv_(rf, X)
        X = X.cpu().numpy()[before:]
        bound = 6 * n * 2.0**-52 * ((np.abs(L) + 1e-4) @ ((np.abs(U) + 1e-4) @ np.abs(X)))
        assert np.all(np.abs(B - A @ X) <= bound), p
