"""block_gmres with the orthogonalization in one launch, at the edges of its tiles and groups.

The basis is checked through what it must give: the CPU oracle's iteration count, and a solution whose
true residual ||B - A X|| agrees with the solver's own estimate.  The estimate is exact in exact
arithmetic; with an orthonormal basis to a few eps the two differ by k eps kappa ||B||, far below the
tolerance of 1e-2 of the stopping bound at rtol 1e-8.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bpf():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import blockpowerflow_b200 as bpf

    return bpf


def _solve(bpf, A, B, **kw):
    import torch

    Ad = bpf.CuSparseMatrixCSR.from_scipy(A)
    N = bpf.ilu0(Ad, B.shape[1])
    X, st = bpf.block_gmres(Ad, torch.as_tensor(B, device="cuda"), N=N, ldiv=True, atol=0.0, rtol=1e-8,
                            history=True, **kw)
    return X.cpu().numpy(), st


# column counts at the edges of the 8-wide tiles; rows: a short last slab, one slab, and more
# rows than SMs x 16 (slabs of 24 rows); other kernels from 65 columns
@pytest.mark.parametrize("nbus,p", [(20, 1), (40, 7), (300, 8), (300, 9), (300, 16), (301, 17), (300, 24),
                                    (300, 25), (300, 31), (300, 32), (300, 33), (1400, 5), (1700, 32), (300, 34), (300, 48), (301, 50), (300, 64), (1700, 64), (300, 66),
                                    (300, 47), (300, 63)])
def test_edges(bpf, nbus, p):
    A = bpf.grid.synthetic_jacobian(nbus, seed=nbus)
    B = np.random.default_rng(p).standard_normal((A.shape[0], p))
    X, st = _solve(bpf, A, B, memory=60)
    _, so = O.block_gmres(A, B, N=(1, O.ilu0(A)), memory=60, atol=0.0, rtol=1e-8, history=True)
    assert st.solved and abs(st.niter - so.niter) <= 1
    nb = np.linalg.norm(B)
    assert abs(np.linalg.norm(B - A @ X) - st.residuals[-1]) <= 1e-2 * 1e-8 * nb


def test_more_blocks_than_a_group(bpf):
    """80 blocks of 32 columns: products go in groups of 64 blocks.  Unpreconditioned and not converged:
    estimate and true residual differ by rounding, at most 10 k eps ||A|| ||X|| + 10 k eps ||B||."""
    import torch

    A = bpf.grid.synthetic_jacobian(1700, seed=3)
    p, k = 32, 80
    B = np.random.default_rng(3).standard_normal((A.shape[0], p))
    X, st = bpf.block_gmres(bpf.CuSparseMatrixCSR.from_scipy(A), torch.as_tensor(B, device="cuda"), memory=k, itmax=k,
                            atol=0.0, rtol=1e-14, history=True)
    X = X.cpu().numpy()
    assert st.niter == k
    bound = 10 * k * 2.0**-52 * (np.sqrt((A.multiply(A)).sum()) * np.linalg.norm(X) + np.linalg.norm(B))
    assert abs(np.linalg.norm(B - A @ X) - st.residuals[-1]) <= bound
    assert bound < 0.1 * st.residuals[-1]


@pytest.mark.parametrize("p", [12, 32, 48, 64])
def test_ill_conditioned_blocks(bpf, p):
    """The identity's columns make numerically rank-deficient blocks: shift, third pass, re-orthogonalization.  The
    estimate and the true residual then agree to the stopping bound (a basis that lost orthogonality would not)."""
    A = bpf.grid.preset_jacobian("case300", 0)
    B = np.eye(A.shape[0], p)
    X, st = _solve(bpf, A, B, memory=60)
    assert st.solved
    assert abs(np.linalg.norm(B - A @ X) - st.residuals[-1]) <= 1e-2 * 1e-8 * np.linalg.norm(B)


@pytest.mark.parametrize("p", [3, 8, 15, 24, 31, 32, 40, 45, 48, 61, 64])
def test_tall_slabs(bpf, p):
    """Slabs of 72 rows (nine row tiles, the last slab short): coefficients through shared memory."""
    A = bpf.grid.synthetic_jacobian(5200, seed=7)
    B = np.random.default_rng(p).standard_normal((A.shape[0], p))
    X, st = _solve(bpf, A, B, memory=300)
    assert st.solved
    assert abs(np.linalg.norm(B - A @ X) - st.residuals[-1]) <= 1e-2 * 1e-8 * np.linalg.norm(B)


@pytest.mark.parametrize("overlap", ["1", "0"])
@pytest.mark.parametrize("nbus,p,ill", [(300, 1, False), (300, 8, False), (300, 16, False), (300, 16, True), (1400, 9, False),
                                        (1400, 8, True), (300, 32, False), (300, 32, True)])
def test_repeated_solves_agree_to_the_bit(bpf, monkeypatch, nbus, p, ill, overlap):
    """Every sum has a fixed order, so CTAs that read one another's partial sums too late or too early are the only
    way for two runs to differ: 10 columns and fewer (16 up to 1,024 rows) sum them in every CTA, more share them out."""
    import torch

    monkeypatch.setenv("BPF_OVERLAP", overlap)
    monkeypatch.setattr(bpf._lib, "_ctxs", {})   # a context made with this setting
    A = bpf.grid.synthetic_jacobian(nbus, seed=nbus)
    n = A.shape[0]
    B = torch.as_tensor(np.eye(n, p) if ill else np.random.default_rng(p).standard_normal((n, p)), device="cuda")
    Ad = bpf.CuSparseMatrixCSR.from_scipy(A)
    N = bpf.ilu0(Ad, p)
    first = None
    for _ in range(40):
        X, st = bpf.block_gmres(Ad, B, N=N, ldiv=True, memory=60, atol=0.0, rtol=1e-8, history=True)
        if first is None:
            first = X.clone(), list(st.residuals)
        assert torch.equal(X, first[0]) and list(st.residuals) == first[1]
