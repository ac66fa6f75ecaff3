"""mul on column-major blocks: the direct and the panel path at their edges, leading dimensions, and X and Y
that share memory.

Each output is a sum of at most k products; the oracle adds them in another order, so they differ by at
most 2 k eps sum |a| |x| (and the scaling's roundings): 4 (k + 4) eps (|alpha| |A| |X| + |beta| |Y|).
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bpf():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import blockpowerflow_b200 as bpf

    return bpf


def _matrix(n, long, seed):
    """Rows of 0 to 17 entries, and one of `long`."""
    rng = np.random.default_rng(seed)
    cnt = rng.integers(0, min(n, 17) + 1, n)
    cnt[n // 2] = min(n, long)
    ci = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in cnt])
    rp = np.concatenate([[0], np.cumsum(cnt)])
    return sp.csr_matrix((rng.standard_normal(len(ci)), ci, rp), shape=(n, n))


# n, p: both sides of the direct path's limit of 2 million products, last tiles of rows and columns in part
# filled, panels of 8, 16, 32 and 64 columns, more than the 256 columns of one pass
@pytest.mark.parametrize("n,p", [(1, 1), (2, 3), (31, 2), (129, 5), (1000, 40), (7001, 5), (9001, 33), (40001, 4), (40001, 7),
                                 (40001, 15), (20001, 31), (20001, 33), (40001, 63), (40001, 130), (3001, 300)])
@pytest.mark.parametrize("pad,beta", [(0, 0.0), (5, 0.25)])
def test_edges(bpf, n, p, pad, beta):
    import torch

    A = _matrix(n, 700, n + p)
    rng = np.random.default_rng(p)
    X, Y = rng.standard_normal((n, p)), rng.standard_normal((n, p))
    Xd = torch.zeros((p, n + pad), dtype=torch.float64, device="cuda")
    Yd = torch.full((p, n + pad), 7.0, dtype=torch.float64, device="cuda")
    Xd[:, :n] = torch.as_tensor(X.T, device="cuda")
    Yd[:, :n] = torch.as_tensor(Y.T if beta else np.full((p, n), np.nan), device="cuda")
    bpf.mul(bpf.CuSparseMatrixCSR.from_scipy(A, index_base=pad & 1), Xd.t()[:n], alpha=-1.5, beta=beta, Y=Yd.t()[:n])
    got = Yd.cpu().numpy()
    k = np.diff(A.indptr).max()
    bound = 4 * (k + 4) * 2.0**-52 * (1.5 * (abs(A) @ abs(X)) + beta * abs(Y))
    assert np.all(abs(got[:, :n].T - (-1.5 * (A @ X) + beta * Y)) <= bound)
    assert np.all(got[:, n:] == 7.0)


@pytest.mark.parametrize("n,p", [(500, 8), (20001, 40), (3001, 300)])
@pytest.mark.parametrize("shift", [0, 1, 17])
def test_shared_memory(bpf, n, p, shift):
    """Y is X's memory, or starts `shift` columns' elements into it: X counts as read first (up to 256 columns)."""
    import torch

    p = min(p, 256) if shift else p
    A = _matrix(n, 40, n)
    buf = torch.as_tensor(np.random.default_rng(n).standard_normal(n * (p + 20)), device="cuda")
    X = buf[: n * p].view(p, n).t()
    Y = buf[n * shift + (3 if shift else 0):][: n * p].view(p, n).t()
    want = bpf.mul(bpf.CuSparseMatrixCSR.from_scipy(A), X.t().clone().t())
    bpf.mul(bpf.CuSparseMatrixCSR.from_scipy(A), X, Y=Y)
    assert torch.equal(Y, want)
