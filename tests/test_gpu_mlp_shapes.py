"""The learned network's gradients and the tensor-core product at the edges of their tiles and K slices.

Tolerances: a gradient is a product of operands rounded to BF16 at up to three levels of the chain; where
FP32 sums differ in their last bits an operand can round the other way, by one BF16 step (2^-8 relative), so
a tensor differs from the oracle's by at most 3 x 2^-8 in the 2-norm; the loss, a sum over all outputs, by 1e-5.
1e-5 relative for the FP32 product of equal BF16 operands (K eps_32 sqrt-growth at K <= 4160).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bpf():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import blockpowerflow_b200 as bpf

    return bpf


# rows: one tile in part, whole tiles, one row beyond; samples around the tiles of 8, 32 and 64 and the
# largest; hidden widths of one and several tiles
@pytest.mark.parametrize("n,p,H", [(1, 1, 128), (31, 7, 128), (128, 33, 128), (129, 64, 384), (1000, 65, 256),
                                   (4161, 127, 640), (9001, 128, 512)])
def test_gradients(bpf, n, p, H):
    import torch

    import mlp_oracle as MO
    from blockpowerflow_b200.learned import PARAMS, WarmStartMLP

    s = 0.05
    mlp = WarmStartMLP(n, hidden=H, seed=1)
    mlp.set_scale(s)
    rng = np.random.default_rng(n)
    npad = (n + 127) // 128 * 128
    bias = np.zeros((1, npad))
    bias[0, :n] = 0.05 * rng.standard_normal(n)
    for k, v in (("b1", 0.1 * rng.standard_normal((1, H))), ("b2", 0.1 * rng.standard_normal((1, H))), ("b3", bias)):
        mlp.set_param(k, torch.as_tensor(v, dtype=torch.float32))
    B = rng.standard_normal((n, p))
    X = s * np.linalg.norm(B, axis=0) * rng.standard_normal((n, p)) / np.sqrt(n)
    pad = np.zeros((p, n + 3))
    pad[:, :n] = B.T
    Bd = torch.as_tensor(pad, device="cuda").t()[:n]   # a leading dimension above n
    loss = mlp.gradients(Bd, bpf.colmajor(torch.as_tensor(X, device="cuda")))
    params = {k: mlp.param(k).cpu().numpy().reshape(-1) if k[0] == "b" else mlp.param(k).cpu().numpy() for k in PARAMS}
    loss_o, g_o = MO.forward_backward(params, B, X, s)
    assert abs(loss - loss_o) <= 1e-5 * abs(loss_o)
    for k in PARAMS:
        g = mlp.param(k, grad=True).cpu().numpy().reshape(g_o[k].shape)
        assert np.linalg.norm(g - g_o[k]) <= 3 * 2.0**-8 * np.linalg.norm(g_o[k]), k


# odd leading dimensions take the scalar stores; splits: slices of unequal length, and added to D
@pytest.mark.parametrize("M,N,K,ldd,splits,acc", [(1, 1, 64, 1, 1, 0), (129, 127, 128, 127, 1, 0), (300, 260, 192, 264, 1, 0),
                                                  (128, 132, 4160, 133, 7, 0), (257, 96, 320, 96, 3, 1), (64, 33, 256, 36, 1, 1)])
def test_product(bpf, M, N, K, ldd, splits, acc):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + K)
    A, B = (torch.randn((r, K), generator=g, device="cuda").to(torch.bfloat16) for r in (M, N))
    D = torch.randn((M, ldd), generator=g, device="cuda")
    want = A.double() @ B.double().t() + (D[:, :N].double() if acc else 0.0)
    rest = D[:, N:].clone()
    ctx = bpf._lib.context(0)
    bpf._lib.check(bpf._lib.load().bpf_tc_gemm_bf16(ctx, M, N, K, A.data_ptr(), K, B.data_ptr(), K, D.data_ptr(), ldd, acc,
                                                    splits), ctx)
    assert float((D[:, :N].double() - want).norm()) <= 1e-5 * float(want.norm())
    if splits == 1 or acc:
        assert torch.equal(D[:, N:], rest)


@pytest.mark.parametrize("exponent", [-560, 560])
def test_targets_of_any_scale(bpf, exponent):
    """X and the scale times a power of two give the same normalized targets, to the bit, although X's squares leave
    the range of FP64; the loss is added up in any order over at most n p terms (2^-52 each)."""
    import torch

    from blockpowerflow_b200.learned import PARAMS, WarmStartMLP

    n, p, H, s = 700, 33, 128, 0.05
    rng = np.random.default_rng(2)
    B = rng.standard_normal((n, p))
    X = s * np.linalg.norm(B, axis=0) * rng.standard_normal((n, p)) / np.sqrt(n)
    out = []
    for k in (0, exponent):
        mlp = WarmStartMLP(n, hidden=H, seed=1)
        mlp.set_scale(s * 2.0**k)
        loss = mlp.gradients(bpf.colmajor(torch.as_tensor(B, device="cuda")), bpf.colmajor(torch.as_tensor(X * 2.0**k, device="cuda")))
        out.append((loss, [mlp.param(q, grad=True).cpu().numpy() for q in PARAMS]))
    assert out[0][0] > 0.5
    assert abs(out[1][0] - out[0][0]) <= n * p * 2.0**-52 * out[0][0]
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)
