"""One activation row in fixed-point limbs (gguf_gemv_fast.cu) against an f64 product with the dequantized weights.

Bound per output: the fixed point rounds an activation at 2^-30 of the power of two above its block's largest, so at most
2^-30 max|x| sum|w|; scales, sums over lanes, warps and blocks are f32, fewer than 64 roundings of terms that together stay below
four times sum|w x| (a Q4_K weight is a difference of two products): 2^-16 sum|w x|."""
import pytest
import torch

from light_b200 import ops, synth

pytestmark = pytest.mark.gpu


def check(y, x, W):
    W, x = W.double(), x.double()
    bound = 2.0**-30 * x.abs().amax() * W.abs().sum(1) + 2.0**-16 * (W.abs() @ x.abs().t()).squeeze(1)
    assert ((y.double().squeeze(0) - W @ x.squeeze(0)).abs() <= bound).all()


def gguf(seed, dt, n, k):
    return ops.QTensor(synth.gaussian_weight(seed, dt, n, k, device="cuda").reshape(-1), dt, (n, k))


# both sides of each change of ring depth (K = 5376 and 14336 with Q4_K), the shortest rows, rows that are no whole tile
@pytest.mark.parametrize("fmt,n,k", [("Q4_K", 16, 256), ("Q4_K", 161, 5376), ("Q4_K", 161, 5632), ("Q4_K", 48, 14336), ("Q4_K", 48, 14592),
                                     ("Q4_K", 5000, 4096), ("Q6_K", 16, 512), ("Q6_K", 161, 1536), ("Q6_K", 5000, 4096), ("Q8_0", 16, 256),
                                     ("Q8_0", 161, 2304), ("Q8_0", 5000, 4096)])
@pytest.mark.parametrize("kind", ["normal", "outlier", "tiny", "huge"])
def test_one_row(cuda, fmt, n, k, kind):
    x = torch.randn(1, k, generator=torch.Generator().manual_seed(n + k)).to(cuda)
    if kind == "outlier":
        x[0, 5] = 1000.0
    x = x * {"tiny": 2.0**-90, "huge": 2.0**90}.get(kind, 1.0)
    w = gguf(n + k, getattr(ops, fmt), n, k)
    check(ops.MatMulQ(x, w), x, ops.Dequantize(w))


@pytest.mark.parametrize("n,k,group", [(16, 256, 64), (161, 2304, 128), (5000, 4096, 256)])
@pytest.mark.parametrize("kind", ["normal", "outlier", "tiny", "huge"])
def test_one_row_int4(cuda, n, k, group, kind):
    """F32 activations and results; sum - z Sx is a difference as in Q4_K."""
    g = torch.Generator().manual_seed(n + k)
    x = torch.randn(1, k, generator=g).to(cuda)
    if kind == "outlier":
        x[0, 5] = 1000.0
    x = x * {"tiny": 2.0**-90, "huge": 2.0**90}.get(kind, 1.0)
    w = ops.Int4(torch.randint(-2**31, 2**31, (n, k // 8), generator=g, dtype=torch.int32).to(cuda), (torch.rand(n, k // group, generator=g) + 0.5).to(cuda),
                 torch.randint(0, 16, (n, k // group), generator=g).float().to(cuda), group)
    check(ops.MatMulInt4(x, w), x, ops.DequantizeInt4(w, torch.float32))


@pytest.mark.parametrize("fmt", ["Q4_K", "Q6_K", "Q8_0"])
def test_a_nan_reaches_every_row(cuda, fmt):
    x = torch.zeros(1, 1024, device=cuda)
    w = gguf(3, getattr(ops, fmt), 40, 1024)
    assert (ops.MatMulQ(x, w) == 0).all()
    for v in (float("nan"), float("inf")):
        x[0, 700] = v
        assert torch.isnan(ops.MatMulQ(x, w)).all()


# eight warps with one block of k, sixteen beyond; one row tile to an SM, two, and more (of 148: 2368 and 4736 rows)
@pytest.mark.parametrize("n", [2368, 2384, 4736, 4752])
@pytest.mark.parametrize("k", [256, 512, 4096, 4352])
def test_one_row_int4_both_sides_of_the_wide_cta(cuda, n, k):
    test_one_row_int4(cuda, n, k, 128, "normal")
