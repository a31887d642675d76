"""Q6_K rows of an odd number of blocks, every second of which starts off a word's boundary, at 1 to 64 activation rows: the one-row kernel and its passes, limbs, and
the row kernel between them, on both sides of the lines.  The last rows of the matrix end where its memory does.

Bound: all three hold f32 accuracy: f32 sums of exact products, 2^-24 of a partial sum per addition, 3e-7 on average over these lengths."""
import pytest
import torch

from helpers import rel_l2
from light_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _check(cuda, M, N, K, off=0):
    raw = synth.gaussian_weight(N + K, ops.Q6_K, N, K, device=cuda).reshape(-1)
    w = raw
    if off:
        w = torch.empty(raw.numel() + 16, dtype=raw.dtype, device=cuda)[off:off + raw.numel()]
        w.copy_(raw)
    x = torch.randn(M, K, generator=torch.Generator(device=cuda).manual_seed(M), device=cuda)
    q = ops.QTensor(w, ops.Q6_K, (N, K))
    y = ops.MatMulQ(x, q)
    assert torch.equal(y, ops.MatMulQ(x, q))
    assert rel_l2(y.cpu().double().numpy(), (x.double() @ ops.Dequantize(ops.QTensor(raw, ops.Q6_K, (N, K))).double().t()).cpu().numpy()) <= 3e-7
    assert ops.prefill_status(0) == 0


@pytest.mark.parametrize("N,K", [(16, 256), (17, 768), (31, 2304), (1000, 1280), (4096, 11008), (4741, 3328)])
def test_one_row(cuda, N, K):
    _check(cuda, 1, N, K)


@pytest.mark.parametrize("M,N,K", [(2, 1024, 3328), (3, 1024, 3328), (4, 1024, 3328), (2, 2048, 768), (8, 3072, 9984), (9, 3072, 9984), (16, 3072, 9984), (4, 16384, 1280), (64, 930, 768), (64, 940, 768),
                                   (33, 1850, 256), (17, 4100, 2816), (3, 15, 768), (64, 15, 768)])
def test_few_rows(cuda, M, N, K):
    _check(cuda, M, N, K)


@pytest.mark.parametrize("M", [1, 3, 40])
@pytest.mark.parametrize("off", [2, 8])
def test_off_the_boundary(cuda, M, off):
    _check(cuda, M, 1600, 3328, off)


def test_infinities_and_nan(cuda):
    """One row and limbs: a row with a NaN or an infinity gives no number or an infinity where plain arithmetic does; the rows beside it are as without."""
    N, K = 1600, 768
    w = ops.QTensor(synth.gaussian_weight(5, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    x = torch.randn(40, K, device=cuda)
    clean = ops.MatMulQ(x, w)
    x[7, 300], x[20, 5] = float("inf"), float("nan")
    y = ops.MatMulQ(x, w)
    keep = [m for m in range(40) if m not in (7, 20)]
    assert torch.equal(y[keep], clean[keep])
    assert not torch.isfinite(y[20]).any() and not torch.isfinite(y[7]).any()
