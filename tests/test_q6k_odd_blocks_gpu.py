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
                                   (33, 1850, 256), (17, 4100, 2816), (3, 15, 768), (64, 15, 768), (1, 3072, 256), (1, 2048, 768)])
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


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("large", [1e3, 1e6, -3e30])
def test_small_activations_beside_a_large_one(cuda, M, large):
    """Outputs whose weights are zero at the large elements: what the others give keeps its f32 accuracy."""
    N, K = 6000, 768
    w = ops.QTensor(synth.gaussian_weight(9, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    deq = ops.Dequantize(w).double()
    x = torch.randn(M, K, generator=torch.Generator(device=cuda).manual_seed(3), device=cuda) * 0.05
    x[:, 130] = large
    rows = deq[:, 130] == 0
    assert int(rows.sum()) > 20
    want = x.double() @ deq.t()
    got = ops.MatMulQ(x, w)
    assert rel_l2(got[:, rows].cpu().double().numpy(), want[:, rows].cpu().numpy()) <= 3e-7
    assert rel_l2(got.cpu().double().numpy(), want.cpu().numpy()) <= 3e-7


def test_one_row_with_infinities_and_nan(cuda):
    """As plain f32 arithmetic over the dequantized weights has it, infinity times zero among it."""
    N, K = 4096, 1280
    w = ops.QTensor(synth.gaussian_weight(11, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    deq = ops.Dequantize(w)
    x = torch.randn(1, K, generator=torch.Generator(device=cuda).manual_seed(3), device=cuda)
    for at, v in ((300, float("inf")), (301, float("-inf")), (5, float("nan"))):
        z = x.clone()
        z[0, at] = v
        y, want = ops.MatMulQ(z, w), (z.double() @ deq.double().t()).float()
        assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
        assert torch.equal(y[torch.isinf(y)], want[torch.isinf(want)])


def _outlier(cuda, M, K, large):
    x = torch.randn(M, K, generator=torch.Generator(device=cuda).manual_seed(3), device=cuda) * 0.05
    x[:, 130] = large
    x[M // 2] = 0
    return x


@pytest.mark.parametrize("M,N", [(4, 16000), (16, 6000), (40, 6000), (64, 6000), (65, 2000), (100, 2000)])
@pytest.mark.parametrize("large", [1e3, 1e6, 1e10, 1e12, -3e30])
def test_limbs_of_small_activations_beside_a_large_one(cuda, M, N, large):
    """As above, where the products are those of limbs: from 60000 outputs on."""
    K = 768
    w = ops.QTensor(synth.gaussian_weight(9, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    deq, x = ops.Dequantize(w).double(), _outlier(cuda, M, K, large)
    rows = deq[:, 130] == 0
    assert int(rows.sum()) > 20
    got, want = ops.MatMulQ(x, w), x.double() @ deq.t()
    assert rel_l2(got[:, rows].cpu().double().numpy(), want[:, rows].cpu().numpy()) <= 3e-7
    assert rel_l2(got.cpu().double().numpy(), want.cpu().numpy()) <= 3e-7
    assert not got[M // 2].any() and torch.equal(got, ops.MatMulQ(x, w))


@pytest.mark.parametrize("large", [1e3, 1e12, -3e30])
@pytest.mark.parametrize("weighted", [False, True])
def test_grouped_limbs_of_small_activations_beside_a_large_one(cuda, large, weighted):
    E, N, K, T, topk = 5, 1500, 768, 150, 2
    w = ops.QTensor(synth.gaussian_weight(9, ops.Q6_K, E * N, K, device=cuda).reshape(-1), ops.Q6_K, (E, N, K))
    deq, x = ops.Dequantize(w).double(), _outlier(cuda, T, K, large)
    g = torch.Generator(device=cuda).manual_seed(8)
    ids = torch.rand(T, E, generator=g, device=cuda).topk(topk, -1).indices
    tw = torch.rand(T * topk, generator=g, device=cuda) + 0.5
    route = ops.MoERouteFromIDs(ids, tw, T, topk)
    got = ops.MoEGemmQ(x, w, route, tw if weighted else None, topk).double()
    e = ids.reshape(-1)
    want = torch.stack([deq[int(e[p])] @ x[p // topk].double() * (float(tw[p]) if weighted else 1.0) for p in range(T * topk)])
    off = deq[e, :, 130] == 0
    assert int(off.sum()) > 1000
    assert float((got - want)[off].norm() / want[off].norm()) <= 3e-7 and float((got - want).norm() / want.norm()) <= 3e-7


@pytest.mark.parametrize("M", [2, 8, 40, 64, 65])
def test_several_matrices_in_one_call(cuda, M):
    """Each gives what it gives alone, bit for bit."""
    K, sizes = 3328, (1600, 96, 2000)
    ws = [ops.QTensor(synth.gaussian_weight(n, ops.Q6_K, n, K, device=cuda).reshape(-1), ops.Q6_K, (n, K)) for n in sizes]
    x = torch.randn(M, K, generator=torch.Generator(device=cuda).manual_seed(M), device=cuda)
    for y, w in zip(ops.MatMulQMulti(x, ws), ws):
        assert torch.equal(y, ops.MatMulQ(x, w))


@pytest.mark.parametrize("M,N,K", [(2, 16384, 256), (2, 4096, 768), (3, 4096, 5376), (4, 3499, 6400), (4, 3500, 6400), (4, 3300, 11008), (5, 2399, 9472), (6, 2400, 9472), (8, 3500, 6400), (8, 6016, 3840),
                                   (8, 6016, 4352), (8, 6016, 8448), (8, 7500, 4352), (8, 3400, 9472)])
def test_both_sides_of_the_passes(cuda, M, N, K):
    _check(cuda, M, N, K)
