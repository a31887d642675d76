"""Q4_K with 9 to 64 rows and Q6_K with 17 to 64 as whole numbers through tensor memory, where it can go wrong: rows that are no whole tile, one block per
row, runs that start and end inside tiles and tiles cut into many runs, token counts on both sides of a chunk.

x is rounded to f16 (taken out of the comparison), a Q4_K weight is exact, a Q6_K weight's scale x code is rounded to 11 bits: 2^-11 of it at
most.  Sums are f32: K terms of like size are off by sqrt(K) 2^-24 of their magnitude in the mean, below 4e-6 of the result here."""
import pytest
import torch

from helpers import rel_l2
from light_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,N,K", [(ops.Q4_K, 65544, 256), (ops.Q4_K, 8200, 2048), (ops.Q4_K, 4097, 4352), (ops.Q4_K, 1500, 14336), (ops.Q4_K, 28672, 768),
                                     (ops.Q6_K, 32800, 512), (ops.Q6_K, 130, 33792), (ops.Q6_K, 4099, 4096)])
def test_whole_numbers(cuda, dt, N, K):
    w = ops.QTensor(synth.gaussian_weight(N + K, dt, N, K, device=cuda).reshape(-1), dt, (N, K))
    W = ops.Dequantize(w).double()
    g = torch.Generator().manual_seed(N)
    for M in (9, 16, 17, 32, 33, 48, 49, 64):
        x = torch.randn(M, K, generator=g).to(cuda)
        y = ops.MatMulQ(x, w)
        assert torch.equal(y, ops.MatMulQ(x, w)), "partial tiles must be added in a fixed order"
        want = x.half().double() @ W.t()
        assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= (4e-6 if dt == ops.Q4_K else 2.0**-11)
    assert ops.prefill_status(0) == 0


def test_calls_of_different_shapes_in_a_graph(cuda):
    """One after the other, and again: flags and partial tiles of a call are not another's."""
    ws = [ops.QTensor(synth.gaussian_weight(i, dt, N, K, device=cuda).reshape(-1), dt, (N, K)) for i, (dt, N, K) in
          enumerate([(ops.Q4_K, 8192, 2048), (ops.Q6_K, 4096, 4096), (ops.Q4_K, 6144, 4096), (ops.Q4_K, 4096, 14336)])]
    xs = [torch.randn(M, w.shape[1], generator=torch.Generator().manual_seed(M)).to(cuda) for M, w in zip((64, 20, 33, 17), ws)]
    want = [ops.MatMulQ(x, w) for x, w in zip(xs, ws)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [ops.MatMulQ(x, w) for x, w in zip(xs, ws)]
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert ops.prefill_status(0) == 0


# on both sides of each line of the dispatch: runs of four, five and six blocks to an SM, tiles cut into four and into eight parts
@pytest.mark.parametrize("dt,N,K", [(ops.Q4_K, 4096, 4096), (ops.Q4_K, 4096, 4864), (ops.Q4_K, 4608, 3840), (ops.Q4_K, 4736, 3584), (ops.Q4_K, 2304, 8192),
                                     (ops.Q4_K, 2432, 7168), (ops.Q4_K, 1024, 23552), (ops.Q4_K, 1024, 24064), (ops.Q6_K, 2304, 9728), (ops.Q6_K, 2432, 7168),
                                     (ops.Q6_K, 1024, 28160), (ops.Q6_K, 1024, 28672), (ops.Q6_K, 2048, 2048)])
def test_both_sides_of_the_dispatch(cuda, dt, N, K):
    w = ops.QTensor(synth.gaussian_weight(N + K, dt, N, K, device=cuda).reshape(-1), dt, (N, K))
    W = ops.Dequantize(w).double()
    for M in (9, 16, 17, 32, 33, 64):
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(cuda)
        want = x.half().double() @ W.t()
        assert rel_l2(ops.MatMulQ(x, w).cpu().double().numpy(), want.cpu().numpy()) <= (4e-6 if dt == ops.Q4_K else 2.0**-11)
    assert ops.prefill_status(0) == 0
