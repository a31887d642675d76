"""Calls whose operands are multiplied as they are stay that way, whichever kernel takes the larger or better aligned ones of the same
format.

Bounds: a product of f32 values summed in f32 over K terms is off by at most about K / 2 * 2^-24 of the sum of magnitudes and by
sqrt(K) * 2^-24 on average, below 1e-5 here; operands rounded to f16 give 2^-11 each at most, 3e-4 on the result."""
import pytest
import torch

from helpers import rel_l2
from light_b200 import _lib, ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(65, 132, 256), (333, 300, 768), (1100, 128, 1280)])
def test_q6_k_with_an_odd_number_of_blocks_per_row(cuda, M, N, K):
    w = ops.QTensor(synth.gaussian_weight(N, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(cuda)
    want = x.double() @ ops.Dequantize(w).double().t()
    assert rel_l2(ops.MatMulQ(x, w).cpu().double().numpy(), want.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("M", [100, 333])   # 200 and 666 pairs
def test_grouped_q6_k_with_an_odd_number_of_blocks_per_row(cuda, M):
    E, N, K, topk = 5, 260, 768, 2
    q = ops.QTensor(synth.gaussian_weight(3, ops.Q6_K, E * N, K, device=cuda).reshape(-1), ops.Q6_K, (E, N, K))
    w = ops.Dequantize(q).double().reshape(E, N, K)
    g = torch.Generator().manual_seed(5)
    x = torch.randn(M, K, generator=g).to(cuda)
    ids = torch.randint(0, E, (M, topk), generator=g).to(cuda)
    r = ops.MoERouteFromIDs(ids, torch.ones(M * topk, device=cuda), M, topk)
    want = torch.einsum("mk,mnk->mn", x.double().repeat_interleave(topk, 0), w[ids.reshape(-1)])
    assert rel_l2(ops.MoEGemmQ(x, q, r, None, topk).cpu().double().numpy(), want.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("G", [64, 256])
@pytest.mark.parametrize("scale", [1e-6, 3e4])
def test_int4_rows_beyond_f16(cuda, G, scale):
    """17 to 64 bf16 rows of a 4-bit matrix whose groups are not 128: x is multiplied as bf16, whatever its range.  bf16 weights (2^-8 of a
    weight at most, 1.1e-3 on average) and the bf16 output's rounding (the same) remain."""
    M, N, K = 33, 4096, 4096
    g = torch.Generator(device=cuda).manual_seed(G)
    w = ops.Int4(torch.randint(-2**31, 2**31, (N, K // 8), generator=g, device=cuda, dtype=torch.int32), torch.rand(N, K // G, generator=g, device=cuda) * 0.02,
                 torch.randint(0, 16, (N, K // G), generator=g, device=cuda).float(), G)
    x = (torch.randn(M, K, generator=g, device=cuda) * scale).bfloat16()
    want = x.double() @ ops.DequantizeInt4(w, torch.float32).double().t()
    assert rel_l2(ops.MatMulInt4(x, w).cpu().double().numpy(), want.cpu().numpy()) <= 2.5e-3


# whole passes of 16 tokens and one more, rows that are no whole tile, one block per row, runs of more than the ring's blocks, more rows
# than limbs are kept of at a time
@pytest.mark.parametrize("M,N,K", [(65, 32, 256), (4100, 48, 256), (80, 33, 768), (81, 300, 1280), (500, 130, 2816)])
@pytest.mark.parametrize("kind", ["normal", "outlier", "tiny", "huge"])
def test_q6_k_in_limbs(cuda, M, N, K, kind):
    """Per output: an activation is held to 2^-23 of itself or 2^-60 of its block's largest, less than 2^-30 max|x| sum|w| in all;
    per block and limb pair the whole sums and their scaling are rounded three times, blocks are added in f32: fewer than 16 + K / 256
    roundings of terms that together stay below four times sum|w x|."""
    w = ops.QTensor(synth.gaussian_weight(N + K, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(cuda)
    if kind == "outlier":
        x[:, 5] = 1000.0
    x = x * {"tiny": 2.0**-90, "huge": 2.0**90}.get(kind, 1.0)
    W, X = ops.Dequantize(w).double(), x.double()
    bound = 2.0**-30 * X.abs().amax(1, keepdim=True) * W.abs().sum(1) + (16 + K / 256) * 2.0**-22 * (X.abs() @ W.abs().t())
    assert bool(((ops.MatMulQ(x, w).double() - X @ W.t()).abs() <= bound).all())


def test_grouped_q6_k_in_limbs_of_many_pairs(cuda):
    """Experts on both sides of the 4096 pairs whose limbs are kept at a time, one of them across."""
    E, T, topk, N, K = 3, 3000, 2, 40, 768
    q = ops.QTensor(synth.gaussian_weight(4, ops.Q6_K, E * N, K, device=cuda).reshape(-1), ops.Q6_K, (E, N, K))
    W = ops.Dequantize(q).double().reshape(E, N, K)
    g = torch.Generator().manual_seed(6)
    x = torch.randn(T, K, generator=g).to(cuda)
    ids = torch.randint(0, E, (T, topk), generator=g).to(cuda)
    wt = torch.rand(T * topk, generator=g).to(cuda)
    y = ops.MoEGemmQ(x, q, ops.MoERouteFromIDs(ids, wt, T, topk), wt, topk)
    want = torch.einsum("mk,mnk->mn", x.double().repeat_interleave(topk, 0), W[ids.reshape(-1)]) * wt.double()[:, None]
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 1e-6
    assert ops.prefill_status(0) == 0


def test_q6_k_in_limbs_infinities_and_nan(cuda):
    """Tokens with infinities or NaN give what f32 products give; the others are not touched by them."""
    M, N, K = 70, 40, 768
    w = ops.QTensor(synth.gaussian_weight(1, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(2)).to(cuda)
    inf = float("inf")
    x[3, 7], x[4, 700], x[5, 0], x[6, 9], x[6, 300], x[69, 1] = inf, -inf, float("nan"), inf, -inf, inf
    W = ops.Dequantize(w).double().cpu()
    want = (x.double().cpu()[:, None, :] * W[None]).sum(-1)
    y = ops.MatMulQ(x, w).double().cpu()
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
    assert torch.equal(y[y.isinf()].sign(), want[want.isinf()].sign())
    fin = want.isfinite()
    assert rel_l2(y[fin].numpy(), want[fin].numpy()) <= 1e-6


def _zero_at(w, N, K, column):
    """The blocks with the code of 0 at this element (of 256) of every block."""
    raw = w.reshape(N, K // 256, 210).clone()
    assert column < 32
    raw[:, :, column] &= 0xF0
    raw[:, :, 128 + column] = (raw[:, :, 128 + column] & 0xFC) | 2
    return raw.reshape(-1)


@pytest.mark.parametrize("M,N,K", [(65, 64, 256), (100, 512, 768), (333, 130, 2816), (200, 64, 11008)])
@pytest.mark.parametrize("large,sigma", [(0, 1.0), (5, 0.05), (1000, 1.0), (1000, 0.05), (1e6, 0.05), (1e9, 0.05)])
def test_q6_k_small_activations_beside_large_ones(cuda, M, N, K, large, sigma):
    """Outputs whose weights are zero where a block's large activation is.  The small ones keep 23 bits (2^-23 each, at random), what is done in
    a block is rounded some 16 times, 2^-24 each: together about 2^-23 = 1.2e-7 (f32 products are 8.1e-8 to 1.46e-7 off at these sizes); without
    large ones the sums of a sub-block are whole numbers and blocks are added exactly: 2.5e-8, and 5e-8 is twice that."""
    raw = synth.gaussian_weight(N + K, ops.Q6_K, N, K, device=cuda)
    w = ops.QTensor(_zero_at(raw, N, K, 9) if large else raw.reshape(-1), ops.Q6_K, (N, K))
    W = ops.Dequantize(w).double()
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(cuda) * sigma
    if large:
        assert not W[:, 9::256].any()
        x[:, 9::256] = large
    y = ops.MatMulQ(x, w).double()
    assert rel_l2(y.cpu().numpy(), (x.double() @ W.t()).cpu().numpy()) <= (2.0**-23 if large else 5e-8)


def test_grouped_q6_k_small_activations_beside_large_ones(cuda):
    E, T, topk, N, K = 4, 200, 2, 96, 768
    raw = synth.gaussian_weight(2, ops.Q6_K, E * N, K, device=cuda)
    q = ops.QTensor(_zero_at(raw, E * N, K, 9), ops.Q6_K, (E, N, K))
    W = ops.Dequantize(q).double().reshape(E, N, K)
    g = torch.Generator().manual_seed(3)
    x = (0.05 * torch.randn(T, K, generator=g)).to(cuda)
    x[:, 9::256] = 1e5
    ids = torch.randint(0, E, (T, topk), generator=g).to(cuda)
    y = ops.MoEGemmQ(x, q, ops.MoERouteFromIDs(ids, torch.ones(T * topk, device=cuda), T, topk), None, topk)
    want = torch.einsum("mk,mnk->mn", x.double().repeat_interleave(topk, 0), W[ids.reshape(-1)])
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 2.0**-23


@pytest.mark.parametrize("kind", ["normal", "silu"])
def test_q6_k_of_ordinary_activations_is_no_less_exact_than_f32_products(cuda, kind):
    M, N, K = 300, 256, 2816
    w = ops.QTensor(synth.gaussian_weight(8, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    g = torch.Generator().manual_seed(9)
    x = torch.randn(M, K, generator=g)
    if kind == "silu":
        x = torch.nn.functional.silu(4 * x) * torch.randn(M, K, generator=g)
    x = x.to(cuda)
    want = x.double() @ ops.Dequantize(w).double().t()
    assert rel_l2(ops.MatMulQ(x, w).cpu().double().numpy(), want.cpu().numpy()) <= 6e-8   # f32 products: 1.0e-7


def test_q6_k_in_limbs_shares_no_memory(cuda):
    """Dense and grouped calls leave the workspace as it is, and several streams have calls at once."""
    N, K, M, E, topk = 96, 1280, 300, 3, 2
    q = ops.QTensor(synth.gaussian_weight(1, ops.Q6_K, E * N, K, device=cuda).reshape(-1), ops.Q6_K, (E, N, K))
    w = ops.QTensor(q.data, ops.Q6_K, (E * N, K))
    g = torch.Generator().manual_seed(2)
    xs = [torch.randn(M, K, generator=g).to(cuda) for _ in range(4)]
    ids = torch.randint(0, E, (M, topk), generator=g).to(cuda)
    r = ops.MoERouteFromIDs(ids, torch.ones(M * topk, device=cuda), M, topk)
    call = lambda x: (ops.MatMulQ(x, w), ops.MoEGemmQ(x, q, r, None, topk), ops.MatMulQMulti(x, [w])[0])  # noqa: E731
    ops.ensure_workspace(0, 1 << 20)
    want = [call(x) for x in xs]
    ws = ops._workspaces[0]
    ws.fill_(0x5A)
    call(xs[0])
    assert bool((ws == 0x5A).all())
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = []
    for _ in range(3):
        for x, s in zip(xs, streams):
            with torch.cuda.stream(s):
                got.append(call(x))
    torch.cuda.synchronize()
    for i, ys in enumerate(got):
        assert all(torch.equal(y, z) for y, z in zip(ys, want[i % 4]))


def test_q6_k_in_limbs_in_a_graph(cuda):
    N, K, M = 64, 768, 100
    w = ops.QTensor(synth.gaussian_weight(3, ops.Q6_K, N, K, device=cuda).reshape(-1), ops.Q6_K, (N, K))
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(4)).to(cuda)
    want = ops.MatMulQ(x, w)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ops.MatMulQ(x, w)
    x.copy_(2 * x)
    graph.replay()
    assert torch.equal(y, 2 * want)


@pytest.mark.parametrize("short", [None, 1])   # no scratch, too little of it
def test_q6_k_without_scratch(cuda, short):
    """f32 products: 8.8e-8 off at this K, whatever the sizes of a block's activations."""
    M, N, K = 100, 64, 768
    w = ops.QTensor(_zero_at(synth.gaussian_weight(4, ops.Q6_K, N, K, device=cuda), N, K, 9), ops.Q6_K, (N, K))
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(5)).to(cuda)
    x[:, 9::256] = 1e6
    L = _lib.lib()
    need = int(L.light_b200_q6k_scratch_bytes(ops.Q6_K, w.data.data_ptr(), M, K, 0))
    own = None if short is None else torch.empty(need - short, dtype=torch.uint8, device=cuda)
    y = torch.empty(M, N, device=cuda)
    _lib.check(L.light_b200_matmul_q_scratch(ops.Q6_K, x.data_ptr(), w.data.data_ptr(), y.data_ptr(), M, N, K, None if own is None else own.data_ptr(),
                                             0 if own is None else own.numel(), 0, torch.cuda.current_stream().cuda_stream))
    want = x.double() @ ops.Dequantize(w).double().t()
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 2.0**-23
