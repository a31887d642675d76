"""Grouped FP8 experts whose scale blocks are whole 128 x 128 blocks (bf16 tokens): f16 operands, the tokens over a power of two each and the
weights over one per block of rows; bf16 operands for the experts whose scales or tokens f16 does not hold.  Where it can go wrong: experts without
tokens and with one, rows per pair, tokens and scales of very uneven size, infinities and NaN, experts of both kinds in a call.

Bounds, f16: a token's elements are exact down to 2^-31 of its largest; scale and weight are rounded to f16, 2^-11 each at most and together, in
the mean, small beside the output's rounding to bf16, 2^-8 at most and 2^-8 / sqrt(3) in the mean.  bf16: the weight is rounded as the output
is, sqrt(2) of that."""
import numpy as np
import pytest
import torch

from helpers import rel_l2
from light_b200 import ops, synth

pytestmark = pytest.mark.gpu
ROUNDING = 2.0**-8 / 3**0.5
BF16_ROUNDING = 2**0.5 * ROUNDING


def _experts(E, N, K, dev, bR=128, bC=128, seed=0):
    codes, scale = synth.random_fp8_block(N + K + seed, E * N, K, bR, bC, device=dev)
    return codes, scale


def _exact(codes, scale, bR, bC):
    return codes.view(torch.float8_e4m3fn).double() * scale.double().repeat_interleave(bR, 0).repeat_interleave(bC, 1)


def _run(x, codes, scale, ids, wt, E, N, K, bR, bC):
    T, topk = ids.shape
    r = ops.MoERouteFromIDs(ids, wt, T, topk)
    return ops.MoEGemmF8Block(x, codes.reshape(E, N, K), scale.reshape(E, N // bR, K // bC), bR, bC, r, wt, topk)


# few pairs (memory of the call), many; pairs of SMs from 64 tokens an expert; blocks of more than 128
@pytest.mark.parametrize("T,E,topk,N,K,bR,bC,per_pair", [(1, 8, 2, 256, 256, 128, 128, False), (5, 300, 3, 128, 128, 128, 128, False), (200, 4, 2, 384, 1024, 128, 128, False),
                                                         (700, 6, 2, 512, 384, 256, 128, False), (90, 16, 4, 256, 512, 128, 256, True), (2000, 12, 2, 640, 256, 128, 128, True),
                                                         (30, 3, 2, 128, 8448, 128, 128, False)])
def test_grouped(cuda, T, E, topk, N, K, bR, bC, per_pair):
    codes, scale = _experts(E, N, K, cuda, bR, bC)
    w = _exact(codes, scale, bR, bC).reshape(E, N, K)
    g = torch.Generator().manual_seed(E)
    x = torch.randn(T * topk if per_pair else T, K, generator=g).to(cuda, torch.bfloat16)
    ids = torch.randint(0, E, (T, topk), generator=g).to(cuda)
    ids[ids == 1] = 0                                    # expert 1 stays empty
    wt = torch.rand(T * topk, generator=g).to(cuda)
    y = _run(x, codes, scale, ids, wt, E, N, K, bR, bC)
    assert torch.equal(y, _run(x, codes, scale, ids, wt, E, N, K, bR, bC))
    rows = x.double() if per_pair else x.double().repeat_interleave(topk, 0)
    want = torch.empty(T * topk, N, dtype=torch.float64, device=cuda)
    flat = ids.reshape(-1)
    for e in range(E):
        at = flat == e
        want[at] = rows[at] @ w[e].t() * wt.double()[at, None]
    assert ops.prefill_status(0) == 0
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= ROUNDING


@pytest.mark.parametrize("T", [20, 300])
@pytest.mark.parametrize("size", [2.0**-120, 1.0, 2.0**100])
@pytest.mark.parametrize("spread", [0, 12])
def test_uneven_tokens_and_scales(cuda, T, size, spread):
    E, topk, N, K = 2, 2, 256, 1024
    codes, scale = _experts(E, N, K, cuda)
    scale *= 2.0 ** -torch.randint(0, spread + 1, scale.shape, generator=torch.Generator().manual_seed(1)).float().to(cuda)
    w = _exact(codes, scale, 128, 128).reshape(E, N, K)
    g = torch.Generator().manual_seed(2)
    x = (torch.randn(T, K, generator=g).sign() * 2.0 ** (-28 * torch.rand(T, K, generator=g)) * size).to(cuda, torch.bfloat16)
    x[3] = 0
    ids = torch.stack([torch.zeros(T, dtype=torch.int64), torch.ones(T, dtype=torch.int64)], 1).to(cuda)
    wt = torch.ones(T * topk, device=cuda)
    y = _run(x, codes, scale, ids, wt, E, N, K, 128, 128).double().reshape(T, topk, N)
    want = torch.einsum("tk,enk->ten", x.double(), w)
    room = 2.0**-8 * want.abs() + 2.0**-10 * torch.einsum("tk,enk->ten", x.double().abs(), w.abs()) + 2.0**-133
    assert bool(((y - want).abs() <= room).all())
    assert bool((y[3] == 0).all())


@pytest.mark.parametrize("T", [20, 300])
def test_infinities_and_nan(cuda, T):
    E, topk, N, K = 2, 2, 128, 256
    codes, scale = _experts(E, N, K, cuda)
    inf = float("inf")
    g = torch.Generator().manual_seed(3)
    x = torch.randn(T, K, generator=g).to(cuda, torch.bfloat16)
    x[3, 7], x[4, 200], x[5, 0], x[6, 9], x[6, 250], x[8, 1], x[8, 2] = inf, -inf, float("nan"), inf, -inf, inf, float("nan")
    codes[10, 7] = 0        # infinity times zero
    codes[77, 30] = 0x7F    # a weight that is no number
    scale[1, 1] = inf       # of expert 1's second 128 k
    with np.errstate(all="ignore"):
        w = _exact(codes, scale, 128, 128).cpu().numpy().reshape(E, N, K)
        want = (x.double().cpu().numpy()[:, None, None, :] * w[None]).sum(-1)
    ids = torch.stack([torch.zeros(T, dtype=torch.int64), torch.ones(T, dtype=torch.int64)], 1).to(cuda)
    y = _run(x, codes, scale, ids, torch.ones(T * topk, device=cuda), E, N, K, 128, 128).cpu().double().numpy().reshape(T, topk, N)
    assert np.array_equal(np.isnan(y), np.isnan(want))
    assert np.array_equal(np.isinf(y), np.isinf(want)) and np.array_equal(np.sign(y[np.isinf(y)]), np.sign(want[np.isinf(want)]))
    fin = np.isfinite(want)
    assert rel_l2(y[fin], want[fin]) <= ROUNDING


@pytest.mark.parametrize("T", [20, 300])   # pairs in memory of the call, in the workspace
@pytest.mark.parametrize("kind", ["scales", "tokens", "both", "neither"])
@pytest.mark.parametrize("per_pair", [False, True])
def test_operands_of_far_apart_sizes(cuda, T, kind, per_pair):
    """What is small beside another block of the row, or another element of the token, counts where the large one meets zeros.  Even tokens
    go to experts 0 and 1, odd ones to 2 and 1; expert 0 has the scales, even tokens have the large elements."""
    E, topk, N, K = 3, 2, 256, 512
    codes, scale = _experts(E, N, K, cuda)
    codes = codes.reshape(E * N, K).clone()
    codes[:, 5] = 0                                      # what the token's large element meets
    x = torch.randn(T, K, generator=torch.Generator().manual_seed(4)).to(cuda, torch.bfloat16)
    if kind in ("scales", "both"):
        scale[:N // 128, 1] *= 2.0**40
        x[:, 128:256] = 0
    if kind in ("tokens", "both"):
        x[::2, 5] = 2.0**60
    w = _exact(codes, scale, 128, 128).reshape(E, N, K)
    even = torch.arange(T) % 2 == 0
    ids = torch.stack([torch.where(even, 0, 2), torch.ones(T, dtype=torch.int64)], 1).to(cuda)
    wt = torch.rand(T * topk, generator=torch.Generator().manual_seed(7)).to(cuda)
    rows = x.repeat_interleave(topk, 0) if per_pair else x
    y = _run(rows, codes, scale, ids, wt, E, N, K, 128, 128).double().reshape(T, topk, N)
    want = torch.einsum("tk,tsnk->tsn", x.double(), w[ids]) * wt.double().reshape(T, topk, 1)
    bf16 = {"scales": (0,), "tokens": (0, 1), "both": (0, 1), "neither": ()}[kind]
    for e in range(E):
        at = ids == e
        assert rel_l2(y[at].cpu().numpy(), want[at].cpu().numpy()) <= (BF16_ROUNDING if e in bf16 else ROUNDING), e
    assert ops.prefill_status(0) == 0


@pytest.mark.parametrize("T", [20, 300])
def test_finite_elements_beside_an_infinity_meet_an_infinite_scale(cuda, T):
    """All terms of one sign: infinity, not NaN."""
    E, topk, N, K = 2, 2, 128, 256
    codes = torch.full((E * N, K), 0x38, dtype=torch.uint8, device=cuda)     # 1.0
    scale = torch.ones(E, K // 128, device=cuda)
    scale[1, 1] = float("inf")
    x = torch.rand(T, K, generator=torch.Generator().manual_seed(5)).add(0.5).to(cuda, torch.bfloat16)
    x[3, 7] = float("inf")
    ids = torch.stack([torch.zeros(T, dtype=torch.int64), torch.ones(T, dtype=torch.int64)], 1).to(cuda)
    y = _run(x, codes, scale, ids, torch.ones(T * topk, device=cuda), E, N, K, 128, 128).reshape(T, topk, N)
    assert bool((y[3] == float("inf")).all()) and bool((y[:, 1] == float("inf")).all())
    assert bool(y[:3, 0].isfinite().all()) and bool(y[4:, 0].isfinite().all())


@pytest.mark.parametrize("T", [20, 300])
@pytest.mark.parametrize("up", [100, -100, 50, -50])   # beyond 2^64 either way: bf16
def test_sizes_that_cancel(cuda, T, up):
    """Scales of 2^up against tokens of 2^-up: neither product nor sum leaves f32's range."""
    E, topk, N, K = 2, 2, 128, 256
    codes, scale = _experts(E, N, K, cuda)
    scale = scale * 2.0**up
    x = (torch.randn(T, K, generator=torch.Generator().manual_seed(6)) * 2.0**-up).to(cuda, torch.bfloat16)
    w = _exact(codes, scale, 128, 128).reshape(E, N, K)
    ids = torch.stack([torch.zeros(T, dtype=torch.int64), torch.ones(T, dtype=torch.int64)], 1).to(cuda)
    y = _run(x, codes, scale, ids, torch.ones(T * topk, device=cuda), E, N, K, 128, 128).double().reshape(T, topk, N)
    want = torch.einsum("tk,enk->ten", x.double(), w)
    assert rel_l2(y.cpu().numpy(), want.cpu().numpy()) <= (BF16_ROUNDING if abs(up) == 100 else ROUNDING)


@pytest.mark.parametrize("T", [20, 300])
def test_small_tokens_with_small_routing_weights(cuda, T):
    """A token's power of two times its routing weight is a subnormal number, the result is not."""
    E, topk, N, K = 2, 2, 128, 256
    codes, scale = _experts(E, N, K, cuda)
    scale = scale * 2.0**60
    x = (torch.randn(T, K, generator=torch.Generator().manual_seed(8)) * 2.0**-120).to(cuda, torch.bfloat16)
    w = _exact(codes, scale, 128, 128).reshape(E, N, K)
    ids = torch.stack([torch.zeros(T, dtype=torch.int64), torch.ones(T, dtype=torch.int64)], 1).to(cuda)
    wt = (torch.rand(T * topk, generator=torch.Generator().manual_seed(9)) * 1e-6 + 1e-7).to(cuda)
    y = _run(x, codes, scale, ids, wt, E, N, K, 128, 128).double().reshape(T, topk, N)
    want = torch.einsum("tk,enk->ten", x.double(), w) * wt.double().reshape(T, topk, 1)
    assert rel_l2((y * 2.0**80).cpu().numpy(), (want * 2.0**80).cpu().numpy()) <= ROUNDING
