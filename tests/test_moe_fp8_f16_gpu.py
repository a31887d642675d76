"""Grouped FP8 experts whose scale blocks are whole 128 x 128 blocks (bf16 tokens): f16 operands, the tokens over a power of two each and the
weights over one per block of rows.  Where it can go wrong: experts without tokens and with one, rows per pair, tokens and scales
of very uneven size, infinities and NaN.

Bounds: a token's elements are exact down to 2^-31 of its largest; scale and weight are rounded to f16, 2^-12 each at most; the output
to bf16, 2^-8 at most and 2^-8 / sqrt(3) in the mean."""
import numpy as np
import pytest
import torch

from helpers import rel_l2
from light_b200 import ops, synth

pytestmark = pytest.mark.gpu
ROUNDING = 2.0**-8 / 3**0.5


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
