"""GPU parity of the decode-step attention trio (KVAppend, DecodeAttention, IncrementI64) through the C ABI:
the cases and tolerances of the reference's own test (ops/decode_attn_cuda_test.go:20-91: 1e-4 of
max(1, |x|) at f32, 3e-2 at bf16), against the CPU oracle and against the reference's kernels
(kernels/cuda/src/decode_attn.cu compiled for sm_100a under oracle/_ref)."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from helpers import RefCuda
from light_b200 import ops
from test_decode_attn_cpu import CASES

pytestmark = pytest.mark.gpu

DTYPES = {"short": torch.float32, "llama-ish": torch.bfloat16, "qwen-ish": torch.bfloat16, "hd256 g1": torch.float32,
          "window mid-block": torch.bfloat16, "window short": torch.float32, "window wider than n": torch.float32,
          "hd512": torch.bfloat16}


def _inputs(case, dt, dev, seed=80):
    _, B, NH, KH, D, cap, n, window = case
    g = torch.Generator().manual_seed(seed)
    mk = lambda *s: torch.randn(*s, generator=g).to(dt)
    return mk(B, KH, cap, D).to(dev), mk(B, KH, cap, D).to(dev), mk(B, NH, 1, D).to(dev), mk(B, KH, 1, D).to(dev), mk(B, KH, 1, D).to(dev)


def _close(got, want, tol):
    got, want = got.float().cpu().numpy().astype(np.float64), np.asarray(want, np.float64)
    return float(np.max(np.abs(got - want) / np.maximum(1, np.abs(want)))) <= tol


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
def test_append_attend_increment(cuda, oracle, case, dt):
    name, B, NH, KH, D, cap, n, window = case
    tol = 1e-4 if dt == torch.float32 else 3e-2
    kbuf, vbuf, q, k, v = _inputs(case, dt, cuda)
    pos = torch.tensor([n - 1], dtype=torch.int64, device=cuda)
    scale = 1 / math.sqrt(D)
    kb2, vb2 = kbuf.clone(), vbuf.clone()
    ops.KVAppend(kbuf, vbuf, k, v, pos)
    assert torch.equal(kbuf[:, :, n - 1], k[:, :, 0]) and torch.equal(vbuf[:, :, n - 1], v[:, :, 0])
    out = ops.DecodeAttention(q, kbuf, vbuf, pos, scale, window)
    want = oracle.decode_attn(q.float().cpu().numpy(), kbuf.float().cpu().numpy(), vbuf.float().cpu().numpy(), n - 1, scale, window)
    assert _close(out, want, tol), name
    # append inside the attention launch: same cache, same bits out
    fused = ops.DecodeAttention(q, kb2, vb2, pos, scale, window, k_new=k, v_new=v)
    assert torch.equal(kb2, kbuf) and torch.equal(vb2, vbuf)
    assert torch.equal(fused, out)
    ops.IncrementI64(pos)
    assert int(pos.item()) == n
    assert ops.decode_attn_status(0) == 0


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_against_reference_kernels(cuda, case):
    """decode_attn_partial_* + decode_attn_combine_* launched as kernels/cuda/decode_attn.go:76-121 does."""
    if not RefCuda.available("decode_attn"):
        pytest.skip("oracle/_ref/decode_attn.cubin not built")
    name, B, NH, KH, D, cap, n, window = case
    dt = DTYPES[name]
    tol = 1e-4 if dt == torch.float32 else 3e-2
    kbuf, vbuf, q, k, v = _inputs(case, dt, cuda, seed=81)
    pos = torch.tensor([n - 1], dtype=torch.int64, device=cuda)
    scale = 1 / math.sqrt(D)
    ref = RefCuda()
    sfx = "f32" if dt == torch.float32 else "bf16"
    P = lambda t: C.c_void_p(t.data_ptr())
    nel = B * KH * D
    ref.launch("decode_attn", "kv_append_" + sfx, [(nel + 255) // 256], [256],
               [P(k), P(v), P(kbuf), P(vbuf), P(pos), C.c_int(B), C.c_int(KH), C.c_int(D), C.c_int(cap)])
    g, splits = NH // KH, (cap + 31) // 32
    part = torch.zeros(B * NH * splits * (D + 2), device=cuda)
    want = torch.empty(B, NH, 1, D, dtype=dt, device=cuda)
    ref.launch("decode_attn", "decode_attn_partial_" + sfx, [B * KH, splits], [128],
               [P(q), P(kbuf), P(vbuf), P(part), P(pos), C.c_int(NH), C.c_int(KH), C.c_int(cap), C.c_int(D), C.c_float(scale), C.c_int(window)],
               shmem=(g * (D + 1) + g * 32) * 4)
    ref.launch("decode_attn", "decode_attn_combine_" + sfx, [B * NH], [min(max(D, 32), 1024)],
               [P(part), P(want), P(pos), C.c_int(splits), C.c_int(D), C.c_int(window)])
    torch.cuda.synchronize()
    got = ops.DecodeAttention(q, kbuf, vbuf, pos, scale, window)
    assert _close(got, want.float().cpu().numpy(), tol), name


def test_one_graph_serves_every_position(cuda, oracle):
    """models/decode_graph.go:27-230: the step is captured once and replayed while the device-side position
    advances; here append + attend + increment, Llama-3-8B head shapes."""
    B, NH, KH, D, cap = 2, 32, 8, 128, 96
    g = torch.Generator().manual_seed(82)
    kbuf, vbuf = torch.zeros(B, KH, cap, D, device=cuda), torch.zeros(B, KH, cap, D, device=cuda)
    ks, vs, qs = torch.randn(5, B, KH, 1, D, generator=g), torch.randn(5, B, KH, 1, D, generator=g), torch.randn(5, B, NH, 1, D, generator=g)
    k, v, q = ks[0].to(cuda), vs[0].to(cuda), qs[0].to(cuda)
    pos = torch.zeros(1, dtype=torch.int64, device=cuda)
    scale = 1 / math.sqrt(D)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        out = ops.DecodeAttention(q, kbuf, vbuf, pos, scale, 0, k_new=k, v_new=v)  # warm-up outside capture
        pos.zero_()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = ops.DecodeAttention(q, kbuf, vbuf, pos, scale, 0, k_new=k, v_new=v)
            ops.IncrementI64(pos)
    kb, vb = np.zeros((B, KH, cap, D), np.float32), np.zeros((B, KH, cap, D), np.float32)
    for t in range(5):
        k.copy_(ks[t]), v.copy_(vs[t]), q.copy_(qs[t])
        graph.replay()
        torch.cuda.synchronize()
        oracle.kv_append(kb, vb, ks[t].numpy(), vs[t].numpy(), t)
        want = oracle.decode_attn(qs[t].numpy(), kb, vb, t, scale, 0)
        assert _close(out, want, 1e-4), t
        assert int(pos.item()) == t + 1
    assert np.array_equal(kbuf.cpu().numpy(), kb)


def test_limits_are_reported_not_asserted(cuda):
    """kernels/cuda/decode_attn.go:36-38,85-87: head dims that are no multiple of 32 and groups above 16 are
    refused (the caller composes the op); a position outside the cache is clamped and recorded."""
    from light_b200 import _lib

    q = torch.zeros(1, 34, 1, 48, device=cuda)
    kbuf = torch.zeros(1, 2, 16, 48, device=cuda)
    pos = torch.zeros(1, dtype=torch.int64, device=cuda)
    with pytest.raises(_lib.Light200Error):
        ops.DecodeAttention(q, kbuf, kbuf.clone(), pos, 1.0)
    q = torch.zeros(1, 34, 1, 64, device=cuda)
    kbuf = torch.zeros(1, 2, 16, 64, device=cuda)
    with pytest.raises(_lib.Light200Error):
        ops.DecodeAttention(q, kbuf, kbuf.clone(), pos, 1.0)
    with pytest.raises(ValueError):
        ops.DecodeAttention(q, kbuf, kbuf.clone(), pos.to(torch.int32), 1.0)


# ---- the tensor-core kernel of bf16 caches: block edges (16 keys a warp, 64 a CTA), one key, head groups on both sides of
# eight, a window that starts inside a block, and a row at pos that held NaN before the append.  Against f64; the bf16 output's
# rounding (2^-8 at most) is what remains.
@pytest.mark.parametrize("B,NH,KH,D,n,win", [(1, 1, 1, 64, 1, 0), (2, 8, 1, 128, 16, 0), (1, 9, 1, 64, 17, 0), (3, 16, 1, 128, 65, 0), (2, 4, 4, 64, 128, 50),
                                             (1, 24, 8, 128, 1000, 300)])
def test_tensor_core_kernel(cuda, B, NH, KH, D, n, win):
    g = torch.Generator().manual_seed(n)
    kb, vb, q, k, v = (torch.randn(s, generator=g).to(cuda, torch.bfloat16)
                       for s in ((B, KH, n, D), (B, KH, n, D), (B, NH, 1, D), (B, KH, 1, D), (B, KH, 1, D)))
    kb[:, :, n - 1], vb[:, :, n - 1] = float("nan"), float("nan")
    pos = torch.full((1,), n - 1, dtype=torch.int64, device=cuda)
    got = ops.DecodeAttention(q, kb, vb, pos, D ** -0.5, win, k, v, rope_base=10000.0)
    ang = (n - 1) * 10000.0 ** (-torch.arange(D // 2, dtype=torch.float64, device=cuda) * 2 / D)

    def rot(x):
        a, b = x.double().chunk(2, -1)
        return torch.cat([a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()], -1)

    assert torch.equal(kb[:, :, n - 1], rot(k)[:, :, 0].float().to(torch.bfloat16)) or (kb[:, :, n - 1].double() - rot(k)[:, :, 0]).abs().max() < 2 ** -6
    assert torch.equal(vb[:, :, n - 1], v[:, :, 0])
    s = max(0, n - win) if win else 0
    K, V = kb.double()[:, :, s:], vb.double()[:, :, s:]
    want = torch.softmax(rot(q).reshape(B, KH, NH // KH, D) @ K.transpose(-1, -2) * D ** -0.5, -1) @ V
    err = (got.double().reshape(want.shape) - want).norm() / want.norm()
    assert float(err) <= 3e-3 and ops.decode_attn_status(0) == 0


def test_position_moves_right_before_the_launch(cuda):
    """The launch starts while the increment before it still runs, and works ahead for the position as it stood: the same bits as with a
    wait between the two."""
    B, NH, KH, D, cap, steps = 2, 8, 2, 128, 256, 40
    g = torch.Generator(device=cuda).manual_seed(5)
    q, k, v = (torch.randn(steps, B, h, 1, D, generator=g, device=cuda) for h in (NH, KH, KH))
    outs = []
    for wait in (False, True):
        kb, vb, pos = torch.zeros(B, KH, cap, D, device=cuda), torch.zeros(B, KH, cap, D, device=cuda), torch.full((1,), 29, device=cuda)
        y = []
        for s in range(steps):
            ops.IncrementI64(pos)
            if wait:
                torch.cuda.synchronize()
            y.append(ops.DecodeAttention(q[s], kb, vb, pos, D ** -0.5, 0, k[s], v[s], rope_base=10000.0))
        outs.append(torch.cat([torch.stack(y).flatten(), kb.flatten(), vb.flatten()]))
    assert torch.equal(*outs)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("D", [32, 64, 128, 256, 512])
def test_position_moves_right_before_the_launch_in_every_kernel(cuda, D, dtype):
    """As above for each kernel: one that keeps the position of its early look overwrites the key before and drops a position."""
    B, NH, KH, cap, steps, dt = 2, 8, 2, 256, 40, {"f32": torch.float32, "bf16": torch.bfloat16}[dtype]
    g = torch.Generator(device=cuda).manual_seed(D)
    q, k, v = (torch.randn(steps, B, h, 1, D, generator=g, device=cuda).to(dt) for h in (NH, KH, KH))
    outs = []
    for wait in (False, True):
        kb, vb = (torch.zeros(B, KH, cap, D, device=cuda, dtype=dt) for _ in range(2))
        pos = torch.full((1,), 29, device=cuda)
        y = []
        for s in range(steps):
            ops.IncrementI64(pos)
            if wait:
                torch.cuda.synchronize()
            y.append(ops.DecodeAttention(q[s], kb, vb, pos, D ** -0.5, 0, k[s], v[s], rope_base=10000.0))
        outs.append(torch.cat([torch.stack(y).flatten(), kb.flatten(), vb.flatten()]))
    assert torch.equal(*outs)


@pytest.mark.parametrize("D,g", [(64, 1), (64, 2), (64, 3), (64, 8), (64, 16), (128, 1), (128, 2), (128, 4), (128, 5), (128, 16)])
@pytest.mark.parametrize("n,window", [(1, 0), (64, 0), (65, 0), (513, 0), (1025, 0), (700, 100)])
def test_f32_kernel(cuda, D, g, n, window):
    """Every count of heads per pass, and tiles of 64 keys with nothing, one or all but one key in the last: against f64, 512 roundings of
    2^-24 in the sums and 2^-20 of the exponentials' arguments stay below 1e-4 of the largest value."""
    B, KH = 2, 3
    gen = torch.Generator(device=cuda).manual_seed(D + g + n)
    kb, vb = (torch.full((B, KH, n + 3, D), float("nan"), device=cuda) for _ in range(2))
    kb[:, :, :n - 1], vb[:, :, :n - 1] = (torch.randn(B, KH, n - 1, D, generator=gen, device=cuda) for _ in range(2))
    q = torch.randn(B, KH * g, 1, D, generator=gen, device=cuda)
    k, v = (torch.randn(B, KH, 1, D, generator=gen, device=cuda) for _ in range(2))
    pos = torch.full((1,), n - 1, device=cuda)
    got = ops.DecodeAttention(q, kb, vb, pos, D ** -0.5, window, k, v)
    assert torch.equal(kb[:, :, n - 1], k[:, :, 0]) and torch.equal(vb[:, :, n - 1], v[:, :, 0])
    s0 = max(0, n - window) if window else 0
    S = (q.double().reshape(B, KH, g, D) @ kb[:, :, s0:n].double().transpose(-1, -2) * D ** -0.5).softmax(-1)
    want = (S @ vb[:, :, s0:n].double()).reshape(B, KH * g, 1, D)
    assert (got.double() - want).abs().max() <= 1e-4 * v.abs().max()


@pytest.mark.parametrize("D,g", [(64, 4), (64, 12), (128, 8), (128, 16)])
@pytest.mark.parametrize("n,append", [(1, False), (37, False), (300, True), (2000, False)])
def test_infinities_in_a_bf16_cache(cuda, D, g, n, append):
    """An infinite value answers an infinity in its dimension alone; a key whose score is -inf counts for nothing; NaN stays NaN: what f32
    arithmetic gives, in a kernel that splits its operands into two bf16 parts.  Against f64; the bf16 output's rounding remains."""
    B, KH = 1, 2
    gen = torch.Generator(device=cuda).manual_seed(n + g)
    kb, vb = (torch.randn(B, KH, n + 1, D, generator=gen, device=cuda).bfloat16() for _ in range(2))
    q = torch.randn(B, KH * g, 1, D, generator=gen, device=cuda).bfloat16()
    q[..., 5] = q[..., 5].abs() + 0.5
    k, v = (torch.randn(B, KH, 1, D, generator=gen, device=cuda).bfloat16() for _ in range(2))
    inf = float("inf")
    vb[0, 0, n // 2, 3] = inf
    vb[0, 0, n - 1, 7] = -inf                               # the last row: read again for the places past it
    kb[0, 1, : n // 2, 5] = -inf                            # the second head's first half: scores of -inf, whole blocks of them
    vb[0, 1, n // 2, 9] = float("nan")
    pos = torch.full((1,), n if append else n - 1, device=cuda)
    new = (k, v) if append else (None, None)
    got = ops.DecodeAttention(q, kb, vb, pos, D ** -0.5, 0, *new).double().reshape(KH, g, D)
    m = int(pos) + 1
    S = (q.double().reshape(KH, g, D) @ kb[0, :, :m].double().transpose(-1, -2) * D ** -0.5).softmax(-1)
    want = S @ vb[0, :, :m].double()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[want.isinf()], want[want.isinf()])
    fin = want.isfinite()
    assert float((got[fin] - want[fin]).norm() / want[fin].norm()) <= 3e-3
    if n > 1:
        assert bool(want[0, :, 3].isinf().all()) and int(fin.sum()) >= KH * g * (D - 4)
