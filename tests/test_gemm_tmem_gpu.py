"""The tensor-memory matmul (weights expanded into TMEM, stream-K over CTAs or CTA pairs) where it can go wrong: one token more
than a tile, ragged row counts (with and without whole 16-byte output rows), the shortest K, runs that start and end inside
tiles, grouped launches with empty experts and single tokens, and launches on two streams.

Bounds: operands are rounded once each to f16 (2^-12 relative on average over a product: 1e-3 with room, the bound of the other
tensor-core paths) or are the bf16 values themselves, when the bf16 output's rounding (2^-8 at most) is what remains."""
import pytest
import torch

from helpers import rel_l2
from light_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _weight(kind, N, K, dev):
    if kind in ("q4_k", "q6_k", "q8_0"):
        dt = {"q4_k": ops.Q4_K, "q6_k": ops.Q6_K, "q8_0": ops.Q8_0}[kind]
        w = ops.QTensor(synth.gaussian_weight(N + K, dt, N, K, device=dev).reshape(-1), dt, (N, K))
        return (lambda x: ops.MatMulQ(x, w)), ops.Dequantize(w).double(), torch.float32
    if kind == "int4":
        g = torch.Generator(device=dev).manual_seed(N + K)
        w = ops.Int4(torch.randint(-2**31, 2**31, (N, K // 8), generator=g, device=dev, dtype=torch.int32), torch.rand(N, K // 64, generator=g, device=dev) * 0.02,
                     torch.randint(0, 31, (N, K // 64), generator=g, device=dev).float() / 2, 64)   # half of the zero points are no whole numbers
        return (lambda x: ops.MatMulInt4(x, w)), ops.DequantizeInt4(w, torch.bfloat16).double(), torch.bfloat16
    codes, scale = synth.random_fp8_block(N + K, N, K, 4, 64, device=dev)
    return (lambda x: ops.MatMulF8Block(x, codes, scale, 4, 64)), ops.DequantizeF8Block(codes, scale, 4, 64, torch.bfloat16).double(), torch.bfloat16


@pytest.mark.parametrize("kind", ["q4_k", "q6_k", "q8_0", "int4", "fp8"])
@pytest.mark.parametrize("M,N,K", [(65, 132, 256), (129, 128, 1280), (200, 300, 512), (257, 4100, 2304), (1100, 1024, 768), (513, 8192, 2048)])
def test_plain(cuda, kind, M, N, K):
    if kind == "fp8" and N % 4:
        pytest.skip("blocks of four rows")
    f, w, dt = _weight(kind, N, K, cuda)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(cuda, dt)
    y = f(x)
    assert torch.equal(y, f(x)), "partial tiles must be added in a fixed order"
    assert ops.prefill_status(0) == 0
    want = x.double() @ w.t()
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= (1e-3 if dt == torch.float32 else 3e-3)


@pytest.mark.parametrize("M,E,topk,N,K", [(1, 8, 2, 256, 256), (5, 300, 3, 132, 128), (40, 4, 1, 128, 1024), (700, 6, 2, 520, 384)])
def test_grouped_fp8(cuda, M, E, topk, N, K):
    codes, scale = synth.random_fp8_block(7, E * N, K, 4, 64, device=cuda)
    w = ops.DequantizeF8Block(codes, scale, 4, 64, torch.bfloat16).double().reshape(E, N, K)
    g = torch.Generator().manual_seed(E)
    x = torch.randn(M, K, generator=g).to(cuda, torch.bfloat16)
    ids = torch.randint(0, E, (M, topk), generator=g).to(cuda)
    ids[ids == 1] = 0                                    # expert 1 stays empty
    wt = torch.rand(M * topk, generator=g).to(cuda)
    r = ops.MoERouteFromIDs(ids, wt, M, topk)
    y = ops.MoEGemmF8Block(x, codes.reshape(E, N, K), scale.reshape(E, N // 4, K // 64), 4, 64, r, wt, topk)
    want = torch.einsum("mk,mnk->mn", x.double().repeat_interleave(topk, 0), w[ids.reshape(-1)]) * wt.double()[:, None]
    assert ops.prefill_status(0) == 0
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 3e-3


def test_grouped_q6_k_rows_at_odd_offsets(cuda):
    E, N, K, M, topk = 5, 260, 768, 333, 2                # 630-byte rows: not a multiple of four
    q = ops.QTensor(synth.gaussian_weight(3, ops.Q6_K, E * N, K, device=cuda).reshape(-1), ops.Q6_K, (E, N, K))
    w = ops.Dequantize(q).double().reshape(E, N, K)
    g = torch.Generator().manual_seed(5)
    x = torch.randn(M, K, generator=g).to(cuda)
    ids = torch.randint(0, E, (M, topk), generator=g).to(cuda)
    r = ops.MoERouteFromIDs(ids, torch.ones(M * topk, device=cuda), M, topk)
    y = ops.MoEGemmQ(x, q, r, None, topk)
    want = torch.einsum("mk,mnk->mn", x.double().repeat_interleave(topk, 0), w[ids.reshape(-1)])
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 1e-3


@pytest.mark.parametrize("M,N,K", [(17, 4096, 4096), (33, 8196, 2048), (48, 732, 14336), (64, 40964, 256)])
def test_narrow_int4(cuda, M, N, K):
    """17 to 64 bf16 rows of a 4-bit matrix of 10 * 2^20 weights or more: f16 operands (2^-12 each on average), then the bf16 output's
    rounding, 2^-8 of a value at most."""
    g = torch.Generator(device=cuda).manual_seed(N)
    w = ops.Int4(torch.randint(-2**31, 2**31, (N, K // 8), generator=g, device=cuda, dtype=torch.int32), torch.rand(N, K // 64, generator=g, device=cuda) * 0.02,
                 torch.randint(0, 31, (N, K // 64), generator=g, device=cuda).float() / 2, 64)
    x = torch.randn(M, K, generator=g, device=cuda).bfloat16()
    y = ops.MatMulInt4(x, w)
    assert torch.equal(y, ops.MatMulInt4(x, w)) and ops.prefill_status(0) == 0
    want = x.double() @ ops.DequantizeInt4(w, torch.float32).double().t()
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 2.5e-3


@pytest.mark.parametrize("M,N,K", [(17, 4096, 4096), (33, 8196, 2048), (48, 732, 14336), (64, 40964, 256)])
def test_narrow_int4_in_groups_of_128(cuda, M, N, K):
    """As test_narrow_int4, for the groups whose 17 to 64 rows this kernel has."""
    g = torch.Generator(device=cuda).manual_seed(N)
    w = ops.Int4(torch.randint(-2**31, 2**31, (N, K // 8), generator=g, device=cuda, dtype=torch.int32), torch.rand(N, K // 128, generator=g, device=cuda) * 0.02,
                 torch.randint(0, 31, (N, K // 128), generator=g, device=cuda).float() / 2, 128)
    x = torch.randn(M, K, generator=g, device=cuda).bfloat16()
    y = ops.MatMulInt4(x, w)
    assert torch.equal(y, ops.MatMulInt4(x, w)) and ops.prefill_status(0) == 0
    want = x.double() @ ops.DequantizeInt4(w, torch.float32).double().t()
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 2.5e-3


def test_launches_of_different_runs_one_after_the_other(cuda):
    """Launches whose tiles are cut in different places leave flags of their own behind: none may pass for a later launch's.  New
    activations every time, so that a partial tile read too early is an old one; no host wait in between."""
    shapes = [("q4_k", 130, 4096, 4096), ("q8_0", 70, 512, 8192), ("int4", 300, 1024, 2048), ("q6_k", 65, 640, 16384), ("fp8", 257, 4096, 1024)]
    calls = [(m, *_weight(kind, n, k, cuda), k) for kind, m, n, k in shapes]
    g = torch.Generator(device=cuda).manual_seed(1)
    got = []
    for i in range(40):
        m, f, w, dt, k = calls[(i * i + i // 5) % len(calls)]
        x = torch.randn(m, k, generator=g, device=cuda).to(dt)
        got.append((f(x), x, w, dt))
    for y, x, w, dt in got:
        assert rel_l2(y.cpu().double().numpy(), (x.double() @ w.t()).cpu().numpy()) <= (1e-3 if dt == torch.float32 else 3e-3)
    assert ops.prefill_status(0) == 0


def _few(dev, seed, T, E, topk, N, K, dense):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, K, generator=g).to(dev, torch.bfloat16)
    ids = torch.rand(T, E, generator=g).topk(topk, -1).indices.to(dev)
    r = ops.MoERouteFromIDs(ids, torch.rand(T * topk, generator=g).to(dev), T, topk)
    if dense:
        w = torch.randn(E, N, K, generator=g).to(dev, torch.bfloat16)
        return lambda: ops.MoEGemm(x, w, r, r.weights, topk)
    codes, scale = synth.random_fp8_block(seed, E * N, K, device=dev)
    return lambda: ops.MoEGemmF8Block(x, codes.reshape(E, N, K), scale.reshape(E, N // 128, K // 128), 128, 128, r, r.weights, topk)


@pytest.mark.parametrize("dense", [False, True])
def test_grouped_calls_of_few_pairs_on_two_streams(cuda, dense):
    """Fewer than 256 pairs share nothing with other calls: flags, partial tiles and gathered tokens are the call's own."""
    calls = [_few(cuda, 1, 9, 24, 3, 512, 4096, dense), _few(cuda, 2, 31, 16, 8, 384, 2048, dense)]
    want = [f() for f in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(40):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(calls[i]())
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(want[i], y) for y in got[i])
    assert ops.prefill_status(0) == 0


def test_scratch_of_a_call_may_hold_anything(cuda):
    """Flags that look raised, and an epoch of any value, are cleared by the call that is given the memory."""
    import ctypes as C

    from light_b200 import _lib

    T, E, topk, N, K = 8, 12, 4, 256, 4096
    g = torch.Generator().manual_seed(4)
    x, w = torch.randn(T, K, generator=g).to(cuda, torch.bfloat16), torch.randn(E, N, K, generator=g).to(cuda, torch.bfloat16)
    ids = torch.rand(T, E, generator=g).topk(topk, -1).indices.to(cuda)
    r = ops.MoERouteFromIDs(ids, torch.ones(T * topk, device=cuda), T, topk)
    M = T * topk
    want = torch.einsum("mk,mnk->mn", x.double().repeat_interleave(topk, 0), w.double()[ids.reshape(-1)])
    counts, offsets = torch.empty(E, dtype=torch.int32, device=cuda), torch.empty(E + 1, dtype=torch.int32, device=cuda)
    L = _lib.lib()
    nbytes = L.light_b200_moe_scratch_bytes(M, K)
    for fill in (1, 0, -1, 0x7f7f7f7f):
        scratch = torch.full((nbytes // 4 + 64,), fill, dtype=torch.int32, device=cuda)
        out = torch.zeros(M, N, dtype=torch.bfloat16, device=cuda)
        a = _lib.MoeArgs(input=x.data_ptr(), weights=w.data_ptr(), sorted_pairs=r.sorted_pairs.data_ptr(), expert_ids=r.sorted_expts.data_ptr(),
                         counts=counts.data_ptr(), offsets=offsets.data_ptr(), topk_weights=0, out=out.data_ptr(), M=M, size_m=M, E=E, N=N, K=K, topk=topk,
                         row_per_pair=0, dtype=_lib.BF16)
        before = _lib.launch_count()
        _lib.check(L.light_b200_moe_gemm_scratch(C.byref(a), None, 0, 0, C.c_void_p(scratch.data_ptr()), nbytes, 0,
                                                 C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert _lib.launch_count() - before == 3      # offsets, token rows, the matmul: not the kernel for calls without scratch (2)
        assert rel_l2(out.cpu().double().numpy(), want.cpu().numpy()) <= 3e-3
        assert L.light_b200_moe_gemm_scratch(C.byref(a), None, 0, 0, C.c_void_p(scratch.data_ptr() + 64), nbytes, 0, None) == -4   # not on 256 bytes
        assert bool((scratch[nbytes // 4:] == fill).all())
    assert ops.prefill_status(0) == 0


@pytest.mark.parametrize("T,N", [(8, 512), (600, 4096)])   # few pairs in memory of the call's own; 4800 pairs with rows looked for
def test_grouped_calls_in_a_graph(cuda, T, N):
    E, topk, K = 16, 8, 1024
    g = torch.Generator().manual_seed(T)
    codes, scale = synth.random_fp8_block(2, E * N, K, device=cuda)
    codes, scale = codes.reshape(E, N, K), scale.reshape(E, N // 128, K // 128)
    x = torch.randn(T, K, generator=g).to(cuda, torch.bfloat16)
    logits = torch.randn(T, E, generator=g).to(cuda)

    def block():
        r = ops.MoERouteSigmoid(logits, None, topk)
        return ops.MoECombine(ops.MoEGemmF8Block(x, codes, scale, 128, 128, r, r.weights, topk), topk)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        block()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            y = block()
    for _ in range(3):                                      # other tokens and another routing at every replay
        x.copy_(torch.randn(T, K, generator=g)), logits.copy_(torch.randn(T, E, generator=g))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, block())
    assert ops.prefill_status(0) == 0
