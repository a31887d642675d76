"""What an operator hands to the library: the addresses of contiguous copies that live until the call returns, two copies never at one address, and only of tensors on
the device that the call runs on.  The library is a stand-in that reads the operands at the addresses it is given, as the kernel would, so that no GPU is needed."""
import ctypes as C

import pytest
import torch

from light_b200 import ops


def _read(address, like):
    """What lies at an address, as a contiguous tensor of this shape and type."""
    n = like.numel() * like.element_size()
    raw = torch.frombuffer(bytearray(C.string_at(getattr(address, "value", address), n)), dtype=torch.uint8)
    return raw.view(like.dtype).reshape(like.shape)


class Library:
    """Every entry point notes the operands it finds at the given arguments; sizes that it is asked for are those given here."""

    def __init__(self, operands, sizes=()):
        self.operands, self.sizes, self.calls = operands, dict(sizes), []

    def __getattr__(self, name):
        def call(*args):
            if name in self.sizes:
                return self.sizes[name]
            self.calls.append([_read(args[i], t) for i, t in self.operands])
            return 0
        return call


@pytest.fixture
def library(monkeypatch):
    def install(operands, **sizes):
        lib = Library(operands, sizes)
        monkeypatch.setattr(ops._lib, "lib", lambda: lib)
        monkeypatch.setattr(ops, "_dev", lambda t, what: 0)
        monkeypatch.setattr(ops, "_stream", lambda dev: C.c_void_p(0))
        monkeypatch.setattr(ops, "ensure_workspace", lambda dev, n: None)
        return lib
    return install


def _views(*shapes, dtype=torch.float32):
    """Tensors that are not contiguous, of one size each, so that a copy fits where the one before was freed."""
    return [torch.randn(*s, generator=torch.Generator().manual_seed(i)).to(dtype).t().contiguous().t() for i, s in enumerate(shapes)]


def test_router_logits(library):
    x, w = _views((512, 256), (512, 256))
    assert not x.is_contiguous() and not w.is_contiguous()
    lib = library([(0, x), (2, w)])
    ops.RouterLogits(x, w)
    (got_x, got_w), = lib.calls
    assert torch.equal(got_x, x) and torch.equal(got_w, w)


def test_router_logits_of_a_weight_elsewhere(library):
    lib = library([])
    with pytest.raises(ValueError, match="router_logits: x on cpu but w on meta"):
        ops.RouterLogits(torch.zeros(4, 8), torch.zeros(4, 8, device="meta"))
    assert not lib.calls


def _i32(*shapes):
    return [v.view(torch.int32) for v in _views(*shapes)]


def _bf16(*shapes):
    return _views(*shapes, dtype=torch.bfloat16)


def _spaced(*values):  # one-dimensional, every second element of its memory
    return [torch.stack([v, v], 1)[:, 0] for v in values]


def _cases():
    S = (256, 256)
    yield "gated_linear", lambda: (lambda x, a, b: ([(0, x), (1, a), (2, b)], lambda: ops.GatedLinear(x, a, b)))(*_spaced(torch.randn(256).bfloat16()), *_bf16(S, S))
    yield "w8a8", lambda: (lambda x, q, s: ([(0, x), (1, q), (2, s)], lambda: ops.MatMulW8A8(x, q, s)))(*_views(S), *_views(S, dtype=torch.int8), *_spaced(torch.randn(256)))
    yield "int4_repack", lambda: (lambda q, z, s: ([(0, q), (1, z), (2, s)], lambda: ops.Int4FromCheckpoint(q, z, s, 8, "gptq")))(*_i32((32, 256), (32, 32)), *_views((32, 256)))
    yield "int4_dequant", lambda: (lambda c, s, z: ([(0, c), (1, s), (2, z)], lambda: ops.DequantizeInt4(ops.Int4(c, s, z, 8), torch.float32)))(*_i32((256, 32)), *_views((256, 32), (256, 32)))
    yield "gather_columns", lambda: (lambda x, i: ([(0, x), (1, i)], lambda: ops.GatherColumns(x, i)))(*_views((2, 256)), *_spaced(torch.randperm(256)))
    yield "int4", lambda: (lambda x, c, s, z: ([(0, x), (1, c), (2, s), (3, z)], lambda: ops.MatMulInt4(x, ops.Int4(c, s, z, 8))))(
        *_views((32, 256)), *_i32((256, 32)), *_views((256, 32), (256, 32)))
    yield "fp8_dequant", lambda: (lambda w, s: ([(0, w), (1, s)], lambda: ops.DequantizeF8Block(w, s, 1, 4, torch.float32)))(*_views((64, 256), dtype=torch.uint8), *_views((64, 64)))
    yield "fp8", lambda: (lambda x, w, s: ([(0, x), (1, w), (2, s)], lambda: ops.MatMulF8Block(x, w, s, 1, 4)))(
        *_views((64, 256)), *_views((256, 256), dtype=torch.uint8), *_views((256, 64)))
    yield "route_topk", lambda: (lambda p: ([(0, p)], lambda: ops.MoERoute(p, 2, True)))(*_views((32, 64)))
    yield "route_deepseek", lambda: (lambda p, b: ([(0, p), (1, b)], lambda: ops.MoERouteDeepseek(p, b, 2)))(*_views((2, 64)), *_spaced(torch.randn(64)))
    yield "route_sigmoid", lambda: (lambda p, b: ([(0, p), (1, b)], lambda: ops.MoERouteSigmoid(p, b, 2)))(*_views((2, 64)), *_spaced(torch.randn(64)))
    yield "sort_pairs", lambda: (lambda i: ([(0, i)], lambda: ops.MoESortPairs(i, 8)))(*_spaced(torch.randint(0, 8, (64,))))
    yield "combine", lambda: (lambda p: ([(0, p)], lambda: ops.MoECombine(p, 2)))(*_views((32, 64)))
    yield "combine_weighted", lambda: (lambda r, i, w: ([(0, r), (1, i), (2, w)], lambda: ops.MoECombineWeighted(r, i, w, 32, 2)))(
        *_views((64, 64)), *_spaced(torch.randperm(64), torch.randn(64)))
    yield "gate_mul", lambda: (lambda h: ([(0, h)], lambda: ops.MoEGateMul(h)))(*_views((32, 64)))
    yield "kv_append", lambda: (lambda k, v, b: ([(0, k), (1, v)], lambda: ops.KVAppend(b, b.clone(), k, v, torch.zeros(1, dtype=torch.int64))))(
        *(t[None, :, None] for t in _views(S, S)), torch.zeros(1, 256, 4, 256))
    yield "rope", lambda: (lambda x, p: ([(0, x), (1, p)], lambda: ops.RoPE(x, p, 1e4)))(*_views((64, 2)), *_spaced(torch.arange(64)))


@pytest.mark.parametrize("make", [pytest.param(m, id=n) for n, m in _cases()])
def test_operators(library, make):
    operands, run = make()
    assert any(not t.is_contiguous() for _, t in operands)
    first = library(operands, light_b200_matmul_q_workspace_bytes=0)
    try:
        run()
    except IndexError:
        pass  # (the sort behind a router takes other arguments)
    for (_, want), got in zip(operands, first.calls[0]):
        assert torch.equal(got, want)


def test_grouped_matmul(library, monkeypatch):
    """The pairs, their experts and weights of a grouped call, and its own memory, which is made after they are."""
    M, E, N, K = 64, 4, 16, 256
    pairs, expts, tw = _spaced(torch.randperm(M), torch.randint(0, E, (M,)).sort().values, torch.randn(M))
    x, = _bf16((M, K))
    w = torch.randn(E, N, K).bfloat16()
    lib = library([], light_b200_moe_scratch_bytes=8 * M)
    seen = []
    lib.light_b200_moe_gemm_scratch = lambda a, *rest: seen.append([_read(p, t) for p, t in ((a._obj.input, x), (a._obj.sorted_pairs, pairs), (a._obj.expert_ids, expts),
                                                                                              (a._obj.topk_weights, tw))]) or 0
    ops.MoEGemm(x, w, ops.MoERouting(None, tw, pairs, expts), tw, 1)
    for got, want in zip(seen[0], (x, pairs, expts, tw)):
        assert torch.equal(got, want)
