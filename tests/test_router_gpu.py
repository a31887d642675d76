"""The router's matmul: f32 in effect.  Bound: f32 products summed in blocks of 32 and then in f32: 2^-24 of the sum of magnitudes per addition, of which K / 32 follow
one another, and far below that on average: 2e-6 of sum |x w| with room."""
import pytest
import torch

from light_b200 import nn, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,E,K", [(1, 8, 8), (16, 256, 7168), (17, 60, 2048), (77, 128, 2040), (333, 33, 520), (1024, 256, 1024), (2400, 250, 264)])
def test_against_64_bits(cuda, dtype, T, E, K):
    g = torch.Generator(device=cuda).manual_seed(T + E)
    x, w = torch.randn(T, K, generator=g, device=cuda).to(dtype), torch.randn(E, K, generator=g, device=cuda)
    w[E // 2] *= 1e20
    y = ops.RouterLogits(x, w)
    assert torch.equal(y, ops.RouterLogits(x, w))
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert float(((y - want).abs() / size).max()) <= 2e-6
    # no further off than the library's f32 matmul, but for chance
    lib = x.float() @ w.t()
    assert float(((y - want) / size).norm()) <= 1.25 * float(((lib - want) / size).norm()) + 1e-9


def test_infinities_and_large_values(cuda):
    x, w = torch.ones(20, 64, device=cuda), torch.ones(40, 64, device=cuda)
    w[3, 5], w[4, 6], w[5, 7] = 3.4e38, float("inf"), float("nan")
    x[7, 0], x[8, 1] = float("-inf"), float("nan")
    y = ops.RouterLogits(x, w)
    want = x @ w.t()
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
    ok = torch.isfinite(want)
    assert torch.allclose(y[ok], want[ok], rtol=1e-6)


def test_sparse_block_takes_the_same_route(cuda):
    """nn.SparseMoE chooses by these logits as by the library's; a gate that requires a gradient goes the library's way."""
    g = torch.Generator(device=cuda).manual_seed(1)
    H, I, E, T, k = 256, 128, 16, 40, 2
    gate = nn.Linear(H, E, W=torch.randn(E, H, generator=g, device=cuda) / 16)
    gu, dn = (torch.randn(E, n, m, generator=g, device=cuda).bfloat16() / 16 for n, m in ((2 * I, H), (H, I)))
    x = torch.randn(T, H, generator=g, device=cuda).bfloat16()
    seen = []
    moe = nn.SparseMoE(gate, gu, dn, TopK=k, RouterF32=True, Router=lambda l: seen.append(l) or ops.MoERouteSigmoid(l, None, k))
    y = moe.forward(x)
    gate.W.requires_grad_()
    z = moe.forward(x)
    assert torch.allclose(seen[0], seen[1], rtol=1e-5, atol=1e-5) and seen[1].requires_grad and not seen[0].requires_grad
    assert torch.equal(y, z)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_operands_that_are_not_contiguous(cuda, dtype):
    g = torch.Generator(device=cuda).manual_seed(2)
    x, w = torch.randn(512, 256, generator=g, device=cuda).to(dtype), torch.randn(512, 256, generator=g, device=cuda)
    xs, ws = x.t().contiguous().t(), w.t().contiguous().t()
    want = ops.RouterLogits(x, w)
    assert torch.equal(ops.RouterLogits(xs, ws), want) and torch.equal(ops.RouterLogits(x, ws), want) and torch.equal(ops.RouterLogits(xs, w), want)


def test_a_weight_on_the_host(cuda):
    with pytest.raises(ValueError, match="router_logits: x on cuda:0 but w on cpu"):
        ops.RouterLogits(torch.zeros(4, 8, device=cuda), torch.zeros(4, 8))


def _block(cuda):
    g = torch.Generator(device=cuda).manual_seed(4)
    moe = nn.SparseMoE(nn.Linear(64, 8, W=torch.randn(8, 64, generator=g, device=cuda)), TopK=2, Router=lambda logits: logits)
    moe.run_experts = lambda flat, route: torch.cat([route] * 8, 1)  # (the block's output is its logits, eight times)
    return moe, torch.randn(40, 64, generator=g, device=cuda), g


def test_tangents_reach_the_router(cuda):
    import torch.autograd.forward_ad as fwd

    moe, x, g = _block(cuda)
    t = torch.randn(40, 64, generator=g, device=cuda)
    with fwd.dual_level():
        value, tangent = fwd.unpack_dual(moe.forward(fwd.make_dual(x, t)))
    assert tangent is not None and torch.equal(tangent[:, :8], t @ moe.Gate.W.t()) and torch.equal(value[:, :8], x @ moe.Gate.W.t())


def test_function_transforms(cuda):
    moe, x, _ = _block(cuda)
    want = torch.cat([x @ moe.Gate.W.t()] * 8, 1)
    assert torch.allclose(torch.vmap(lambda v: moe.forward(v[None])[0])(x), want, rtol=1e-5, atol=1e-5)
    value, tangent = torch.func.jvp(moe.forward, (x,), (x,))
    assert torch.allclose(value, want) and torch.allclose(tangent, want)


def test_modes_see_the_matmul(cuda):
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    seen = []

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", ""))
            return func(*args, **(kwargs or {}))

    moe, x, _ = _block(cuda)
    for mode, name in ((Dispatch, "mm"), (Function, "matmul")):
        seen.clear()
        with mode():
            moe.forward(x)
        assert any(name in s for s in seen), seen


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("of_x,of_w", [(0, -100), (0, -112), (0, -120), (-20, -100), (-112, 0), (-120, 0), (-130, 8), (-60, -60), (60, -118), (60, 40)])
@pytest.mark.parametrize("T", [5, 70])
def test_powers_of_two(cuda, dtype, of_x, of_w, T):
    """Small operands keep their bits, down to subnormal ones; a sum is within the bound above, and an output's own last place where that is subnormal."""
    g = torch.Generator(device=cuda).manual_seed(T)
    x, w = (torch.randn(T, 512, generator=g, device=cuda) * 2.0**of_x).to(dtype), torch.randn(72, 512, generator=g, device=cuda) * 2.0**of_w
    y = ops.RouterLogits(x, w).double()
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert float(want.abs().max()) > 0 and bool(((y - want).abs() <= 2e-6 * size + 2.0**-149).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,E,K", [(16, 513, 7168), (17, 33, 256), (64, 512, 2048), (65, 512, 2048), (1024, 64, 2040), (1025, 64, 1024), (8192, 32, 256), (8193, 32, 256), (1, 1, 8)])
def test_both_sides_of_the_tiles(cuda, dtype, T, E, K):
    test_against_64_bits(cuda, dtype, T, E, K)
