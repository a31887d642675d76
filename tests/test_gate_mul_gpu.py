"""The gated activation's quotient where exp overflows, at infinities and beside them, and row lengths on both sides of the divisions that place an element.

Bound: one rounding each of exp, the sum, the quotient (one ulp) and the product, exp itself two ulp: 6e-7 of the value."""
import pytest
import torch

from light_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,I", [(1, 8), (3, 264), (257, 1000), (5, 70000)])
def test_gate_mul(cuda, M, I):
    g = torch.Generator(device=cuda).manual_seed(I)
    h = torch.randn(M, 2 * I, generator=g, device=cuda) * 30
    y = ops.MoEGateMul(h)
    x = h[:, :I].double()
    want = x / (1 + torch.exp(-x)) * h[:, I:].double()
    # (where exp passes f32's range the quotient is zero: it would be 89 / 2^128 = 2.7e-37 at most)
    assert bool(((y - want).abs() <= 6e-7 * want.abs() + 3e-37 * (1 + h[:, I:].double().abs())).all())


def test_extremes(cuda):
    v = torch.tensor([0.0, -0.0, 1e-30, -1e-30, 87.0, -87.0, -88.0, -88.6, -88.8, -89.0, -103.9, -1000.0, 3e38, -3e38, float("inf"), float("-inf"), float("nan"), 1.0, -1.0, 20.0, -20.0,
                      50.0, -50.0, -127.5], device=cuda)
    y = ops.MoEGateMul(torch.cat([v, torch.ones_like(v)])[None])[0]
    want = (v / (1 + torch.exp(-v)))
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
    ok = torch.isfinite(want)
    assert bool(((y - want)[ok].abs() <= 4e-7 * want[ok].abs() + 2.0**-148).all())


def test_bits_of_the_division(cuda):
    """f32 gates of every exponent and both signs, zeros and infinities among them (every 1021st bit pattern): the bits that a correctly rounded division gives."""
    bits = torch.arange(-2**31, 2**31, 1021, device=cuda, dtype=torch.int64)
    v = torch.cat([bits.to(torch.int32).view(torch.float32), torch.tensor([0.0, -0.0, float("inf"), float("-inf")], device=cuda)])
    v = torch.cat([v, v.new_full((-v.numel() % 8,), -0.0)]).reshape(-1, 8)
    y, want = ops.MoEGateMul(torch.cat([v, torch.ones_like(v)], 1)), v / (1 + torch.exp(-v))
    assert torch.equal(torch.isnan(y), torch.isnan(want))
    number = ~torch.isnan(want)
    assert torch.equal(y.view(torch.int32)[number], want.view(torch.int32)[number])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_zeros_keep_their_sign(cuda, dtype):
    v = torch.tensor([0.0, -0.0] * 4, device=cuda, dtype=dtype)
    for u in (1.0, -1.0):
        y = ops.MoEGateMul(torch.cat([v, torch.full_like(v, u)])[None])[0]
        assert torch.equal(torch.signbit(y), torch.signbit(v * u)) and not y.any()
