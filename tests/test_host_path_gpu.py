"""The native host path of the hot operators under conditions that a server has to survive."""
import pytest
import torch

from light_b200 import ops, synth
from light_b200.nn import Linear

pytestmark = pytest.mark.gpu


def _calls(dev):
    """Calls whose outputs are 64 MB or more each."""
    M, K, N = 4096, 256, 4096
    ops.ensure_workspace(0, 256 << 20)
    x = torch.ones(M, K, device=dev)
    lin = Linear(K, N, W=ops.QTensor(synth.gaussian_weight(1, ops.Q4_K, N, K, device=dev).reshape(-1), ops.Q4_K, (N, K)))
    w4 = ops.Int4(torch.zeros(2 * N, K // 8, dtype=torch.int32, device=dev), torch.ones(2 * N, 2, device=dev), torch.zeros(2 * N, 2, device=dev), 128)
    codes, scale = synth.random_fp8_block(1, 2 * N, K, device=dev)
    h = torch.ones(4096, 8192, device=dev)
    ids = torch.zeros(M, 1, dtype=torch.int64, device=dev)
    r = ops.MoERouteFromIDs(ids, torch.ones(M, device=dev), M, 1)
    b = x.bfloat16()
    return {"linear_q": lambda: lin.forward(x), "linear_int4": lambda: ops.MatMulInt4(b, w4), "linear_f8": lambda: ops.MatMulF8Block(b, codes, scale, 128, 128),
            "gate_mul": lambda: ops.MoEGateMul(h), "combine": lambda: ops.MoECombine(h, 2),
            "moe_gemm": lambda: ops.MoEGemmF8Block(b, codes.reshape(1, 2 * N, K), scale.reshape(1, 2 * N // 128, K // 128), 128, 128, r, None, 1)}


@pytest.mark.parametrize("name", ["linear_q", "linear_int4", "linear_f8", "gate_mul", "combine", "moe_gemm"])
def test_no_memory_for_the_output_is_an_exception(cuda, name):
    """torch.OutOfMemoryError, which a server can catch, and the same call runs once there is memory."""
    call = _calls(cuda)[name]
    want = call().clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction(1e-4)   # the caching allocator refuses to grow: nothing is exhausted
    try:
        kept = []                                       # (until what other tests left in the allocator's cache is used up)
        with pytest.raises(torch.OutOfMemoryError):
            for _ in range(torch.cuda.memory_reserved() // (64 << 20) + 2):
                kept.append(call())
    finally:
        kept.clear()
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(call(), want)


def test_grouped_fp8_scale_of_another_shape_is_refused(cuda):
    """A scale with the right number of elements and another shape: refused, as before the call went through the native path."""
    E, N, K, bR, bC, M = 2, 256, 512, 64, 128, 8
    codes, scale = synth.random_fp8_block(1, E * N, K, bR, bC, device=cuda)
    codes, scale = codes.reshape(E, N, K), scale.reshape(E, N // bR, K // bC)
    x = torch.randn(M, K, device=cuda).bfloat16()
    r = ops.MoERouteFromIDs(torch.arange(M, device=cuda).reshape(M, 1) % E, torch.ones(M, device=cuda), M, 1)
    good = ops.MoEGemmF8Block(x, codes, scale, bR, bC, r, None, 1)
    assert torch.isfinite(good.float()).all()
    s2 = torch.cat([scale, scale], 1)[:, :2, :].contiguous()      # (E, 2, 4) for blocks of (128, 128)
    for bad, br, bc in ((s2.transpose(1, 2).contiguous(), 128, 128), (s2.reshape(E, 8, 1), 128, 128), (scale.reshape(-1), bR, bC), (scale[:, None], bR, bC)):
        with pytest.raises(ValueError):
            ops.MoEGemmF8Block(x, codes, bad, br, bc, r, None, 1)


def test_linear_whose_weight_has_another_shape_is_refused(cuda):
    """A weight that was put into the layer without set_weight / set_int4 and is not (out, in): the general path's error."""
    x = torch.randn(4, 256, device=cuda)
    q = ops.QTensor(synth.gaussian_weight(1, ops.Q8_0, 256, 512, device=cuda).reshape(-1), ops.Q8_0, (256, 512))
    with pytest.raises(ValueError, match="inner dim mismatch"):
        Linear(256, 512, W=q).forward(x)                       # (in, out): as many blocks
    w4 = ops.Int4(torch.zeros(512, 32, dtype=torch.int32, device=cuda), torch.ones(512, 2, device=cuda), torch.zeros(512, 2, device=cuda), 128)
    codes, scale = synth.random_fp8_block(1, 512, 256, device=cuda)
    for layer in (Linear(256, 384, W4=w4), Linear(256, 384, W=codes.view(torch.float8_e4m3fn), WBlockScale=scale, WBlock=(128, 128))):
        with pytest.raises(RuntimeError):
            layer.forward(x.bfloat16())
