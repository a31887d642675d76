"""Tuning switches of the tensor-memory matmul at values that are no multiple of what it works in: each is read once, so in a process of its own."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

RUN = """
import json
import torch
from light_b200 import ops, synth
dev = torch.device("cuda", 0)
g = torch.Generator().manual_seed(1)
err = []
E, N, K, topk, T = 3, 256, 512, 2, 300                    # experts of 200 tokens in the mean, bf16 and f32
codes, scale = synth.random_fp8_block(2, E * N, K, device=dev)
w = (codes.view(torch.float8_e4m3fn).double() * scale.double().repeat_interleave(128, 0).repeat_interleave(128, 1)).reshape(E, N, K)
ids = torch.randint(0, E, (T, topk), generator=g).to(dev)
one = torch.ones(T * topk, device=dev)
for dt in (torch.bfloat16, torch.float32):
    x = torch.randn(T, K, generator=g).to(dev, dt)
    y = ops.MoEGemmF8Block(x, codes.reshape(E, N, K), scale.reshape(E, N // 128, K // 128), 128, 128, ops.MoERouteFromIDs(ids, one, T, topk), None, topk)
    want = torch.einsum("mk,mnk->mn", x.double().repeat_interleave(topk, 0), w[ids.reshape(-1)])
    err.append(float((y.double() - want).norm() / want.norm()))
q = ops.QTensor(synth.gaussian_weight(3, ops.Q4_K, 300, 1024, device=dev).reshape(-1), ops.Q4_K, (300, 1024))
x = torch.randn(333, 1024, generator=g).to(dev)
want = x.double() @ ops.Dequantize(q).double().t()
err.append(float((ops.MatMulQ(x, q).double() - want).norm() / want.norm()))
print(json.dumps([err, ops.prefill_status(0)]))
"""


@pytest.mark.parametrize("name,value", [("NT", 100), ("NT", 8), ("NT", 40), ("CG", 3), ("CG", 2), ("RUN", 0), ("WMIN", 0), ("WMIN", 1 << 30)])
def test_any_value(cuda, name, value):
    """bf16 operands and output 2^-8 each at most (FP8), operands of 11 bits (f32 tokens, GGUF)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RUN], cwd=root, env=dict(os.environ, **{"LIGHT_B200_TMEM_" + name: str(value)}), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    (fp8, fp8_f32, q4), status = json.loads(r.stdout.splitlines()[-1])
    assert status == 0 and fp8 <= 2.0**-8 and fp8_f32 <= 2.0**-10 and q4 <= 2.0**-10, (fp8, fp8_f32, q4)
