"""The native host path (light_b200._host) as a Python extension: what goes wrong inside it is a Python exception or None, as from the
Python code that does the same.  Fake tensors say that they are on a GPU and have no storage, so that no GPU is needed."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEAD = f"""
import sys
sys.path.insert(0, {ROOT!r})
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from light_b200 import ops
"""


def _child(code):
    r = subprocess.run([sys.executable, "-c", HEAD + code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "CASE OK" in r.stdout, (r.returncode, r.stdout + r.stderr[-2000:])


def test_what_torch_throws_is_a_python_exception():
    _child("""
with FakeTensorMode():
    x = torch.empty(4, 256, device="cuda")
    h, c = torch.empty(4, 64, device="cuda"), torch.empty(64, 128, dtype=torch.uint8, device="cuda")
    s, i32 = torch.empty(64, 4, device="cuda"), torch.empty(64, 32, dtype=torch.int32, device="cuda")
    i64 = torch.empty(8, dtype=torch.int64, device="cuda")
    q, kb = torch.empty(1, 4, 1, 64, device="cuda"), torch.empty(1, 2, 16, 64, device="cuda")
    ops._host.set_workspace(0, 1 << 40)
    experts = torch.empty(2, 64, 256, dtype=torch.uint8, device="cuda")
    calls = {
        "moe_gemm": lambda: ops._host.moe_gemm(x, experts, torch.empty(2, 64, 4, device="cuda"), 1, 64, -1, 2, 64, 256, i64[:4], i64[:4], None, 1),
        "gate_mul": lambda: ops._host.gate_mul(h, False),
        "combine": lambda: ops._host.combine(h, 2),
        "linear_q": lambda: ops._host.linear_q(x[:1], torch.empty(16 * 144, dtype=torch.uint8, device="cuda"), ops.Q4_K, 16, 256),
        "linear_int4": lambda: ops._host.linear_int4(x[:1], i32, s, s, 64),
        "linear_f8": lambda: ops._host.linear_f8(x[:1], torch.empty(64, 256, dtype=torch.uint8, device="cuda"), s, 1, 64),
        "moe_route": lambda: ops._host.moe_route(h, None, 2, False, True),
        "decode_attention": lambda: ops._host.decode_attention(q, kb, kb, i64[:1], 0.125, 0, None, None, 0.0),
        "public": lambda: ops.MoEGateMul(h),
    }
    for name, call in calls.items():
        try:
            call()
        except RuntimeError:
            continue
        raise SystemExit(name + ": no exception")
print("CASE OK")
""")


def test_numbers_beyond_64_bits_are_not_the_common_form():
    """None, and no Python error left behind (which made it a SystemError)."""
    import pytest
    import torch

    from light_b200 import ops

    x, u8, big = torch.zeros(1, 256), torch.zeros(144, dtype=torch.uint8), 2**70
    assert ops._host.linear_q(x, u8, ops.Q4_K, big, 256) is None
    assert ops._host.linear_int4(x, x, x, x, big) is None
    assert ops._host.linear_f8(x, x, x, -big, 1) is None
    assert ops._host.combine(x, big) is None
    assert ops._host.moe_route(x, None, big, True, True) is None
    assert ops._host.decode_attention(x, x, x, x, 1.0, big, None, None, 0.0) is None
    with pytest.raises(ValueError):
        ops._host.set_workspace(64, 1)
