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
