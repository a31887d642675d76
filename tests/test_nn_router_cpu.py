"""What a program puts in the place of a sparse block's route or of its gate's forward is called, however it is put there: the native form of the router's matmul stands
in for the plain ones alone.  (The native function is a stand-in that fails the test, so that no GPU is needed.)"""
import types

import pytest
import torch

from light_b200 import nn, ops

H, E = 32, 8


def _block(cls=nn.SparseMoE, gate=None):
    g = torch.Generator().manual_seed(1)
    moe = cls(gate or nn.Linear(H, E, W=torch.randn(E, H, generator=g)), TopK=2, Router=lambda logits: logits)
    moe.run_experts = lambda flat, route: route.sum() + flat
    return moe, torch.randn(5, H, generator=g)


@pytest.fixture
def native(monkeypatch):
    calls = []
    monkeypatch.setattr(ops._host, "router_logits", lambda x, w: calls.append(1) or x @ w.t())
    return calls


def test_a_plain_block_takes_the_native_form(native):
    moe, x = _block()
    want = (x @ moe.Gate.W.t()).sum() + x
    assert torch.equal(moe.forward(x), want) and native


class Doubled(nn.Linear):
    def forward(self, x):
        return 2 * super().forward(x)


class Routed(nn.SparseMoE):
    def route(self, gate_in):
        return 2 * super().route(gate_in)


def _gate_on_the_object():
    moe, x = _block()
    plain = moe.Gate.forward
    moe.Gate.forward = lambda v: 2 * plain(v)
    return moe, x


def _gate_on_the_object_as_a_method():
    moe, x = _block()
    moe.Gate.forward = types.MethodType(lambda self, v: 2 * nn.Linear.forward(self, v), moe.Gate)
    return moe, x


def _route_on_the_object():
    moe, x = _block()
    plain = moe.route
    moe.route = lambda v: 2 * plain(v)
    return moe, x


@pytest.mark.parametrize("make", [_gate_on_the_object, _gate_on_the_object_as_a_method, _route_on_the_object, lambda: _block(Routed),
                                  lambda: _block(gate=Doubled(H, E, W=torch.randn(E, H, generator=torch.Generator().manual_seed(1))))])
def test_what_a_program_puts_in_its_place(native, make):
    moe, x = make()
    assert torch.equal(moe.forward(x), 2 * (x @ moe.Gate.W.t()).sum() + x) and not native


@pytest.mark.parametrize("cls,name", [(nn.Linear, "forward"), (nn.SparseMoE, "route")])
def test_on_the_class(native, monkeypatch, cls, name):
    plain = getattr(cls, name)
    monkeypatch.setattr(cls, name, lambda self, v: 2 * plain(self, v))
    moe, x = _block()
    assert torch.equal(moe.forward(x), 2 * (x @ moe.Gate.W.t()).sum() + x) and not native
