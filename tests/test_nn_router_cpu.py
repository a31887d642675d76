"""What a program puts in the place of a sparse block's route or of its gate's forward is called, however it is put there: the native form of the router's matmul stands
in for the plain ones alone.  (The native function is a stand-in that fails the test, so that no GPU is needed.)"""
import types

import pytest
import torch

from light_b200 import nn, ops

H, E = 1024, 8


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


@pytest.mark.parametrize("T,E,K,f32,bf16", [(1, 64, 2048, True, True), (1, 256, 2048, False, True), (1, 256, 1024, True, True), (1, 64, 7168, False, False), (1, 256, 7168, False, False),
                                            (8, 256, 7168, True, True), (77, 128, 2048, True, True), (17, 64, 256, True, True), (16, 64, 256, False, True), (512, 256, 768, False, True),
                                            (1024, 8, 1280, True, True), (1500, 8, 1280, False, True), (4096, 64, 1024, True, True), (4097, 64, 4096, False, True), (4096, 256, 7168, False, True),
                                            (4096, 4, 512, False, False), (8192, 8, 1280, False, False), (4096, 40, 256, False, False), (16384, 8, 2560, False, True)])
def test_sizes_where_it_is_the_faster_one(T, E, K, f32, bf16):
    assert nn._router_is_faster(T, E, K, True) == f32 and nn._router_is_faster(T, E, K, False) == bf16


def test_a_size_where_the_library_is(native):
    g = torch.Generator().manual_seed(2)
    moe = nn.SparseMoE(nn.Linear(64, E, W=torch.randn(E, 64, generator=g)), TopK=2, Router=lambda logits: logits)
    moe.run_experts = lambda flat, route: route.sum() + flat
    x = torch.randn(3, 64, generator=g)
    assert torch.equal(moe.forward(x), (x @ moe.Gate.W.t()).sum() + x) and not native
