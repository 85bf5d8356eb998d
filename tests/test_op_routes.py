"""Which calls take which route through the Python layer, on the CPU with the library calls replaced."""

import pytest
import torch
from torch.autograd import forward_ad

from flash_moe_b200.ops import flash_expert, flash_mlp, flash_router


def expert(x):
    return flash_expert.flash_expert_func(x, x, x, torch.zeros(2, 1, dtype=torch.int64), torch.ones(2, 1))


def mlp(x):
    return flash_mlp.flash_mlp_func(x, x, x, x)


def router(x):
    return flash_router.flash_router_func(x[None], 3, 1)[0][0]


OPS = [expert, mlp, router]


@pytest.fixture(autouse=True)
def ops_without_a_gpu(monkeypatch):
    """Each op doubles its first argument, out of autograd's sight as the library does."""
    monkeypatch.setattr(flash_expert, "_expert_forward", lambda x, *a, **k: torch.from_numpy(2 * x.detach().numpy()))
    monkeypatch.setattr(flash_mlp, "_mlp_forward", lambda x, *a, **k: torch.from_numpy(2 * x.detach().numpy()))
    monkeypatch.setattr(flash_router, "_router_forward",
                        lambda x, *a, **k: (torch.from_numpy(2 * x.detach().numpy()), torch.zeros(2, 1, dtype=torch.int64)))


@pytest.mark.parametrize("op", OPS)
def test_tangents_are_refused_not_dropped(op):
    with torch.no_grad(), forward_ad.dual_level():
        dual = forward_ad.make_dual(torch.ones(2, 3), torch.ones(2, 3))
        with pytest.raises(RuntimeError, match="jvp"):
            op(dual)
    with torch.no_grad():
        assert torch.equal(op(torch.ones(2, 3)), torch.full((2, 3), 2.0))


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning", "ignore::DeprecationWarning")
@pytest.mark.parametrize("op", OPS)
def test_a_trace_records_the_op(op):
    with torch.no_grad():
        traced = torch.jit.trace(op, (torch.ones(2, 3),), check_trace=False)
        assert torch.equal(traced(torch.full((2, 3), 3.0)), torch.full((2, 3), 6.0))


def wrap_forward(layer):
    inner = layer.router_gate.forward
    layer.router_gate.forward = lambda x: inner(x)


def hook(layer):
    layer.router_gate.register_forward_hook(lambda *a: None)


@pytest.fixture
def taken(monkeypatch):
    """(layer, call): which of the two differentiable forms of the layer a call takes."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig
    from flash_moe_b200.modules import training

    layer = FlashMoE(FlashMoEConfig(16, 16, "silu", 16, 2))
    route = []

    def node(x, *a):
        route.append("node")
        return x, x.new_zeros(x.shape[0], 8), None, None

    monkeypatch.setattr(training.LayerTrainingStep, "apply", node)
    monkeypatch.setattr(layer, "_forward_chain", lambda *a: route.append("chain"))

    def call():
        layer._forward_differentiable(torch.ones(1, 4, 16))
        return route.pop()

    return layer, call


def test_a_plain_layer_trains_in_one_node(taken):
    assert taken[1]() == "node"


@pytest.mark.parametrize("change", [wrap_forward, hook])
def test_a_router_gate_that_does_more_is_called(taken, change):
    layer, call = taken
    change(layer)
    assert call() == "chain"


def test_global_hooks_see_the_router_gate(taken):
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert taken[1]() == "chain"
    finally:
        handle.remove()
    assert taken[1]() == "node"
