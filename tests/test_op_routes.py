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
