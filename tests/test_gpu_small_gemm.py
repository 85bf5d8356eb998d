"""GEMM kernels of the shared MLP off the large-tile path: float32 register tiles."""
import pytest
import torch

from tests.helpers import randn

pytestmark = pytest.mark.gpu


def mlp_case(T, H, I, dtype):
    x = randn((T, H), 1, dtype, 0.5).cuda()
    wg = randn((I, H), 2, dtype, 1.0 / H**0.5).cuda()
    wu = randn((I, H), 3, dtype, 1.0 / H**0.5).cuda()
    wd = randn((H, I), 4, dtype, 1.0 / I**0.5).cuda()
    h = torch.nn.functional.silu(x.double() @ wg.double().t()) * (x.double() @ wu.double().t())
    return x, wg, wu, wd, h


@pytest.mark.parametrize(
    "T,H,I",
    [(1, 4, 4), (33, 36, 68), (31, 1028, 132), (256, 256, 1024), (300, 192, 1500), (1030, 512, 2300)],
)
def test_mlp_float32_tiles(T, H, I):
    """32 x 32 tiles with K split over thread groups, 64 x 64 and 128-row tiles, remainders in every dimension."""
    from flash_moe_b200.ops.flash_mlp import flash_mlp_add

    x, wg, wu, wd, h = mlp_case(T, H, I, torch.float32)
    addend = randn((T, H), 5, torch.float32).cuda()
    want = h @ wd.double().t() + addend.double()
    got = flash_mlp_add(x, wg, wu, wd, addend)
    assert (got.double() - want).norm() <= 2e-6 * want.norm()
    assert torch.equal(got, flash_mlp_add(x, wg, wu, wd, addend))
