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
    [(1, 4, 4), (33, 36, 68), (31, 1028, 132), (256, 256, 1024), (300, 192, 1500), (1030, 512, 2300), (100, 2052, 4100),
     (16, 200, 1028), (700, 516, 1500)],
)
def test_mlp_float32_tiles(T, H, I):
    """32 x 32 tiles with K split over thread groups and clusters of 2 and 4, 64 x 64 and 128-row tiles, remainders in every
    dimension, a cluster with fewer k-steps than CTAs."""
    from flash_moe_b200.ops.flash_mlp import flash_mlp_add

    x, wg, wu, wd, h = mlp_case(T, H, I, torch.float32)
    addend = randn((T, H), 5, torch.float32).cuda()
    want = h @ wd.double().t() + addend.double()
    got = flash_mlp_add(x, wg, wu, wd, addend)
    assert (got.double() - want).norm() <= 2e-6 * want.norm()
    assert torch.equal(got, flash_mlp_add(x, wg, wu, wd, addend))


@pytest.mark.parametrize(
    "T,H,I",
    [(1, 8, 8), (16, 1024, 4096), (17, 72, 200), (64, 2048, 1024), (129, 128, 8), (257, 256, 1000), (500, 1000, 520),
     (1100, 512, 2000)],
)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_mlp_few_tokens(T, H, I, dtype):
    """Weight-row tiles of 64 and 128 rows, 16 to 256 token columns, remainders in every dimension; with the addend, and the
    pre-activations kept for the backward."""
    from flash_moe_b200 import check_status
    from flash_moe_b200.ops.flash_mlp import _mlp_forward, flash_mlp_add

    x, wg, wu, wd, _ = mlp_case(T, H, I, dtype)
    g, u = x.float() @ wg.float().t(), x.float() @ wu.float().t()
    h = (torch.nn.functional.silu(g) * u).to(dtype).float()
    addend = randn((T, H), 5, torch.float32).cuda()
    ulp = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    want = h @ wd.float().t() + addend
    got = flash_mlp_add(x, wg, wu, wd, addend)
    assert (got.float() - want).norm() <= ulp * want.norm()
    assert torch.equal(got, flash_mlp_add(x, wg, wu, wd, addend))
    out, a, b = _mlp_forward(x, wg, wu, wd, save_preacts=True)
    assert (out.float() - (want - addend)).norm() <= ulp * (want - addend).norm()
    for kept, ref in ((a, g), (b, u)):
        if kept is not None:
            assert (kept.float() - ref).norm() <= ulp * ref.norm()
    check_status()


@pytest.mark.parametrize("T,H,I,dtype", [((1 << 23) + 300, 8, 8, torch.bfloat16), (2_100_001, 64, 8, torch.float32)])
def test_mlp_with_more_tokens_than_one_grid_takes(T, H, I, dtype):
    """More token tiles than the grid's second dimension holds: rows around the seam, at both ends and in between."""
    from flash_moe_b200 import check_status
    from flash_moe_b200.ops.flash_mlp import flash_mlp_func

    gen = torch.Generator(device="cuda").manual_seed(T)
    x, wg, wu, wd = (torch.empty(shape, device="cuda", dtype=dtype).normal_(0, std, generator=gen)
                     for shape, std in (((T, H), 0.5), ((I, H), H**-0.5), ((I, H), H**-0.5), ((H, I), I**-0.5)))
    with torch.no_grad():
        got = flash_mlp_func(x, wg, wu, wd)
    check_status()
    for rows in (slice(0, 400), slice(T // 2, T // 2 + 400), slice(T - 700, T)):
        xs = x[rows].double()
        h = torch.nn.functional.silu(xs @ wg.double().t()) * (xs @ wu.double().t())
        want = (h if dtype == torch.float32 else h.to(dtype).double()) @ wd.double().t()
        assert (got[rows].double() - want).norm() <= (2e-6 if dtype == torch.float32 else 2.0**-8) * want.norm()
