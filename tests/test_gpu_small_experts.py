"""Expert passes for few tokens (one task spread over the warps of a CTA) and the float32 scores pass."""
import pytest
import torch

from tests.helpers import randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "T,H,N,k",
    [(1, 8, 4, 1), (1, 1024, 16384, 64), (3, 136, 50, 17), (64, 2048, 4096, 32), (37, 1000, 300, 9), (590, 512, 1000, 32),
     (593, 512, 1000, 32)],
)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_expert_passes_for_few_tokens(T, H, N, k, dtype):
    """Edges of the split over warps: fewer slots than warps, a group of 17 slots, ragged columns, both sides of the token
    count at which the one-warp-per-task kernels take over; empty and out-of-range slots."""
    from flash_moe_b200 import _lib
    from flash_moe_b200.ops.flash_expert import flash_expert_fp32

    x, d, u = (randn(shape, s, dtype, sc).cuda() for shape, s, sc in (((T, H), 1, 0.5), ((N, H), 2, 0.1), ((N, H), 3, 1.0)))
    gen = torch.Generator().manual_seed(T + k)
    idx = torch.randint(0, N, (T, k), generator=gen)
    idx[0, -1] = -1
    idx = idx.cuda()
    gates = torch.softmax(randn((T, k), 4, torch.float32), -1).to(dtype).cuda()
    ok = (idx >= 0).double()
    rows = idx.clamp(min=0)
    want = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for j in range(k):
        s = (x.double() * d[rows[:, j]].double()).sum(-1)
        want += (torch.nn.functional.silu(s) * gates[:, j].double() * ok[:, j])[:, None] * u[rows[:, j]].double()
    for _ in range(3):  # back to back: each pass may start beside the one before it
        got = flash_expert_fp32(x, d, u, idx, gates)
    assert (got.double() - want).norm() <= 5e-6 * want.norm() + 1e-12
    assert torch.equal(got, flash_expert_fp32(x, d, u, idx, gates))
    assert _lib.read_status() == 0
    idx[0, 0] = N  # skipped and reported
    flash_expert_fp32(x, d, u, idx, gates)
    assert _lib.read_status() == _lib.STATUS_BAD_EXPERT_ID


@pytest.mark.parametrize("H,offset", [(1040, 0), (1040, 8), (2048, 0), (1032, 0)])
def test_scores_over_tables_beyond_the_tlb(H, offset):
    """Tables of more than 384 MiB: whole-line loads, at both alignments and with a ragged last block of columns; 1032 has no
    16-column pieces."""
    from flash_moe_b200.ops.flash_expert import flash_expert_fp32

    T, k, N = 801, 16, (400 << 20) // (2 * H)
    gen = torch.Generator(device="cuda").manual_seed(H)

    def normal(rows, std):
        flat = torch.empty(rows * H + offset, device="cuda", dtype=torch.bfloat16).normal_(0, std, generator=gen)
        return flat[offset:].view(rows, H)

    x, d, u = normal(T, 0.5), normal(N, 0.1), normal(N, 1.0)
    idx = torch.randint(0, N, (T, k), device="cuda", generator=gen)
    gates = torch.rand(T, k, device="cuda", generator=gen).bfloat16()
    want = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for j in range(k):
        s = (x.double() * d[idx[:, j]].double()).sum(-1)
        want += (torch.nn.functional.silu(s) * gates[:, j].double())[:, None] * u[idx[:, j]].double()
    assert (flash_expert_fp32(x, d, u, idx, gates).double() - want).norm() <= 5e-6 * want.norm()


@pytest.mark.parametrize("H,N", [(1040, 3000), (1040, (400 << 20) // 2080), (1032, (400 << 20) // 2064)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_a_token_alone_has_the_bits_it_has_in_a_batch(H, N, dtype):
    """The order of a sum depends on the table alone, not on the number of tokens: few-token kernels (1 and 40 tokens) against
    the one-warp-per-task kernels (801 tokens), for tables below and above 384 MiB (whole-line loads, where H allows them)."""
    from flash_moe_b200.ops.flash_expert import _expert_forward

    T, k = 801, 16
    gen = torch.Generator(device="cuda").manual_seed(N)
    x, d, u = (torch.empty(rows, H, device="cuda", dtype=dtype).normal_(0, std, generator=gen)
               for rows, std in ((T, 0.5), (N, 0.1), (N, 1.0)))
    idx = torch.randint(0, N, (T, k), device="cuda", generator=gen)
    gates = torch.rand(T, k, device="cuda", generator=gen).to(dtype)
    out, scores = _expert_forward(x, d, u, idx, gates, torch.float32, save_scores=True)
    for rows in (slice(5, 6), slice(800, 801), slice(100, 140)):
        few, few_scores = _expert_forward(x[rows], d, u, idx[rows], gates[rows], torch.float32, save_scores=True)
        assert torch.equal(few_scores, scores[rows]) and torch.equal(few, out[rows])


@pytest.mark.parametrize("H,T,k", [(520, 430, 17), (1000, 1500, 17), (1024, 1500, 32), (1544, 801, 16)])
def test_tables_beyond_l2(H, T, k):
    """Tables of more than 144 MiB, whose accumulate pass runs with the CTAs that are resident at once: last column blocks of 8,
    488, 512 and 8 columns give the bits of the few-token kernels and the float64 sums up to float32 rounding; empty slots stay
    empty."""
    from flash_moe_b200.ops.flash_expert import _expert_forward

    N = (150 << 20) // (2 * H)
    gen = torch.Generator(device="cuda").manual_seed(H)
    x, d, u = (torch.empty(rows, H, device="cuda", dtype=torch.bfloat16).normal_(0, std, generator=gen)
               for rows, std in ((T, 0.5), (N, 0.1), (N, 1.0)))
    idx = torch.randint(0, N, (T, k), device="cuda", generator=gen)
    idx[::7, k // 2] = -1
    gates = torch.rand(T, k, device="cuda", generator=gen).bfloat16()
    out, scores = _expert_forward(x, d, u, idx, gates, torch.float32, save_scores=True)
    for rows in (slice(0, 20), slice(T - 20, T)):
        few, few_scores = _expert_forward(x[rows], d, u, idx[rows], gates[rows], torch.float32, save_scores=True)
        assert torch.equal(few_scores, scores[rows]) and torch.equal(few, out[rows])
    want = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for j in range(k):
        e = idx[:, j].clamp(min=0)
        s = (x.double() * d[e].double()).sum(-1)
        want += (torch.nn.functional.silu(s) * gates[:, j].double() * (idx[:, j] >= 0))[:, None] * u[e].double()
    assert (out.double() - want).norm() <= 5e-6 * want.norm()


@pytest.mark.parametrize("H,offset,dtype", [(1040, 0, torch.bfloat16), (1040, 8, torch.float16), (2048, 8, torch.bfloat16)])
def test_whole_line_loads_over_several_tasks(H, offset, dtype):
    """Tables of more than 384 MiB with two to four tasks for each warp, the next one's rows fetched behind the present one, at
    both alignments: the bits of the few-token kernels."""
    from flash_moe_b200.ops.flash_expert import _expert_forward

    T, k, N = 2500, 33, (400 << 20) // (2 * H)
    gen = torch.Generator(device="cuda").manual_seed(H + offset)

    def normal(rows, std):
        flat = torch.empty(rows * H + offset, device="cuda", dtype=dtype).normal_(0, std, generator=gen)
        return flat[offset:].view(rows, H)

    x, d, u = normal(T, 0.5), normal(N, 0.1), normal(N, 1.0)
    idx = torch.randint(0, N, (T, k), device="cuda", generator=gen)
    gates = torch.rand(T, k, device="cuda", generator=gen).to(dtype)
    out, scores = _expert_forward(x, d, u, idx, gates, torch.float32, save_scores=True)
    for start in range(0, T, 100):
        rows = slice(start, start + 100)
        few, few_scores = _expert_forward(x[rows], d, u, idx[rows], gates[rows], torch.float32, save_scores=True)
        assert torch.equal(few_scores, scores[rows]) and torch.equal(few, out[rows])


@pytest.mark.parametrize(
    "H,T,k,N,offset,dtype",
    [(2048, 1184, 32, 37500, 0, torch.bfloat16), (1000, 2500, 33, 78643, 0, torch.float16), (520, 4800, 32, 151233, 0, torch.bfloat16),
     (1040, 6200, 33, 201649, 0, torch.bfloat16), (2048, 3200, 33, 102400, 8, torch.float16), (1032, 6200, 33, 203212, 0, torch.bfloat16)],
)
def test_columns_in_slabs(H, T, k, N, offset, dtype):
    """A layer's scores pass walks tables of more than 144 MiB, rows wanted more than once, in slabs of 512 columns, the sums so
    far kept in registers (2048: warps with one task) or in memory: last slabs of 512, 488, 8 and 16 columns, loads of 8 columns,
    of whole lines (above 384 MiB) and of whole lines in two pieces.  With a down projection of zeros the layer returns the
    experts' sum, and the op walks whole rows: the same bits."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig, check_status
    from flash_moe_b200.ops.flash_expert import flash_expert_fp32

    gen = torch.Generator(device="cuda").manual_seed(H)
    with torch.device("cuda"):
        layer = FlashMoE(FlashMoEConfig(H, 64, "silu", N, k, True)).to(dtype).eval()
    with torch.no_grad():
        layer.down_proj.weight.zero_()
        for table, std in ((layer.down_embed, 0.1), (layer.up_embed, 1.0)):
            flat = torch.empty(N * H + offset, device="cuda", dtype=dtype).normal_(0, std, generator=gen)
            table.weight.data = flat[offset:].view(N, H)
        xs = [torch.empty(1, T, H, device="cuda", dtype=dtype).normal_(0, 0.5, generator=gen) for _ in range(2)]
        got = []
        for x in xs:
            y, _ = layer(x, return_routing=True)
            got.append((y, layer.last_indices.clone(), layer.last_gates.clone()))
        for x, (y, idx, gates) in zip(xs, got):
            want = flash_expert_fp32(x[0], layer.down_embed.weight, layer.up_embed.weight, idx, gates)
            assert torch.equal(y[0], want.to(dtype)) and bool(want.abs().max() > 0.1)
    check_status()


@pytest.mark.parametrize("T,k", [(5, 3), (64, 20), (1200, 20), (1200, 33)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_row_that_nobody_selects_has_no_effect(T, k, dtype):
    """Slots beyond top-k, empty slots and out-of-range ids read no row: infinities and NaN in the first rows of the tables
    reach only the tokens that select them."""
    from flash_moe_b200 import _lib
    from flash_moe_b200.ops.flash_expert import _expert_backward, flash_expert_fp32

    N, H = 300, 264
    x, d, u, dout = (randn(shape, s, dtype).cuda() for shape, s in (((T, H), 1), ((N, H), 2), ((N, H), 3), ((T, H), 4)))
    gen = torch.Generator().manual_seed(k)
    idx = torch.randint(2, N, (T, k), generator=gen)
    idx[1, 0], idx[2, -1], idx[3, 0] = -1, N, 0
    idx = idx.cuda()
    gates = torch.rand(T, k, generator=gen).to(dtype).cuda()
    want, grads = flash_expert_fp32(x, d, u, idx, gates), _expert_backward(dout, x, d, u, idx, gates)
    for t in (d, u):
        t[0], t[1] = float("inf"), float("nan")
    got, bad = flash_expert_fp32(x, d, u, idx, gates), _expert_backward(dout, x, d, u, idx, gates)
    others = torch.arange(T, device="cuda") != 3
    assert torch.equal(got[others], want[others]) and torch.equal(bad[0][others], grads[0][others])
    assert not torch.isfinite(got[3]).any()
    _lib.read_status()
