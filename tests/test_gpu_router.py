"""Router parity on the GPU, through the C ABI (fmoe_router_topk / fmoe_router_front)."""

import os

import numpy as np
import pytest
import torch

from oracle import flashmoe_oracle as O
from tests.helpers import bf16_ulp_close, log_probs, randn

pytestmark = pytest.mark.gpu


def run_router(lp, nk, k):
    from flash_moe_b200.ops.flash_router import flash_router_func

    s, i = flash_router_func(lp.cuda(), nk, k)
    torch.cuda.synchronize()
    return s.cpu(), i.cpu()


@pytest.mark.parametrize(
    "T,nk,k",
    [(64, 32, 8), (256, 128, 64), (33, 100, 7), (5, 16, 1), (9, 16, 16), (17, 1, 1), (40, 256, 32), (12, 512, 128),
     (7, 48, 48), (3, 1000, 10)],
)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_router_topk_exact(T, nk, k, dtype):
    """Scores, indices and their order are bit-identical to the reference semantics, ties included
    (16-bit inputs produce many exactly equal pair sums)."""
    lp = log_probs(T, nk, seed=T * 1000 + nk, dtype=dtype)
    want_s, want_i = O.router_topk(lp, nk, k)
    got_s, got_i = run_router(lp, nk, k)
    assert got_i.dtype == torch.int64 and got_s.dtype == dtype
    assert torch.equal(got_s.float(), want_s.float())
    assert torch.equal(got_i, want_i)
    assert all(v == 0 for v in O.check_router_threshold(lp, nk, k, got_i).values())


@pytest.mark.parametrize(
    "name", ["triton_router_nk16_k4", "triton_router_nk16_k4_tied", "triton_router_nk32_k8_tied", "triton_router_nk128_k16"]
)
def test_router_topk_matches_reference_kernel_fixture(golden_dir, name):
    z = np.load(os.path.join(golden_dir, name + ".npz"))
    got_s, got_i = run_router(torch.from_numpy(z["log_probs"]), int(z["nk"]), int(z["k"]))
    assert np.array_equal(got_s.numpy(), z["scores"])
    assert np.array_equal(got_i.numpy(), z["indices"])


@pytest.mark.parametrize("T,nk,k", [(16, 64, 32), (8, 128, 64), (8, 256, 32), (6, 512, 16)])
def test_router_heavy_ties_and_infinities(T, nk, k):
    """Log-probabilities on a grid of 0.5: hundreds of candidates tie with the threshold (short tie lists ranked by
    shuffles, long ones by the bitwise search, overflowing ones by the per-row search), float32 through the kernel that sorts
    whole rows and 16-bit through the one that drops keys."""
    lp = torch.round(randn((2, T, nk), 3) * 2) / 2 - 3.0
    lp[0, 0, :] = -1.0  # a whole half tied
    lp[1, 1, :] = float("-inf")  # every sum is -inf for this token
    lp[0, 2, 5] = float("-inf")
    for dtype in (torch.float32, torch.bfloat16):
        x = lp.to(dtype)
        want_s, want_i = O.router_topk(x, nk, k)
        got_s, got_i = run_router(x, nk, k)
        assert torch.equal(got_s.float(), want_s.float())
        assert torch.equal(got_i, want_i)


def test_router_empty_and_argument_errors():
    from flash_moe_b200.ops.flash_router import flash_router_func

    lp = log_probs(4, 16, 1, torch.float32).cuda()
    s, i = flash_router_func(lp, 16, 0)
    assert s.shape == (4, 0) and i.shape == (4, 0)
    s, i = flash_router_func(lp[:, :0], 16, 4)
    assert s.shape == (0, 4)
    with pytest.raises(AssertionError):
        flash_router_func(lp, 16, 17)
    with pytest.raises(AssertionError):
        flash_router_func(lp[0], 16, 4)
    with pytest.raises(Exception):
        flash_router_func(lp.cpu(), 16, 4)


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_gates(norm, dtype):
    from flash_moe_b200.ops.flash_router import flash_router_with_gates

    T, nk, k = 128, 64, 16
    lp = log_probs(T, nk, 11, dtype)
    s, i, g = flash_router_with_gates(lp.cuda(), nk, k, norm)
    want = O.routing_weights(s.cpu(), norm)
    if dtype == torch.float32:
        torch.testing.assert_close(g.cpu(), want, rtol=2e-6, atol=0)
    else:
        assert bf16_ulp_close(g.cpu(), want, 1).all()
        assert (g.cpu() == want).float().mean() > 0.98


@pytest.mark.parametrize("T,H,nk", [(256, 256, 32), (300, 1024, 128), (130, 512, 256), (64, 128, 24), (200, 64, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("training", [False, True])
def test_router_front(T, H, nk, dtype, training):
    """logits against a float32 evaluation of BN -> Linear on the same stored operands (2e-2 x RMS for
    16-bit), log-probs against torch's log-softmax of OUR logits (one rounding step), and the
    batch-norm running-statistics side effect."""
    from flash_moe_b200.ops.router_front import router_front

    x = randn((T, H), 5, dtype) + (0.25 if training else 0.0)
    w = randn((2 * nk, H), 6, dtype, scale=1.0 / H**0.5)
    rm = randn((H,), 7, dtype, scale=0.1)
    rv = (randn((H,), 8).abs() + 0.5).to(dtype)
    rm_g, rv_g = rm.clone().cuda(), rv.clone().cuda()
    logits, logp = router_front(x.cuda(), w.cuda(), rm_g, rv_g, training=training)
    torch.cuda.synchronize()
    rm32, rv32 = rm.float().clone(), rv.float().clone()
    want_logits, _ = O.router_front(x.float(), w.float(), rm32, rv32, training)
    tol = 2e-2 if dtype != torch.float32 else 1e-4
    assert O.rel_rms_error(logits.cpu().float(), want_logits) < tol
    chained = torch.log_softmax(logits.cpu().view(T, 2, nk).transpose(0, 1).float(), dim=-1).to(dtype)
    if dtype == torch.float32:
        torch.testing.assert_close(logp.cpu(), chained.contiguous(), rtol=1e-5, atol=2e-6)
    else:
        assert bf16_ulp_close(logp.cpu(), chained.contiguous(), 1).all()
        assert (logp.cpu() == chained).float().mean() > 0.99
    if training:
        torch.testing.assert_close(rm_g.cpu().float(), rm32, rtol=1e-2, atol=1e-2 if dtype != torch.float32 else 1e-5)
        torch.testing.assert_close(rv_g.cpu().float(), rv32, rtol=1e-2, atol=1e-2 if dtype != torch.float32 else 1e-5)
    else:
        assert torch.equal(rm_g.cpu(), rm) and torch.equal(rv_g.cpu(), rv)


def test_router_full_size_properties():
    """Config-3 shape (16384 tokens, nk=512, k=128, bf16): properties that need no brute force -
    sorted output, no duplicates, ids in range, scores equal the in-dtype pair sum of their id;
    plus exact parity on a 64-token sample."""
    T, nk, k = 16384, 512, 128
    lp = log_probs(T, nk, 21, torch.bfloat16)
    s, i = run_router(lp, nk, k)
    assert ((i >= 0) & (i < nk * nk)).all()
    sf = s.float()
    assert (sf[:, :-1] >= sf[:, 1:]).all()
    assert (torch.sort(i, dim=-1).values.diff(dim=-1) > 0).all()
    a = lp[0].gather(-1, i // nk)
    b = lp[1].gather(-1, i % nk)
    assert torch.equal((a + b).float(), sf)
    tie = sf[:, :-1] == sf[:, 1:]
    assert (i[:, :-1][tie] < i[:, 1:][tie]).all()
    sel = torch.arange(0, T, T // 64)
    want_s, want_i = O.router_topk(lp[:, sel], nk, k)
    assert torch.equal(s[sel].float(), want_s.float()) and torch.equal(i[sel], want_i)


@pytest.mark.parametrize(
    "T,nk,k",
    [(33, 33, 16), (70, 64, 32), (70, 65, 33), (65, 128, 64), (41, 129, 128), (37, 256, 71), (37, 256, 34), (19, 513, 127),
     (9, 1024, 128)],
)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("scale", [0.05, 1.0, 12.0])
def test_router_pruned_rows(T, nk, k, dtype, scale):
    """Rows whose keys are dropped below a bound: nearly flat ones (everything stays, many ties), ordinary and peaked ones,
    at the edges of the keys per lane and of the candidates per lane."""
    lp = torch.log_softmax(randn((2, T, nk), T + nk + k, torch.float32) * scale, -1).to(dtype).contiguous()
    want_s, want_i = O.router_topk(lp, nk, k)
    got_s, got_i = run_router(lp, nk, k)
    assert torch.equal(got_s.float(), want_s.float())
    assert torch.equal(got_i, want_i)


@pytest.mark.parametrize("T,nk,k", [(40, 33, 16), (40, 40, 17), (40, 64, 32), (40, 128, 64), (30, 256, 65), (20, 512, 128), (12, 1000, 33)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["masked", "one_hot", "few_values", "infinite", "opposite_signs", "dominant", "half_dominant"])
def test_router_rare_rows(T, nk, k, dtype, kind):
    """Rows that the usual few candidates do not cover, in one call with rows that they do: keys of -inf (down to fewer finite
    sums than slots), sums too many levels apart for 32-bit keys, more ties than candidates are kept, +inf, sums around 0, keys that hold most of the
    probability of their half, or of one half (the k sums are then a row and a column)."""
    x = randn((2, T, nk), T + nk + k, torch.float32)
    if kind == "masked":
        x[torch.rand(x.shape, generator=torch.Generator().manual_seed(nk)) < 0.5] = float("-inf")
        x[:, ::5, 3:] = float("-inf")
    elif kind == "one_hot":
        x[:, ::2, nk // 3] += 40.0
    elif kind == "few_values":
        x[:, ::2] = x[:, ::2].round()
        x[:, 1] = 0.0
    elif kind == "infinite":
        x[0, ::3, nk // 2] = float("inf")
    elif kind == "dominant":
        x[:, ::2, nk // 3] += 12.0
        x[0, 1::4, 0] += 7.0
    elif kind == "half_dominant":
        x[0, :, nk // 2] += 9.0
        x[1, ::3, :3] += 9.0
    else:
        x[1] = -x[0].flip(-1)
    lp = (torch.log_softmax(x, -1) if kind in ("one_hot", "few_values", "dominant", "half_dominant") else x).to(dtype).contiguous()
    want_s, want_i = O.router_topk(lp, nk, k)
    got_s, got_i = run_router(lp, nk, k)
    assert torch.equal(got_s.float(), want_s.float())
    assert torch.equal(got_i, want_i)


@pytest.mark.parametrize("nk,k", [(65, 36), (72, 60), (100, 50), (100, 71), (128, 40), (128, 64), (128, 72)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_router_in_more_than_one_wave(nk, k, dtype):
    """The result of a token does not depend on the tokens beside it: 65 to 128 keys, both sides of half the keys wanted, where the
    kernel changes, ordinary rows and rows full of ties, more tokens than are resident at once
    against the same tokens in small batches and, for some of them, against the oracle."""
    T = 6001
    lp = torch.log_softmax(randn((2, T, nk), nk * k, torch.float32), -1)
    lp[:, ::3] = torch.round(lp[:, ::3] * 2) / 2
    lp[0, 9, 3] = float("-inf")
    lp[1, 12] = float("-inf")
    lp = lp.to(dtype).contiguous()
    got_s, got_i = run_router(lp, nk, k)
    for t0 in (0, 1000, T - 500):
        s, i = run_router(lp[:, t0:t0 + 500], nk, k)
        assert torch.equal(s.float(), got_s[t0:t0 + 500].float()) and torch.equal(i, got_i[t0:t0 + 500])
    want_s, want_i = O.router_topk(lp[:, :200].contiguous(), nk, k)
    assert torch.equal(got_s[:200].float(), want_s.float()) and torch.equal(got_i[:200], want_i)
