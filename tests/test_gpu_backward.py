"""Backward of the three ops and of the layer through the C ABI, against the oracle's float32 restatements and the
gradients of the reference's own eager module (golden fixtures)."""

import os

import numpy as np
import pytest
import torch

from oracle import flashmoe_oracle as O
from tests.helpers import randn

pytestmark = pytest.mark.gpu


def rel_err(got, want):
    want = want.float()
    return float((got.detach().float().cpu() - want).abs().max() / want.abs().max().clamp_min(1e-12))


def tol(dtype):
    return {torch.float32: 2e-5, torch.bfloat16: 1.2e-2, torch.float16: 2e-3}[dtype]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,nk,k", [(1, 4, 1), (33, 16, 4), (257, 128, 64), (64, 100, 100)])
def test_router_backward(dtype, T, nk, k):
    from flash_moe_b200.ops.flash_router import flash_router_func

    lp = torch.log_softmax(randn((2, T, nk), T + nk, torch.float32), -1).to(dtype).cuda().requires_grad_()
    scores, idx = flash_router_func(lp, nk, k)
    ds = randn((T, k), 5, torch.float32).to(dtype).cuda()
    scores.backward(ds)
    want = O.router_backward(ds.cpu(), idx.cpu(), nk)
    assert lp.grad.shape == (2, T, nk) and lp.grad.dtype == dtype
    assert rel_err(lp.grad, want) <= (1e-6 if dtype == torch.float32 else tol(dtype))
    # every slot's gradient arrives exactly twice (once per half)
    assert abs(float(lp.grad.float().sum()) - 2 * float(ds.float().sum())) <= 1e-2 * (1 + float(ds.float().abs().sum()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_swiglu_backward(dtype):
    from flash_moe_b200.ops.flash_mlp import swiglu_backward

    a, b, dh = (randn((37, 256), s, torch.float32).mul(2).to(dtype).cuda() for s in (1, 2, 3))
    da, db, h = swiglu_backward(dh, a, b, want_h=True)
    wa, wb = O.swiglu_backward(dh.cpu(), a.cpu(), b.cpu())
    wh = torch.nn.functional.silu(a.cpu().float()) * b.cpu().float()
    for got, want in ((da, wa), (db, wb), (h, wh)):
        assert rel_err(got, want) <= tol(dtype)


def expert_case(T, H, N, k, dtype, zipf=False, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(T, H, generator=g) * 0.5).to(dtype)
    d = (torch.randn(N, H, generator=g) * 0.2).to(dtype)
    u = (torch.randn(N, H, generator=g) * 0.2).to(dtype)
    if zipf:
        p = torch.arange(1, N + 1, dtype=torch.float64).pow(-1.1)
        idx = torch.multinomial((p / p.sum()).float(), T * k, replacement=True, generator=g).view(T, k)
    else:
        idx = torch.randint(0, N, (T, k), generator=g)
    if k > 1:
        idx[0, 1] = idx[0, 0]
    gates = torch.softmax(torch.randn(T, k, generator=g), -1).to(dtype)
    dout = torch.randn(T, H, generator=g).to(dtype)
    return x, d, u, idx, gates, dout


def run_expert_backward(x, d, u, idx, gates, dout):
    from flash_moe_b200.ops.flash_expert import flash_expert_func

    xs, ds_, us, gs = (t.cuda().requires_grad_() for t in (x, d, u, gates))
    out = flash_expert_func(xs, ds_, us, idx.cuda(), gs)
    out.backward(dout.cuda())
    torch.cuda.synchronize()
    return xs.grad, ds_.grad, us.grad, gs.grad


@pytest.mark.parametrize(
    "T,H,N,k,dtype,zipf",
    [
        (5, 8, 7, 1, torch.float32, False),
        (64, 72, 50, 3, torch.float32, False),      # ragged column block
        (300, 256, 64, 8, torch.float32, True),     # hot experts: rows assembled from several chunk partials
        (128, 64, 4096, 4, torch.bfloat16, False),  # most experts untouched
        (512, 1280, 96, 16, torch.bfloat16, True),  # two column blocks, hot experts
        (200, 128, 33, 6, torch.float16, True),
        (2048, 1024, 16384, 16, torch.bfloat16, False),
    ],
)
def test_expert_backward(T, H, N, k, dtype, zipf):
    from flash_moe_b200 import check_status

    x, d, u, idx, gates, dout = expert_case(T, H, N, k, dtype, zipf, seed=T + N)
    got = run_expert_backward(x, d, u, idx, gates, dout)
    check_status()
    want = O.expert_backward(dout, x, d, u, idx, gates)
    for name, g_, w_ in zip(("dx", "ddown", "dup", "dgates"), got, want):
        assert g_.dtype == dtype
        assert rel_err(g_, w_) <= tol(dtype), name
    untouched = torch.ones(N, dtype=torch.bool)
    untouched[idx.unique()] = False
    if untouched.any():  # experts nobody selected get exact zero rows
        assert float(got[1][untouched.cuda()].abs().max()) == 0.0 and float(got[2][untouched.cuda()].abs().max()) == 0.0
    again = run_expert_backward(x, d, u, idx, gates, dout)
    assert all(torch.equal(a, b) for a, b in zip(got, again))  # fixed summation order: bit-equal reruns


def test_expert_backward_skips_out_of_range_ids():
    from flash_moe_b200 import read_status, _lib

    x, d, u, idx, gates, dout = expert_case(40, 64, 20, 4, torch.float32, seed=3)
    idx[3, 2] = -2
    idx[7, 0] = 20
    read_status()
    got = run_expert_backward(x, d, u, idx, gates, dout)
    assert read_status() & _lib.STATUS_BAD_EXPERT_ID
    g0 = gates.clone()
    g0[3, 2] = 0
    g0[7, 0] = 0
    want = O.expert_backward(dout, x, d, u, idx.clamp(0, 19), g0)
    for g_, w_ in zip(got[:3], want[:3]):
        assert rel_err(g_, w_) <= 2e-5
    assert float(got[3][3, 2]) == 0.0 and float(got[3][7, 0]) == 0.0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_mlp_backward(dtype):
    from flash_moe_b200.ops.flash_mlp import flash_mlp_func

    T, H, I = 200, 128, 384
    x = (randn((T, H), 1, torch.float32) * 0.5).to(dtype)
    wg, wu = ((randn((I, H), s, torch.float32) * 0.1).to(dtype) for s in (2, 3))
    wd = (randn((H, I), 4, torch.float32) * 0.1).to(dtype)
    dy = randn((T, H), 5, torch.float32).to(dtype)
    leaves = [t.cuda().requires_grad_() for t in (x, wg, wu, wd)]
    flash_mlp_func(*leaves).backward(dy.cuda())
    want = O.mlp_backward(dy, x, wg, wu, wd)
    for leaf, w_ in zip(leaves, want):
        assert leaf.grad.dtype == dtype
        assert rel_err(leaf.grad, w_) <= (1e-4 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("name", ["eager_mini_fp32_grads", "eager_mini_fp32_grads_norm_train"])
def test_layer_gradients_match_reference_eager_module(golden_dir, name):
    """float32 layer with the fixture's parameters: gradients of sum(y * w) equal the reference's autograd result."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig, check_status

    z = np.load(os.path.join(golden_dir, name + ".npz"))
    H, I, N, k, norm, B, S, train = (int(v) for v in z["cfg"])
    layer = FlashMoE(FlashMoEConfig(H, I, "silu", N, k, bool(norm)))
    layer.load_state_dict({n[len("param."):]: torch.from_numpy(z[n]) for n in z.files if n.startswith("param.")})
    layer = layer.cuda().train(bool(train))
    x = torch.from_numpy(z["x"]).cuda().requires_grad_()
    y, _ = layer(x)
    assert rel_err(y, torch.from_numpy(z["y"])) < 1e-4
    (y * torch.from_numpy(z["w"]).cuda()).sum().backward()
    torch.cuda.synchronize()
    check_status()
    grads = dict({"x": x.grad}, **{n: p.grad for n, p in layer.named_parameters()})
    for n, got in grads.items():
        assert rel_err(got, torch.from_numpy(z["grad." + n])) < 5e-4, n


def test_layer_backward_bf16_runs_and_no_grad_path_is_unchanged():
    from flash_moe_b200 import FlashMoE, FlashMoEConfig, check_status

    torch.manual_seed(0)
    layer = FlashMoE(FlashMoEConfig(256, 512, "silu", 1024, 8, True)).to(torch.bfloat16).cuda().train()
    x = randn((2, 64, 256), 3, torch.bfloat16).cuda().requires_grad_()
    y, logits = layer(x)
    assert y.requires_grad and logits.requires_grad
    y.float().pow(2).mean().backward()
    torch.cuda.synchronize()
    check_status()
    for n, p in layer.named_parameters():
        assert p.grad is not None and torch.isfinite(p.grad.float()).all(), n
        assert float(p.grad.float().abs().max()) > 0, n
    assert torch.isfinite(x.grad.float()).all()
    layer.eval()
    with torch.no_grad():
        y2, _ = layer(x)
    assert not y2.requires_grad


def test_training_step_replays_from_a_cuda_graph():
    """Forward + backward of the layer captured as one CUDA graph (every launch of the library, the ordering of the pairs
    included, is capturable): replayed gradients are bit-equal to the eager step's."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig, check_status

    torch.manual_seed(0)
    layer = FlashMoE(FlashMoEConfig(256, 512, "silu", 1024, 8, True)).to(torch.bfloat16).cuda().eval()
    x = randn((2, 64, 256), 3, torch.bfloat16).cuda().requires_grad_()
    dy = randn((2, 64, 256), 4, torch.bfloat16).cuda()

    def step():
        for p in layer.parameters():
            p.grad = None
        x.grad = None
        y, _ = layer(x)
        y.backward(dy)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    want = {n: p.grad.clone() for n, p in layer.named_parameters()}
    want_x = x.grad.clone()
    for p in layer.parameters():
        p.grad = None
    x.grad = None
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y, _ = layer(x)
        y.backward(dy)
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    check_status()
    assert torch.equal(x.grad, want_x)
    for n, p in layer.named_parameters():
        assert torch.equal(p.grad, want[n]), n


def test_backward_with_no_pairs():
    """k = 0: the expert op's gradients are all zero (and every table row is written)."""
    from flash_moe_b200.ops.flash_expert import _expert_backward

    dt = torch.float32
    x, dout = randn((6, 32), 1, dt).cuda(), randn((6, 32), 2, dt).cuda()
    d, u = randn((10, 32), 3, dt).cuda(), randn((10, 32), 4, dt).cuda()
    idx = torch.empty(6, 0, dtype=torch.int64, device="cuda")
    gates = torch.empty(6, 0, dtype=dt, device="cuda")
    dx, dd, du, dg = _expert_backward(dout, x, d, u, idx, gates)
    torch.cuda.synchronize()
    assert float(dx.abs().max()) == 0.0 and float(dd.abs().max()) == 0.0 and float(du.abs().max()) == 0.0
    assert dg.shape == (6, 0)


def test_mlp_backward_with_kept_preactivations():
    """The forward keeps x Wg^T and x Wu^T, the backward uses them."""
    from flash_moe_b200.ops.flash_mlp import FlashMLPFunc, _mlp_forward

    dtype = torch.bfloat16
    T, H, I = 1024, 256, 512
    x = (randn((T, H), 1, torch.float32) * 0.5).to(dtype)
    wg, wu = ((randn((I, H), s, torch.float32) * 0.1).to(dtype) for s in (2, 3))
    wd = (randn((H, I), 4, torch.float32) * 0.1).to(dtype)
    dy = randn((T, H), 5, torch.float32).to(dtype)
    out, a, b = _mlp_forward(x.cuda(), wg.cuda(), wu.cuda(), wd.cuda(), save_preacts=True)
    assert a is not None and rel_err(a, x.float() @ wg.float().t()) < 1e-2 and rel_err(b, x.float() @ wu.float().t()) < 1e-2
    assert torch.equal(out, _mlp_forward(x.cuda(), wg.cuda(), wu.cuda(), wd.cuda()))  # same kernels, same output
    leaves = [t.cuda().requires_grad_() for t in (x, wg, wu, wd)]
    FlashMLPFunc.apply(*leaves).backward(dy.cuda())
    want = O.mlp_backward(dy, x, wg, wu, wd)
    for leaf, w_ in zip(leaves, want):
        assert rel_err(leaf.grad, w_) <= 2e-2


@pytest.mark.parametrize("T,H,N,k,dtype", [(3000, 64, 9, 8, torch.float32), (600, 1096, 40, 33, torch.bfloat16),
                                           (70000, 64, 5, 8, torch.float16), (37, 520, 4000, 5, torch.bfloat16)])
def test_expert_backward_segments(T, H, N, k, dtype):
    """Segments sorted in a warp (up to 256 pairs) and through the bitmap (longer; more pair ids than one bitmap pass),
    experts whole in a chunk and split over many, chunks of every size."""
    from flash_moe_b200 import check_status
    from flash_moe_b200.ops.flash_expert import _expert_backward

    x, d, u, idx, gates, dout = expert_case(T, H, N, k, dtype, False, seed=T + N)
    idx[0, 0] = -1
    x, d, u, idx, gates, dout = (t.cuda() for t in (x, d, u, idx, gates, dout))
    got = _expert_backward(dout, x, d, u, idx, gates)
    again = _expert_backward(dout, x, d, u, idx, gates)
    assert all(torch.equal(a, b) for a, b in zip(got, again))
    ddown, dup = torch.zeros(N, H, device="cuda", dtype=torch.float64), torch.zeros(N, H, device="cuda", dtype=torch.float64)
    for j in range(k):
        e, ok = idx[:, j].clamp(min=0), (idx[:, j] >= 0).double()[:, None]
        s = (x.double() * d[e].double()).sum(-1, keepdim=True)
        q = (dout.double() * u[e].double()).sum(-1, keepdim=True)
        g, sig = gates[:, j].double()[:, None], torch.sigmoid(s)
        ddown.index_add_(0, e, ok * q * g * sig * (1 + s * (1 - sig)) * x.double())
        dup.index_add_(0, e, ok * s * sig * g * dout.double())
    tol = {torch.float32: 2e-5, torch.bfloat16: 4e-3, torch.float16: 1e-3}[dtype]
    for a, b in ((got[1], ddown), (got[2], dup)):
        assert (a.double() - b).norm() <= tol * b.norm()
    check_status()


@pytest.mark.parametrize("nk", [6145, 8192])
def test_training_step_with_the_widest_routers(nk):
    """Router halves up to the widest that the top-k takes (their sums do not fit four tokens to a CTA): float32 gradients
    against the same layer in float64 on the experts that it selected."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig, check_status

    T, H, I, k = 6, 8, 16, 4
    torch.manual_seed(nk)
    with torch.device("cuda"):
        layer = FlashMoE(FlashMoEConfig(H, I, "silu", nk * nk, k, True)).eval()
        x, dy = torch.randn(1, T, H), torch.randn(1, T, H)
    x.requires_grad_()
    y, _ = layer(x, return_routing=True)
    y.backward(dy)
    check_status()
    idx = layer.last_indices
    leaf = {n: getattr(layer, n).weight.detach().double().requires_grad_()
            for n in ("router_gate", "gate_proj", "up_proj", "down_proj")}
    leaf.update({n: getattr(layer, n).weight.detach()[idx].double().requires_grad_() for n in ("down_embed", "up_embed")})
    xr = x.detach()[0].double().requires_grad_()
    logits = (xr / (1.0 + layer.router_norm.eps) ** 0.5) @ leaf["router_gate"].t()
    lp = torch.log_softmax(logits.view(T, 2, nk), -1)
    gates = torch.exp(lp[:, 0].gather(1, idx // nk) + lp[:, 1].gather(1, idx % nk))
    gates = gates / gates.sum(-1, keepdim=True)
    s = (xr[:, None] * leaf["down_embed"]).sum(-1)
    experts = ((torch.nn.functional.silu(s) * gates)[..., None] * leaf["up_embed"]).sum(1)
    h = torch.nn.functional.silu(xr @ leaf["gate_proj"].t()) * (xr @ leaf["up_proj"].t())
    want = experts + h @ leaf["down_proj"].t()
    want.backward(dy[0].double())
    assert rel_err(y[0], want.detach().cpu()) < 1e-5
    assert rel_err(x.grad[0], xr.grad.cpu()) < 2e-5
    for n, w in leaf.items():
        got = getattr(layer, n).weight.grad
        if n.endswith("embed"):  # a row's gradient is the sum over its slots; rows that no slot selects get zeros
            rows, at = idx.unique(return_inverse=True)
            ref = torch.zeros(len(rows), H, dtype=torch.float64, device="cuda").index_add_(0, at.flatten(), w.grad.flatten(0, 1))
            assert rel_err(got[rows], ref.cpu()) < 2e-5, n
            assert int(got.count_nonzero()) <= rows.numel() * H
        else:
            assert rel_err(got, w.grad.cpu()) < 2e-5, n


def test_autocast_selects_on_float32_log_probabilities():
    """Under autocast the log-softmax returns float32, whatever the layer's type, and the selection is made on that."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig

    torch.manual_seed(2)
    with torch.device("cuda"):
        layer = FlashMoE(FlashMoEConfig(256, 512, "silu", 4096, 16, False)).to(torch.bfloat16).eval()
        x = torch.randn(2, 200, 256).to(torch.bfloat16)
    with torch.autocast("cuda", torch.bfloat16):
        y, logits = layer(x, return_routing=True)
        lp = torch.log_softmax(logits.detach(), -1)
    assert lp.dtype == torch.float32
    scores, idx = O.router_topk(lp.cpu(), 64, 16)
    assert torch.equal(layer.last_indices.cpu(), idx)
    y.float().sum().backward()
    assert torch.isfinite(layer.router_gate.weight.grad.float()).all()


@pytest.mark.parametrize("T,H,I,pair", [(512, 256, 256, False), (515, 264, 264, False), (545, 256, 392, False),
                                        (2100, 512, 2048, True), (2100, 512, 1992, True), (2100, 512, 2056, True),
                                        (1030, 256, 2072, True), (4100, 256, 1064, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_kept_products(T, H, I, pair, dtype):
    """Both GEMMs that keep the two products, the pair GEMM with boxes of 32 rows x 32 columns that end inside, at and beyond the
    last row and column: the output has the bits of the forward that keeps nothing, the products are the float32 ones rounded
    once (half a step of the type, and the float32 sums' own rounding where it moves a value across: 1e-6 of the sum of
    magnitudes), nothing is written behind them."""
    from flash_moe_b200 import _lib
    from flash_moe_b200.ops.flash_mlp import _mlp_forward
    from tests.helpers import kernels_of

    x, wg, wu, wd = (randn(shape, 20 + i, dtype, sc).cuda()
                     for i, (shape, sc) in enumerate([((T, H), 1.0), ((I, H), 0.05), ((I, H), 0.05), ((H, I), 0.05)]))
    dev, code = x.device, _lib.dtype_code(x)
    ws_bytes = _lib.lib().fmoe_mlp_workspace_bytes(T, H, I, code)
    sizes = (T * H, T * I, T * I, ws_bytes // 2)
    bufs = [torch.full((n + 512,), -3.0, dtype=dtype, device=dev) for n in sizes]
    names = kernels_of(lambda: _lib.check(_lib.call(
        "fmoe_mlp_forward_saving_preacts", dev, x.data_ptr(), wg.data_ptr(), wu.data_ptr(), wd.data_ptr(),
        *[t.data_ptr() for t in bufs[:3]], code, T, H, I, bufs[3].data_ptr(), ws_bytes, _lib.status_ptr(dev)), "mlp"))
    assert "gemm_tcgen05_pair_kernel" in names[0] if pair else "gemm_narrow_kernel" in names[0], names
    for t, n in zip(bufs, sizes):
        assert bool((t[n:] == -3.0).all())
    out, a, b = (t[:n].view(T, -1) for t, n in zip(bufs, sizes[:3]))
    assert torch.equal(out, _mlp_forward(x, wg, wu, wd))
    step = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for got, w in ((a, wg), (b, wu)):
        want = x.double() @ w.double().t()
        slack = 1e-6 * (x.double().abs() @ w.double().abs().t())
        assert ((got.double() - want).abs() <= step * want.abs() + slack + 2.0 ** -24).all()


@pytest.mark.parametrize("T,H,I,R", [(1, 4, 4, 4), (2, 8, 260, 68), (65, 64, 128, 64), (64, 132, 68, 36), (500, 512, 768, 128)])
@pytest.mark.parametrize("leave_out", [(), ("dx", "dwd"), ("dxn", "dwr")])
def test_dense_backward_float32(T, H, I, R, leave_out):
    """All dense gradients in two launches: partial tiles of 64 in every direction, steps of k cut off inside (T, H, I and R are
    each somebody's k), outputs left out; float32 sums against float64 ones (5e-6 as for the other float32 sums here)."""
    from flash_moe_b200 import _lib

    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(T + H)
    sizes = dict(dy=(T, H), x=(T, H), a=(T, I), b=(T, I), wg=(I, H), wu=(I, H), wd=(H, I), dl=(T, R), xn=(T, H), wr=(R, H))
    t = {n: torch.randn(*s, device=dev, generator=gen) for n, s in sizes.items()}
    outs = dict(dab=(T, 2 * I), h=(T, I), dx=(T, H), dxn=(T, H), dw=(2 * I, H), dwd=(H, I), dwr=(R, H))
    o = {n: torch.full(s, float("nan"), device=dev) for n, s in outs.items()}
    o["dx"].copy_(t["x"])  # added to
    rc = _lib.call_struct("fmoe_dense_backward_f32", dev, _lib.DENSE_BACKWARD_ARGS.pack(
        *[v.data_ptr() for v in t.values()], *[0 if n in leave_out else v.data_ptr() for n, v in o.items()],
        _lib.current_stream_ptr(torch.device("cuda", torch.cuda.current_device())), T, H, I, R))
    assert rc == 0
    d = {n: v.double() for n, v in t.items()}
    sig = torch.sigmoid(d["a"])
    dh, act = d["dy"] @ d["wd"], d["a"] * sig
    da, db, h = dh * d["b"] * (sig * (1 + d["a"] * (1 - sig))), dh * act, act * d["b"]
    dab = torch.cat([da, db], 1)
    want = dict(dab=dab, h=h, dx=d["x"] + da @ d["wg"] + db @ d["wu"], dxn=d["dl"] @ d["wr"], dw=dab.t() @ d["x"],
                dwd=d["dy"].t() @ h, dwr=d["dl"].t() @ d["xn"])
    for n, w in want.items():
        if n in leave_out:
            assert n == "dx" or torch.isnan(o[n]).all()
        else:
            assert (o[n].double() - w).norm() <= 5e-6 * w.norm(), n


def test_dense_backward_float32_refuses_ragged_rows():
    from flash_moe_b200 import _lib

    dev = torch.device("cuda", torch.cuda.current_device())
    z = [torch.zeros(64, 64, device=dev).data_ptr()] * 17
    pack = lambda *n: _lib.DENSE_BACKWARD_ARGS.pack(*z, _lib.current_stream_ptr(dev), *n)
    assert _lib.call_struct("fmoe_dense_backward_f32", dev, pack(4, 6, 8, 8)) == _lib.ERR_UNSUPPORTED
    assert _lib.call_struct("fmoe_dense_backward_f32", dev, pack(4, 8, 8, 6)) == _lib.ERR_UNSUPPORTED
    z[3] += 4
    assert _lib.call_struct("fmoe_dense_backward_f32", dev, pack(4, 8, 8, 8)) == _lib.ERR_ALIGNMENT


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_saved_tensors_may_come_back_with_other_strides(dtype):
    """Hooks on saved tensors may return them in another layout: the same gradients."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig, check_status

    def columns_first(t):
        return t.t().contiguous().t() if t.dim() == 2 else t

    torch.manual_seed(5)
    with torch.device("cuda"):
        layer = FlashMoE(FlashMoEConfig(64, 96, "silu", 400, 8, True)).to(dtype).eval()
        x, dy = torch.randn(3, 20, 64).to(dtype), torch.randn(3, 20, 64).to(dtype)
    x.requires_grad_()
    grads = []
    for hook in (lambda t: t, columns_first):
        layer.zero_grad()
        x.grad = None
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, hook):
            y, _ = layer(x)
            y.backward(dy)
        grads.append([x.grad.clone()] + [p.grad.clone() for p in layer.parameters()])
    assert all(torch.equal(a, b) for a, b in zip(*grads))
    check_status()


def test_captured_float32_step_takes_torch_products():
    """A step replayed from a graph has no host time to gain from fewer launches: torch's products, and the eager step's gradients
    up to float32 sums in another order."""
    from flash_moe_b200 import FlashMoE, FlashMoEConfig, _lib, check_status

    torch.manual_seed(6)
    with torch.device("cuda"):
        layer = FlashMoE(FlashMoEConfig(64, 96, "silu", 400, 8, True)).eval()
        x, dy = torch.randn(3, 20, 64), torch.randn(3, 20, 64)
    called, call_struct = [], _lib.call_struct

    def step():
        called.clear()
        layer(x)[0].backward(dy)
        return set(called)

    _lib.call_struct = lambda name, *args: called.append(name) or call_struct(name, *args)
    try:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                layer.zero_grad(set_to_none=True)
                assert "fmoe_dense_backward_f32" in step()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        want = [p.grad.clone() for p in layer.parameters()]
        layer.zero_grad(set_to_none=True)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            names = step()
        assert "fmoe_train_backward" in names and "fmoe_dense_backward_f32" not in names
    finally:
        _lib.call_struct = call_struct
    for p in layer.parameters():
        p.grad.fill_(float("nan"))
    graph.replay()
    for p, w in zip(layer.parameters(), want):
        assert (p.grad.double() - w.double()).norm() <= 5e-6 * w.double().norm()
    check_status()
