"""Performance cases of the framework: what a program that uses it asks of it, from one decoded token to a whole batch of
training or prefill tokens.

Five kinds of work, each through the public entry point that a program calls:

  layer    `FlashMoE` under no_grad (eager, or as a `GraphedFlashMoE`)
  stack    `FlashMoEStack`, pre-norm residual blocks, under no_grad
  train    forward and backward of `FlashMoE` in training mode (batch statistics, all gradients)
  router   `flash_router_func` on log-probabilities
  experts  `flash_expert_func` on given ids and gates
  mlp      `flash_mlp_func`

Sizes are those of the benchmark configurations, the tests and generic ones around them.
"""

import math

import numpy as np
import torch

from flash_moe_b200 import FlashMoE, FlashMoEConfig, GraphedFlashMoE, flash_expert_func, flash_mlp_func, flash_router_func
from flash_moe_b200.modules.stack import FlashMoEStack

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}


def layer_case(kind, dtype, batch, seq, hidden, intermediate, experts, top_k, norm, **more):
    return dict(kind=kind, dtype=dtype, batch=batch, seq=seq, hidden=hidden, intermediate=intermediate, experts=experts,
                top_k=top_k, norm=norm, **more)


def listed():
    return [
        # one token of one sequence being generated, default layer, plain module call: latency and host work
        dict(layer_case("layer", "bfloat16", 1, 1, 1024, 4096, 16384, 64, False, graph=False), name="decode_1"),
        # a batch of 64 sequences being generated, decoder-sized layer, replayed from a CUDA graph as servers do
        dict(layer_case("layer", "bfloat16", 64, 1, 2048, 5632, 65536, 32, True, graph=True), name="decode_64_graph"),
        # the small float32 layer (256 tokens): checks, ports and small experiments
        dict(layer_case("layer", "float32", 1, 256, 256, 1024, 1024, 8, False, graph=False), name="layer_256_f32"),
        # a short ragged batch in float16: 3 x 259 tokens, sizes that no tile divides
        dict(layer_case("layer", "float16", 3, 259, 1000, 2728, 10000, 24, True, graph=False), name="layer_777_f16"),
        # the default layer at its headline size
        dict(layer_case("layer", "bfloat16", 1, 4096, 1024, 4096, 16384, 64, False, graph=False), name="layer_4096"),
        # four pre-norm blocks of the decoder configuration over 8 x 2048 tokens
        dict(layer_case("stack", "bfloat16", 8, 2048, 2048, 5632, 65536, 32, True, layers=4), name="stack_4x16384"),
        # one layer of the decoder configuration over its full global batch
        dict(layer_case("layer", "bfloat16", 64, 2048, 2048, 5632, 65536, 32, True, graph=False), name="layer_131072"),
        # a training step of the default layer
        dict(layer_case("train", "bfloat16", 2, 2048, 1024, 4096, 16384, 64, False), name="train_4096"),
        # a small ragged float32 training step with renormalised gates
        dict(layer_case("train", "float32", 4, 125, 512, 768, 4096, 16, True), name="train_500_f32"),
        # router alone: 512 + 512 sub-keys, top-128
        dict(kind="router", dtype="bfloat16", tokens=16384, keys=512, top_k=128, name="router_16384"),
        # experts alone: a million experts whose popularity follows Zipf's law, tables far larger than the caches
        dict(kind="experts", dtype="bfloat16", tokens=32768, hidden=2048, experts=1 << 20, top_k=16, zipf=1.1,
             name="experts_32768"),
        # shared MLP alone, wide
        dict(kind="mlp", dtype="bfloat16", tokens=2048, hidden=4096, intermediate=16384, name="mlp_2048"),
    ]


def log_int(rng, lo, hi, step=1):
    """An integer of [lo, hi], even over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, round(v / step) * step))


def draw(rng):
    kind = rng.choice(["layer"] * 5 + ["stack"] + ["train"] * 2 + ["router", "experts", "mlp"])
    dtype = rng.choice(["bfloat16"] * 4 + ["float16"] * 2 + ["float32"])
    f32 = dtype == "float32"
    if kind in ("layer", "stack", "train"):
        train = kind == "train"
        keys = log_int(rng, 32, 128 if train else 256)
        tokens = log_int(rng, 32, 2048 if f32 else 8192) if train else log_int(rng, 1, 1024 if f32 else 65536)
        if kind == "stack":
            tokens = max(1, tokens // 4)
        batch = rng.choice([b for b in (1, 2, 4, 8) if b <= tokens])
        case = layer_case(kind, dtype, batch, max(tokens // batch, 2 if train else 1),
                          log_int(rng, 256, 1024 if train else 2048, 8), log_int(rng, 512, 4096 if train else 5632, 8),
                          keys * keys + rng.choice([0, 0, rng.randrange(2 * keys)]), log_int(rng, 4, min(64, keys)),
                          rng.random() < 0.5)
        if kind == "layer":
            case["graph"] = tokens <= 256 and rng.random() < 0.5
        if kind == "stack":
            case["layers"] = rng.randint(2, 4)
        return case
    if kind == "router":
        keys = log_int(rng, 32, 512)
        return dict(kind=kind, dtype=dtype, tokens=log_int(rng, 16, 32768), keys=keys, top_k=log_int(rng, 4, min(128, keys)))
    if kind == "experts":
        return dict(kind=kind, dtype=dtype, tokens=log_int(rng, 16, 4096 if f32 else 32768), hidden=log_int(rng, 256, 2048, 8),
                    experts=log_int(rng, 1024, 1 << (17 if f32 else 20)), top_k=log_int(rng, 4, 64),
                    zipf=rng.choice([0.0, 0.7, 1.1]))
    return dict(kind="mlp", dtype=dtype, tokens=log_int(rng, 1, 512 if f32 else 8192), hidden=log_int(rng, 256, 4096, 8),
                intermediate=log_int(rng, 512, 4096 if f32 else 16384, 8))


def popularity(case):
    """Share of the (token, slot) pairs that goes to each expert, most popular first."""
    p = np.arange(1, case["experts"] + 1, dtype=np.float64) ** -case["zipf"]
    return p / p.sum()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]

    def normal(*shape, std=1.0):
        return torch.randn(*shape, device="cuda", dtype=dt, generator=gen).mul_(std)

    kind = case["kind"]
    state = dict(kind=kind)
    if kind in ("layer", "stack", "train"):
        config = FlashMoEConfig(case["hidden"], case["intermediate"], "silu", case["experts"], case["top_k"], case["norm"])
        torch.manual_seed(seed)
        with torch.device("cuda"):
            module = FlashMoEStack(config, case["layers"], pre_norm=True) if kind == "stack" else FlashMoE(config)
        module = module.to(dt).train(kind == "train")
        for layer in module.layers if kind == "stack" else [module]:  # statistics as training leaves them
            layer.router_norm.running_mean.copy_(normal(case["hidden"], std=0.1))
            layer.router_norm.running_var.copy_(normal(case["hidden"], std=0.25).abs_().add_(0.8))
        x = normal(case["batch"], case["seq"], case["hidden"])
        if kind == "train":
            x.requires_grad_()
            state["dy"] = normal(case["batch"], case["seq"], case["hidden"])
        state["module"] = GraphedFlashMoE(module, x) if case.get("graph") else module
        state["x"] = x
    elif kind == "router":
        logits = torch.randn(2, case["tokens"], case["keys"], device="cuda", generator=gen)
        state["args"] = (torch.log_softmax(logits, -1).to(dt), case["keys"], case["top_k"])
    elif kind == "experts":
        N, H, k = case["experts"], case["hidden"], case["top_k"]
        cdf = torch.from_numpy(np.cumsum(popularity(case))).cuda()
        at = torch.rand(case["tokens"], k, device="cuda", dtype=torch.float64, generator=gen)
        rank = torch.searchsorted(cdf, at).clamp_(max=N - 1)
        ids = torch.randperm(N, device="cuda", generator=gen)[rank]  # popular experts lie anywhere in the tables
        gates = torch.softmax(torch.randn(case["tokens"], k, device="cuda", generator=gen), -1).to(dt)
        state["args"] = (normal(case["tokens"], H), normal(N, H, std=H**-0.5), normal(N, H), ids, gates)
    else:
        H, I = case["hidden"], case["intermediate"]
        state["args"] = (normal(case["tokens"], H, std=0.5), normal(I, H, std=H**-0.5), normal(I, H, std=H**-0.5),
                         normal(H, I, std=I**-0.5))
    return state


def run(state):
    kind = state["kind"]
    if kind == "train":
        module, x = state["module"], state["x"]
        module.zero_grad(set_to_none=True)
        x.grad = None
        y, logits = module(x)
        y.backward(state["dy"])
        norm = module.router_norm
        return dict(y=y, logits=logits, dx=x.grad, mean=norm.running_mean, var=norm.running_var,
                    grads={name: p.grad for name, p in module.named_parameters()})
    with torch.no_grad():
        if kind in ("layer", "stack"):
            return state["module"](state["x"])
        op = {"router": flash_router_func, "experts": flash_expert_func, "mlp": flash_mlp_func}[kind]
        return op(*state["args"])


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    kind = case["kind"]
    if kind == "router":
        T, nk, k = case["tokens"], case["keys"], case["top_k"]
        # the sums that can reach the k largest, (p + 1)(q + 1) <= k over the ranks of the two halves
        return dict(bytes=T * (2 * nk * size + k * (size + 8)), flops=T * sum(k // (p + 1) for p in range(k)))
    if kind == "experts":
        T, H, k = case["tokens"], case["hidden"], case["top_k"]
        rows = float(np.sum(-np.expm1(T * k * np.log1p(-np.minimum(popularity(case), 1 - 1e-12)))))  # distinct experts
        return dict(bytes=2 * rows * H * size + T * (2 * H * size + k * (8 + size)), flops=4 * T * k * H)
    if kind == "mlp":
        T, H, I = case["tokens"], case["hidden"], case["intermediate"]
        return dict(bytes=(3 * H * I + 2 * T * H) * size, flops=6 * T * H * I)
    T = case["batch"] * case["seq"]
    H, I, N, k = case["hidden"], case["intermediate"], case["experts"], case["top_k"]
    nk = math.isqrt(N)
    rows = N * -math.expm1(-T * k / N)  # distinct experts, were they equally popular
    weights = 3 * H * I + 2 * nk * H
    flops = T * (6 * H * I + 4 * H * nk + 4 * k * H)
    layers = case.get("layers", 1)
    if kind == "train":
        # both directions; the gradients of the whole tables are written
        moved = 2 * weights + 2 * rows * H + 2 * N * H + T * (4 * H + 2 * nk)
        return dict(bytes=moved * size, flops=3 * flops)
    return dict(bytes=(layers * (weights + 2 * rows * H + T * 2 * nk) + 2 * T * H) * size, flops=layers * flops)


def tolerance(case):
    if case["kind"] == "router":
        return "exact"  # sums in the type of the input, and which of equal sums comes first is defined
    f32 = case["dtype"] == "float32"
    if case["kind"] in ("experts", "mlp"):
        return dict(rel=1e-5 if f32 else 1e-2)
    # a token whose k-th and following experts tie to within the rounding of a logit may take the other one
    return dict(rel=5e-5 if f32 else 1e-2, max=1e-2 if f32 else 0.5)
