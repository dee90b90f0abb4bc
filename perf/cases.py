"""The work that a user of this package has it do, as cases that can be timed and compared.

A case is one layer of one configuration on one batch, driven through the public modules: ``LatentMoELayer`` (bf16, or with
its routed experts in e4m3), the non-latent ``MoELayer``, ``NormedResidualFFN`` around the layer, and ``GraphedLatentMoE``.
``direction`` "infer" is a forward pass under ``no_grad`` (generation, prompt processing, validation); "train" is what one
micro-step of a training loop does with the layer: forward, backward from the upstream gradient and the router's z-loss,
and the router's bias update.  Widths, expert counts and dtypes are those of the package's own workloads
(``swamla_b200/workloads.py``: the moe-1b and moe-2b shapes, 64 base experts, the non-latent layer).
"""
import gc
import math
from types import SimpleNamespace

import torch

from swamla_b200.block import NormedResidualFFN
from swamla_b200.graphs import GraphedLatentMoE
from swamla_b200.layer import create_moe_layer

BF16 = torch.bfloat16
D = 1024                 # n_embd of every benchmark configuration
RATIO = 4                # latent_ratio

#: base experts, base activated experts, expert_dim (the latent layer multiplies the first two by RATIO)
SHAPES = {"1b": (32, 3, 1024), "2b": (32, 3, 3072), "64e": (64, 4, 1024)}


def _case(name, layer, direction, shape, batch, seq, dtype="bf16", skew=0.0, update=True):
    """``layer``: latent | fp8 | moe | block | graphed.  ``dtype``: "bf16", or "mixed" for an fp32 residual stream with fp32
    linear weights and bf16 expert weights.  ``skew``: height of a Zipf(1.2) selection bias over the experts.
    ``update``: whether this micro-step ends an optimizer step, i.e. the selection bias is updated after it."""
    return dict(name=name, layer=layer, direction=direction, shape=shape, batch=batch, seq=seq, dtype=dtype, skew=skew,
                update=update)


def listed():
    return [
        # generation, one stream: the smallest call there is
        _case("decode_1x1", "latent", "infer", "1b", 1, 1),
        # generation, an odd number of streams
        _case("decode_23x1", "latent", "infer", "1b", 23, 1),
        # a prompt of ragged length
        _case("prefill_1x777", "latent", "infer", "1b", 1, 777),
        # validation batch of the wide layer
        _case("eval_4x2048_2b", "latent", "infer", "2b", 4, 2048),
        # small micro-batch of training
        _case("train_2x512", "latent", "train", "1b", 2, 512),
        # the benchmark's own step, replayed as CUDA graphs
        _case("train_8x2048_graphed", "graphed", "train", "1b", 8, 2048),
        # the block around the layer under mixed-precision training, ragged sequences
        _case("block_3x1365_mixed", "block", "train", "1b", 3, 1365, dtype="mixed"),
        # large batch of the wide layer with skewed load; a micro-step inside gradient accumulation (no bias update)
        _case("train_32x2048_2b_skewed", "latent", "train", "2b", 32, 2048, skew=0.25, update=False),
        # 256 experts, top-16
        _case("train_16x2048_64e", "latent", "train", "64e", 16, 2048),
        # e4m3 experts: a ragged mid-size batch and the largest one
        _case("fp8_5x411", "fp8", "train", "1b", 5, 411),
        _case("fp8_64x2048", "fp8", "train", "1b", 64, 2048),
        # the non-latent layer (experts at the model width)
        _case("moe_2x2048", "moe", "train", "1b", 2, 2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    layer = rng.choice(["latent", "latent", "latent", "fp8", "block", "graphed", "moe"])
    direction = "train" if layer == "graphed" else rng.choice(["infer", "train"])
    shape = rng.choice(["1b", "2b", "64e"]) if layer in ("latent", "block") else "1b"
    skew = rng.choice([0.0, 0.0, 0.25]) if layer == "latent" else 0.0
    dtype = rng.choice(["bf16", "mixed"]) if layer == "block" else "bf16"
    if direction == "infer" and rng.random() < 0.5:
        batch, seq = _log_int(rng, 1, 128), 1                                    # generation
    else:
        most = {"graphed": 16384, "moe": 8192, "fp8": 65536}.get(layer, 32768)
        if direction == "infer":
            most = min(most, 16384)
        tokens = _log_int(rng, 64 if direction == "infer" else 256, most)
        batch = min(rng.choice([1, 2, 3, 4, 8, 16]), max(1, tokens // 64))
        seq = max(1, tokens // batch)
    return {k: v for k, v in _case("", layer, direction, shape, batch, seq, dtype, skew, direction == "train" and skew == 0).items()
            if k != "name"}


def _config(case):
    n_experts, n_activated, expert_dim = SHAPES[case["shape"]]
    return SimpleNamespace(n_embd=D, n_experts=n_experts, n_activated=n_activated, n_shared_experts=1, latent_ratio=RATIO,
                           expert_dim=expert_dim, bias=False, dropout=0.0, router_z_loss_coef=0.001,
                           use_latent_moe=case["layer"] != "moe", moe_fp8=case["layer"] == "fp8")


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(dev).manual_seed(seed)
    with torch.device(dev):
        layer = create_moe_layer(_config(case), use_latent=case["layer"] != "moe")
    mixed = case["dtype"] == "mixed"
    with torch.no_grad():
        for name, p in layer.named_parameters():
            p.normal_(0.0, 0.02, generator=g)
            if not (mixed and "experts." not in name.replace("shared_experts", "shared")):
                p.data = p.data.to(BF16)          # the routed experts are bf16 in either mode
        if case["skew"] > 0:
            E = layer.n_experts
            height = case["skew"] * torch.arange(1, E + 1, device=dev, dtype=torch.float32).pow(-1.2)
            layer.router.expert_bias[torch.randperm(E, device=dev, generator=g)] = height
    x_dtype = torch.float32 if mixed else BF16
    shape = (case["batch"], case["seq"], D)
    x = torch.randn(shape, device=dev, generator=g, dtype=torch.float32).to(x_dtype)
    train = case["direction"] == "train"
    layer.train(train)
    module = layer
    if case["layer"] == "block":
        module = NormedResidualFFN(layer, D).to(dev).train(train)
        if not mixed:
            module.ffn_norm.to(BF16)
    state = SimpleNamespace(case=case, layer=layer, module=module, x=x)
    if train:
        state.dy = torch.randn(shape, device=dev, generator=g, dtype=torch.float32).to(x_dtype)
        state.x.requires_grad_(True)
        state.d_aux = torch.ones((), device=dev)
        if case["layer"] == "graphed":
            gc.collect()                 # an earlier replayed layer must not be destroyed while this one is captured
            state.module = GraphedLatentMoE(layer, x)
        state.params = list(layer.parameters() if case["layer"] == "graphed" else module.parameters())
    return state


def run(state):
    if state.case["direction"] == "infer":
        with torch.no_grad():
            return state.module(state.x)
    state.x.grad = None
    for p in state.params:
        p.grad = None
    y = state.module(state.x)
    aux = state.layer.get_aux_loss()
    torch.autograd.backward((y, aux), (state.dy, state.d_aux))
    router = state.layer.router
    out = [y, aux, state.x.grad, [p.grad for p in state.params]]
    if state.case["update"]:
        router.update_bias_from_last_forward()
        out += [router.expert_bias, router.load_history]
    return out


def work(case):
    n_experts, n_activated, Fs = SHAPES[case["shape"]]
    latent = case["layer"] != "moe"
    r = RATIO if latent else 1
    E, K, L, F = n_experts * r, n_activated * r, D // r, Fs // r
    T = case["batch"] * case["seq"]
    flops = T * (2 * D * E + 6 * D * Fs + 6 * K * L * F + (4 * D * L if latent else 0))
    dense = D * E + 3 * D * Fs + (2 * D * L if latent else 0)
    experts = E * 3 * L * F
    wide = 4 if case["dtype"] == "mixed" else 2
    if case["direction"] == "infer":
        used = 1.0 - (1.0 - K / E) ** T                      # share of the experts that the tokens meet
        return {"bytes": 2 * wide * T * D + wide * dense + 2 * experts * used, "flops": flops}
    # x, dy in; y, dx out; every parameter in, its gradient out
    return {"bytes": 4 * wide * T * D + 2 * wide * dense + 2 * 2 * experts, "flops": 3 * flops}


def tolerance(case):
    if case["layer"] == "fp8":
        # e4m3 operands: a difference of one bf16 ulp before a quantisation moves results across e4m3 steps
        return {"rel": 2e-2, "max": 0.4}
    return {"rel": 1e-2, "max": 0.2}
