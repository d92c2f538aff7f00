"""Timing cases of the MoE layer: the calls a program makes on it, over the sizes it is used at.

A case is one forward pass of a layer (or a stack of layers) on tokens the program already holds.  The kinds:

  "resident"  experts in device memory, tokens in and out on the device (MoELayer.forward), on one stream
  "stack"     `layers` layers one behind the other, clones that share the first one's experts
  "host"      experts resident, tokens in and out in page-locked host memory (MoELayer.forward_host_ptr)
  "streamed"  experts in page-locked host memory, copied to the device by every call (max_concurrency slots)
  "cached"    the same with the layer's expert cache large enough for every expert: only a first call copies
"""
import math

import numpy as np
import torch

from infmoe_b200 import MoELayer

VARIANTS = ("default", "cpm_2", "base_layer")


def _case(name, kind, variant, E, D, F, T, zipf=0.0, layers=1):
    return {"name": name, "kind": kind, "variant": variant, "experts": E, "d_model": D, "d_ff": F, "tokens": T,
            "zipf": zipf, "layers": layers}


def listed():
    return [
        # a layer of a test or a toy model: nothing but launches and latency
        _case("tiny", "resident", "default", 4, 64, 256, 32),
        # token-by-token generation on a large layer: one, eight and 64 sequences at once
        _case("decode_1", "resident", "cpm_2", 32, 4096, 10240, 1),
        _case("decode_8", "resident", "cpm_2", 32, 4096, 10240, 8),
        _case("decode_64", "resident", "cpm_2", 32, 4096, 10240, 64),
        # encoding a batch of 8 x 512 tokens, about 128 tokens per expert: the benchmark's workload
        _case("batch_4096", "resident", "cpm_2", 32, 4096, 10240, 4096),
        # the largest batches: 512 tokens per expert
        _case("batch_16384", "resident", "cpm_2", 32, 4096, 10240, 16384),
        # skewed routing: a few of 64 experts take most of the tokens
        _case("skewed_16384", "resident", "base_layer", 64, 1024, 4096, 16384, zipf=1.1),
        # a mid-sized layer and a token count that fills no tile
        _case("ragged_777", "resident", "default", 12, 1000, 2724, 777),
        # three layers of a small model back to back, the demo program's sizes
        _case("stack_3", "stack", "cpm_2", 8, 1024, 4096, 4096, layers=3),
        # a serving process that gets its tokens in host memory and hands them back there
        _case("host_4096", "host", "cpm_2", 32, 1024, 4096, 4096),
        # experts that do not stay on the device: every call streams those it needs
        _case("streamed_64", "streamed", "cpm_2", 8, 1024, 4096, 64),
        # widths that are no multiple of four floats, which take the exact kernels
        _case("odd_width", "resident", "cpm_2", 6, 510, 1022, 300),
    ]


def _weight_bytes(c):
    return 12.0 * c["experts"] * c["d_model"] * c["d_ff"]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case; none costs more than batch_16384."""
    kind = rng.choice(["resident"] * 6 + ["stack", "host", "streamed", "cached"])
    odd = kind == "resident" and rng.random() < 0.12
    host_weights = kind in ("streamed", "cached")
    while True:
        D = 8 * _log_int(rng, 8, 512)
        F = 4 * int(round(D * rng.uniform(1.5, 4.0) / 4))
        c = _case("", kind, rng.choice(VARIANTS), _log_int(rng, 2, 64), D, F, _log_int(rng, 1, 16384))
        if odd:
            c["d_model"] -= rng.randint(1, 3)
            c["d_ff"] += rng.randint(1, 3)
        if rng.random() < 0.3:
            c["zipf"] = 1.1
        if kind == "stack":
            c["layers"] = rng.randint(2, 4)
        work = float(c["tokens"]) * c["d_model"] * c["d_ff"] * c["layers"]
        if work > (3e9 if odd else 6.8e11) or _weight_bytes(c) > (4e8 if host_weights else 1.6e10):
            continue
        del c["name"]
        return c


def _expert(gen, D, F):
    """Weights of one expert: LayerNorm near one, matrices of variance 1 / fan-in."""
    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32)

    return 1.0 + 0.01 * normal(D), normal(F, D).div_(math.sqrt(D)), normal(F, D).div_(math.sqrt(D)), normal(D, F).div_(math.sqrt(F))


def _inputs(case, seed):
    """Routing parameters, tokens and the generator that the experts' weights come from, all made from the seed."""
    E, D, T = case["experts"], case["d_model"], case["tokens"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    centroids = (0.02 * rng.standard_normal((E, D))).astype(np.float32)
    gating_ln = (1.0 + 0.01 * rng.standard_normal(D)).astype(np.float32) if case["variant"] == "cpm_2" else None
    x = torch.randn(T, D, generator=gen, device="cuda", dtype=torch.float32)
    if case["zipf"] > 0 and gating_ln is None:
        # skewed routing through the data: feature 0 is one, and centroid column 0 carries the experts' log shares,
        # scaled by the width of the scores' distribution
        share = (rng.permutation(E) + 1.0) ** -case["zipf"]
        scale = math.sqrt(6.0) / math.pi * 0.02 * math.sqrt(max(1, D - 1))
        x[:, 0] = 1.0
        centroids[:, 0] = scale * np.log(share / share.sum())
    return centroids, gating_ln, x, gen


def prepare(case, seed):
    E, D, F = case["experts"], case["d_model"], case["d_ff"]
    centroids, gating_ln, x, gen = _inputs(case, seed)
    layer = MoELayer.create(E, D, F, 2, centroids, None, "T5_FF", case["variant"], gating_ln)
    host = case["kind"] in ("streamed", "cached")
    for e in range(E):
        weights = _expert(gen, D, F)
        layer.set_expert(e, *([w.cpu().numpy() for w in weights] if host else weights))
    layer.set_residency(0 if host else 1)
    if case["kind"] == "cached":
        layer.set_expert_cache(E)
    state = {"kind": case["kind"], "layers": [layer] + [layer.clone() for _ in range(case["layers"] - 1)], "x": x}
    if case["kind"] == "host":
        state["x"] = x.cpu().pin_memory()
        state["out"] = torch.empty_like(state["x"]).pin_memory()
    return state


def run(state):
    x = state["x"]
    if state["kind"] == "host":
        state["layers"][0].forward_host_ptr(x.data_ptr(), state["out"].data_ptr(), x.shape[0])
        return state["out"]
    for layer in state["layers"]:
        x = layer.forward(x)
    return x


def work(case):
    E, D, F, T = case["experts"], case["d_model"], case["d_ff"], case["tokens"]
    share = (np.arange(E) + 1.0) ** -(case["zipf"] if case["variant"] != "cpm_2" else 0.0)
    active = float((1.0 - (1.0 - share / share.sum()) ** T).sum())                 # experts that get a token, on average
    one = 12.0 * active * D * F + 4.0 * E * D + 8.0 * T * D                        # weights, centroids, rows in and out
    return {"bytes": case["layers"] * one, "flops": case["layers"] * (6.0 * T * D * F + 2.0 * T * D * E)}


def tolerance(case):
    # FP32 in and out.  The layer output x + FFN(x) of the split-operand tensor-core products is 1e-6 to 3e-6
    # (2-norm) from an evaluation in 64 bits; a stack adds its layers' errors.
    return {"rel": 1e-5 * case["layers"], "max": 2e-4 * case["layers"]}


def exact(case, seed):
    """The layer's definition in 64 bits."""
    centroids, gating_ln, x, gen = _inputs(case, seed)
    D, F = case["d_model"], case["d_ff"]
    experts = [_expert(gen, D, F) for _ in range(case["experts"])]
    centroids = torch.from_numpy(centroids).cuda().double()

    def layer_norm(v, gamma):
        centred = v - v.mean(1, keepdim=True)
        return gamma.double() * centred / torch.sqrt(centred.square().mean(1, keepdim=True) + 1e-6)

    x = x.double()
    for _ in range(case["layers"]):
        scored = x if gating_ln is None else layer_norm(x, torch.from_numpy(gating_ln).cuda())
        score, gate = (scored @ centroids.T).max(1)
        out = x.clone()
        for e, (ln, wi0, wi1, wo) in enumerate(experts):
            rows = (gate == e).nonzero()[:, 0]
            if rows.numel():
                h = layer_norm(x[rows], ln)
                g = torch.nn.functional.gelu(h @ wi0.double().T, approximate="tanh") * (h @ wi1.double().T)
                out[rows] += g @ wo.double().T
        if case["variant"] == "base_layer":
            alpha = torch.sigmoid(score)[:, None]
            out = alpha * out + (1.0 - alpha) * x
        x = out
    return x.cpu() if case["kind"] == "host" else x
