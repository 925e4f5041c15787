"""What this library is asked to do in earnest, as timed cases over its public entry points.

Paths (`case["path"]`):
  forward   `provider.apply` without gradients: decode steps and prefill of a served layer
  train     `provider.apply` and `torch.autograd.grad`: one layer's share of a training step
  lora      `lora.expert_lora` on a frozen base and the factors' gradients
  gemm      `ops.grouped_gemm_fp8` alone, for hosts that orchestrate the layer themselves
  publish   `BlockFP8Weight.copy_(master)`: the fp32 master weights quantised into the expert
            container after an optimizer step

The expert weights are block-FP8 containers (`experts="fp8"`) or plain bf16 tensors. Layer
shapes are the ones the benchmark runs (see `SHAPES`) and, in `draw`, others of the same ranges.
"""

import math

import torch

from mlops_b200 import lora, ops, provider
from mlops_b200.weights import BlockFP8Weight

# D hidden width, F expert width, E experts, K experts per token
SHAPES = {
    # the small layer of the CPU-runnable configuration
    "small": dict(D=256, F=512, E=8, K=2, mode="softmax_then_topk"),
    # few wide experts (Mixtral-8x7B-shaped)
    "wide": dict(D=4096, F=14336, E=8, K=2, mode="softmax_then_topk"),
    # many narrow experts (Qwen3-30B-A3B-shaped)
    "fine": dict(D=2048, F=768, E=128, K=8, mode="softmax_then_topk"),
    # group-limited sigmoid routing beside a shared expert (DeepSeek-V3-shaped)
    "grouped": dict(D=7168, F=2048, E=256, K=8, mode="sigmoid_noaux_tc", n_group=8, topk_group=4, scaling=2.5,
                    shared=True),
}
LAYER = dict(n_group=1, topk_group=1, scaling=1.0, shared=False, experts="fp8", grad="bf16", zipf=0.0)
WEIGHT_STD = 0.02
BIAS_STD = 0.001  # a trained selection bias balances the load; this exercises it near balance


def _layer(path, shape, T, **changes):
    return dict(LAYER, path=path, T=T, **{**SHAPES[shape], **changes})


def listed():
    return [
        # one sequence's next token: the smallest call, launches and host time only
        dict(_layer("forward", "fine", 1), name="fine_decode_1"),
        # a decode batch over all 256 experts: every expert's weights read for a few rows each
        dict(_layer("forward", "grouped", 64), name="grouped_decode_64"),
        # a prompt of odd length
        dict(_layer("forward", "fine", 3001), name="fine_prefill_3001"),
        # a full prefill batch over all 256 experts, about 256 rows per expert
        dict(_layer("forward", "grouped", 8192), name="grouped_prefill_8192"),
        # the small layer's training step
        dict(_layer("train", "small", 512), name="small_train_512"),
        # an ordinary training micro-batch of odd length, gradients for fp32 masters
        dict(_layer("train", "fine", 4099, grad="fp32"), name="fine_train_4099"),
        # the wide layer's full training batch: the largest products
        dict(_layer("train", "wide", 16384), name="wide_train_16384"),
        # one GPU's share of the 256-expert layer sharded over four: 1024 rows per expert
        dict(_layer("train", "grouped", 8192, E=64), name="grouped_train_8192"),
        # adapter fine-tuning with skewed expert load, from one row to most of the batch per expert
        dict(_layer("lora", "fine", 65536, zipf=1.2, rank=16), name="fine_lora_65536"),
        # experts kept in bf16
        dict(_layer("train", "wide", 4096, experts="bf16"), name="wide_bf16_train_4096"),
        # the grouped product alone, skewed groups of 415 to 18668 rows
        dict(path="gemm", groups=32, rows=65536, D=4096, N=2048, zipf=1.1, along="rows", scales="1x128",
             name="gemm_zipf_65536"),
        # one optimizer step's publication of both expert weights
        dict(path="publish", D=2048, F=768, E=128, name="fine_publish"),
    ]


def _spread(rng, low, high):
    """A whole number, spread evenly over the logarithm of [low, high]."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    path = rng.choices(["forward", "train", "lora", "bf16", "gemm", "publish"], weights=[5, 5, 2, 2, 2, 1])[0]
    if path == "gemm":
        return dict(path="gemm", groups=rng.randint(1, 64), rows=_spread(rng, 64, 65536), D=128 * rng.randint(4, 56),
                    N=128 * rng.randint(4, 32), zipf=rng.choice([0.0, 1.1]), along=rng.choice(["rows", "columns"]),
                    scales=rng.choice(["1x128", "row"]))
    if path == "publish":
        return dict(path="publish", D=128 * _spread(rng, 2, 56), F=128 * _spread(rng, 2, 24), E=_spread(rng, 4, 64))
    shape = rng.choice(["small", "wide", "fine", "grouped", "other"])
    if shape == "other":
        experts = rng.choice([8, 16, 32, 64])
        changes = dict(D=128 * rng.randint(4, 40), F=128 * rng.randint(4, 24), E=experts, K=rng.choice([1, 2, 4, 6, 8]),
                       mode=rng.choice(["softmax_then_topk", "topk_then_softmax", "sigmoid_noaux_tc"]))
        shape = "fine"
    elif shape == "grouped":
        changes = dict(E=rng.choice([64, 256]) if path == "forward" else rng.choice([32, 64]))
    else:
        changes = {}
    if path == "forward":
        return _layer("forward", shape, _spread(rng, 2, 8192), **changes)
    if path == "train":
        return _layer("train", shape, _spread(rng, 64, 8192), grad=rng.choice(["bf16", "bf16", "fp32"]),
                      zipf=rng.choice([0.0, 0.0, 1.2]), **changes)
    if path == "bf16":
        changes["shared"] = False
        return _layer("train", shape, _spread(rng, 64, 4096), experts="bf16", **changes)
    changes["shared"] = False
    return _layer("lora", shape, _spread(rng, 64, 16384), rank=rng.choice([8, 16, 32, 64]), zipf=rng.choice([0.0, 1.2]),
                  **changes)


# ------------------------------------------------------------------------------ inputs
def _randn(generator, *shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=generator, device="cuda", dtype=dtype).mul_(std)


def _experts(generator, kind, experts, out, inner, dtype):
    """`[E, out, in]` expert weights, drawn and quantised a few experts at a time."""
    if kind == "bf16":
        return _randn(generator, experts, out, inner, std=WEIGHT_STD)
    data = torch.empty((experts, out, inner), dtype=torch.float8_e4m3fn, device="cuda")
    scale = torch.empty((experts, out // 128, inner // 128), dtype=torch.float32, device="cuda")
    step = max(1, (1 << 29) // (out * inner))
    for low in range(0, experts, step):
        part = _randn(generator, min(step, experts - low), out, inner, std=WEIGHT_STD)
        data[low:low + step], scale[low:low + step] = ops.quantize_blocks(part)
    return BlockFP8Weight(data, scale, dtype=dtype)


def _offsets(generator, groups, rows, zipf):
    """Row ranges of the groups: a multinomial split of `rows` with Zipf popularity."""
    popularity = torch.arange(1, groups + 1, device="cuda", dtype=torch.float32).pow(-zipf)
    drawn = torch.multinomial(popularity, rows, replacement=True, generator=generator)
    counts = torch.bincount(drawn, minlength=groups)
    return torch.cat([counts.new_zeros(1), counts.cumsum(0)]).to(torch.int32)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["path"] == "gemm":
        inner, out = case["D"], case["N"]
        a_q, a_scale = ops.quantize_rows(_randn(g, case["rows"], inner),
                                         mode="1x128" if case["scales"] == "1x128" else "row")
        shape = (out, inner) if case["along"] == "rows" else (inner, out)
        b_q, b_scale = ops.quantize_blocks(_randn(g, case["groups"], *shape))
        return dict(case=case, operands=(a_q, a_scale, b_q, b_scale,
                                         _offsets(g, case["groups"], case["rows"], case["zipf"])))
    D, F, E = case["D"], case["F"], case["E"]
    if case["path"] == "publish":
        masters = [_randn(g, E, 2 * F, D, std=WEIGHT_STD, dtype=torch.float32),
                   _randn(g, E, D, F, std=WEIGHT_STD, dtype=torch.float32)]
        return dict(case=case, masters=masters,
                    containers=[BlockFP8Weight(torch.zeros(m.shape, dtype=torch.float8_e4m3fn, device="cuda"),
                                               torch.zeros((E, m.shape[1] // 128, m.shape[2] // 128), device="cuda"))
                                for m in masters])

    trains = case["path"] == "train"
    x, residual = _randn(g, case["T"], D), _randn(g, case["T"], D)
    router = _randn(g, E, D, std=WEIGHT_STD, dtype=torch.float32)
    if case["zipf"]:  # the skew lives in the data: x[:, 0] = 1 and router[:, 0] = log popularity
        popularity = torch.arange(1, E + 1, device="cuda", dtype=torch.float32).pow(-case["zipf"])
        router[:, 0] = torch.log(popularity / popularity.sum())
        x[:, 0] = 1.0
    logical = torch.float32 if case["grad"] == "fp32" else torch.bfloat16
    w13 = _experts(g, case["experts"], E, 2 * F, D, logical)
    w2 = _experts(g, case["experts"], E, D, F, logical)
    state = dict(case=case, x=x, residual=residual, router=router, w13=w13, w2=w2, extra=[], shared={},
                 routing=dict(top_k=case["K"], routing_mode=case["mode"], n_group=case["n_group"],
                              topk_group=case["topk_group"], routed_scaling=case["scaling"]))
    if case["mode"] == "sigmoid_noaux_tc":
        state["routing"]["router_bias"] = _randn(g, E, std=BIAS_STD, dtype=torch.float32)
    if case["path"] == "lora":
        r = case["rank"]
        state["extra"] = [_randn(g, E, r, D, std=0.02), _randn(g, E, 2 * F, r, std=0.01),
                          _randn(g, E, r, F, std=0.02), _randn(g, E, D, r, std=0.01)]
    elif case["shared"]:
        state["extra"] = [_randn(g, 2 * F, D, std=WEIGHT_STD), _randn(g, D, F, std=WEIGHT_STD)]
        state["shared"] = dict(shared_w13=state["extra"][0], shared_w2=state["extra"][1])
    if case["path"] != "forward":
        state["dy"] = _randn(g, case["T"], D)
        # what a trainer differentiates: the inputs, and every weight that is not frozen
        state["leaves"] = [x, residual, *([router, w13, w2] if trains else []), *state["extra"]]
        for leaf in state["leaves"]:
            leaf.requires_grad_(True)
    return state


# ------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    if case["path"] == "gemm":
        return ops.grouped_gemm_fp8(*state["operands"], b_mn_major=case["along"] == "columns")
    if case["path"] == "publish":
        with torch.no_grad():
            for container, master in zip(state["containers"], state["masters"]):
                container.copy_(master)
        return [container.components() for container in state["containers"]]
    layer = (state["x"], state["residual"], state["router"], state["w13"], state["w2"])
    if case["path"] == "forward":
        with torch.no_grad():
            return provider.apply(*layer, **state["routing"], **state["shared"])
    if case["path"] == "lora":
        results = lora.expert_lora(*layer, *state["extra"], scale=1.0, **state["routing"])
    else:
        results = provider.apply(*layer, **state["routing"], **state["shared"])
    return [*(t.detach() for t in results), *torch.autograd.grad(results[0], state["leaves"], state["dy"])]


# --------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: each input read once (of the experts, those that get rows), each output written once.
    FLOPs: the products."""
    if case["path"] == "gemm":
        rows, inner, out, groups = case["rows"], case["D"], case["N"], min(case["groups"], case["rows"])
        return dict(bytes=rows * inner * 1.03 + groups * inner * out + 2 * rows * out, flops=2 * rows * inner * out)
    D, F, E = case["D"], case["F"], case["E"]
    expert = 3 * D * F  # elements of one expert's weights
    if case["path"] == "publish":
        return dict(bytes=5 * E * expert, flops=0)
    T, rows = case["T"], case["T"] * case["K"]
    bf16 = case["experts"] == "bf16"
    active = E * (1 - (1 - case["K"] / E) ** T)  # expected number of experts that get a token
    nbytes = 2 * 3 * T * D + 4 * E * D + active * expert * (2 if bf16 else 1)
    flops = 2 * T * D * E + 2 * rows * expert
    if case["shared"]:
        nbytes += 2 * expert
        flops += 2 * T * expert
    if case["path"] == "forward":
        return dict(bytes=nbytes, flops=flops)
    nbytes *= 2  # the weights and the tokens are read again; gradients of the tokens go out
    factors = case["rank"] * (2 * D + 3 * F) if case["path"] == "lora" else 0
    if case["path"] == "lora":
        nbytes += 2 * 3 * E * factors
        return dict(bytes=nbytes, flops=2 * flops + 6 * rows * factors)
    nbytes += E * expert * (4 if case["grad"] == "fp32" else 2) + 4 * E * D + (2 * expert if case["shared"] else 0)
    return dict(bytes=nbytes, flops=3 * flops)


def tolerance(case):
    """About four times what the path shows against itself with its products' sums in 64 bits (from
    the same operands): single bf16 results round the other way, and through them single E4M3
    operands of the next product. The rank-r terms of adapters are rounded to bf16 themselves."""
    if case["path"] == "publish":
        return "exact"
    if case["path"] == "gemm":  # measured 2e-5, at most one bf16 step
        return {"rel": 1e-4, "max": 3e-2}
    if case["path"] == "lora":  # measured 1.5e-3; 0.26 on a single value where a block's scale moved
        return {"rel": 6e-3, "max": 0.9}
    if case["experts"] == "bf16":  # measured 1.8e-3; 4.4e-2 on a single value
        return {"rel": 7e-3, "max": 2e-1}
    return {"rel": 2e-3, "max": 1e-1}  # measured 4.8e-4; 2.7e-2 on a single value
