"""Timed cases of the MoE layer: what a training or serving program asks of it on one GPU, through `mok.functional`,
`mok.moe_layer` and `mok.MoKMoE`.

Shapes are those of the repository's configurations - a small layer (hidden 512), Qwen3-MoE-shaped (hidden 2048, 128
experts of 768, top-8), Mixtral-shaped (hidden 4096, 8 experts of 14336, top-2, skewed routing) and DeepSeek-V3-shaped
(hidden 7168, experts of 2048, top-8; 32 or 128 of its 256 experts, the share of one rank) - plus a generic odd one.
A case is one rank: the process group has world size 1.
"""
import math
import os
import sys

import torch
import torch.distributed as dist

_PACKAGE = os.path.join(os.getcwd(), "mixture-of-kittens_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import mok  # noqa: E402

QWEN3 = dict(hidden=2048, intermediate=768, experts=128, topk=8, weight_std=0.02)
MIXTRAL = dict(hidden=4096, intermediate=14336, experts=8, topk=2, weight_std=0.02)
DEEPSEEK = dict(hidden=7168, intermediate=2048, topk=8, weight_std=0.006)

# macrobatch: rows of the activation ring; 131072 is MoKConfig's default (several windows and the backward replay at the
# largest sizes), 0 = one window over the whole schedule.  skew: expert bias of the router logits, N(0, skew) when
# positive, Zipf(-skew) when negative.  limit: SwiGLU clamp, 0 = none.
DEFAULTS = dict(api="functional", mode="train", mxfp8=False, recompute=False, macrobatch=131072, limit=0.0, skew=0.5)


def listed():
    cases = [
        # a serving step: the smallest batch the layer takes, every expert's weights read for a few rows each
        dict(name="decode_qwen3_t512", mode="forward", tokens=512, **QWEN3),
        # prefill of a prompt batch, balanced experts of a few hundred rows
        dict(name="prefill_qwen3_t4096", mode="forward", tokens=4096, **QWEN3),
        # prefill with weights quantized once at load time, one rank's experts of a large model
        dict(name="prefill_deepseek_mxfp8_t4096", mode="forward", mxfp8=True, tokens=4096, experts=32, **DEEPSEEK),
        # the small layer as a module, device router included: forward + backward are bound by launches
        dict(name="train_small_module_t2048", api="module", tokens=2048, hidden=512, intermediate=1024, experts=8, topk=2,
             weight_std=0.02),
        # odd sizes: ragged expert loads, tile counts that divide nothing, clamped SwiGLU
        dict(name="train_odd_clamped_t3328", api="layer", tokens=3328, hidden=1792, intermediate=1280, experts=12, topk=6,
             limit=7.0, weight_std=0.02),
        # full training step of the Qwen3-MoE-shaped layer in the default ring (a second, nearly empty window)
        dict(name="train_qwen3_t16384", tokens=16384, **QWEN3),
        # low-precision training with activation checkpointing: weights quantized in the step, context recomputed
        dict(name="train_qwen3_mxfp8_recompute_t8192", api="layer", mxfp8=True, recompute=True, tokens=8192, **QWEN3),
        # few wide experts, one of them hot
        dict(name="train_mixtral_zipf_t16384", tokens=16384, skew=-1.2, **MIXTRAL),
        # low-precision training step, weights quantized in it as after every optimizer step
        dict(name="train_deepseek_mxfp8_t16384", api="layer", mxfp8=True, macrobatch=0, tokens=16384, experts=32, **DEEPSEEK),
        # many experts of about 1000 rows: what one GPU sees with few expert-parallel ranks
        dict(name="train_deepseek_128_t16384", api="layer", macrobatch=0, tokens=16384, experts=128, **DEEPSEEK),
        # 32 experts of about 8000 rows, one rank of eight, in the default ring with its backward replay: the largest
        dict(name="train_deepseek_32_t32768", tokens=32768, experts=32, **DEEPSEEK),
    ]
    return [{**DEFAULTS, **c} for c in cases]


def _log_uniform(rng, low, high, step):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))) / step) * step))


def draw(rng):
    while True:
        mxfp8 = rng.random() < 0.4
        api = rng.choice(("functional", "layer", "module"))
        c = dict(DEFAULTS, api=api, mode=rng.choice(("forward", "train", "train")), mxfp8=mxfp8,
                 recompute=api == "layer" and rng.random() < 0.4,
                 tokens=_log_uniform(rng, 512, 32768, 256), hidden=_log_uniform(rng, 512, 7168, 256),
                 intermediate=_log_uniform(rng, 512, 14336, 256), experts=_log_uniform(rng, 4, 128, 1),
                 macrobatch=rng.choice((131072, 131072, 0, 32768)), limit=rng.choice((0.0, 0.0, 7.0)),
                 skew=rng.choice((0.5, 0.5, 0.0, -1.2)))
        c["topk"] = rng.randint(1, min(8, c["experts"] // 2))
        c["weight_std"] = 0.02 if c["hidden"] <= 4096 else 0.006
        # no drawn case costs more, or holds more memory, than the largest listed one of its kind
        rows, per_row = c["tokens"] * c["topk"] + 128 * c["experts"], c["hidden"] * c["intermediate"]
        replay = 1.0 if rows <= (c["macrobatch"] or rows) or c["mode"] == "forward" else 4 / 3
        if 18 * (rows + c["tokens"]) * per_row * replay > 7e13 or c["experts"] * per_row > 1.9e9:
            continue
        if rows * (c["hidden"] + 2 * c["intermediate"]) > 4e9:
            continue
        return c


def _group():
    if not dist.is_initialized():
        torch.cuda.set_device(0)
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    return dist.group.WORLD


def _config(case):
    """The ring of the case, and a capacity that the padding of every expert to 256 rows cannot overflow."""
    routes = case["tokens"] * case["topk"]
    multiplier = max(0.5, math.ceil((routes + 256 * case["experts"]) / routes) if 256 * case["experts"] > routes else 0.5)
    macrobatch = case["macrobatch"] or -(-(routes + 256 * case["experts"]) // 4096) * 4096
    chunk = 2048 if routes * 4 % 2048 == 0 else 1024
    return mok.functional.MoKConfig(macrobatch_size=macrobatch, schedule_capacity_multiplier=multiplier,
                                    all_gather_top_experts_chunk_bytes=chunk)


def prepare(case, seed):
    group = _group()
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(seed)
    T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "intermediate", "experts", "topk"))
    train = case["mode"] == "train"

    def normal(*shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=dev).normal_(0.0, std, generator=gen)

    config = _config(case)
    state = dict(case=case, config=config, limit=case["limit"] or None, x=normal(T, H))
    if train:
        state["d_out"] = normal(T, H)
    shapes = ((I, H), (I, H), (H, I), (E, I, H), (E, I, H), (E, H, I))
    weights = [normal(*s, std=case["weight_std"]) for s in shapes]
    bias = torch.zeros(E, device=dev)
    if case["skew"] > 0:
        bias = normal(E, std=case["skew"], dtype=torch.float32)
    elif case["skew"] < 0:
        bias = (case["skew"] * torch.log(torch.arange(1, E + 1, device=dev)))[torch.randperm(E, device=dev, generator=gen)]
    if case["api"] == "module":
        layer = mok.MoKMoE(H, I, E, K, group=group, config=config, swiglu_limit=state["limit"], mxfp8=case["mxfp8"], device=dev)
        names = ("w_shared_gate", "w_shared_up", "w_shared_down", "w_routed_gate", "w_routed_up", "w_routed_down")
        with torch.no_grad():
            layer.router.copy_(normal(E, H, std=H ** -0.5, dtype=torch.float32))
            for name, w in zip(names, weights):
                getattr(layer, name).copy_(w)
        state.update(layer=layer, params=[layer.router] + [getattr(layer, n) for n in names])
        state["x"].requires_grad_(train)
        return state
    logits = normal(T, E, dtype=torch.float32) + bias
    top, experts = torch.topk(logits, K, dim=-1)
    state.update(experts=experts.contiguous(), router_weights=torch.softmax(top, dim=-1).contiguous(), weights=weights)
    state["workspace"] = mok.functional.get_workspace(config, group, device=dev, num_local_tokens=T, hidden_size=H, topk=K)
    if case["mxfp8"] and case["api"] == "functional":
        state["quantized"] = mok.quantize_routed_weights(*weights[3:])
        if not train:
            state["weights"] = weights[:3]     # a serving process keeps the quantized copies only
    if case["api"] == "layer" and train:
        for t in (state["x"], state["router_weights"], *weights):
            t.requires_grad_(True)
    return state


def _run_functional(s):
    F, case, config, ws = mok.functional, s["case"], s["config"], s["workspace"]
    schedule = F.build_schedule(ws, config, s["experts"], num_local_experts=case["experts"])
    shared, routed = s["weights"][:3], s["weights"][3:]
    backward_routed = routed
    if case["mxfp8"]:
        gate, up, down = s["quantized"]
        routed, backward_routed = (gate[:2], up[:2], down[:2]), (gate, up, down[2:])
    out, context = F.forward(config, ws, schedule, s["x"], s["router_weights"], *shared, *routed, swiglu_limit=s["limit"])
    if case["mode"] == "forward":
        return out
    grads = F.backward(config, ws, schedule, context, s["d_out"], s["x"], s["router_weights"], *shared, *backward_routed,
                       swiglu_limit=s["limit"])
    return (out, *grads)


def _run_layer(s):
    case = s["case"]
    inputs = (s["x"], s["router_weights"], *s["weights"])

    def layer():
        return mok.moe_layer(s["x"], s["experts"], s["router_weights"], *s["weights"], config=s["config"], swiglu_limit=s["limit"],
                             recompute=case["recompute"], mxfp8=case["mxfp8"])
    if case["mode"] == "forward":
        with torch.no_grad():
            return layer()
    out = layer()
    return (out.detach(), *torch.autograd.grad(out, inputs, s["d_out"]))


def _run_module(s):
    if s["case"]["mode"] == "forward":
        with torch.no_grad():
            return s["layer"](s["x"])
    out = s["layer"](s["x"])
    return (out.detach(), *torch.autograd.grad(out, [s["x"], *s["params"]], s["d_out"]))


_RUN = {"functional": _run_functional, "layer": _run_layer, "module": _run_module}


def run(state):
    return _RUN[state["case"]["api"]](state)


def work(case):
    """Each input read once, each output written once; padding rows, replayed or recomputed activations and every
    intermediate (routed rows, slots, quantized copies made in the pass) are not counted."""
    T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "intermediate", "experts", "topk"))
    train, module = case["mode"] == "train", case["api"] == "module"
    shared, routed = 3 * H * I, 3 * E * H * I
    quantized_input = case["mxfp8"] and case["api"] == "functional"
    weight_bytes = 2 * shared + routed * (1 + 1 / 32 if quantized_input else 2)
    io = 2 * T * H * 2 + (E * H * 4 if module else T * K * 12)          # x, output; router matrix, or routes and their weights
    flops = 6 * (K + 1) * T * H * I + (2 * T * H * E if module else 0)
    if train:
        weight_bytes += routed * (1 + 1 / 32) if quantized_input else 0  # the transposed copies
        weight_bytes += 2 * (shared + routed)                            # weight gradients
        io += 2 * T * H * 2 + (E * H * 4 if module else T * K * 4)       # d_output, d_x; router gradient
        flops *= 3
    return {"bytes": weight_bytes + io, "flops": flops}


def tolerance(case):
    """bf16 results (fp32 accumulation, bf16 between the steps) are 3.9e-3 away from float64 in the 2-norm and up to 0.12
    in the largest element; an MXFP8 layer that sums in another order is 1.7e-3 away."""
    return {"rel": 0.01, "max": 0.4}
