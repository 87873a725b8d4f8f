"""Performance cases of the routed-expert layer: what a training or serving program has it do.

Every case is one MoE layer on one GPU (all of the named experts local), called through the public entry points
(``create_context``, ``prepare_block_scaled_weight``, ``routed_experts``).  The configurations are the ones the
benchmark and the tests of this repository name, plus ragged ones of the same ranges:

* training (BF16, MXFP8): forward and backward of ``routed_experts`` in eager mode, returning the output and all
  gradients; weight gradients either come back from autograd or are accumulated in place into ``.grad``;
* inference (BF16, MXFP8, NVFP4): the forward; prefill is called eagerly, decode replays a CUDA graph that the
  program captured once, after copying the step's tokens and routing into the graph's input tensors.
"""

from __future__ import annotations

import math
import random

import torch

import dist_moe_b200 as dm

DEVICE = "cuda:0"

_DEFAULTS = dict(
    family="bf16",        # bf16 | mxfp8 | nvfp4
    train=False,          # forward + backward, or forward only
    T=16, D=256, F=256, E=8, K=2,
    routing="uniform",    # uniform | zipf (skewed expert popularity) | hot (half of the routes on E/8 experts) | cyclic
    scores="softmax",     # softmax over the chosen experts | sigmoid | equal
    score_dtype="float32",
    ids="int64",
    clamped=False,        # clamped SwiGLU (limit 7.0)
    norm=False,           # fused post-expert RMSNorm
    slots="default",      # default (layer input kept, the rest recomputed) | full (activations kept)
    grads="fresh",        # fresh (returned by autograd) | accumulate (added into .grad in place)
    grad_dtype="bfloat16",
    weights="prepared",   # MXFP8 training: prepared (quantised once for many micro-batches) | tensor (in every call)
    graph=False,          # inference: replay of a captured CUDA graph
)


def _case(name=None, **fields):
    unknown = set(fields) - set(_DEFAULTS)
    if unknown:
        raise ValueError(f"unknown case fields {sorted(unknown)}")
    case = {**_DEFAULTS, **fields}
    return {"name": name, **case} if name else case


def listed():
    layer = dict(T=4096, D=2048, F=1408, K=6)                       # the BF16 training layer of the benchmark
    mx_layer = dict(family="mxfp8", D=4096, F=1536, E=128, K=8)     # the MXFP8 training layer of the benchmark
    mx_infer = dict(family="mxfp8", D=2816, F=2816, E=128, K=4, clamped=True, norm=True)
    nv_share = dict(family="nvfp4", D=7168, F=2048, E=32, K=8, scores="sigmoid")  # one rank's experts of 256 at EP=8
    return [
        # a first program (the quick start of the README's configuration list): launches and host work count
        _case("bf16-train-quickstart", train=True, T=16, routing="cyclic", scores="equal"),
        # a training step's layer, one micro-batch of a gradient-accumulation step
        _case("bf16-train-layer", train=True, E=64, slots="full", grads="accumulate", **layer),
        # the same layer as one of eight expert-parallel ranks sees it (8 large experts), fp32 main gradients
        _case("bf16-train-ep8-share", train=True, E=8, slots="full", grads="accumulate", grad_dtype="float32", **layer),
        # fine-tuning on ragged sizes with the default memory policy (activations recomputed), bf16 scores, int32 ids
        _case("bf16-train-ragged", train=True, T=1531, D=1088, F=704, E=24, K=3, clamped=True, score_dtype="bfloat16",
              ids="int32"),
        # decoding a batch of 32 sequences with BF16 weights
        _case("bf16-decode", T=32, D=2048, F=1408, E=64, K=6, graph=True),
        # scoring / prefill of one long prompt with BF16 weights
        _case("bf16-prefill", T=1999, D=2048, F=1408, E=64, K=6),
        # the largest training step: skewed expert popularity, weights prepared once per optimiser step
        _case("mxfp8-train-layer", train=True, T=8192, routing="zipf", slots="full", grads="accumulate", **mx_layer),
        # a small MXFP8 training layer with tensor weights (quantised in the call) and the default memory policy
        _case("mxfp8-train-small", family="mxfp8", train=True, T=777, D=1024, F=640, E=16, K=4, weights="tensor"),
        # serving: prefill of 4096 tokens, clamped SwiGLU, fused RMSNorm
        _case("mxfp8-prefill", T=4096, **mx_infer),
        # serving: decoding 16 sequences, half of the routes on the first experts
        _case("mxfp8-decode", T=16, routing="hot", graph=True, **mx_infer),
        # serving: decoding 128 sequences with NVFP4 weights
        _case("nvfp4-decode", T=128, graph=True, **nv_share),
        # serving: prefill of 8192 tokens with NVFP4 weights
        _case("nvfp4-prefill", T=8192, **nv_share),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the listed ranges."""
    bound = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["bf16-train", "bf16-infer", "mxfp8-train", "mxfp8-infer", "nvfp4-infer"])
        family, mode = kind.split("-")
        train = mode == "train"
        c = dict(family=family, train=train, ids=rng.choice(["int64", "int32"]),
                 score_dtype=rng.choice(["float32", "float32", "bfloat16"]), clamped=rng.random() < 0.3,
                 routing=rng.choice(["uniform", "uniform", "zipf", "hot"]))
        if family == "bf16":
            c.update(T=_log_int(rng, 8 if train else 1, 4096), D=64 * rng.randint(4, 32), F=64 * rng.randint(4, 24),
                     E=rng.choice([4, 8, 16, 24, 32, 48, 64]))
        elif family == "mxfp8":
            c.update(T=_log_int(rng, 16 if train else 1, 8192), D=128 * rng.randint(4, 32), F=128 * rng.randint(3, 22),
                     E=rng.choice([8, 16, 32, 64, 128]))
        else:
            c.update(T=_log_int(rng, 1, 8192), D=256 * rng.randint(8, 28), F=256 * rng.randint(3, 8),
                     E=rng.choice([8, 16, 32]), scores="sigmoid")
        c["K"] = rng.randint(1, min(8, c["E"] // 2))
        if train:
            c.update(slots=rng.choice(["default", "full"]), grads=rng.choice(["fresh", "accumulate"]),
                     grad_dtype=rng.choice(["bfloat16", "bfloat16", "float32"]),
                     weights=rng.choice(["prepared", "tensor"]) if family == "mxfp8" else "prepared")
        else:
            c.update(norm=rng.random() < 0.25, graph=c["T"] <= 256)
        case = _case(**c)
        if _cost(case) <= bound:
            return case


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 300.0)


def work(case):
    """Bytes and operations one pass cannot do without: inputs read once, outputs written once."""
    T, D, F, E, K = (case[k] for k in ("T", "D", "F", "E", "K"))
    rows = T * K
    per_element = {"bf16": 2.0, "mxfp8": 1.0 + 1.0 / 32, "nvfp4": 0.5 + 1.0 / 16}[case["family"]]
    if case["train"] and case["weights"] == "tensor" and case["family"] == "mxfp8":
        per_element = 2.0
    hit = E * (1.0 - (1.0 - K / E) ** T)  # experts some token is expected to choose
    tokens = T * D * 2 + T * K * ((8 if case["ids"] == "int64" else 4) + (4 if case["score_dtype"] == "float32" else 2))
    weights = 3.0 * D * F * hit * per_element
    total, flops = tokens + weights + T * D * 2, 6.0 * rows * D * F
    if case["train"]:
        grad = 3.0 * D * F * (4 if case["grad_dtype"] == "float32" else 2)
        total += 2 * T * D * 2 + T * K * 4  # output gradient in, input and score gradients out
        total += 2 * grad * hit if case["grads"] == "accumulate" else grad * E
        flops *= 3.0
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Largest difference another correct implementation at the same precision would show.

    Measured on a B200 against the same layer in 64-bit arithmetic with the same quantisation points and no other
    rounding (777 to 4096 tokens, D 256 to 7168): BF16 relative 4e-3 and largest 4.5e-2, over outputs and all gradients;
    MXFP8 1.8e-2 to 3.2e-2 and 0.42, because a bf16 rounding more or less in front of a quantiser moves whole E4M3
    steps; NVFP4 likewise 7e-2 and 0.54.  The block-scaled paths are held to less than that, 3e-2.
    """
    if case["family"] == "bf16":
        return {"rel": 1e-2, "max": 0.15}
    return {"rel": 3e-2, "max": 0.9}


# ------------------------------------------------------------------------------------------------------------------
class _State:
    """What a program keeps: the context, its weights, this step's tokens, routing and output gradient."""

    def __init__(self):
        self.graph = None
        self.context = None

    def __del__(self):
        if self.graph is not None:
            torch.cuda.synchronize(DEVICE)
            self.graph = None
        if self.context is not None:
            self.context.close()
            self.context = None


def _routing(case, gen):
    T, E, K = case["T"], case["E"], case["K"]
    if case["routing"] == "cyclic":
        ids = (torch.arange(T, device=DEVICE)[:, None] * K + torch.arange(K, device=DEVICE)[None, :]) % E
        values = torch.zeros(T, K, device=DEVICE)
    else:
        logits = torch.randn(T, E, device=DEVICE, generator=gen)
        if case["routing"] == "zipf":
            # a popularity of its own for every expert, drawn with the rest of the inputs
            rank = torch.randperm(E, device=DEVICE, generator=gen).float() + 1.0
            logits = logits - 0.5 * torch.log(rank)
        if case["routing"] == "hot" and K > 1:
            hot = max(K // 2, E // 8)
            a, b = torch.topk(logits[:, :hot], K // 2), torch.topk(logits[:, hot:], K - K // 2)
            values, ids = torch.cat([a.values, b.values], 1), torch.cat([a.indices, b.indices + hot], 1)
        else:
            values, ids = torch.topk(logits, K)
    if case["scores"] == "equal":
        scores = torch.full((T, K), 1.0 / K, device=DEVICE)
    elif case["scores"] == "sigmoid":
        scores = torch.sigmoid(values)
    else:
        scores = torch.softmax(values, -1)
    return ids.to(getattr(torch, case["ids"])).contiguous(), scores.to(getattr(torch, case["score_dtype"])).contiguous()


def _config(case):
    policy = None
    if case["family"] != "bf16":
        fmt = dm.BlockScaledFormat.NVFP4 if case["family"] == "nvfp4" else dm.BlockScaledFormat.MXFP8_E4M3
        policy = dm.BlockScaledConfig(format=fmt)
    extra = dict(activation="swiglu_clamped", swiglu_limit=7.0) if case["clamped"] else {}
    if case["train"]:
        extra["wgrad_dtype"] = getattr(torch, case["grad_dtype"])
        if case["slots"] == "full":
            extra["activation_slot_capacity_factor"] = 1.0
    else:
        extra.update(inference=True, num_activation_slots=0)
    return dm.Config(max_num_local_input_tokens=case["T"], hidden_dim=case["D"], intermediate_dim=case["F"],
                     top_k=case["K"], num_experts=case["E"], max_moe_layers_per_activation_slot=1, block_scaled=policy,
                     **extra)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    T, D, F, E, K = (case[k] for k in ("T", "D", "F", "E", "K"))

    def normal(*shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(*shape, device=DEVICE, dtype=dtype).normal_(0.0, std, generator=gen)

    s = _State()
    s.case = case
    s.x = normal(T, D)
    s.ids, s.scores = _routing(case, gen)
    cfg = _config(case)
    s.context = dm.create_context(group=None, config=cfg, device=DEVICE)
    std = 0.02 if D >= 1024 else D ** -0.5
    s.w13, s.w2 = normal(E, 2, F, D, std=std), normal(E, D, F, std=std)
    post = dm.RMSNormPostprocess(eps=1e-6, norm_output_dtype=torch.float32, output_dtype=torch.bfloat16) \
        if case["norm"] else None
    if case["train"]:
        s.grad_out = normal(T, D)
        s.w13.requires_grad_(True)
        s.w2.requires_grad_(True)
        s.operands = (s.w13, s.w2)
        if case["family"] == "mxfp8" and case["weights"] == "prepared":
            s.operands = (dm.prepare_block_scaled_weight(s.w13, cfg), dm.prepare_block_scaled_weight(s.w2, cfg))
        accumulate = case["grads"] == "accumulate"
        if accumulate:  # gradients of earlier micro-batches
            dtype = getattr(torch, case["grad_dtype"])
            for w in (s.w13, s.w2):
                if dtype != w.dtype:
                    w.grad_dtype = dtype
                w.grad = normal(*w.shape, std=0.5, dtype=dtype)
        s.options = dm.ExecutionOptions(inplace_wgrad_accum=accumulate, experts_output_postprocess=post)
        return s
    s.options = dm.ExecutionOptions(experts_output_postprocess=post)
    if case["family"] == "bf16":
        s.operands = (s.w13, s.w2)
    else:
        s.operands = (dm.prepare_block_scaled_weight(s.w13, cfg, fuse_swiglu=True, inference=True),
                      dm.prepare_block_scaled_weight(s.w2, cfg, inference=True))
    if case["graph"]:
        # the program's captured decode step, reading its tokens and routing from tensors of its own
        s.graph_inputs = tuple(t.clone() for t in (s.x, s.ids, s.scores))
        side = torch.cuda.Stream(device=DEVICE)
        side.wait_stream(torch.cuda.current_stream(DEVICE))
        with torch.cuda.stream(side), torch.no_grad():
            dm.routed_experts(*s.graph_inputs, *s.operands, s.context, options=s.options)
        torch.cuda.current_stream(DEVICE).wait_stream(side)
        torch.cuda.synchronize(DEVICE)
        s.graph = torch.cuda.CUDAGraph()
        with torch.no_grad(), torch.cuda.graph(s.graph):
            s.graph_output = dm.routed_experts(*s.graph_inputs, *s.operands, s.context, options=s.options)
    return s


def run(s):
    if s.graph is not None:
        for dst, src in zip(s.graph_inputs, (s.x, s.ids, s.scores)):
            dst.copy_(src)
        s.graph.replay()
        return s.graph_output
    if not s.case["train"]:
        with torch.no_grad():
            return dm.routed_experts(s.x, s.ids, s.scores, *s.operands, s.context, options=s.options)
    if s.case["grads"] == "fresh":
        s.w13.grad = s.w2.grad = None
    x, scores = s.x.detach().requires_grad_(True), s.scores.detach().requires_grad_(True)
    out = dm.routed_experts(x, s.ids, scores, *s.operands, s.context, options=s.options)
    out.backward(s.grad_out)
    return {"out": out, "grad_x": x.grad, "grad_scores": scores.grad, "grad_w13": s.w13.grad, "grad_w2": s.w2.grad}


if __name__ == "__main__":
    for c in listed() + [draw(random.Random(i)) for i in range(8)]:
        w = work(c)
        print(f"{c.get('name', 'drawn'):24s} {w['bytes'] / 1e6:10.2f} MB {w['flops'] / 1e9:10.2f} GFLOP  "
              f"{ {k: v for k, v in c.items() if k != 'name'} }")
