"""Performance cases of the MoE layer: the calls a user's program makes through `mok.functional` and `mok.ops`, one rank.

A case is a dict of plain values:
  mode       "train"      build_schedule + forward + backward: one layer of a training step
             "infer"      build_schedule + forward: one layer of a serving step
             "recompute"  build_schedule + recompute_forward_context + backward: the backward half of a step with
                          activation checkpointing
             "quantize"   mxfp8_quantize of the layer's three routed weight tensors, both orientations: what an MXFP8
                          training step does after every optimizer update
  precision  "bf16" | "mxfp8" (routed experts; the shared expert is always bf16)
  tokens, hidden, inter, experts, topk, routing ("gaussian" | "zipf" | "router"), limit (SwiGLU clamp, 0 = none)
  minibatch, macrobatch (0: large enough for the worst padding, otherwise as given: more rows are replayed)
"""
import math
import os
import sys

import torch

PACKAGE = os.path.join(os.getcwd(), "mixture-of-kittens_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

PAD = 256          # expert segments are padded to this many rows


def _case(name, mode, precision, tokens, hidden, inter, experts, topk, routing="gaussian", limit=0.0, minibatch=4096, macrobatch=0):
    return {"name": name, "mode": mode, "precision": precision, "tokens": tokens, "hidden": hidden, "inter": inter, "experts": experts,
            "topk": topk, "routing": routing, "limit": limit, "minibatch": minibatch, "macrobatch": macrobatch}


def listed():
    return [
        # the smallest training layer (benchmark configuration 1): launches and host time count
        _case("train_bf16_1k", "train", "bf16", 1024, 1024, 512, 8, 2, routing="router", minibatch=256),
        _case("train_mxfp8_1k", "train", "mxfp8", 1024, 1024, 512, 8, 2, routing="router", minibatch=256),
        # a decode-like serving step: the fewest tokens the layer takes, every expert's weights touched for few rows
        _case("infer_bf16_512", "infer", "bf16", 512, 5120, 1408, 64, 6, minibatch=2048),
        # a short prefill with a skewed expert popularity, block-scaled weights, many experts
        _case("infer_mxfp8_2k", "infer", "mxfp8", 2048, 4096, 1536, 128, 8, routing="zipf", minibatch=2048),
        # an ordinary training layer with a small micro-batch
        _case("train_bf16_4k", "train", "bf16", 4096, 5120, 1408, 64, 6, minibatch=2048),
        # the same model with a full micro-batch, MXFP8
        _case("train_mxfp8_16k", "train", "mxfp8", 16384, 5120, 1408, 64, 6, minibatch=8192),
        # skewed routing and the default macrobatch: the routed rows do not fit it, so the backward replays the rest
        _case("train_bf16_16k_zipf", "train", "bf16", 16384, 4096, 1536, 128, 8, routing="zipf", macrobatch=131072),
        _case("train_mxfp8_8k_zipf", "train", "mxfp8", 8192, 4096, 1536, 128, 8, routing="zipf", limit=7.0, minibatch=8192),
        # activation checkpointing on odd sizes, with the clamped SwiGLU
        _case("recompute_bf16_6k_ragged", "recompute", "bf16", 5888, 2816, 1408, 24, 5, limit=7.0),
        # the largest: one rank's share of the 256-expert benchmark layer at EP=8, both precisions
        _case("train_bf16_16k_large", "train", "bf16", 16384, 7168, 2048, 32, 8, minibatch=8192),
        _case("train_mxfp8_16k_large", "train", "mxfp8", 16384, 7168, 2048, 32, 8, minibatch=8192),
        # re-quantising that layer's routed weights after an optimizer update
        _case("quantize_weights_large", "quantize", "mxfp8", 0, 7168, 2048, 32, 0),
    ]


def _log_pick(rng, low, high, step):
    """A multiple of `step` in [low, high], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(low), math.log(high + step)))
    return min(max(int(v) // step * step, low), high)


def draw(rng):
    mode = rng.choice(["train", "train", "train", "infer", "infer", "recompute", "quantize"])
    precision = "mxfp8" if mode == "quantize" else rng.choice(["bf16", "mxfp8"])
    tokens = _log_pick(rng, 512, 16384, 256)
    hidden = _log_pick(rng, 1024, 7168, 256)
    inter = _log_pick(rng, 512, 2048, 128)
    experts = _log_pick(rng, 8, 128, 1)
    topk = rng.randint(1, 8)
    while experts > 8 and experts * hidden * inter > 128 * 4096 * 1536:
        experts -= 1
    case = _case("", mode, precision, tokens, hidden, inter, experts, topk, routing=rng.choice(["gaussian", "gaussian", "zipf"]),
                 limit=rng.choice([0.0, 0.0, 7.0]), minibatch=256 * rng.choice([1, 3, 8, 16, 32]))
    if mode == "quantize":
        case.update(tokens=0, topk=0, routing="gaussian", limit=0.0)
    else:
        # no more multiplications than the largest listed case, padding rows counted
        while (case["tokens"] * (topk + 1) + experts * PAD) * hidden * inter > 16384 * 9 * 7168 * 2048 and case["tokens"] > 512:
            case["tokens"] -= 256
        if mode == "train" and rng.random() < 0.25:      # a macrobatch that only holds part of the rows
            rows = (case["tokens"] * topk * 2 // 3) // case["minibatch"] * case["minibatch"]
            case["macrobatch"] = max(rows, case["minibatch"])
            case["inter"] = -(-inter // 256) * 256
    del case["name"]
    return case


def _group():
    import torch.distributed as dist
    if not dist.is_initialized():
        dev = torch.cuda.current_device()
        torch.cuda.set_device(dev)
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", dev))
    return dist.group.WORLD


def prepare(case, seed):
    from mok import functional as F, ops
    dev = torch.device("cuda", torch.cuda.current_device())
    T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "inter", "experts", "topk"))
    gen = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape, std):
        return torch.empty(*shape, dtype=torch.bfloat16, device=dev).normal_(0.0, std, generator=gen)

    weights = [normal(E, I, H, std=0.02), normal(E, I, H, std=0.02), normal(E, H, I, std=0.02)]
    state = {"mode": case["mode"], "experts": E, "limit": case["limit"] or None}
    if case["mode"] == "quantize":
        state["weights"] = weights
        return state
    state["shared"] = (normal(I, H, std=0.02), normal(I, H, std=0.02), normal(H, I, std=0.02))
    if case["precision"] == "mxfp8":
        q = [ops.mxfp8_quantize(w, True, True) for w in weights]
        state["fwd_weights"] = ((q[0][0], q[0][1]), (q[1][0], q[1][1]), (q[2][0], q[2][1]))
        state["bwd_weights"] = (q[0], q[1], (q[2][2], q[2][3]))
    else:
        state["fwd_weights"] = state["bwd_weights"] = tuple(weights)
    del weights
    state["x"] = normal(T, H, std=1.0)
    state["grad_output"] = normal(T, H, std=1.0)
    if case["routing"] == "router":
        logits = state["x"].float() @ (torch.randn(H, E, generator=gen, device=dev) * 0.02)
    else:
        logits = torch.randn(T, E, generator=gen, device=dev)
    if case["routing"] == "zipf":
        popularity = torch.randperm(E, generator=gen, device=dev)
        bias = torch.empty(E, device=dev)
        bias[popularity] = -1.2 * torch.log(torch.arange(1, E + 1, dtype=torch.float32, device=dev))
        logits = logits + bias
    values, chosen = torch.topk(logits, K, dim=1)
    state["top_experts"] = chosen.to(torch.int64).contiguous()
    state["router_weights"] = torch.softmax(values.float(), -1).contiguous()
    worst = T * K + E * PAD                           # rows with the most padding any routing can need
    mb = case["minibatch"]
    state["config"] = F.MoKConfig(minibatch_size=mb, macrobatch_size=case["macrobatch"] or -(-worst // mb) * mb,
                                  schedule_capacity_multiplier=float(max(2, -(-worst // (T * K)))),
                                  all_gather_top_experts_chunk_bytes=2048 if T * K * 4 % 2048 == 0 else 1024)
    state["workspace"] = F.create_workspace(state["config"], _group(), device=dev, num_local_tokens=T, hidden_size=H, topk=K)
    return state


def run(state):
    from mok import functional as F, ops
    if state["mode"] == "quantize":
        return [ops.mxfp8_quantize(w, True, True) for w in state["weights"]]
    cfg, ws, x, rw, limit = state["config"], state["workspace"], state["x"], state["router_weights"], state["limit"]
    sched = F.build_schedule(ws, cfg, state["top_experts"], num_local_experts=state["experts"])
    out = {"peer_rank": sched.peer_rank, "peer_token_idx": sched.peer_token_idx, "num_tokens": sched.num_tokens,
           "tokens_per_expert": sched.tokens_per_expert}
    if state["mode"] == "recompute":
        ctx = F.recompute_forward_context(cfg, ws, sched, x, *state["shared"][:2], *state["fwd_weights"][:2], limit)
    else:
        out["y"], ctx = F.forward(cfg, ws, sched, x, rw, *state["shared"], *state["fwd_weights"], limit)
    if state["mode"] != "infer":
        out["grads"] = F.backward(cfg, ws, sched, ctx, state["grad_output"], x, rw, *state["shared"], *state["bwd_weights"], limit)
    return out


def work(case):
    T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "inter", "experts", "topk"))
    routed = 3 * E * H * I
    mx = 1.0 + 1.0 / 32                               # bytes of an E4M3 element with its share of the scales
    if case["mode"] == "quantize":
        return {"bytes": routed * (2 + 2 * mx), "flops": 0}
    per_row = {"train": 18, "infer": 6, "recompute": 16}[case["mode"]]
    backward = case["mode"] != "infer"
    data = 2 * T * H + T * K * (8 + 4)                # x, routing choices and weights
    data += 2 * 3 * H * I                             # the shared expert's weights
    # routed weights: only experts that can have a row; MXFP8 reads the other orientation in the backward
    used = min(E, T * K) / E
    data += routed * used * ((mx * (2 if backward else 1)) if case["precision"] == "mxfp8" else 2)
    if case["mode"] != "recompute":
        data += 2 * T * H                             # the layer's output
    if backward:
        data += 2 * 2 * T * H + 4 * T * K             # grad_output in; d_x, router-weight gradients out
        data += 2 * (3 * H * I + routed)              # weight gradients
    return {"bytes": data, "flops": per_row * T * (K + 1) * H * I}


def tolerance(case):
    if case["mode"] == "quantize":
        return "exact"
    # Against a float64 restatement of the layer with the same rounding points, over five of the listed cases: bf16 at most
    # rel 1.2e-3 and max 0.033, mxfp8 rel 9.1e-4 and max 0.21 (a value that crosses a bf16 step can cross an E4M3 step,
    # which moves a product by 1/16); about four times that.
    return {"rel": 5e-3, "max": 0.15} if case["precision"] == "bf16" else {"rel": 5e-3, "max": 0.8}
