"""Workloads of the routed-expert step, as a serving program issues them.

A case is a dict of plain values:
  entry     how the program calls the step
              graph     GraphedStep on device tensors (a decode loop replaying a captured step)
              host      HostMappedStep on pinned host tensors (a step that starts and ends on the host)
              call      kernel_fn launched directly (prefill chunks, mixed batches, layers with their own graph)
              okc       compat.OkcExt.okc_run (a decode layer that routes itself and passes local ids)
              prefill   compat.PrefillMoe.moe_forward (a prefill layer that routes itself)
              load      prepare(weights) and export_weights(state): a program that takes the weights of a
                        checkpoint in and gives them back in the checkpoint's own layout
  H, I, E, k, lo, nloc   hidden, expert width, experts, routes per token, local expert range
  T         tokens of the pass (0 for load)
  route     logits  router logits are given, the step takes the top-k
            weight  the router's matrix belongs to the state, the step computes the logits too
            ids     expert ids and weights are given
  load_kind how the tokens spread over the experts: uniform / normal (near even), zipf (a few experts take
            most tokens, several get none), skew (a rank's view: 1.6 local routes a token, two experts
            take 70 % of them)
  sigmoid   sigmoid scores with a selection bias instead of softmax over the chosen logits
  pre, post pre-expert and post-expert RMS norm
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "muse-spark-kernels_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import muse_moe_w4a16 as moe  # noqa: E402
from muse_moe_w4a16 import compat, inputs  # noqa: E402

# (H, I, E, k, lo, nloc): the single-GPU shape, one rank of eight of the layer call sites, one rank of eight of
# the expert-parallel shape, and a smaller model
ONE_GPU = (4096, 1536, 128, 8, 0, 128)
LAYER_RANK = (4096, 4096, 256, 8, 0, 32)
EP_RANK = (7168, 2048, 256, 8, 96, 32)
SMALL = (2048, 1024, 64, 4, 0, 64)


def _case(entry, shape, T, route, load_kind, sigmoid=False, pre=False, post=False, **more):
    H, I, E, k, lo, nloc = shape
    return dict(more, entry=entry, H=H, I=I, E=E, k=k, lo=lo, nloc=nloc, T=T, route=route, load_kind=load_kind,
                sigmoid=sigmoid, pre=pre, post=post)


def listed():
    return [
        # one user decoding: the step is replayed from a graph for every token and layer
        _case("graph", ONE_GPU, 1, "logits", "uniform", name="decode_1"),
        # the same for a program that keeps hidden states and results on the host
        _case("host", ONE_GPU, 1, "logits", "normal", name="host_1"),
        # a verify step of two tokens in a layer with sigmoid routing and both expert norms, launched directly
        _case("call", ONE_GPU, 2, "weight", "normal", sigmoid=True, pre=True, post=True, name="layer_2"),
        # a small decode batch
        _case("graph", ONE_GPU, 8, "logits", "normal", name="decode_8"),
        # a decode batch at the call site of the decode layer: local ids, -1 for another rank's expert
        _case("okc", LAYER_RANK, 24, "ids", "skew", post=True, name="okc_24"),
        # a full decode batch: every expert is touched, the weights set the pace
        _case("graph", ONE_GPU, 64, "logits", "normal", name="batch_64"),
        # a large decode batch or a short prompt
        _case("graph", ONE_GPU, 256, "logits", "normal", name="batch_256"),
        # an odd-sized prefill chunk in a layer that leaves routing and both norms to the step
        _case("call", ONE_GPU, 777, "weight", "normal", sigmoid=True, pre=True, post=True, name="chunk_777"),
        # a prompt at the call site of the prefill layer, with the skew of one rank's experts
        _case("prefill", LAYER_RANK, 3012, "ids", "skew", pre=True, post=True, name="prefill_layer_3012"),
        # what one of eight ranks computes for the tokens of two source ranks (4096 each)
        _case("call", EP_RANK, 8192, "ids", "uniform", name="ep_rank_8192"),
        # a long prompt whose tokens favour a few experts
        _case("call", ONE_GPU, 8192, "logits", "zipf", name="prefill_8192"),
        # start-up: a checkpoint's weights are taken in, and given back in their own layout
        _case("load", ONE_GPU, 0, "ids", "uniform", name="load"),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    entry = rng.choice(["graph", "graph", "call", "call", "call", "host", "okc", "prefill", "ep", "load"])
    flag = lambda: rng.random() < 0.5  # noqa: E731
    if entry == "okc":
        return _case("okc", LAYER_RANK, _log_uniform(rng, 1, 384), "ids", "skew", post=True)
    if entry == "prefill":
        return _case("prefill", LAYER_RANK, _log_uniform(rng, 200, 8000), "ids", "skew", pre=True, post=True)
    if entry == "ep":
        return _case("call", EP_RANK, _log_uniform(rng, 64, 8192), "ids", "uniform", post=flag())
    if entry == "load":
        n = rng.randrange(8, 129)
        return _case("load", (4096, 1536, n, 8, 0, n), 0, "ids", "uniform")
    shape = rng.choice([ONE_GPU, ONE_GPU, ONE_GPU, SMALL])
    kind = rng.choice(["uniform", "normal", "zipf"])
    if entry == "host":
        return _case("host", shape, _log_uniform(rng, 1, 48), rng.choice(["logits", "ids"]), kind, post=flag())
    if entry == "graph":
        return _case("graph", shape, _log_uniform(rng, 1, 512), rng.choice(["logits", "ids"]), kind, sigmoid=flag(), post=flag())
    return _case("call", shape, _log_uniform(rng, 1, 7000), rng.choice(["logits", "weight", "ids"]), kind, sigmoid=flag(), pre=flag(),
                 post=flag())


def _skewed_ids(case, gen, dev):
    """Local ids [T, k] as a rank of the layer call sites sees them, -1 for another rank's expert: two experts
    with 0.56 routes a token each, the other thirty share 0.48."""
    T, k, n = case["T"], case["k"], case["nloc"]
    p = torch.full((n,), 0.48 / (n - 2), device=dev)
    p[torch.randperm(n, generator=gen, device=dev)[:2]] = 0.56
    on = torch.rand((T, n), generator=gen, device=dev) < p
    score = on.float() + 0.5 * torch.rand((T, n), generator=gen, device=dev)
    val, idx = score.topk(k, dim=1)
    ids = torch.where(val >= 1.0, idx, torch.full_like(idx, -1))
    slot = torch.rand((T, k), generator=gen, device=dev).argsort(1)      # local routes sit at any of the k places
    w = torch.rand((T, k), generator=gen, device=dev) + 0.1
    return ids.gather(1, slot).to(torch.int32).contiguous(), (w / w.sum(1, keepdim=True)).contiguous()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    H, E, k, lo, nloc, T = (case[n] for n in ("H", "E", "k", "lo", "nloc", "T"))
    weights = inputs.make_weights(H, case["I"], nloc, seed, dev, post_norm=case["post"])
    if case["entry"] == "load":
        return {"entry": "load", "weights": weights, "E": E, "k": k}
    gen = torch.Generator(device=dev).manual_seed(seed * 15485863 + 29)
    if case["pre"]:
        weights["pre_norm_w"] = (torch.randn((H,), generator=gen, device=dev) * 0.1).to(torch.bfloat16)
    data = {"hidden_states": torch.randn((T, H), generator=gen, device=dev).to(torch.bfloat16)}
    if case["sigmoid"]:
        weights["route_bias"] = torch.randn((E,), generator=gen, device=dev) * 0.05
    if case["route"] == "weight":
        weights["router"] = torch.randn((E, H), generator=gen, device=dev) * 0.02
    elif case["load_kind"] == "skew":
        data["topk_ids"], data["topk_weights"] = _skewed_ids(case, gen, dev)
    else:
        logits = inputs.make_logits(T, E, case["load_kind"], seed, dev)
        if case["route"] == "ids":
            val, ids = logits.topk(k, dim=1)
            data["topk_ids"], data["topk_weights"] = ids.to(torch.int32).contiguous(), val.softmax(1).contiguous()
        else:
            data["router_logits"] = logits
    # a server prepares one state for all its token counts; the layer call sites state their own limits
    room = {"okc": 384, "prefill": max(T, 4096)}.get(case["entry"], 8192)
    state = moe.prepare(weights, local_start=lo, n_experts=E, top_k=k, max_tokens=room,
                        routing_mode="sigmoid_bias" if case["sigmoid"] else "softmax_topk")
    del weights
    got = {"entry": case["entry"], "state": state, "data": data}
    if case["entry"] == "graph":
        got["step"] = moe.GraphedStep(state, data)
    elif case["entry"] == "host":
        got["data"] = {n: t.cpu().pin_memory() for n, t in data.items()}
        got["step"] = moe.HostMappedStep(state, got["data"])
    elif case["entry"] == "okc":
        got["ext"] = compat.OkcExt(state)
        got["ext"].okc_set_pdl(1)
    elif case["entry"] == "prefill":
        got["layer"] = compat.PrefillMoe(state)
    return got


def run(state):
    entry, data = state["entry"], state.get("data")
    if entry in ("graph", "host"):
        return state["step"](data)
    if entry == "call":
        return moe.kernel_fn(data, state["state"], return_routing=True)
    if entry == "okc":
        x = data["hidden_states"]
        out = torch.empty_like(x)
        state["ext"].okc_run(None, None, x, data["topk_ids"], data["topk_weights"], out, 0, state["state"]["cnt"], 148)
        return out
    if entry == "prefill":
        x = data["hidden_states"]
        return state["layer"].moe_forward(x, data["topk_ids"], None, None, x.shape[0], data["topk_weights"])["out"]
    loaded = moe.prepare(state["weights"], n_experts=state["E"], top_k=state["k"])
    return moe.export_weights(loaded)


def _routes_and_touched(case):
    """Expected (token, local expert) pairs and local experts that get at least one."""
    T, E, k, n = case["T"], case["E"], case["k"], case["nloc"]
    if case["load_kind"] == "skew":
        p = [0.56, 0.56] + [0.48 / (n - 2)] * (n - 2)
    elif case["load_kind"] == "zipf" and case["route"] != "weight":
        # chance of each expert to be among a token's k: noise of unit variance on the logarithm of the
        # popularity, with the threshold at which k experts pass on average
        mu = [-1.2 * math.log(r + 2.0) for r in range(E)]
        above = lambda t: [0.5 * math.erfc((t - m) / math.sqrt(2.0)) for m in mu]  # noqa: E731
        a, b = -12.0, 8.0
        for _ in range(60):
            c = 0.5 * (a + b)
            a, b = (c, b) if sum(above(c)) > k else (a, c)
        p = above(a)[:n]
    else:
        p = [k / E] * n
    return T * sum(p), sum(1.0 - (1.0 - v) ** T for v in p)


def work(case):
    H, I, E, k, T, n = (case[x] for x in ("H", "I", "E", "k", "T", "nloc"))
    per_expert = 3 * I * H * (0.5 + 1.0 / 16.0) + 8
    if case["entry"] == "load":     # each way every byte is read once and written once
        return {"bytes": 2 * 2 * n * (per_expert - 8), "flops": 0}
    routes, touched = _routes_and_touched(case)
    nbytes = touched * per_expert + 2 * 2 * T * H + {"logits": 4 * T * E, "weight": 4 * E * H, "ids": 8 * T * k}[case["route"]]
    flops = 2.0 * routes * 3 * I * H + (2.0 * T * E * H if case["route"] == "weight" else 0.0)
    return {"bytes": nbytes + 2 * H * (case["pre"] + case["post"]), "flops": flops}


def tolerance(case):
    if case["entry"] == "load":
        return "exact"
    # BF16 rows out of a BF16 intermediate, summed in FP32; ids of a router computed here may flip at a tie
    return {"rel": 1e-2, "differ": 1e-3 if case["route"] == "weight" else 0.0}
