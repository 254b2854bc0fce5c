"""The calls a user of the MoE layer makes, as cases that can be timed and compared.

One case = one forward of the layer (or of its activation quantiser) through the package's public entry points, with the
shapes and distributions of `justgoal_b200.inputs`: logits ~ N(0,1), selection bias ~ N(0,0.1) for the DeepSeek-V3
shape, hidden states ~ N(0,1) quantised per 1x128, weights ~ N(0,0.02) quantised per 128x128.  A case is a dict:

  entry   run / run_dps      the operator entry points (DeepSeek-V3 routing), output returned / written in place
          forward            MoELayer.forward (handle kept by the caller; other shapes than the operator's own)
          forward_routed     MoELayer.forward_routed, fp16 rows: the expert-parallel receive side
          quantize           quantize_1x128, the step before the layer
  model   deepseek_v3 / qwen3_moe
  tokens  rows of the call;  local: experts held;  rank: whose share (local_expert_offset = rank * local)
  skew    four of the local experts drawn about four times as often as the others
"""
from __future__ import annotations

import functools
import math

import torch

import justgoal_b200 as jg
from justgoal_b200 import inputs as I

MODELS = {"deepseek_v3": I.DEEPSEEK_V3, "qwen3_moe": I.QWEN3_MOE}
SKEW_DELTA = 0.328      # added to the selection bias of local experts 0, 8, 16, 24: about 4x the mean load


def _case(name, entry, model, tokens, local, rank=0, skew=False):
    return {"name": name, "entry": entry, "model": model, "tokens": tokens, "local": local, "rank": rank, "skew": skew}


def listed():
    return [
        # one user generating text: one token per step, a rank that holds 32 of 256 experts
        _case("decode_1", "run", "deepseek_v3", 1, 32),
        # a handful of users, odd count, output written into the caller's buffer; not the first rank's share
        _case("decode_7", "run_dps", "deepseek_v3", 7, 32, rank=5),
        # the ordinary decode batch
        _case("decode_64", "run", "deepseek_v3", 64, 32),
        # a full decode batch, or 64 users with one speculated token each
        _case("decode_128", "run_dps", "deepseek_v3", 128, 32, rank=2),
        # decode batch with a short prompt mixed in: just past a power of two
        _case("mixed_257", "run", "deepseek_v3", 257, 32, rank=7),
        # a chunk of a chunked prefill, ragged
        _case("chunk_901", "run", "deepseek_v3", 901, 32, rank=1),
        # a long prompt whose topic loads a few experts heavily
        _case("prefill_4096_skew", "run", "deepseek_v3", 4096, 32, skew=True),
        # several long prompts in one ragged batch
        _case("prefill_14107", "run_dps", "deepseek_v3", 14107, 32),
        # the whole layer on one GPU
        _case("full_8192", "forward", "deepseek_v3", 8192, 256),
        # one rank's share of the softmax-routed shape
        _case("qwen3_2048", "forward", "qwen3_moe", 2048, 16, rank=3),
        # expert-parallel receive side: tokens that other ranks routed to this one
        _case("routed_4201", "forward_routed", "deepseek_v3", 4201, 32, rank=4),
        # the activations of a prompt, quantised for the layer
        _case("quantize_4096", "quantize", "deepseek_v3", 4096, 0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.random()
    if kind < 0.10:
        c = _case("", "quantize", rng.choice(sorted(MODELS)), log_int(64, 14107), 0)
    elif kind < 0.25:
        local = rng.choice((8, 16, 32, 64))
        c = _case("", "forward", "qwen3_moe", log_int(1, 8192), local, rng.randrange(128 // local))
    elif kind < 0.40:
        local = rng.choice((32, 64, 128))
        c = _case("", "forward_routed", "deepseek_v3", log_int(8, 6144), local, rng.randrange(256 // local), rng.random() < 0.25)
    elif kind < 0.50:
        local = rng.choice((64, 128))
        c = _case("", "forward", "deepseek_v3", log_int(1, 8192), local, rng.randrange(256 // local), rng.random() < 0.25)
    else:
        c = _case("", rng.choice(("run", "run_dps")), "deepseek_v3", log_int(1, 14107), 32, rng.randrange(8), rng.random() < 0.25)
    del c["name"]
    return c


def _shape(case):
    return MODELS[case["model"]].with_local(max(1, case["local"]))


def _boost(case):
    if not case["skew"]:
        return None
    off, local = case["rank"] * case["local"], case["local"]
    return tuple(off + i * (local // 4) for i in range(4)), SKEW_DELTA


def _received(case):
    """Tokens the other ranks had to route so that `tokens` of them have an expert here (with room to spare)."""
    return case["tokens"] * _shape(case).num_experts // case["local"] + 512


def prepare(case, seed):
    shape, T, dev = _shape(case), case["tokens"], "cuda"
    if case["entry"] == "quantize":
        g = torch.Generator(device=dev)
        g.manual_seed(int(seed))
        return {"entry": "quantize", "x": torch.randn(T, shape.hidden, generator=g, device=dev).to(torch.bfloat16)}
    off, scale = case["rank"] * case["local"], 2.5 if case["model"] == "deepseek_v3" else 1.0
    w = I.make_weights(shape, seed, dev, off)
    weights = (w["gemm1_weights"], w["gemm1_weights_scale"], w["gemm2_weights"], w["gemm2_weights_scale"])
    if case["entry"] == "forward_routed":
        layer = jg.MoELayer(shape)
        d = I.make_tokens(shape, _received(case), seed, dev, _boost(case))
        idx, topk_w = layer.route(d["routing_logits"], d["routing_bias"], scale)
        mine = ((idx >= off) & (idx < off + case["local"])).any(dim=1).nonzero().flatten()
        assert mine.numel() >= T
        mine = mine[:T]
        args = (idx[mine].contiguous(), topk_w[mine].contiguous(),
                d["hidden_states"].view(torch.uint8)[mine].contiguous().view(torch.float8_e4m3fn),
                d["hidden_states_scale"][:, mine].contiguous(), *weights, off)
        return {"entry": "forward_routed", "layer": layer, "args": args}
    d = I.make_tokens(shape, T, seed, dev, _boost(case))
    args = (d["routing_logits"], d["routing_bias"], d["hidden_states"], d["hidden_states_scale"], *weights, off, scale)
    state = {"entry": case["entry"], "args": args}
    if case["entry"] == "forward":
        state["layer"] = jg.MoELayer(shape)
    elif case["entry"] == "run_dps":
        state["out"] = torch.empty(T, shape.hidden, dtype=torch.bfloat16, device=dev)
    return state


def run(state):
    entry = state["entry"]
    if entry == "run":
        return jg.run(*state["args"])
    if entry == "run_dps":
        return jg.run_dps(*state["args"], state["out"])
    if entry == "forward":
        return state["layer"].forward(*state["args"])
    if entry == "forward_routed":
        return state["layer"].forward_routed(*state["args"], out_dtype=torch.float16)
    q, scale = jg.quantize_1x128(state["x"])
    return q.view(torch.uint8), scale


@functools.lru_cache(maxsize=None)
def _routing(model, entry, tokens, local, rank, skew):
    """(pairs, experts that get a token) of a call on this rank: means over a few drawn routings."""
    case = dict(model=model, entry=entry, tokens=tokens, local=local, rank=rank, skew=skew)
    shape, off = _shape(case), rank * local
    E, pairs, active, draws = shape.num_experts, 0.0, 0.0, max(1, min(64, 4096 // tokens))
    for k in range(draws):
        g = torch.Generator().manual_seed(9000 + k)
        n = tokens if entry != "forward_routed" else _received(case)
        s = torch.randn(n, E, generator=g)
        if shape.routing_mode == I.ROUTING_DS:
            s = torch.sigmoid(s)
        bias = torch.randn(E, generator=g) * 0.1 if shape.routing_mode == I.ROUTING_DS else torch.zeros(E)
        boost = _boost(case)
        if boost is not None:
            bias[list(boost[0])] += boost[1]
        v = s + bias
        if shape.routing_mode == I.ROUTING_DS:
            groups = v.view(n, shape.n_group, -1)
            keep = groups.topk(2, dim=2).values.sum(2).topk(shape.topk_group, dim=1).indices
            mask = torch.zeros(n, shape.n_group, dtype=torch.bool).scatter_(1, keep, True)
            v = groups.masked_fill(~mask.unsqueeze(2), -1e9).view(n, E)
        idx = v.topk(shape.top_k, dim=1).indices
        mine = (idx >= off) & (idx < off + local)
        if entry == "forward_routed":
            hit = mine.any(dim=1).nonzero().flatten()[:tokens]
            idx, mine = idx[hit], mine[hit]
        pairs += float(mine.sum()) / draws
        active += float(idx[mine].unique().numel()) / draws
    return pairs, active


def work(case):
    shape, T = _shape(case), case["tokens"]
    H, inter, E, K = shape.hidden, shape.intermediate, shape.num_experts, shape.top_k
    if case["entry"] == "quantize":
        return {"bytes": 3 * T * H + 4 * T * (H // 128), "flops": 0}
    pairs, active = _routing(case["model"], case["entry"], T, case["local"], case["rank"], case["skew"])
    weights = active * (3 * H * inter + 4 * (3 * H * inter // (128 * 128)))
    routing = 8 * T * K if case["entry"] == "forward_routed" else 4 * T * E + 2 * E
    return {"bytes": weights + routing + T * H + 4 * T * (H // 128) + 2 * T * H, "flops": 6 * pairs * H * inter}


def tolerance(case):
    if case["entry"] == "quantize":
        return "exact"
    # bf16 result (8 significant bits: 1.7e-3 in the 2-norm) of fp32 sums over fp8 products; the activations between the
    # two GEMMs carry seven to eight significant bits
    return {"rel": 5e-3}
