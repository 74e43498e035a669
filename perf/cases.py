"""The work this package is timed on: what a serving or training-style program has it do, through its public calls.

A case is a dict of plain values. ``kind`` is the call it makes:

    decode        ``gdn2_decode_step`` (n = 1) / ``gdn2_decode`` (n draft tokens), the state updated in place
    prefill       ``gdn2_prefill``: a batch of prompts, optionally continuing from a state
    packed        ``gdn2_attention`` with ``cu_seqlens``: prompts of unequal lengths in one row
    attention     ``gdn2_attention``: the functional op over a batch, with the final state
    forward       ``chunk_gdn2_fwd(return_chunk_states=True)``: the training-style forward that keeps every chunk's state
    layer_prefill ``GatedDeltaNet2.prefill`` of a prompt
    layer_step    ``GatedDeltaNet2.step`` / ``GraphedStep``: one token through the whole layer

``H`` value heads read ``HK`` key heads; ``g`` and the recurrent state are float32 whatever ``dtype`` is. The input
distributions are the ones the benchmark uses: q, k normal and L2-normalised per head, v normal, g = logsigmoid(normal) / 16,
b, w sigmoids of normals, recurrent states normal with standard deviation 0.02.
"""

from __future__ import annotations

import random

import torch
import torch.nn.functional as F

import gdn2_tilelang_b200 as gdn2

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
BYTES = {"bf16": 2, "f16": 2, "f32": 4}


def listed():
    return [
        # one token for one conversation: the latency of the op itself
        _op("step_b1", "decode", B=1, S=1),
        # one token for each of 256 conversations, the decode batch of the benchmark: the state streams through once
        _op("step_b256", "decode", B=256, S=1),
        # eight draft tokens for each of them (speculative decoding at full batch)
        _op("drafts_b256_n8", "decode", B=256, S=8),
        # five draft tokens for a middling batch, key heads shared by two value heads, half precision
        _op("drafts_b24_n5_f16", "decode", B=24, S=5, HK=8, dtype="f16"),
        # the benchmark's serving prefill: four long prompts, 250 chunks and a ragged tail each
        _op("prefill_serving", "prefill", B=4, S=16037),
        # what one of eight head-sharded GPUs does of it
        _op("prefill_two_heads", "prefill", B=4, S=16037, H=2, HK=2),
        # the next segment of one conversation's prompt, key heads shared, continuing from its state
        _op("prompt_segment", "prefill", B=1, S=1037, HK=8, state=True),
        # ten prompts of unequal lengths packed into one row
        _packed("packed_prompts", seqs=10, tokens=6007, lengths=1),
        # training-style forward with the state entering every chunk kept
        _op("forward_states", "forward", B=2, S=4096),
        # full precision at the smaller head size
        _op("attention_f32", "attention", B=2, S=1000, H=8, HK=8, DK=64, DV=64, dtype="f32"),
        # the whole token mixer on two prompts of 4096 tokens
        _layer("layer_prefill", "layer_prefill", B=2, S=4096),
        # one token through the whole token mixer, called as a generation loop calls it
        _layer("layer_step", "layer_step", B=2, graphed=False),
    ]


def _op(name, kind, B, S, H=16, HK=16, DK=128, DV=128, dtype="bf16", state=False):
    return dict(name=name, kind=kind, B=B, S=S, H=H, HK=HK, DK=DK, DV=DV, dtype=dtype, state=state)


def _packed(name, seqs, tokens, lengths, H=16, HK=16, dtype="bf16"):
    return dict(name=name, kind="packed", seqs=seqs, tokens=tokens, lengths=lengths, B=1, S=tokens, H=H, HK=HK, DK=128, DV=128,
                dtype=dtype, state=False)


def _layer(name, kind, B, S=1, hidden=2048, H=16, HK=8, graphed=False):
    return dict(name=name, kind=kind, B=B, S=S, hidden=hidden, H=H, HK=HK, DK=128, DV=128, dtype="bf16", graphed=graphed)


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "prefill", "packed", "attention", "forward",
                       "layer_prefill", "layer_step"])
    H = rng.choice([2, 4, 8, 16, 16])
    HK = H if rng.random() < 0.6 else H // 2
    if kind == "decode":
        D = rng.choice([64, 128, 128, 128])
        case = _op("", kind, _log_uniform(rng, 1, 256), rng.choice([1, 1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 16]), H, HK, D, D,
                   rng.choice(["bf16", "bf16", "bf16", "f16", "f32"]))
    elif kind == "prefill":
        B = rng.choice([1, 1, 2, 3, 4, 8])
        case = _op("", kind, B, _log_uniform(rng, 17, min(32000, 900000 // (B * H))), H, HK, state=rng.random() < 0.5)
    elif kind == "packed":
        seqs = rng.randint(2, 9)
        case = _packed("", seqs, _log_uniform(rng, 40 * seqs, 16000), rng.randint(1, 10**6), H, HK)
    elif kind == "attention":
        DK, DV = rng.choice([(64, 64), (64, 128), (128, 128)])
        B = rng.choice([1, 2, 3])
        most = 16000 * 4096 // (B * H * DK * DV)
        case = _op("", kind, B, _log_uniform(rng, 65, max(130, most)), H, HK, DK, DV, rng.choice(["f32", "f16"]))
    elif kind == "forward":
        B = rng.choice([1, 2, 4])
        case = _op("", kind, B, 64 * _log_uniform(rng, 2, 2048 // (B * H)), H, HK)
    elif kind == "layer_prefill":
        B = rng.choice([1, 2, 4])
        case = _layer("", kind, B, _log_uniform(rng, 33, 8192 // B), rng.choice([1024, 2048]), H, HK)
    else:
        case = _layer("", kind, _log_uniform(rng, 1, 64), 1, rng.choice([1024, 2048]), H, HK, rng.random() < 0.5)
    del case["name"]
    return case


def _sequence_offsets(case):
    """``cu_seqlens`` of a packed case: the token axis cut at random places, every sequence at least one token long."""
    rng = random.Random(case["lengths"])
    return [0] + sorted(rng.sample(range(1, case["tokens"]), case["seqs"] - 1)) + [case["tokens"]]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    B, S, H, HK, DK, DV = (case[n] for n in ("B", "S", "H", "HK", "DK", "DV"))
    st = {"case": case}
    if case["kind"] in ("layer_prefill", "layer_step"):
        st["layer"] = layer = _make_layer(case, gen)
        st["x"] = normal(*((B, S) if case["kind"] == "layer_prefill" else (B,)), case["hidden"]).to(dt)
        if case["kind"] == "layer_step":
            cache = layer.init_cache(B)
            cache.recurrent_state.copy_(0.02 * normal(*cache.recurrent_state.shape))
            cache.conv_state.copy_(normal(*cache.conv_state.shape))
            st["cache"] = cache
            if case["graphed"]:
                st["step"] = gdn2.GraphedStep(layer, cache)
        return st
    q = F.normalize(normal(B, S, HK, DK), dim=-1).to(dt)
    k = F.normalize(normal(B, S, HK, DK), dim=-1).to(dt)
    v = normal(B, S, H, DV).to(dt)
    g = F.logsigmoid(normal(B, S, HK, DK)) / 16.0
    b = torch.sigmoid(normal(B, S, HK, DK)).to(dt)
    w = torch.sigmoid(normal(B, S, H, DV)).to(dt)
    st["ins"] = (q, k, v, g, b, w)
    if case["kind"] == "decode" and S == 1:
        st["ins"] = tuple(t[:, 0].contiguous() for t in st["ins"])
    if case["kind"] == "decode" or case["state"]:
        st["state"] = 0.02 * normal(B, H, DK, DV)
    if case["kind"] == "packed":
        st["cu_seqlens"] = torch.tensor(_sequence_offsets(case), dtype=torch.int32)      # a scheduler has the lengths on the host
    return st


def _make_layer(case, gen):
    cfg = gdn2.GatedDeltaNet2Config(hidden_size=case["hidden"], num_heads=case["H"], num_kv_heads=case["HK"],
                                    head_dim_k=case["DK"], head_dim_v=case["DV"])
    with torch.device("cuda"):
        layer = gdn2.GatedDeltaNet2(cfg)
    with torch.no_grad():
        for name, p in layer.named_parameters():
            if name == "A_log":
                p.copy_(torch.empty_like(p).uniform_(*cfg.a_init_range, generator=gen).log())
            elif name == "dt_bias":
                p.copy_(torch.empty_like(p).uniform_(*cfg.dt_init_range, generator=gen).expm1().log())
            elif name != "o_norm.weight":
                p.copy_(0.02 * torch.randn(p.shape, generator=gen, device=p.device))
    return layer.to(DTYPES[case["dtype"]]).eval()


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "decode":
        call = gdn2.gdn2_decode_step if case["S"] == 1 else gdn2.gdn2_decode
        return call(*state["ins"], state["state"]), state["state"]
    if kind == "prefill":
        return gdn2.gdn2_prefill(*state["ins"], state.get("state"))
    if kind == "packed":
        return gdn2.gdn2_attention(*state["ins"], output_final_state=True, cu_seqlens=state["cu_seqlens"])
    if kind == "attention":
        return gdn2.gdn2_attention(*state["ins"], output_final_state=True)
    if kind == "forward":
        return gdn2.chunk_gdn2_fwd(*state["ins"], case["DK"] ** -0.5, output_final_state=True, return_chunk_states=True)
    if kind == "layer_prefill":
        out, cache = state["layer"].prefill(state["x"])
    elif case["graphed"]:
        out, cache = state["step"](state["x"]), state["cache"]
    else:
        out, cache = state["layer"].step(state["x"], state["cache"])
    return out, cache.recurrent_state, cache.conv_state


def work(case):
    """Each input once and each output once; the recurrence's own 7 operations per token and state entry (decay, read,
    write, query), and the layer's projections."""
    B, S, H, HK, DK, DV, e = (*(case[n] for n in ("B", "S", "H", "HK", "DK", "DV")), BYTES[case["dtype"]])
    tokens, kind = B * S, case["kind"]
    states = 4 * DK * DV * H * (case["seqs"] if kind == "packed" else B)
    flops = 7.0 * tokens * H * DK * DV
    if kind in ("layer_prefill", "layer_step"):
        hid = case["hidden"]
        columns = 4 * HK * DK + 3 * H * DV                                         # q, k, b, f and v, w, o_gate
        conv = (2 * HK * DK + H * DV) * 3 * B * e
        weights = hid * (columns + H * DV) * e
        moved = weights + 2 * tokens * hid * e + (2 if kind == "layer_step" else 1) * (states + conv)
        return {"bytes": moved, "flops": flops + 2.0 * tokens * hid * (columns + H * DV)}
    moved = tokens * (HK * DK * (3 * e + 4) + H * DV * 3 * e) + states             # q, k, b, g; v, w and o; the final state
    if kind == "decode" or case["state"]:
        moved += states
    if kind == "forward":
        moved += tokens // 64 * H * DK * DV * 4
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """Four times the largest error of the calls against the same recurrence (and layer) in 64-bit arithmetic, over the
    listed cases and a few drawn ones; measured (2-norm, largest): decode 1.7e-3, 3.9e-3 in bf16 (the rounding of o)
    and 2.1e-4, 4.9e-4 in f16; the chunkwise forms 2.9e-3, 2.1e-2 in bf16 (their erase and query operands are bf16);
    float32 2.8e-7, 2.1e-6; the layer 5.5e-3, 4.3e-2 for prompts and 4.1e-3, 1.7e-2 for one token (its projections
    are rounded to bf16)."""
    kind = case["kind"]
    if kind == "layer_prefill":
        return {"rel": 2.2e-2, "max": 0.17}
    if kind == "layer_step":
        return {"rel": 1.6e-2, "max": 7e-2}
    if case["dtype"] == "f32":
        return {"rel": 1.1e-6, "max": 8e-6}
    if case["dtype"] == "f16":
        return {"rel": 9e-4, "max": 2e-3}
    return {"rel": 7e-3, "max": 1.6e-2} if kind == "decode" else {"rel": 1.2e-2, "max": 8e-2}
