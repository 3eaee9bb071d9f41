"""What is measured: the work that a step of this engine gives the GPU, layer kind by layer kind and as a whole model.

A case is one step of one part — a mixer or feed-forward, built from its registered kind and fed through ``Part.forward`` — or of a
whole decoder (``DecoderModel.forward``).  A step is any mix of ``portions`` prompt portions with ``tokens`` tokens together (each
behind ``behind`` tokens that earlier steps left in the cache) and ``singles`` sequences that decode one token at a context of
about ``context``.  As in the engine, steps of up to 1,024 tokens are recorded once in a CUDA graph and replayed, larger ones
are launched kernel by kernel.  Sizes are those of the shape files and of the benchmark's designs at widths 1,024, 2,048, 4,096.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

from dli_b200.cache.pools import CachePools, LayerCache
from dli_b200.config.registry import resolve_architecture
from dli_b200.config.spec import PartSpec
from dli_b200.engine.batch import GroupView, StepBatch
from dli_b200.parts.base import BuildEnv, build_part
from dli_b200.parts.model import DecoderModel

DEVICE = "cuda:0"
PAGE = 16
GRAPH_TOKENS = 1024
ROPE = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}

ATTENTION = ("gqa", "latent", "diff")
RECURRENT = ("mamba2", "gated_delta", "shift_decay", "channel_delta", "matrix_memory")
FEED_FORWARD = ("swiglu", "routed_glu")


def case(kind, dtype="bfloat16", width=2048, portions=0, tokens=0, behind=0, singles=0, context=0, window=0, layers=0):
    return {"kind": kind, "dtype": dtype, "width": width, "portions": portions, "tokens": tokens, "behind": behind, "singles": singles,
            "context": context, "window": window, "layers": layers}


def listed():
    return [
        # the headline: eight users' chat turns decode side by side through a whole Llama-3.2-1B
        dict(case("llama", layers=16, singles=8, context=2100), name="llama_decode_8"),
        # the other headline: one 2,048-token prompt through the whole model, logits at its last token
        dict(case("llama", layers=16, portions=1, tokens=2048), name="llama_prefill_2048"),
        # a full batch of decoding users: a Llama layer's feed-forward on 64 rows
        dict(case("swiglu", singles=64), name="swiglu_decode_64"),
        # one user's decode step through an attention layer: as small as a call gets
        dict(case("gqa", singles=1, context=700), name="gqa_decode_1"),
        # documents of several users at once in Mamba-2 layers, none of a round length
        dict(case("mamba2", portions=3, tokens=3001), name="mamba2_portions"),
        # one long prompt through a gated delta rule layer
        dict(case("gated_delta", portions=1, tokens=2048), name="gated_delta_prompt"),
        # one long prompt through attention over a cached latent
        dict(case("latent", portions=1, tokens=4096), name="latent_prompt"),
        # the second portion of a chunked prompt beside decoding users, differential attention with its window
        dict(case("diff", portions=1, tokens=1535, behind=1024, singles=9, context=1500, window=1024), name="diff_chunk_and_decode"),
        # a model checked in float32: short prompts through a token-shift recurrence
        dict(case("shift_decay", dtype="float32", portions=2, tokens=501), name="shift_decay_f32"),
        # two long prompts through a delta rule with a decay per channel
        dict(case("channel_delta", portions=2, tokens=3500), name="channel_delta_prompts"),
        # a short prompt that arrives while others decode, matrix memory
        dict(case("matrix_memory", portions=1, tokens=600, singles=7, context=900), name="matrix_memory_mixed"),
        # a long prompt's routed feed-forward
        dict(case("routed_glu", portions=1, tokens=2048), name="routed_prompt"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("llama",) + ATTENTION + RECURRENT + RECURRENT + FEED_FORWARD)
    width = rng.choice((1024, 2048, 2048, 4096))
    window = rng.choice((0, 512, 1024)) if kind in ("latent", "diff") else 0
    layers = rng.randint(2, 8) if kind == "llama" else 0
    if kind == "llama":
        width = 2048
    elif rng.random() < 0.15:  # the float32 path: what a model is checked with, at small sizes
        tokens = log(16, 512)
        return case(kind, "float32", min(width, 2048), rng.randint(1, min(3, tokens // 8)), tokens, 0, 0, 0, window)
    form = rng.choice(("prompts", "prompts", "decode", "mixed"))
    if kind in RECURRENT and form == "decode":
        form = "mixed"
    portions, tokens, behind, singles, context = 0, 0, 0, 0, 0
    if form != "decode":
        tokens = log(24, 1024 if form == "mixed" else 4096)
        portions = rng.randint(1, max(1, min(4, tokens // 16)))
        if kind in ATTENTION + ("llama",) and tokens > 512:
            behind = rng.choice((0, 512))
    if form != "prompts":
        singles, context = log(1, 64 if form == "decode" else 24), log(32, 4096)
    return case(kind, "bfloat16", width, portions, tokens, behind, singles, context, window, layers)


# ------------------------------------------------------------------------------------------------ sizes


def step_lengths(c):
    """Per sequence, single tokens first: (tokens this step, tokens before it)."""
    out = [(1, max(1, int(c["context"] * (0.5 + (i + 0.5) / c["singles"])))) for i in range(c["singles"])]
    left, parts = c["tokens"], c["portions"]
    share = [i + 2 for i in range(parts)]
    for i in range(parts):
        n = left if i == parts - 1 else max(2, c["tokens"] * share[i] // sum(share))
        out.append((n, c["behind"]))
        left -= n
    return out


def sizes(c):
    """The sizes of a kind at a width."""
    W, kind = c["width"], c["kind"]
    s = W / 2048
    if kind == "gqa":  # Llama-3.2-1B's heads; at width 4,096 heads of 128
        return dict(H=W, nh=32 if W > 1024 else 16, nkv=8 if W > 1024 else 4, d=128 if W == 4096 else 64)
    if kind == "latent":
        return dict(H=W, nh=int(16 * s), d=128, dr=64, dv=128, rank=192)
    if kind == "diff":
        return dict(H=W, nh=int(16 * s), nkv=int(4 * s), d=64, dv=128)
    if kind == "mamba2":
        return dict(H=W, nh=int(64 * s), P=64, N=64 if W == 1024 else 128, groups=8, taps=4)
    if kind in ("gated_delta", "channel_delta"):
        return dict(H=W, nh=int(16 * s), nkv=int(8 * s), d=128, taps=4, low=64)
    if kind == "shift_decay":
        return dict(H=W, nh=int(16 * s), d=64, low=64)
    if kind == "matrix_memory":
        return dict(H=W, nh=int(16 * s), d=128)
    if kind == "swiglu":
        return dict(H=W, ff=4 * W)
    if kind == "routed_glu":
        return dict(H=W, ff=W, E=16, top=4)
    return dict(H=2048, nh=32, nkv=8, d=64, ff=8192, V=128256)


def part_spec(c):
    z, kind = sizes(c), c["kind"]
    window = c["window"] or None
    if kind == "gqa":
        return "mixer", PartSpec("gqa_attention", {"hidden_size": z["H"], "num_heads": z["nh"], "num_kv_heads": z["nkv"], "head_dim": z["d"], "scale": z["d"] ** -0.5,
                                                   "window": window, "position": PartSpec("rotary", {"head_dim": z["d"], "rotary_dim": z["d"], "theta": 500000.0})})
    if kind == "latent":
        return "mixer", PartSpec("latent_attention", {"hidden_size": z["H"], "num_heads": z["nh"], "head_dim": z["d"], "rot_dim": z["dr"], "value_dim": z["dv"],
                                                      "kv_rank": z["rank"], "scale": (z["d"] + z["dr"]) ** -0.5, "window": window, "gate": True, "eps": 1e-6,
                                                      "rotary_dim": z["dr"], "theta": 500000.0})
    if kind == "diff":
        return "mixer", PartSpec("diff_attention", {"hidden_size": z["H"], "num_heads": z["nh"], "num_kv_heads": z["nkv"], "head_dim": z["d"], "value_dim": z["dv"],
                                                    "scale": z["d"] ** -0.5, "window": window, "keep_first": 16 if window else 0, "diff": 0.8, "eps": 1e-6,
                                                    "rotary_dim": z["d"], "theta": 500000.0})
    if kind == "mamba2":
        return "mixer", PartSpec("mamba2", {"hidden_size": z["H"], "num_heads": z["nh"], "head_dim": z["P"], "state_size": z["N"], "groups": z["groups"],
                                            "conv_taps": z["taps"], "norm_groups": z["groups"], "eps": 1e-6})
    if kind == "gated_delta":
        return "mixer", PartSpec("gated_delta", {"hidden_size": z["H"], "num_heads": z["nh"], "num_kv_heads": z["nkv"], "head_dim": z["d"], "value_dim": z["d"],
                                                 "conv_taps": z["taps"], "eps": 1e-6})
    if kind == "channel_delta":
        return "mixer", PartSpec("channel_delta", {"hidden_size": z["H"], "num_heads": z["nh"], "num_kv_heads": z["nkv"], "head_dim": z["d"], "value_dim": z["d"],
                                                   "conv_taps": z["taps"], "eps": 1e-6, "decay_rank": z["low"], "gate_rank": z["low"]})
    if kind == "shift_decay":
        return "mixer", PartSpec("shift_decay_recurrence", {"hidden_size": z["H"], "num_heads": z["nh"], "head_dim": z["d"], "eps": 1e-6, "decay_rank": z["low"]})
    if kind == "matrix_memory":
        return "mixer", PartSpec("matrix_memory", {"hidden_size": z["H"], "num_heads": z["nh"], "head_dim": z["d"], "value_dim": z["d"], "gate_cap": 15.0, "eps": 1e-6})
    if kind == "swiglu":
        return "feed_forward", PartSpec("swiglu", {"hidden_size": z["H"], "intermediate_size": z["ff"]})
    return "feed_forward", PartSpec("routed_glu", {"hidden_size": z["H"], "intermediate_size": z["ff"], "num_experts": z["E"], "top": z["top"], "route_scale": 2.5,
                                                   "group_count": 4, "group_keep": 2})


# ------------------------------------------------------------------------------------------------ inputs


def weights(c, seed):
    """Tensors by name: matrices N(0, 0.02) in the step's dtype, and float32 vectors with the spread that trained models give them."""
    z, kind, dt = sizes(c), c["kind"], getattr(torch, c["dtype"])
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 1)
    H, t = z["H"], {}

    def mat(name, *shape, std=0.02):
        t[name] = torch.empty(shape, dtype=dt, device=DEVICE).normal_(0.0, std, generator=g)

    def vec(name, n, lo, hi):
        t[name] = torch.empty(n, dtype=torch.float32, device=DEVICE).uniform_(lo, hi, generator=g)

    def steps(name, n):  # a bias whose softplus is spread over 0.001 .. 0.1, evenly over its logarithm
        vec(name, n, math.log(1e-3), math.log(0.1))
        t[name] = torch.log(torch.expm1(torch.exp(t[name])))

    def conv(name, rows):
        t[name] = torch.empty((rows, z["taps"]), dtype=torch.float32, device=DEVICE).uniform_(-0.5, 0.5, generator=g)

    if kind == "llama":
        mat("model.embed_tokens.weight", z["V"], H)
        vec("model.norm.weight", H, 0.9, 1.1)
        for i in range(c["layers"]):
            p = f"model.layers.{i}."
            for name, rows, cols in (("self_attn.q_proj", z["nh"] * z["d"], H), ("self_attn.k_proj", z["nkv"] * z["d"], H), ("self_attn.v_proj", z["nkv"] * z["d"], H),
                                     ("self_attn.o_proj", H, z["nh"] * z["d"]), ("mlp.gate_proj", z["ff"], H), ("mlp.up_proj", z["ff"], H), ("mlp.down_proj", H, z["ff"])):
                mat(p + name + ".weight", rows, cols)
            vec(p + "input_layernorm.weight", H, 0.9, 1.1)
            vec(p + "post_attention_layernorm.weight", H, 0.9, 1.1)
    elif kind == "gqa":
        mat("q_proj.weight", z["nh"] * z["d"], H), mat("k_proj.weight", z["nkv"] * z["d"], H), mat("v_proj.weight", z["nkv"] * z["d"], H)
        mat("o_proj.weight", H, z["nh"] * z["d"])
    elif kind == "latent":
        mat("q_proj.weight", z["nh"] * (z["d"] + z["dr"]), H), mat("kv_down_proj.weight", z["rank"] + z["dr"], H)
        mat("k_up_proj.weight", z["nh"] * z["d"], z["rank"], std=z["rank"] ** -0.5), mat("v_up_proj.weight", z["nh"] * z["dv"], z["rank"], std=z["rank"] ** -0.5)
        mat("g_proj.weight", z["nh"] * z["dv"], H), mat("o_proj.weight", H, z["nh"] * z["dv"])
        vec("kv_norm.weight", z["rank"], 0.9, 1.1)
    elif kind == "diff":
        mat("q_proj.weight", z["nh"] * 2 * z["d"], H), mat("k_proj.weight", z["nkv"] * 2 * z["d"], H), mat("v_proj.weight", z["nkv"] * z["dv"], H)
        mat("g_proj.weight", z["nh"], H), mat("o_proj.weight", H, z["nh"] * z["dv"])
        vec("q_norm.weight", z["d"], 0.9, 1.1), vec("k_norm.weight", z["d"], 0.9, 1.1)
        for name in ("lambda_q1", "lambda_k1", "lambda_q2", "lambda_k2"):
            vec(name, z["d"], -0.1, 0.1)
    elif kind == "mamba2":
        inner = z["nh"] * z["P"]
        channels = inner + 2 * z["groups"] * z["N"]
        mat("in_proj.weight", inner + channels + z["nh"], H), mat("out_proj.weight", H, inner)
        conv("conv1d.weight", channels), vec("conv1d.bias", channels, -0.2, 0.2)
        steps("dt_bias", z["nh"]), vec("A_log", z["nh"], 0.0, math.log(16.0)), vec("D", z["nh"], 0.5, 1.5), vec("norm.weight", inner, 0.9, 1.1)
    elif kind in ("gated_delta", "channel_delta"):
        qk, inner = z["nkv"] * z["d"], z["nh"] * z["d"]
        mat("q_proj.weight", qk, H), mat("k_proj.weight", qk, H), mat("v_proj.weight", inner, H), mat("b_proj.weight", z["nh"], H), mat("o_proj.weight", H, inner)
        if kind == "gated_delta":
            mat("a_proj.weight", z["nh"], H), mat("g_proj.weight", inner, H), steps("dt_bias", z["nh"])
        else:
            mat("a1.weight", z["low"], H), mat("a2.weight", inner, z["low"]), mat("g1.weight", z["low"], H), mat("g2.weight", inner, z["low"], std=0.1)
            steps("dt_bias", inner)
        vec("A_log", z["nh"], 0.0, math.log(16.0)), vec("norm.weight", z["d"], 0.9, 1.1)
        conv("q_conv.weight", qk), conv("k_conv.weight", qk), conv("v_conv.weight", inner)
    elif kind == "shift_decay":
        inner = z["nh"] * z["d"]
        for name in ("r_proj", "k_proj", "v_proj", "g_proj"):
            mat(name + ".weight", inner, H)
        mat("o_proj.weight", H, inner), mat("w1.weight", z["low"], H), mat("w2.weight", inner, z["low"])
        vec("w0", inner, -6.0, -0.5), vec("bonus", (z["nh"], z["d"]), -0.5, 1.0), vec("norm.weight", inner, 0.9, 1.1)
        for s in "rkvgw":
            vec("mu_" + s, H, 0.0, 1.0)
    elif kind == "matrix_memory":
        inner = z["nh"] * z["d"]
        for name in ("q_proj", "k_proj", "v_proj", "g_proj"):
            mat(name + ".weight", inner, H)
        mat("i_gate.weight", z["nh"], H), mat("f_gate.weight", z["nh"], H), mat("o_proj.weight", H, inner)
        vec("i_gate.bias", z["nh"], -10.0, 0.0), vec("f_gate.bias", z["nh"], 3.0, 6.0), vec("norm.weight", inner, 0.9, 1.1)
    elif kind == "swiglu":
        mat("gate_proj.weight", z["ff"], H), mat("up_proj.weight", z["ff"], H), mat("down_proj.weight", H, z["ff"])
    else:
        t["router.weight"] = torch.empty((z["E"], H), dtype=torch.float32, device=DEVICE).normal_(0.0, 0.02, generator=g)
        vec("router.correction", z["E"], -0.05, 0.05)
        for e in range(z["E"]):
            mat(f"experts.{e}.gate_proj.weight", z["ff"], H), mat(f"experts.{e}.up_proj.weight", z["ff"], H), mat(f"experts.{e}.down_proj.weight", H, z["ff"])
    return t


def step_tables(c, seed):
    """The step's integers on the host; a sequence's pages are scattered over the pool, as they are in a pool that has been in use."""
    lens = step_lengths(c)
    blocks = [-(-(n + before) // PAGE) for n, before in lens]
    pages = list(range(sum(blocks)))
    random.Random(seed * 31 + 7).shuffle(pages)
    tables, at = np.zeros((len(lens), max(blocks)), dtype=np.int32), 0
    positions, seq_of, slots = [], [], []
    for s, (n, before) in enumerate(lens):
        own = pages[at : at + blocks[s]]
        at += blocks[s]
        tables[s, : blocks[s]] = own
        p = np.arange(before, before + n)
        positions.append(p), seq_of.append(np.full(n, s))
        slots.append(np.asarray(own)[p // PAGE] * PAGE + p % PAGE)
    q_lens, starts = [n for n, _ in lens], [b for _, b in lens]
    return {"q_lens": q_lens, "starts": starts, "pages": sum(blocks), "tables": tables, "positions": np.concatenate(positions), "seq_of_token": np.concatenate(seq_of),
            "slots": np.concatenate(slots), "q_start": np.concatenate([[0], np.cumsum(q_lens)]), "kv_len": np.asarray(q_lens) + np.asarray(starts)}


def inputs(c, seed):
    """What the step reads besides weights: rows (or token ids), the cache that earlier steps left, the recurrent states."""
    z, kind, dt = sizes(c), c["kind"], getattr(torch, c["dtype"])
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 2)
    h = step_tables(c, seed)
    n, S, fresh = int(sum(h["q_lens"])), len(h["q_lens"]), torch.tensor([b == 0 for b in h["starts"]], device=DEVICE)

    def normal(shape, dtype, std=1.0):
        return torch.empty(shape, dtype=dtype, device=DEVICE).normal_(0.0, std, generator=g)

    x = torch.randint(0, z["V"], (n,), dtype=torch.int32, device=DEVICE, generator=g) if kind == "llama" else normal((n, z["H"]), dt)
    pools, states = [], []
    if kind in ("gqa", "llama"):
        layers = max(1, c["layers"])
        pools = [normal((layers, h["pages"] + 1, z["nkv"], PAGE, z["d"]), dt, 0.9) for _ in range(2)]
    elif kind == "latent":
        pools = [normal((1, h["pages"] + 1, 1, PAGE, z["rank"] + z["dr"]), dt)]
    elif kind == "diff":
        pools = [normal((1, h["pages"] + 1, z["nkv"], PAGE, 2 * z["d"]), dt), normal((1, h["pages"] + 1, z["nkv"], PAGE, z["dv"]), dt, 0.9)]
    elif kind == "mamba2":
        channels = z["nh"] * z["P"] + 2 * z["groups"] * z["N"]
        states = [normal((S, z["nh"], z["P"], z["N"]), torch.float32, 0.1), normal((S, z["taps"] - 1, channels), dt, 0.9)]
    elif kind in ("gated_delta", "channel_delta"):
        channels = 2 * z["nkv"] * z["d"] + z["nh"] * z["d"]
        states = [normal((S, z["nh"], z["d"], z["d"]), torch.float32, 0.05), normal((S, z["taps"] - 1, channels), dt, 0.9)]
    elif kind == "shift_decay":
        states = [normal((S, z["nh"], z["d"], z["d"]), torch.float32, 2.0), normal((S, 1, z["H"]), dt)]
    elif kind == "matrix_memory":
        states = [normal((S, z["nh"], z["d"] + 1, z["d"]), torch.float32, 0.5), torch.ones((S, z["nh"], z["d"] + 1), device=DEVICE)]
    for s in states:
        s[fresh] = 0  # a prompt's first portion starts from nothing
    return x, pools, states, h


def prepare(c, seed):
    """The part or model with its weights, the step's batch, and the cache and state slots as earlier steps left them."""
    dt = getattr(torch, c["dtype"])
    x, pools, starts, h = inputs(c, seed)
    n, S = int(sum(h["q_lens"])), len(h["q_lens"])

    def ints(a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEVICE)

    singles = c["singles"]
    batch = StepBatch(
        n=n, num_seqs=S, num_single=singles, token_ids=x if c["kind"] == "llama" else ints(np.zeros(n)), positions=ints(h["positions"]),
        seq_of_token=ints(h["seq_of_token"]), q_start=ints(h["q_start"]), kv_len=ints(h["kv_len"]), state_slot=ints(np.arange(S)),
        logit_rows=ints(h["q_start"][1:] - 1), groups=[GroupView(ints(h["tables"]), ints(h["slots"]))], q_lens=h["q_lens"], starts=h["starts"],
        state_slots=list(range(S)), max_q_len=max(h["q_lens"]), max_kv_len=int(max(h["kv_len"])),
        max_kv_len_single=max((k for k, q in zip(h["kv_len"].tolist(), h["q_lens"]) if q == 1), default=0), logits_all_rows=singles == S)
    states = ()
    if c["kind"] == "llama":
        arch = resolve_architecture({"model_type": "llama"})
        z = sizes(c)
        cfg = arch.parse_config({"model_type": "llama", "num_hidden_layers": c["layers"], "hidden_size": z["H"], "num_attention_heads": z["nh"],
                                 "num_key_value_heads": z["nkv"], "head_dim": z["d"], "intermediate_size": z["ff"], "vocab_size": z["V"], "rope_theta": 500000.0,
                                 "rope_scaling": ROPE, "tie_word_embeddings": True, "rms_norm_eps": 1e-5, "max_position_embeddings": 131072, "hidden_act": "silu"})
        model = DecoderModel(arch.model_spec(cfg), dt, DEVICE)
        model.load(weights(c, seed))
        cache = CachePools(model.cache_needs(), model.spec.run_order, [h["pages"]], PAGE, 1, dt, DEVICE)
        cache.k[0].copy_(pools[0]), cache.v[0].copy_(pools[1])
        pools = [cache.k[0], cache.v[0]]

        def forward():
            return model.forward(batch, cache.layer_caches)
    else:
        category, spec = part_spec(c)
        part = build_part(category, spec, BuildEnv(dt, torch.device(DEVICE)))
        part.load(weights(c, seed))
        if category == "feed_forward":
            def forward():
                return part.forward(x)
        else:
            states = tuple(torch.empty((S + 1, *s.shape[1:]), dtype=s.dtype, device=DEVICE) for s in starts)
            k = pools[0][0] if pools else None
            cache = LayerCache(0 if pools else None, k, (pools[1][0] if len(pools) > 1 else k), PAGE, states=states)

            def forward():
                return part.forward(x, batch, cache)

    @torch.inference_mode()
    def step():
        for slot, start in zip(states, starts):  # the states that the step begins with, as they were bound to its sequences
            slot[:S].copy_(start)
        return forward()

    state = {"step": step, "graph": None, "out": None, "kept": [*pools, *(s[:S] for s in states)]}
    if n <= GRAPH_TOKENS:
        side = torch.cuda.Stream(device=DEVICE)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                step()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["out"] = step()
        state["graph"] = graph
    return state


def run(state):
    """One step: its output rows (or logits), and the pools and state slots that it has written."""
    if state["graph"] is not None:
        state["graph"].replay()
        return [state["out"], *state["kept"]]
    return [state["step"](), *state["kept"]]


# ------------------------------------------------------------------------------------------------ work and tolerance


def work(c):
    z, kind = sizes(c), c["kind"]
    e = 2 if c["dtype"] == "bfloat16" else 4
    lens = step_lengths(c)
    n, S = sum(q for q, _ in lens), len(lens)
    W, window = z["H"], c["window"]
    fresh = sum(1 for _, b in lens if b == 0)
    if window:
        pairs = sum(min(b + i + 1, window) for q, b in lens for i in range(q))
        seen = sum(min(q + b, window + q) for q, b in lens)
    else:
        pairs = sum(q * b + q * (q + 1) // 2 for q, b in lens)
        seen = sum(q + b for q, b in lens)
    matrix, extra_flops, other = 0, 0, 0  # matrix elements, operations that are not products with a weight, other bytes
    if kind in ("gqa", "llama"):
        per = (z["nh"] * 2 + z["nkv"] * 2) * z["d"] * W
        att, kv = 4 * z["nh"] * z["d"] * pairs, 2 * z["nkv"] * z["d"] * e
        if kind == "gqa":
            matrix, extra_flops, other = per, att, kv * (seen - n) + kv * n
        else:
            per += 3 * z["ff"] * W
            matrix, extra_flops, other = per * c["layers"], att * c["layers"] + 2 * z["V"] * W * S, kv * seen * c["layers"] + z["V"] * W * e + S * z["V"] * 4 + n * W * e
            return {"bytes": matrix * e + other, "flops": 2 * matrix * n + extra_flops}
    elif kind == "latent":
        row = z["rank"] + z["dr"]
        matrix = W * (z["nh"] * (z["d"] + z["dr"]) + row + 2 * z["nh"] * z["dv"]) + z["nh"] * z["rank"] * (z["d"] + z["dv"])
        extra_flops, other = 2 * z["nh"] * (row + z["rank"]) * pairs, row * e * seen
    elif kind == "diff":
        matrix = W * (z["nh"] * 2 * z["d"] + z["nkv"] * (2 * z["d"] + z["dv"]) + z["nh"] + z["nh"] * z["dv"])
        extra_flops, other = 2 * z["nh"] * (2 * z["d"] + 2 * z["dv"]) * pairs, z["nkv"] * (2 * z["d"] + z["dv"]) * e * seen
    elif kind == "mamba2":
        inner = z["nh"] * z["P"]
        channels = inner + 2 * z["groups"] * z["N"]
        matrix = W * (inner + channels + z["nh"]) + W * inner
        extra_flops = n * (5 * z["nh"] * z["P"] * z["N"] + 2 * z["taps"] * channels)
        other = (2 * S - fresh) * (z["nh"] * z["P"] * z["N"] * 4 + (z["taps"] - 1) * channels * e)
    elif kind in ("gated_delta", "channel_delta"):
        qk, inner = z["nkv"] * z["d"], z["nh"] * z["d"]
        channels = 2 * qk + inner
        matrix = W * (channels + inner + z["nh"]) + (W * (inner + z["nh"]) if kind == "gated_delta" else 2 * z["low"] * (W + inner))
        extra_flops = n * (7 * z["nh"] * z["d"] * z["d"] + 2 * z["taps"] * channels)
        other = (2 * S - fresh) * (z["nh"] * z["d"] * z["d"] * 4 + (z["taps"] - 1) * channels * e)
    elif kind == "shift_decay":
        inner = z["nh"] * z["d"]
        matrix = 5 * W * inner + z["low"] * (W + inner)
        extra_flops, other = n * 6 * inner * z["d"], (2 * S - fresh) * (inner * z["d"] * 4 + W * e)
    elif kind == "matrix_memory":
        inner = z["nh"] * z["d"]
        matrix = 5 * W * inner + 2 * z["nh"] * W
        extra_flops, other = n * 5 * z["nh"] * z["d"] * (z["d"] + 1), (2 * S - fresh) * z["nh"] * (z["d"] + 1) * (z["d"] + 1) * 4
    elif kind == "swiglu":
        matrix = 3 * z["ff"] * W
    else:
        used = min(z["E"], n * z["top"])
        return {"bytes": 2 * n * W * e + z["E"] * W * 4 + used * 3 * z["ff"] * W * e, "flops": 6 * z["ff"] * W * n * z["top"] + 2 * n * z["E"] * W}
    return {"bytes": matrix * e + other + 2 * n * W * e, "flops": 2 * matrix * n + extra_flops}


def tolerance(c):
    if c["kind"] == "llama":
        return {"rel": 0.03, "max": 0.5}  # sixteen bits through up to sixteen layers
    if c["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-3}
    return {"rel": 0.01, "max": 0.25}


# ------------------------------------------------------------------------------------------------ the same in 64 bits


def sigmoid(v):
    return torch.sigmoid(v)


def rms(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def unit(v):
    return v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6)


def rotate(v, pos, d, base, pairs, scaling=None):
    """v [T, heads, >= d]: its first d numbers turned by position; pairs: (2i, 2i + 1), otherwise (i, i + d / 2)."""
    f = base ** (-torch.arange(0, d, 2, dtype=torch.float64, device=v.device) / d)
    if scaling:
        old, wave = scaling["original_max_position_embeddings"], 2 * math.pi / f
        smooth = (old / wave - scaling["low_freq_factor"]) / (scaling["high_freq_factor"] - scaling["low_freq_factor"])
        mid = (1 - smooth) * f / scaling["factor"] + smooth * f
        f = torch.where(wave > old / scaling["low_freq_factor"], f / scaling["factor"], torch.where(wave < old / scaling["high_freq_factor"], f, mid))
    ang = pos.double()[:, None, None] * f
    cos, sin, out = torch.cos(ang), torch.sin(ang), v.clone()
    a, b = (slice(0, d, 2), slice(1, d, 2)) if pairs else (slice(0, d // 2), slice(d // 2, d))
    out[..., a], out[..., b] = v[..., a] * cos - v[..., b] * sin, v[..., b] * cos + v[..., a] * sin
    return out


def attend(q, k, v, start, scale, window, keep):
    """q [T, d], k [K, d], v [K, dv] of one head; query t stands at position start + t."""
    T, K = q.shape[0], k.shape[0]
    out = torch.empty((T, v.shape[1]), dtype=torch.float64, device=q.device)
    j = torch.arange(K, device=q.device)[None, :]
    for t in range(0, T, 2048):
        i = torch.arange(start + t, start + min(T, t + 2048), device=q.device)[:, None]
        hidden = j > i
        if window:
            hidden |= (i - j >= window) & (j >= keep)
        s = (q[t : t + 2048] @ k.T) * scale
        out[t : t + 2048] = torch.softmax(s.masked_fill_(hidden, -math.inf), 1) @ v
    return out


def convolve(u, w, before):
    """u [T, C] behind before [taps - 1, C]; w [C, taps].  Returns the sums and the last taps - 1 inputs."""
    full, taps = torch.cat([before, u], 0), w.shape[1]
    return sum(full[j : j + u.shape[0]] * w[:, j] for j in range(taps)), full[full.shape[0] - (taps - 1) :]


def silu(v):
    return v * torch.sigmoid(v)


class Pages:
    """One layer's pools of one case in 64 bits: a sequence's rows, and what the step writes."""

    def __init__(self, pools, h):
        self.p, self.h = [p.double() for p in pools], h

    def write(self, rows, which):
        pos = torch.from_numpy(self.h["slots"]).to(DEVICE)
        self.p[which][pos // PAGE, :, pos % PAGE] = rows

    def rows(self, s, which):
        n = int(self.h["kv_len"][s])
        own = torch.from_numpy(self.h["tables"][s][: -(-n // PAGE)].astype(np.int64)).to(DEVICE)
        got = self.p[which][own]
        return got.transpose(1, 2).reshape(-1, got.shape[1], got.shape[3])[:n]


def gqa_exact(z, w, x, pages, h, pos, base, scaling, window):
    n = x.shape[0]
    q = rotate((x @ w["q_proj.weight"].T).view(n, z["nh"], z["d"]), pos, z["d"], base, False, scaling)
    pages.write(rotate((x @ w["k_proj.weight"].T).view(n, z["nkv"], z["d"]), pos, z["d"], base, False, scaling), 0)
    pages.write((x @ w["v_proj.weight"].T).view(n, z["nkv"], z["d"]), 1)
    out = torch.empty_like(q)
    for s, (t, start) in enumerate(zip(h["q_start"], h["starts"])):
        k, v, end = pages.rows(s, 0), pages.rows(s, 1), h["q_start"][s + 1]
        for a in range(z["nh"]):
            g = a // (z["nh"] // z["nkv"])
            out[t:end, a] = attend(q[t:end, a], k[:, g], v[:, g], start, z["d"] ** -0.5, window, 0)
    return out.view(n, -1) @ w["o_proj.weight"].T


def llama_exact(c, w, ids, pools, h, pos):
    z = sizes(c)
    x = w["model.embed_tokens.weight"][ids.long()].double()
    for i in range(c["layers"]):
        p = f"model.layers.{i}."
        lw = {k[len(p) :]: v.double() for k, v in w.items() if k.startswith(p)}
        pages = Pages([pools[0][i], pools[1][i]], h)
        y = rms(x, 1e-5) * lw["input_layernorm.weight"]
        x = x + gqa_exact(z, {k[len("self_attn.") :]: v for k, v in lw.items()}, y, pages, h, pos, 500000.0, ROPE, 0)
        y = rms(x, 1e-5) * lw["post_attention_layernorm.weight"]
        x = x + (silu(y @ lw["mlp.gate_proj.weight"].T) * (y @ lw["mlp.up_proj.weight"].T)) @ lw["mlp.down_proj.weight"].T
    last = torch.from_numpy(h["q_start"][1:] - 1).to(DEVICE)
    return (rms(x[last], 1e-5) * w["model.norm.weight"].double()) @ w["model.embed_tokens.weight"].double().T


def latent_exact(c, w, x, pages, h, pos):
    z, n = sizes(c), x.shape[0]
    q = (x @ w["q_proj.weight"].T).view(n, z["nh"], z["d"] + z["dr"])
    down = x @ w["kv_down_proj.weight"].T
    turned = rotate(down[:, None, z["rank"] :], pos, z["dr"], 500000.0, False)[:, 0]
    pages.write(torch.cat([rms(down[:, : z["rank"]], 1e-6) * w["kv_norm.weight"], turned], 1)[:, None], 0)
    q_turned = rotate(q[..., z["d"] :], pos, z["dr"], 500000.0, False)
    uk, uv = w["k_up_proj.weight"].view(z["nh"], z["d"], z["rank"]), w["v_up_proj.weight"].view(z["nh"], z["dv"], z["rank"])
    out = torch.empty((n, z["nh"], z["dv"]), dtype=torch.float64, device=x.device)
    for s, (t, start) in enumerate(zip(h["q_start"], h["starts"])):
        rows, end = pages.rows(s, 0)[:, 0], h["q_start"][s + 1]
        for a in range(z["nh"]):
            mine = torch.cat([q[t:end, a, : z["d"]] @ uk[a], q_turned[t:end, a]], 1)
            out[t:end, a] = attend(mine, rows, rows[:, : z["rank"]], start, (z["d"] + z["dr"]) ** -0.5, c["window"], 0) @ uv[a].T
    return (out.view(n, -1) * sigmoid(x @ w["g_proj.weight"].T)) @ w["o_proj.weight"].T


def diff_exact(c, w, x, pages, h, pos):
    z, n = sizes(c), x.shape[0]
    q = rms((x @ w["q_proj.weight"].T).view(n, z["nh"] * 2, z["d"]), 1e-6) * w["q_norm.weight"]
    k = rms((x @ w["k_proj.weight"].T).view(n, z["nkv"] * 2, z["d"]), 1e-6) * w["k_norm.weight"]
    q = rotate(q, pos, z["d"], 500000.0, True).view(n, z["nh"], 2, z["d"])
    pages.write(rotate(k, pos, z["d"], 500000.0, True).view(n, z["nkv"], 2 * z["d"]), 0)
    pages.write((x @ w["v_proj.weight"].T).view(n, z["nkv"], z["dv"]), 1)
    lam = math.exp(float(w["lambda_q1"] @ w["lambda_k1"])) - math.exp(float(w["lambda_q2"] @ w["lambda_k2"])) + 0.8
    out = torch.empty((n, z["nh"], z["dv"]), dtype=torch.float64, device=x.device)
    keep = 16 if c["window"] else 0
    for s, (t, start) in enumerate(zip(h["q_start"], h["starts"])):
        ks, vs, end = pages.rows(s, 0), pages.rows(s, 1), h["q_start"][s + 1]
        for a in range(z["nh"]):
            g = a // (z["nh"] // z["nkv"])
            maps = [attend(q[t:end, a, m], ks[:, g, m * z["d"] : (m + 1) * z["d"]], vs[:, g], start, z["d"] ** -0.5, c["window"], keep) for m in range(2)]
            out[t:end, a] = rms(maps[0] - lam * maps[1], 1e-6) * 0.2
    out *= sigmoid(x @ w["g_proj.weight"].T)[..., None]
    return out.view(n, -1) @ w["o_proj.weight"].T


def mamba2_exact(c, w, x, states):
    z, T = sizes(c), x.shape[0]
    S, before = states
    inner, gn = z["nh"] * z["P"], z["groups"] * z["N"]
    u = x @ w["in_proj.weight"].T
    channels = inner + 2 * gn
    mixed, before = convolve(u[:, inner : inner + channels], w["conv1d.weight"], before)
    mixed = silu(mixed + w["conv1d.bias"])
    v, per = mixed[:, :inner].view(T, z["nh"], z["P"]), z["nh"] // z["groups"]
    B = mixed[:, inner : inner + gn].view(T, z["groups"], z["N"]).repeat_interleave(per, 1)
    C = mixed[:, inner + gn :].view(T, z["groups"], z["N"]).repeat_interleave(per, 1)
    dt = torch.nn.functional.softplus(u[:, inner + channels :] + w["dt_bias"])
    keep, y = torch.exp(-torch.exp(w["A_log"]) * dt), torch.empty_like(v)
    write = dt[..., None] * v
    for t in range(T):
        S = keep[t, :, None, None] * S + write[t, :, :, None] * B[t, :, None, :]
        y[t] = (S @ C[t, :, :, None])[..., 0]
    y = (y + w["D"][:, None] * v).reshape(T, inner) * silu(u[:, :inner])
    return (rms(y.view(T, z["groups"], -1), 1e-6).view(T, inner) * w["norm.weight"]) @ w["out_proj.weight"].T, (S, before)


def delta_exact(c, w, x, states):
    """Both delta rules: a decay per head, or per head and key channel."""
    z, T = sizes(c), x.shape[0]
    S, before = states  # S [heads, value, key]
    qk, inner, per = z["nkv"] * z["d"], z["nh"] * z["d"], z["nh"] // z["nkv"]
    u = torch.cat([x @ w[r + "_proj.weight"].T for r in "qkv"], 1)
    mixed, before = convolve(u, torch.cat([w[r + "_conv.weight"] for r in "qkv"], 0), before)
    mixed = silu(mixed)
    q = (unit(mixed[:, :qk].view(T, z["nkv"], z["d"])) * z["d"] ** -0.5).repeat_interleave(per, 1)
    k = unit(mixed[:, qk : 2 * qk].view(T, z["nkv"], z["d"])).repeat_interleave(per, 1)
    v = mixed[:, 2 * qk :].view(T, z["nh"], z["d"])
    beta = sigmoid(x @ w["b_proj.weight"].T)
    if c["kind"] == "gated_delta":
        keep = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a_proj.weight"].T + w["dt_bias"]))[..., None]
        gate = silu(x @ w["g_proj.weight"].T)
    else:
        step = torch.nn.functional.softplus((x @ w["a1.weight"].T) @ w["a2.weight"].T + w["dt_bias"]).view(T, z["nh"], z["d"])
        keep = torch.exp(-torch.exp(w["A_log"])[:, None] * step)
        gate = sigmoid((x @ w["g1.weight"].T) @ w["g2.weight"].T)
    o = torch.empty_like(v)
    for t in range(T):
        S = S * keep[t, :, None, :]
        S = S + (beta[t, :, None] * (v[t] - (S @ k[t, :, :, None])[..., 0]))[:, :, None] * k[t, :, None, :]
        o[t] = (S @ q[t, :, :, None])[..., 0]
    o = (rms(o, 1e-6) * w["norm.weight"]).view(T, inner) * gate
    return o @ w["o_proj.weight"].T, (S, before)


def shift_decay_exact(c, w, x, states):
    z, T = sizes(c), x.shape[0]
    S, before = states  # S [heads, value, key]
    old = torch.cat([before, x[:-1]], 0)
    mix = {s: x + (old - x) * w["mu_" + s] for s in "rkvgw"}
    r, k, v = ((mix[s] @ w[s + "_proj.weight"].T).view(T, z["nh"], z["d"]) for s in "rkv")
    keep = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w["w1.weight"].T) @ w["w2.weight"].T + w["w0"])).view(T, z["nh"], z["d"])
    o = torch.empty_like(v)
    for t in range(T):
        kv = v[t, :, :, None] * k[t, :, None, :]
        o[t] = ((S + kv * w["bonus"][:, None, :]) @ r[t, :, :, None])[..., 0]
        S = S * keep[t, :, None, :] + kv
    o = rms(o, 1e-6).view(T, -1) * w["norm.weight"] * silu(mix["g"] @ w["g_proj.weight"].T)
    return o @ w["o_proj.weight"].T, (S, x[-1:])


def matrix_memory_exact(c, w, x, states):
    z, T, cap = sizes(c), x.shape[0], 15.0
    S, top = states[0], states[1][:, 0]  # S [heads, value + 1, key]: the vector n is the last value column
    q, k, v = ((x @ w[s + "_proj.weight"].T).view(T, z["nh"], z["d"]) for s in "qkv")
    q, v = q * z["d"] ** -0.5, torch.cat([v, torch.ones_like(v[..., :1])], 2)
    gi = cap * torch.tanh((x @ w["i_gate.weight"].T + w["i_gate.bias"]) / cap)
    gf = torch.nn.functional.logsigmoid(cap * torch.tanh((x @ w["f_gate.weight"].T + w["f_gate.bias"]) / cap))
    o = torch.empty((T, z["nh"], z["d"]), dtype=torch.float64, device=x.device)
    for t in range(T):
        new = torch.maximum(gf[t] + top, gi[t])
        S = torch.exp(gf[t] + top - new)[:, None, None] * S + torch.exp(gi[t] - new)[:, None, None] * v[t, :, :, None] * k[t, :, None, :]
        top = new
        read = (S @ q[t, :, :, None])[..., 0]
        o[t] = read[:, :-1] / (torch.maximum(read[:, -1].abs(), torch.exp(-top)) + 1e-6)[:, None]
    y = rms(o, 1e-6).view(T, -1) * w["norm.weight"] * sigmoid(x @ w["g_proj.weight"].T)
    return y @ w["o_proj.weight"].T, (S, top[:, None].expand(-1, z["d"] + 1))


def routed_exact(c, w, x):
    z = sizes(c)
    score = sigmoid(x @ w["router.weight"].T)
    choice = score + w["router.correction"]
    per = z["E"] // 4
    mark = choice.view(-1, 4, per).topk(2, 2).values.sum(2)
    best = mark.topk(2, 1).indices
    allowed = torch.zeros_like(mark).scatter_(1, best, 1.0).repeat_interleave(per, 1) > 0
    ids = choice.masked_fill(~allowed, -math.inf).topk(z["top"], 1).indices
    share = score.gather(1, ids)
    share = share / (share.sum(1, keepdim=True) + 1e-20) * 2.5
    out = torch.zeros_like(x)
    for e in range(z["E"]):
        t, j = torch.nonzero(ids == e, as_tuple=True)
        y = x[t]
        y = (silu(y @ w[f"experts.{e}.gate_proj.weight"].T) * (y @ w[f"experts.{e}.up_proj.weight"].T)) @ w[f"experts.{e}.down_proj.weight"].T
        out.index_add_(0, t, y * share[t, j][:, None])
    return out


@torch.no_grad()
def exact(c, seed):
    kind = c["kind"]
    w = weights(c, seed)
    x, pools, starts, h = inputs(c, seed)
    pos = torch.from_numpy(h["positions"]).to(DEVICE)
    if kind == "llama":
        return [llama_exact(c, w, x, pools, h, pos), None, None]
    w, x = {k: v.double() for k, v in w.items()}, x.double()
    if kind in ATTENTION:
        pages = Pages([p[0] for p in pools], h)
        if kind == "gqa":
            out = gqa_exact(sizes(c), w, x, pages, h, pos, 500000.0, None, c["window"])
        else:
            out = (latent_exact if kind == "latent" else diff_exact)(c, w, x, pages, h, pos)
        return [out, *(p[None] for p in pages.p)]
    if kind in RECURRENT:
        rule = {"mamba2": mamba2_exact, "gated_delta": delta_exact, "channel_delta": delta_exact, "shift_decay": shift_decay_exact, "matrix_memory": matrix_memory_exact}[kind]
        out, after = [], []
        for s in range(len(h["q_lens"])):
            y, states = rule(c, w, x[h["q_start"][s] : h["q_start"][s + 1]], [t[s].double() for t in starts])
            out.append(y), after.append(states)
        return [torch.cat(out, 0), *(torch.stack([a[i] for a in after], 0) for i in range(len(starts)))]
    if kind == "swiglu":
        return [(silu(x @ w["gate_proj.weight"].T) * (x @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T]
    return [routed_exact(c, w, x)]
