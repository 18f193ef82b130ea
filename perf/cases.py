"""The work by which this library's speed is judged, case by case.

A case is a call that a program makes through the public entry points: whole requests through ``Engine`` and its
step function, or one part of a layer (a mixer, a feed-forward, a whole block) through ``bind`` and ``forward`` with
the library's own cache and step description. Steps of one token per sequence replay a captured graph, as the step
function itself does. ``exact`` restates every part in 64 bits with plain torch.

Sizes are the configurations' own: Qwen3 at 4B, 8B and 14B, the 1.5k- and 2.5k-wide presets of the hybrid designs and
the 2k-wide presets of the designs with routed experts. Weights are drawn like a fresh model's (normal, 0.02), decays
and gates over the ranges that trained models use.
"""

from __future__ import annotations

import json
import math
import os
import shutil
import tempfile

import torch
import torch.nn.functional as F

DEVICE = "cuda:0"
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

QWEN = {
    "4b": dict(hidden=2560, inter=9728, heads=32, kv=8, dim=128, vocab=151936, theta=5e6, tied=True),
    "8b": dict(hidden=4096, inter=12288, heads=32, kv=8, dim=128, vocab=151936, theta=1e6, tied=False),
    "14b": dict(hidden=5120, inter=17408, heads=40, kv=8, dim=128, vocab=151936, theta=1e6, tied=False),
}

# mixers of the other designs, with the sizes of their presets
MIXERS = {
    "delta_1b": dict(kind="delta", hidden=1536, heads=12, kv=4, window=1024, d_heads=8, d_dim=64, rank=16),
    "delta_4b": dict(kind="delta", hidden=2560, heads=32, kv=8, window=1024, d_heads=16, d_dim=64, rank=16),
    "timemix_1b": dict(kind="timemix", hidden=1536, d_heads=24, d_dim=64, rank=16),
    "timemix_4b": dict(kind="timemix", hidden=2560, d_heads=40, d_dim=64, rank=16),
    "ssm_1b": dict(kind="ssm", hidden=1536, d_heads=48, d_dim=64, state=128, groups=4, taps=4),
    "gla_lite": dict(kind="gla", hidden=2048, d_heads=8, d_dim=128, vdim=256, rank=16),
    "mlstm_lite": dict(kind="mlstm", hidden=2048, d_heads=8, d_dim=128, vdim=256),
    "window_lite": dict(kind="window", hidden=2048, heads=16, kv=4, window=1024, softcap=0.0),
    "capped_lite": dict(kind="window", hidden=2048, heads=16, kv=4, window=4096, softcap=30.0),
}

EXPERTS = {
    "disorax_lite": dict(hidden=2048, experts=64, top=6, inter=1408, shared=2816, gate=True, clamp=0.0, ways="chosen"),
    "givizen_lite": dict(hidden=2048, experts=64, top=6, inter=1408, shared=2816, gate=False, clamp=7.0, ways="input"),
    "zadunex_1b": dict(hidden=1536, experts=16, top=2, inter=3072, shared=0, gate=False, clamp=0.0, ways="all"),
}


def listed():
    return [
        # a batch of chats: eight unequal prompts start together and are answered (headline workload, fewer layers)
        {"name": "chat_8", "kind": "chat", "model": "4b", "layers": 4, "dtype": "bfloat16", "batch": 8, "low": 100, "high": 600, "steps": 16},
        # the 32-bit path: a short batch replayed for its logits
        {"name": "replay_float32", "kind": "chat", "model": "4b", "layers": 2, "dtype": "float32", "batch": 3, "low": 40, "high": 200, "steps": 6},
        # one user waiting for the next token: the smallest call, a layer at one row
        {"name": "layer_token_1", "kind": "layer", "model": "4b", "dtype": "bfloat16", "batch": 1, "tokens": 1, "low": 1024, "high": 1024},
        # a full server: 64 sequences, one token each
        {"name": "layer_tokens_64", "kind": "layer", "model": "4b", "dtype": "bfloat16", "batch": 64, "tokens": 1, "low": 900, "high": 1300},
        # one long prompt
        {"name": "layer_prompt_2048", "kind": "layer", "model": "4b", "dtype": "bfloat16", "batch": 1, "tokens": 2048, "low": 0, "high": 0},
        # unequal prompts of the 14B sizes
        {"name": "layer_prompts_14b", "kind": "layer", "model": "14b", "dtype": "bfloat16", "batch": 4, "tokens": 1531, "low": 0, "high": 0},
        # windowed attention beside a delta rule, a long prompt
        {"name": "delta_prompt_2048", "kind": "mixer", "model": "delta_1b", "batch": 1, "tokens": 2048, "low": 0, "high": 0},
        # time mixing, three unequal prompts
        {"name": "timemix_prompts_3", "kind": "mixer", "model": "timemix_4b", "batch": 3, "tokens": 1021, "low": 0, "high": 0},
        # a state-space layer, a long prompt
        {"name": "ssm_prompt_2048", "kind": "mixer", "model": "ssm_1b", "batch": 1, "tokens": 2048, "low": 0, "high": 0},
        # attention with distance biases over a window, a long prompt
        {"name": "window_prompt_2048", "kind": "mixer", "model": "window_lite", "batch": 1, "tokens": 2048, "low": 0, "high": 0},
        # routed experts, eight sequences' next tokens
        {"name": "experts_tokens_8", "kind": "experts", "model": "disorax_lite", "batch": 8, "tokens": 1},
        # routed experts, a long prompt
        {"name": "experts_prompt_2048", "kind": "experts", "model": "givizen_lite", "batch": 1, "tokens": 2048},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["chat", "layer", "layer", "layer", "mixer", "mixer", "mixer", "experts", "experts"])
    if kind == "chat":
        dtype = rng.choice(["bfloat16", "float32"])
        batch = _log_int(rng, 1, 8) if dtype == "bfloat16" else rng.randint(1, 3)
        high = _log_int(rng, 40, 600) if dtype == "bfloat16" else _log_int(rng, 20, 200)
        return {"kind": "chat", "model": "4b", "layers": rng.randint(1, 2), "dtype": dtype, "batch": batch,
                "low": max(1, high // rng.randint(1, 8)), "high": high, "steps": rng.randint(2, 16 if dtype == "bfloat16" else 6)}
    one_token = rng.random() < 0.5
    if kind == "layer":
        if one_token:
            low = _log_int(rng, 16, 2000)
            return {"kind": "layer", "model": rng.choice(["4b", "8b", "14b"]), "dtype": "bfloat16", "batch": _log_int(rng, 1, 64),
                    "tokens": 1, "low": low, "high": low + rng.randint(0, low // 2)}
        batch = rng.randint(1, 4)
        first = rng.choice([0, 0, rng.randint(1, 1000)])
        return {"kind": "layer", "model": rng.choice(["4b", "8b", "14b"]), "dtype": "bfloat16", "batch": batch,
                "tokens": _log_int(rng, 20, 4000 // batch), "low": first, "high": first}
    if kind == "mixer":
        batch = _log_int(rng, 1, 32) if one_token else rng.randint(1, 4)
        first = rng.randint(1, 1500) if one_token else rng.choice([0, 0, rng.randint(1, 1500)])
        return {"kind": "mixer", "model": rng.choice(sorted(MIXERS)), "batch": batch,
                "tokens": 1 if one_token else _log_int(rng, 30, 3000 // batch), "low": first, "high": first}
    return {"kind": "experts", "model": rng.choice(sorted(EXPERTS)), "batch": _log_int(rng, 1, 64) if one_token else 1,
            "tokens": 1 if one_token else _log_int(rng, 20, 4000)}


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------

class _Draw:
    def __init__(self, seed, dtype):
        self.g = torch.Generator(DEVICE).manual_seed(seed)
        self.dtype = dtype

    def normal(self, *shape, std=0.02, mean=0.0, dtype=None):
        # the values of a checkpoint, which is in bfloat16 on either path
        t = torch.empty(shape, dtype=torch.float32, device=DEVICE).normal_(mean, std, generator=self.g)
        return t.to(torch.bfloat16).to(dtype or self.dtype)

    def between(self, low, high, *shape):
        t = torch.empty(shape, dtype=torch.float32, device=DEVICE).uniform_(low, high, generator=self.g)
        return t.to(torch.bfloat16).to(self.dtype)

    def rows(self, *shape, std=1.0):
        return torch.empty(shape, dtype=torch.float32, device=DEVICE).normal_(0.0, std, generator=self.g).to(self.dtype)


def _lengths(case):
    """Tokens that each sequence brings, and the tokens that it holds already. Unequal unless there is one sequence
    or one token each: sequence i of a step of prompts brings between half of ``tokens`` and all of them."""
    n, t = case["batch"], case["tokens"]
    brings = [1] * n if t == 1 else [max(1, t - (t * i) // (2 * n)) for i in range(n)]
    low, high = case.get("low", 0), case.get("high", 0)
    holds = [low + ((high - low) * ((i * 37) % 64)) // 64 for i in range(n)]
    return brings, holds


def _qwen_layer(d, m, prefix=""):
    H, D = m["hidden"], m["dim"]
    w = {"input_layernorm": d.normal(H, mean=1.0), "post_attention_layernorm": d.normal(H, mean=1.0),
         "self_attn.q_proj": d.normal(m["heads"] * D, H), "self_attn.k_proj": d.normal(m["kv"] * D, H),
         "self_attn.v_proj": d.normal(m["kv"] * D, H), "self_attn.o_proj": d.normal(H, m["heads"] * D),
         "self_attn.q_norm": d.normal(D, mean=1.0), "self_attn.k_norm": d.normal(D, mean=1.0),
         "mlp.gate_proj": d.normal(m["inter"], H), "mlp.up_proj": d.normal(m["inter"], H), "mlp.down_proj": d.normal(H, m["inter"])}
    return {f"{prefix}{k}.weight": v for k, v in w.items()} if prefix else w


def _chat_inputs(case, seed):
    m = QWEN[case["model"]]
    d = _Draw(seed, torch.bfloat16)
    w = {"model.embed_tokens.weight": d.normal(m["vocab"], m["hidden"]), "model.norm.weight": d.normal(m["hidden"], mean=1.0)}
    for i in range(case["layers"]):
        w.update(_qwen_layer(d, m, f"model.layers.{i}."))
    g = torch.Generator().manual_seed(seed)
    lens = torch.randint(case["low"], case["high"] + 1, (case["batch"],), generator=g).tolist()
    prompts = [torch.randint(0, m["vocab"], (n,), generator=g).tolist() for n in lens]
    given = torch.randint(0, m["vocab"], (case["steps"], case["batch"]), generator=g).tolist()
    return w, prompts, given


def _context(d, brings, holds, kv, dim, vdim):
    """Keys and values that the sequences hold before the step, [tokens, kv heads, size] each."""
    return [(d.rows(n, kv, dim), d.rows(n, kv, vdim)) for n in holds]


def _layer_inputs(case, seed):
    m = QWEN[case["model"]]
    d = _Draw(seed, DTYPES[case["dtype"]])
    brings, holds = _lengths(case)
    w = _qwen_layer(d, m)
    return w, d.rows(sum(brings), m["hidden"]), _context(d, brings, holds, m["kv"], m["dim"], m["dim"]), brings, holds


def _attention_weights(d, m):
    H, D = m["hidden"], 128
    return {"q": d.normal(m["heads"] * D, H), "k": d.normal(m["kv"] * D, H), "v": d.normal(m["kv"] * D, H),
            "o": d.normal(H, m["heads"] * D), "sink": d.normal(m["heads"], std=0.5)}


def _decayed_weights(d, m, low, high):
    C, HN, R = m["hidden"], m["d_heads"] * m["d_dim"], m["rank"]
    w = {k: d.normal(HN, C) for k in ("r", "k", "v", "g")}
    w.update({"w1": d.normal(R, C), "w2": d.normal(HN, R, std=0.1), "w0": d.between(low, high, HN),
              "norm": d.normal(HN, mean=1.0), "o": d.normal(C, HN)})
    return w


def _mixer_inputs(case, seed):
    """(weights, rows, keys and values held, states held [sequences, ...], tokens brought, tokens held)"""
    m = MIXERS[case["model"]]
    d = _Draw(seed, torch.bfloat16)
    brings, holds = _lengths(case)
    n, C, kind = case["batch"], m["hidden"], m["kind"]
    context, states = None, []
    state = lambda *shape, std=1.0: torch.empty((n,) + shape, dtype=torch.float32, device=DEVICE).normal_(
        0.0, std if holds[0] else 0.0, generator=d.g)
    if kind == "delta":
        HN = m["d_heads"] * m["d_dim"]
        w = {"left." + k: v for k, v in _attention_weights(d, m).items()}
        right = _decayed_weights(d, m, -6.0, 1.0)
        right.update({"a": d.normal(HN, C), "a.b": d.normal(HN, std=0.5)})
        w.update({"right." + k: v for k, v in right.items()})
        context = _context(d, brings, holds, m["kv"], 128, 128)
        states = [state(m["d_heads"], m["d_dim"], m["d_dim"])]
    elif kind == "timemix":
        w = _decayed_weights(d, m, -6.0, 0.0)
        w.update({"mu." + s: d.between(0.0, 1.0, C) for s in "rkvgw"})
        w["u"] = d.normal(m["d_heads"], m["d_dim"], std=0.5)
        states = [state(m["d_heads"], m["d_dim"], m["d_dim"]), state(C)]
    elif kind == "ssm":
        HP, GN, H = m["d_heads"] * m["d_dim"], m["groups"] * m["state"], m["d_heads"]
        step = torch.exp(d.between(math.log(0.001), math.log(0.1), H).float())
        w = {"in": d.normal(2 * HP + 2 * GN + H, C), "conv": d.between(-0.5, 0.5, HP + 2 * GN, m["taps"]),
             "conv.b": d.normal(HP + 2 * GN), "dt_bias": torch.log(torch.expm1(step)).to(torch.bfloat16),
             "A_log": torch.log(d.between(1.0, 16.0, H).float()).to(torch.bfloat16), "D": d.normal(H, mean=1.0),
             "norm": d.normal(HP, mean=1.0), "o": d.normal(C, HP)}
        states = [state(H, m["state"], m["d_dim"]), state(m["taps"] - 1, HP + 2 * GN).to(torch.bfloat16)]
    elif kind in ("gla", "mlstm"):
        HN, HP, H = m["d_heads"] * m["d_dim"], m["d_heads"] * m["vdim"], m["d_heads"]
        w = {"q": d.normal(HN, C), "k": d.normal(HN, C), "v": d.normal(HP, C), "g": d.normal(HP, C), "o": d.normal(C, HP)}
        if kind == "gla":
            w.update({"a1": d.normal(m["rank"], C), "a2": d.normal(HN, m["rank"], std=0.1), "a2.b": d.normal(HN, std=1.0),
                      "norm": d.normal(m["vdim"], mean=1.0)})
            states = [state(H, m["d_dim"], m["vdim"])]
        else:
            w.update({"i": d.normal(H, C), "i.b": d.normal(H, std=0.1), "f": d.normal(H, C), "f.b": d.between(3.0, 6.0, H),
                      "norm": d.normal(HP, mean=1.0)})
            beside = state(H, m["d_dim"] + 1)
            beside[..., -1].abs_()
            states = [state(H, m["d_dim"], m["vdim"]), beside]
    else:
        w = _attention_weights(d, m)
        if m["softcap"]:
            del w["sink"]
            w["g"] = d.normal(m["heads"], C)
        else:
            w.update({"q.norm": d.normal(128, mean=1.0), "k.norm": d.normal(128, mean=1.0)})
        context = _context(d, brings, holds, m["kv"], 128, 128)
    return w, d.rows(sum(brings), C), context, states, brings, holds


def _experts_inputs(case, seed):
    m = EXPERTS[case["model"]]
    d = _Draw(seed, torch.bfloat16)
    H, E, I = m["hidden"], m["experts"], m["inter"]
    w = {"router": d.normal(E, H)}
    gate, up, down = d.normal(E, I, H), d.normal(E, I, H), d.normal(E, H, I)
    for e in range(E):
        w.update({f"e{e}.gate": gate[e], f"e{e}.up": up[e], f"e{e}.down": down[e]})
    if m["ways"] == "chosen":
        w["router.b"] = d.normal(E, std=0.1)
    if m["shared"]:
        w.update({"shared.gate": d.normal(m["shared"], H), "shared.up": d.normal(m["shared"], H), "shared.down": d.normal(H, m["shared"])})
        if m["gate"]:
            w["shared.sg"] = d.normal(1, H)
    return w, d.rows(case["batch"] * case["tokens"], H)


# ---------------------------------------------------------------------------
# the library's side
# ---------------------------------------------------------------------------

def _write_folder(folder, config, tensors):
    """config.json and one safetensors file: eight bytes of header length, a JSON header, the tensors' bytes."""
    header, at = {}, 0
    for name, t in tensors.items():
        size = t.numel() * t.element_size()
        header[name] = {"dtype": "BF16", "shape": list(t.shape), "data_offsets": [at, at + size]}
        at += size
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(config, f)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(len(text).to_bytes(8, "little") + text)
        for t in tensors.values():
            t.view(torch.uint8).cpu().numpy().tofile(f)


def _prepare_chat(case, seed):
    from kernel_rush_kawk_b200 import Engine

    m = QWEN[case["model"]]
    w, prompts, given = _chat_inputs(case, seed)
    config = {"architectures": ["Qwen3ForCausalLM"], "hidden_size": m["hidden"], "intermediate_size": m["inter"],
              "num_hidden_layers": case["layers"], "num_attention_heads": m["heads"], "num_key_value_heads": m["kv"],
              "head_dim": m["dim"], "vocab_size": m["vocab"], "rope_theta": m["theta"], "rms_norm_eps": 1e-6,
              "tie_word_embeddings": True, "max_position_embeddings": 4096}
    folder = tempfile.mkdtemp(prefix="chat_")
    try:
        _write_folder(folder, config, w)
        del w
        engine = Engine(folder, dtype=case["dtype"], device=DEVICE)
    finally:
        shutil.rmtree(folder)
    pages = sum(-(-(len(p) + case["steps"]) // 64) for p in prompts)
    engine.open_cache(pages * 64, case["batch"])
    return {"engine": engine, "prompts": prompts, "given": given}


def _run_chat(state):
    from kernel_rush_kawk_b200.engine import StepEntry

    engine = state["engine"]
    slots = [engine.cache.alloc() for _ in state["prompts"]]
    logits = [engine.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, state["prompts"])])]
    for row in state["given"]:  # the step's buffer is the next step's too: what is kept is copied
        logits.append(engine.step([StepEntry(s, [t], [0]) for s, t in zip(slots, row)]).clone())
    for s in slots:
        engine.cache.free(s)
    return logits


def _prepare_part(part, dtype, weights, rows, brings, holds, context=None, states=(), forward=None):
    """What a program keeps around a part: its cache, the step's description, the rows, and a captured graph where
    every sequence brings one token."""
    from kernel_rush_kawk_b200.cache.store import KVView, SequenceCache
    from kernel_rush_kawk_b200.csrc import load_kernels
    from kernel_rush_kawk_b200.engine import BatchMeta, Runtime, StepContext

    ops = load_kernels(tuple(getattr(part, "attention_head_dims", lambda: ())()), DEVICE)
    runtime = Runtime(torch.device(DEVICE), dtype, ops)
    part.bind(weights, runtime)
    n, total = len(brings), sum(-(-(a + b) // 64) * 64 for a, b in zip(brings, holds))
    longest = max(a + b for a, b in zip(brings, holds))
    need = part.cache_need() if hasattr(part, "cache_need") else None
    cache = SequenceCache([need], total, n, longest, DEVICE, dtype, step_tokens=max(brings))
    slots = []
    for a, b in zip(brings, holds):
        slots.append(cache.alloc())
        cache.reserve(slots[-1], a + b)
        cache.advance(slots[-1], b)
    cache.sync()
    view = cache.view(0)
    views = view if isinstance(view, tuple) else () if view is None else (view,)
    kept, given = [], list(states)
    for v in views:
        if isinstance(v, KVView):
            kept += [v.k, v.v]
            for slot, (k, val) in zip(slots, context):
                p = torch.arange(k.shape[0], device=DEVICE)
                if v.window is not None:  # a ring of pages holds the last positions only
                    p = p[max(0, k.shape[0] - v.window):]
                page = v.table[slot].long()[(p // 64) % v.width]
                v.k[page, :, p % 64] = k[p].to(dtype)
                v.v[page, :, p % 64] = val[p].to(dtype)
        else:
            kept.append(v.state)
            v.state[slots] = given.pop(0).to(v.state.dtype)
    fresh = [(v.state, v.state.clone()) for v in views if not isinstance(v, KVView)]
    meta = BatchMeta(sum(brings), n, 0, DEVICE)
    meta.fill(slots, holds, [[0] * a for a in brings], [])
    forward = forward or (lambda ctx: part.forward(ctx, rows, ctx.cache_view(0)))
    call = lambda: forward(StepContext(ops, meta, cache))
    state = {"call": call, "fresh": fresh, "kept": kept, "graph": None, "part": part, "rows": rows}
    if max(brings) == 1:
        side = torch.cuda.Stream(device=DEVICE)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            call()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["out"] = call()
    return state


def _run_part(state):
    for s, start in state["fresh"]:  # each pass continues from the same state
        s.copy_(start)
    if state["graph"] is not None:
        state["graph"].replay()
        out = state["out"]
    else:
        out = state["call"]()
    return list(out if isinstance(out, (list, tuple)) else [out]) + state["kept"]


class _Layer:
    """A whole decoder layer as one part: norms, attention and feed-forward in their block."""

    def __init__(self, m, positions):
        from kernel_rush_kawk_b200 import parts
        from kernel_rush_kawk_b200.parts import base

        norm = lambda: base.norm_class("rmsnorm")({"size": m["hidden"], "eps": 1e-6})
        self.rope = parts.RotaryTable({"theta": m["theta"], "dim": m["dim"], "positions": positions})
        self.mixer = base.mixer_class("gqa_attention")({"hidden": m["hidden"], "heads": m["heads"], "kv_heads": m["kv"],
                                                        "head_dim": m["dim"], "eps": 1e-6})
        self.mixer.set_position(self.rope)
        self.ffn = base.feed_forward_class("swiglu")({"hidden": m["hidden"], "intermediate": m["inter"]})
        self.norms = (norm(), norm())
        self.block = base.block_class("prenorm")(self.norms[0], self.mixer, self.norms[1], self.ffn)

    def attention_head_dims(self):
        return self.mixer.attention_head_dims()

    def cache_need(self):
        return self.mixer.cache_need()

    def bind(self, w, runtime):
        self.rope.bind({}, runtime)
        self.norms[0].bind({"weight": w["input_layernorm"]}, runtime)
        self.norms[1].bind({"weight": w["post_attention_layernorm"]}, runtime)
        self.mixer.bind({k[10:]: v for k, v in w.items() if k.startswith("self_attn.")}, runtime)
        self.ffn.bind({k[4:]: v for k, v in w.items() if k.startswith("mlp.")}, runtime)


def _prepare_layer(case, seed):
    from kernel_rush_kawk_b200.parts import Stream

    w, rows, context, brings, holds = _layer_inputs(case, seed)
    layer = _Layer(QWEN[case["model"]], 8192)

    def forward(ctx):
        stream = layer.block.forward(ctx, Stream(rows), ctx.cache_view(0))
        return [stream.x, stream.branch]

    return _prepare_part(layer, DTYPES[case["dtype"]], w, rows, brings, holds, context, forward=forward)


def _attention_params(m):
    return {"hidden": m["hidden"], "heads": m["heads"], "kv_heads": m["kv"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
            "window": m["window"], "eps": 1e-6}


def _mixer_part(m):
    import kernel_rush_kawk_b200.parts  # noqa: F401  (registers the kinds)
    from kernel_rush_kawk_b200.parts.base import mixer_class

    C, kind = m["hidden"], m["kind"]
    if kind == "delta":
        left = dict(_attention_params(m), rot_dims=128, rot_base=10000.0, value_norm=True, sink=True)
        right = {"hidden": C, "heads": m["d_heads"], "dim": m["d_dim"], "rank": m["rank"], "eps": 1e-6}
        return mixer_class("parallel")({"hidden": C, "branches": [
            {"name": "left", "kind": "sink_window_attention", "scale": 1.0, "params": left},
            {"name": "right", "kind": "delta_rule", "scale": 1.0, "params": right}]})
    if kind == "timemix":
        return mixer_class("wkv_time_mix")({"hidden": C, "heads": m["d_heads"], "dim": m["d_dim"], "rank": m["rank"], "eps": 1e-6})
    if kind == "ssm":
        return mixer_class("mamba2")({"hidden": C, "heads": m["d_heads"], "head_dim": m["d_dim"], "state": m["state"],
                                      "groups": m["groups"], "taps": m["taps"], "norm_groups": 4, "eps": 1e-6})
    if kind in ("gla", "mlstm"):
        params = {"hidden": C, "heads": m["d_heads"], "dim": m["d_dim"], "vdim": m["vdim"], "eps": 1e-5}
        params.update({"rank": m["rank"], "tau": 16.0} if kind == "gla" else {"gate_cap": 15.0})
        return mixer_class(kind)(params)
    params = dict(_attention_params(m), q_temp=(0.1, 4096), distance_bias=True)
    params.update({"qk_norm": "head_rms", "softcap": m["softcap"], "gate": "head"} if m["softcap"] else {"qk_norm": "head", "sink": True})
    return mixer_class("sink_window_attention")(params)


def _prepare_mixer(case, seed):
    w, rows, context, states, brings, holds = _mixer_inputs(case, seed)
    return _prepare_part(_mixer_part(MIXERS[case["model"]]), torch.bfloat16, w, rows, brings, holds, context, states)


def _prepare_experts(case, seed):
    import kernel_rush_kawk_b200.parts  # noqa: F401
    from kernel_rush_kawk_b200.parts.base import feed_forward_class

    m = EXPERTS[case["model"]]
    w, rows = _experts_inputs(case, seed)
    params = {"hidden": m["hidden"], "experts": m["experts"], "top": m["top"], "intermediate": m["inter"],
              "shared_intermediate": m["shared"] or None, "shared_gate": m["gate"]}
    if m["ways"] == "chosen":
        params["router_bias"] = True
    elif m["ways"] == "all":
        params.update(router_bias=False, weights="all")
    else:
        params.update(activation="swish_clamped", limit=m["clamp"], shared_limit=m["clamp"], scoring="sigmoid", weigh_input=True)
    part = feed_forward_class("routed_experts")(params)
    brings = [case["tokens"]] * case["batch"]
    return _prepare_part(part, torch.bfloat16, w, rows, brings, [0] * case["batch"],
                         forward=lambda ctx: part.forward(ctx, rows))


def prepare(case, seed):
    with torch.no_grad():
        return {"chat": _prepare_chat, "layer": _prepare_layer, "mixer": _prepare_mixer, "experts": _prepare_experts}[case["kind"]](case, seed)


def run(state):
    return _run_chat(state) if "engine" in state else _run_part(state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _seen(brings, holds, window=None):
    """(query, key) pairs that attention looks at, and keys that it reads."""
    pairs = keys = 0
    for a, b in zip(brings, holds):
        if window is None or a + b <= window:
            pairs += a * b + a * (a + 1) // 2
            keys += a + b
        else:
            pairs += sum(min(window, b + i + 1) for i in range(a))
            keys += min(a + b, window + a)
    return pairs, keys


def _layer_work(m, rows, brings, holds, esz):
    D = m["dim"]
    params = m["hidden"] * D * (2 * m["heads"] + 2 * m["kv"]) + 3 * m["hidden"] * m["inter"]
    pairs, keys = _seen(brings, holds)
    return esz * (params + 2 * keys * m["kv"] * D), 2 * rows * params + 4 * pairs * m["heads"] * D


def work(case):
    kind = case["kind"]
    if kind == "chat":
        m, esz = QWEN[case["model"]], 4 if case["dtype"] == "float32" else 2
        g = torch.Generator().manual_seed(0)
        lens = torch.randint(case["low"], case["high"] + 1, (case["batch"],), generator=g).tolist()
        total = [0, 0]
        for step in range(case["steps"] + 1):
            brings = lens if step == 0 else [1] * len(lens)
            holds = [0] * len(lens) if step == 0 else [n + step - 1 for n in lens]
            b, f = _layer_work(m, sum(brings), brings, holds, esz)
            total[0] += case["layers"] * b + esz * m["vocab"] * m["hidden"] + 4 * len(lens) * m["vocab"]
            total[1] += case["layers"] * f + 2 * len(lens) * m["vocab"] * m["hidden"]
        return {"bytes": total[0], "flops": total[1]}
    if kind == "experts":
        m = EXPERTS[case["model"]]
        rows = case["batch"] * case["tokens"]
        used = m["experts"] * (1.0 - (1.0 - m["top"] / m["experts"]) ** rows)
        one, shared = 3 * m["hidden"] * m["inter"], 3 * m["hidden"] * m["shared"]
        return {"bytes": 2 * (used * one + shared + m["experts"] * m["hidden"] + 2 * rows * m["hidden"]),
                "flops": 2 * rows * (m["top"] * one + shared + m["experts"] * m["hidden"])}
    brings, holds = _lengths(case)
    rows = sum(brings)
    if kind == "layer":
        m = QWEN[case["model"]]
        b, f = _layer_work(m, rows, brings, holds, 4 if case["dtype"] == "float32" else 2)
        return {"bytes": b + 3 * 2 * rows * m["hidden"], "flops": f}
    m = MIXERS[case["model"]]
    C, params, pairs, keys, state, scan = m["hidden"], 0, 0, 0, 0, 0
    if "heads" in m:
        params += C * 128 * (2 * m["heads"] + 2 * m["kv"])
        pairs, keys = _seen(brings, holds, m["window"])
    if "d_heads" in m:
        N, P = m.get("state", m["d_dim"]), m.get("vdim", m["d_dim"])
        inner = m["d_heads"] * m["d_dim"]
        params += {"delta": 6 * C * inner, "timemix": 5 * C * inner, "ssm": C * (3 * inner + 2 * m.get("groups", 0) * N)}.get(
            m["kind"], 2 * C * inner + 3 * C * m["d_heads"] * P)
        state = 4 * m["d_heads"] * N * P * case["batch"]
        scan = (8 if m["kind"] == "delta" else 6) * rows * m["d_heads"] * N * P
    return {"bytes": 2 * params + 4 * keys * m.get("kv", 0) * 128 + 2 * state + 4 * rows * C,
            "flops": 2 * rows * params + 4 * pairs * m.get("heads", 0) * 128 + scan}


TOLERANCE = {"chat": 4e-2, "layer": 2e-2, "delta": 2e-2, "timemix": 2e-2, "ssm": 2e-2, "gla": 2e-2, "mlstm": 2e-2, "window": 2e-2,
             "experts": 2e-2}


def tolerance(case):
    """Of a bfloat16 path: a few roundings in a row, which another order of the sums moves by a step each. Of the 32-bit
    path: sums of some thousand terms."""
    if case.get("dtype") == "float32":
        return {"rel": 2e-5}
    return {"rel": TOLERANCE[MIXERS[case["model"]]["kind"] if case["kind"] == "mixer" else case["kind"]]}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, first, base):
    """x [T, heads, D], positions from ``first`` on; element i turns with element i + D/2."""
    half = x.shape[-1] // 2
    freq = base ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a = (first + torch.arange(x.shape[0], dtype=torch.float64, device=x.device))[:, None, None] * freq
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _attend(q, k, v, first, scale, window=None, sink=None, slopes=None, softcap=0.0):
    """q [T, H, D] at positions from ``first`` on over k, v [first + T, G, D]."""
    T, H, D = q.shape
    G = k.shape[1]
    out = torch.empty_like(q)
    for t in range(0, T, 512):
        n = min(512, T - t)
        low = 0 if window is None else max(0, first + t - window + 1)
        kk, vv = k[low:first + t + n], v[low:first + t + n]
        s = torch.einsum("tgrd,kgd->grtk", q[t:t + n].view(n, G, H // G, D), kk) * scale
        gap = (first + t + torch.arange(n, device=q.device))[:, None] - (low + torch.arange(kk.shape[0], device=q.device))
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if slopes is not None:
            s = s - slopes.view(G, H // G, 1, 1) * gap
        s = s.masked_fill((gap < 0) | (gap >= (window or 1 << 40)), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.view(G, H // G, 1, 1).expand(-1, -1, n, 1)], -1)
        p = s.softmax(-1)
        out[t:t + n] = torch.einsum("grtk,kgd->tgrd", p[..., :kk.shape[0]], vv).reshape(n, H, D)
    return out


def _pieces(brings):
    at = 0
    for n in brings:
        yield slice(at, at + n)
        at += n


def _exact_layer(x, w, m, context, brings, holds):
    """(x after the attention, the feed-forward's output) of rows in 64 bits; ``context`` is added to."""
    T, D = x.shape[0], m["dim"]
    h = _rms(x, 1e-6) * w["input_layernorm"].double()
    q, k, v = (h @ w[f"self_attn.{n}_proj"].double().T for n in "qkv")
    q = _rms(q.view(T, m["heads"], D), 1e-6) * w["self_attn.q_norm"].double()
    k = _rms(k.view(T, m["kv"], D), 1e-6) * w["self_attn.k_norm"].double()
    v = v.view(T, m["kv"], D)
    o = torch.empty_like(q)
    for i, rows in enumerate(_pieces(brings)):
        ks = torch.cat([context[i][0].double(), _rotate(k[rows], holds[i], m["theta"])])
        vs = torch.cat([context[i][1].double(), v[rows]])
        o[rows] = _attend(_rotate(q[rows], holds[i], m["theta"]), ks, vs, holds[i], D ** -0.5)
        context[i] = (ks, vs)
    x = x + o.reshape(T, -1) @ w["self_attn.o_proj"].double().T
    h = _rms(x, 1e-6) * w["post_attention_layernorm"].double()
    return x, (F.silu(h @ w["mlp.gate_proj"].double().T) * (h @ w["mlp.up_proj"].double().T)) @ w["mlp.down_proj"].double().T


def _exact_chat(case, seed):
    """All tokens of a sequence at once: each row sees its own past only."""
    m = QWEN[case["model"]]
    w, prompts, given = _chat_inputs(case, seed)
    table = w["model.embed_tokens.weight"]
    brings = [len(p) + case["steps"] for p in prompts]
    ids = [t for i, p in enumerate(prompts) for t in p + [row[i] for row in given]]
    x = table[torch.tensor(ids, device=DEVICE)].double()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        mine = {k[len(p):-7]: v for k, v in w.items() if k.startswith(p)}
        empty = [(x.new_zeros(0, m["kv"], m["dim"]),) * 2 for _ in brings]
        x, branch = _exact_layer(x, mine, m, empty, brings, [0] * len(brings))
        x = x + branch
    x = _rms(x, 1e-6) * w["model.norm.weight"].double()
    last = torch.tensor([s.start + len(p) - 1 for s, p in zip(_pieces(brings), prompts)], device=DEVICE)
    out = []
    for t in range(case["steps"] + 1):
        rows = x[last + t]
        out.append(torch.cat([rows @ part.double().T for part in table.split(16384)], -1))
    return out


def _decays(h, w, p=""):
    return torch.tanh(h @ w[p + "w1"].double().T) @ w[p + "w2"].double().T + w[p + "w0"].double()


def _exact_delta(h, w, m, S):
    T, H, N = h.shape[0], m["d_heads"], m["d_dim"]
    r, k, v = ((h @ w["right." + n].double().T).view(T, H, N) for n in "rkv")
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(_decays(h, w, "right."))).view(T, H, N, 1)
    rate = torch.sigmoid(h @ w["right.a"].double().T + w["right.a.b"].double()).view(T, H, N)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au, out = (rate * u).unsqueeze(-1), torch.empty_like(r)
    for t in range(T):
        S = decay[t] * S - au[t] * (u[t].unsqueeze(1) @ S) + k[t].unsqueeze(-1) * v[t].unsqueeze(1)
        out[t] = (r[t].unsqueeze(1) @ S).squeeze(1)
    out = _rms(out, 1e-6).view(T, H * N) * w["right.norm"].double() * torch.sigmoid(h @ w["right.g"].double().T)
    return out @ w["right.o"].double().T, S


def _exact_timemix(h, w, m, S, before):
    T, H, N = h.shape[0], m["d_heads"], m["d_dim"]
    prev = torch.cat([before[None], h[:-1]])
    mix = {s: h + (prev - h) * w["mu." + s].double() for s in "rkvgw"}
    r, k, v = ((mix[n] @ w[n].double().T).view(T, H, N) for n in "rkv")
    decay = torch.exp(-torch.exp(_decays(mix["w"], w))).view(T, H, N, 1)
    bonus, out = w["u"].double().unsqueeze(-1), torch.empty_like(r)
    for t in range(T):
        kv = k[t].unsqueeze(-1) * v[t].unsqueeze(1)
        out[t] = (r[t].unsqueeze(1) @ (S + bonus * kv)).squeeze(1)
        S = decay[t] * S + kv
    out = _rms(out, 1e-6).view(T, H * N) * w["norm"].double() * F.silu(mix["g"] @ w["g"].double().T)
    return out @ w["o"].double().T, S, h[-1]


def _exact_ssm(h, w, m, S, tail):
    T, H, P, N, G, taps = h.shape[0], m["d_heads"], m["d_dim"], m["state"], m["groups"], m["taps"]
    z, xbc, dt = (h @ w["in"].double().T).split([H * P, H * P + 2 * G * N, H], -1)
    seq = torch.cat([tail, xbc])
    conv = sum(seq[i:i + T] * w["conv"][:, i].double() for i in range(taps)) + w["conv.b"].double()
    x, B, C = F.silu(conv).split([H * P, G * N, G * N], -1)
    x, B, C = x.view(T, H, P), B.view(T, G, N).repeat_interleave(H // G, 1), C.view(T, G, N).repeat_interleave(H // G, 1)
    dt = F.softplus(dt + w["dt_bias"].double())
    decay, out = torch.exp(-torch.exp(w["A_log"].double()) * dt), torch.empty_like(x)
    for t in range(T):
        S = decay[t].view(H, 1, 1) * S + (dt[t].unsqueeze(-1) * B[t]).unsqueeze(-1) * x[t].unsqueeze(1)
        out[t] = (C[t].unsqueeze(1) @ S).squeeze(1)
    y = (out + w["D"].double()[:, None] * x).reshape(T, H * P) * F.silu(z)
    y = _rms(y.view(T, 4, -1), 1e-6).view(T, H * P) * w["norm"].double()
    return y @ w["o"].double().T, S, seq[T:]


def _exact_memory(h, w, m, S, beside=None):
    T, H, N, P = h.shape[0], m["d_heads"], m["d_dim"], m["vdim"]
    q, k, v = ((h @ w[n].double().T).view(T, H, -1) for n in "qkv")
    q, g, out = q * N ** -0.5, h @ w["g"].double().T, torch.empty_like(v)
    if beside is None:
        decay = torch.exp(F.logsigmoid((h @ w["a1"].double().T) @ w["a2"].double().T + w["a2.b"].double()) / 16.0).view(T, H, N, 1)
        for t in range(T):
            S = decay[t] * S + k[t].unsqueeze(-1) * v[t].unsqueeze(1)
            out[t] = (q[t].unsqueeze(1) @ S).squeeze(1)
        out = (_rms(out, 1e-5) * w["norm"].double()).view(T, H * P) * F.silu(g)
        return out @ w["o"].double().T, S, None
    cap = lambda z: 15.0 * torch.tanh(z / 15.0)
    i, f = cap(h @ w["i"].double().T + w["i.b"].double()), F.logsigmoid(cap(h @ w["f"].double().T + w["f.b"].double()))
    n, top = beside[:, :-1], beside[:, -1]
    for t in range(T):
        new = torch.maximum(f[t] + top, i[t])
        keep, take, top = torch.exp(f[t] + top - new)[:, None], torch.exp(i[t] - new)[:, None], new
        S = keep.unsqueeze(-1) * S + (take * k[t]).unsqueeze(-1) * v[t].unsqueeze(1)
        n = keep * n + take * k[t]
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out[t] = (q[t].unsqueeze(1) @ S).squeeze(1) / den[:, None]
    out = _rms(out, 1e-5).view(T, H * P) * w["norm"].double() * torch.sigmoid(g)
    return out @ w["o"].double().T, S, torch.cat([n, top[:, None]], -1)


def _exact_window(h, w, m, context, first, p=""):
    T, H, G = h.shape[0], m["heads"], m["kv"]
    q, k, v = (h @ w[p + "q"].double().T).view(T, H, 128), (h @ w[p + "k"].double().T).view(T, G, 128), (h @ w[p + "v"].double().T).view(T, G, 128)
    slopes, cap = None, m.get("softcap", 0.0)
    if m["kind"] == "delta":
        q, k, v = _rotate(q, first, 10000.0), _rotate(k, first, 10000.0), _rms(v, 1e-6)
    else:
        q, k = _rms(q, 1e-6), _rms(k, 1e-6)
        if not cap:
            q, k = q * w["q.norm"].double(), k * w["k.norm"].double()
        at = first + torch.arange(T, dtype=torch.float64, device=DEVICE)
        q = q * (1.0 + 0.1 * torch.log(torch.floor((at + 1) / 4096) + 1.0))[:, None, None]
        slopes = 2.0 ** (-8.0 * (torch.arange(H, dtype=torch.float64, device=DEVICE) + 1) / H)
    sink = w[p + "sink"].double() if p + "sink" in w else None
    o = _attend(q, torch.cat([context[0].double(), k]), torch.cat([context[1].double(), v]), first, 128 ** -0.5, m["window"], sink, slopes, cap)
    if cap:
        o = o * torch.sigmoid(h @ w["g"].double().T)[:, :, None]
    return o.reshape(T, -1) @ w[p + "o"].double().T


def _exact_mixer(case, seed):
    m = MIXERS[case["model"]]
    w, rows, context, states, brings, holds = _mixer_inputs(case, seed)
    outs, after = [], []
    for i, piece in enumerate(_pieces(brings)):
        h, s = rows[piece].double(), [t[i].double() for t in states]
        if m["kind"] == "delta":
            o, S = _exact_delta(h, w, m, *s)
            got = (_exact_window(h, w, m, context[i], holds[i], "left.") + o, S)
        elif m["kind"] == "window":
            got = (_exact_window(h, w, m, context[i], holds[i]),)
        else:
            got = {"timemix": _exact_timemix, "ssm": _exact_ssm}.get(m["kind"], _exact_memory)(h, w, m, *s)
        outs.append(got[0])
        after.append([t for t in got[1:] if t is not None])
    kept = [torch.stack(t) for t in zip(*after)]
    return [torch.cat(outs)] + ([None, None] if context is not None else []) + kept


def _exact_experts(case, seed):
    m = EXPERTS[case["model"]]
    w, rows = _experts_inputs(case, seed)
    h = rows.double()

    def expert(x, p):
        g, u = x @ w[p + "gate"].double().T, x @ w[p + "up"].double().T
        if m["clamp"]:
            g, u = g.clamp(max=m["clamp"]), u.clamp(-m["clamp"], m["clamp"])
            return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[p + "down"].double().T
        return (F.silu(g) * u) @ w[p + "down"].double().T

    z = h @ w["router"].double().T
    if m["ways"] == "chosen":
        z = z + w["router.b"].double()
    top, chosen = z.topk(m["top"], -1)
    weight = {"chosen": lambda: top.softmax(-1), "all": lambda: z.softmax(-1).gather(-1, chosen), "input": lambda: torch.sigmoid(top)}[m["ways"]]()
    out = torch.zeros_like(h)
    for e in range(m["experts"]):
        at, j = (chosen == e).nonzero(as_tuple=True)
        if at.numel():
            by = weight[at, j][:, None]
            out[at] += expert(by * h[at], f"e{e}.") if m["ways"] == "input" else by * expert(h[at], f"e{e}.")
    if m["shared"]:
        base = expert(h, "shared.")
        out = out + (base * torch.sigmoid(h @ w["shared.sg"].double().T) if m["gate"] else base)
    return [out]


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "chat":
            return _exact_chat(case, seed)
        if case["kind"] == "mixer":
            return _exact_mixer(case, seed)
        if case["kind"] == "experts":
            return _exact_experts(case, seed)
        m = QWEN[case["model"]]
        w, x, context, brings, holds = _layer_inputs(case, seed)
        return list(_exact_layer(x.double(), w, m, context, brings, holds)) + [None, None]
