"""Workloads of the library whose time is followed, and what each must compute.

`listed()` names twelve: a conversation of the dense decoder at batch 1, 8 and 64 through `InferenceSession` (prompts, then
one token at a time), and single layers through the parts a model is assembled from: the dense feed-forward (bfloat16 and
true 32-bit), grouped-query attention over prompts, mixtures of experts over a prompt and in a one-token step, the three
recurrent mixers over prompts, and one-token latent attention over long caches.  Layer sizes are those of the repository's
presets (Mistral 7B v0.1 / v0.3, Mistral NeMo 12B, and the other architectures "at 7B sizes").  `draw()` gives more of the
same ranges.

Weights, token ids and activations are made on the GPU from a seed; `exact()` makes them again and computes the same
results in 64 bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

DEV = "cuda:0"
PAGE = 64


# ---------------------------------------------------------------------------------------
# the cases


def listed():
    return [
        # one person waiting for an answer: a prompt of a few tokens (the reference measures its time to first token with
        # six), then one token at a time; launches and weights are all there is
        {"name": "turn_b1", "kind": "turn", "hidden": 4096, "vocab": 32000, "batch": 1, "prompt": 6, "steps": 24, "window": 4096},
        # the benchmark's batch and context: eight prompts of about 2,048 tokens, then one token each
        {"name": "turn_b8", "kind": "turn", "hidden": 4096, "vocab": 32000, "batch": 8, "prompt": 2048, "steps": 48, "window": 4096},
        # a full server: 64 shorter conversations at once
        {"name": "turn_b64", "kind": "turn", "hidden": 4096, "vocab": 32768, "batch": 64, "prompt": 256, "steps": 48, "window": 0},
        # the dense feed-forward of a 7B layer over one prompt of 2,048 tokens
        {"name": "mlp_prompt", "kind": "mlp", "dtype": "bfloat16", "tokens": 2048, "hidden": 4096, "inter": 14336},
        # the same layer in a run that asks for true 32-bit arithmetic, over a prompt of an odd length
        {"name": "mlp_f32", "kind": "mlp", "dtype": "float32", "tokens": 333, "hidden": 4096, "inter": 14336},
        # grouped-query attention of a 7B layer over one prompt of 2,048 tokens (projections, rotation, cache write included)
        {"name": "attention_prompt", "kind": "attention", "tokens": 2048, "batch": 1, "hidden": 4096, "window": 4096},
        # mixture of experts (two of sixteen and a shared one, 7B sizes) over a prompt of 2,048 tokens
        {"name": "moe_prompt", "kind": "moe", "router": "softmax", "tokens": 2048, "hidden": 4096},
        # mixture of experts (four of sixteen, grouped sigmoid router, 7B sizes) in a one-token step of 32 conversations
        {"name": "moe_step", "kind": "moe", "router": "sigmoid", "tokens": 32, "hidden": 4096},
        # the gated delta rule over one prompt of 2,048 tokens
        {"name": "delta_prompt", "kind": "delta", "tokens": 2048, "batch": 1, "kv_heads": 8},
        # the recurrence with token shift and a decay per key channel, over one prompt of 2,048 tokens
        {"name": "wkv_prompt", "kind": "wkv", "tokens": 2048, "batch": 1, "hidden": 4096},
        # the selective scan over four prompts of about 1,024 tokens in one step
        {"name": "scan_prompt", "kind": "scan", "tokens": 4096, "batch": 4, "hidden": 4096},
        # one-token latent attention of 64 conversations with up to 4,096 cached positions each
        {"name": "latent_step", "kind": "latent", "batch": 64, "context": 4096},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["turn", "turn", "mlp", "mlp", "attention", "moe", "moe", "delta", "wkv", "scan", "latent"])
    hidden = rng.choice([4096, 5120])
    if kind == "turn":
        batch = _log(rng, 1, 64)
        return {"kind": kind, "hidden": 4096, "vocab": rng.choice([32000, 32768]), "batch": batch,
                "prompt": _log(rng, 6, min(2048, 16384 // batch)), "steps": rng.randint(8, 48), "window": rng.choice([0, 1024, 4096])}
    if kind == "mlp":
        f32 = rng.random() < 0.3
        return {"kind": kind, "dtype": "float32" if f32 else "bfloat16", "tokens": _log(rng, 1, 400 if f32 else 8192),
                "hidden": 4096 if f32 else hidden, "inter": 14336}
    if kind == "attention":
        batch = rng.choice([1, 1, 2, 3, 5, 8])
        return {"kind": kind, "tokens": max(batch, _log(rng, 64, 8192)), "batch": batch, "hidden": hidden,
                "window": rng.choice([0, 1024, 4096])}
    if kind == "moe":
        return {"kind": kind, "router": rng.choice(["softmax", "sigmoid"]), "tokens": _log(rng, 1, 4096), "hidden": hidden}
    if kind == "delta":
        batch = rng.choice([1, 1, 2, 3, 6])
        return {"kind": kind, "tokens": max(batch, _log(rng, 64, 4096)), "batch": batch, "kv_heads": rng.choice([8, 32])}
    if kind in ("wkv", "scan"):
        batch = rng.choice([1, 1, 2, 3, 6])
        return {"kind": kind, "tokens": max(batch, _log(rng, 64, 4096)), "batch": batch, "hidden": 4096}
    return {"kind": "latent", "batch": _log(rng, 8, 64), "context": _log(rng, 300, 4096)}


# ---------------------------------------------------------------------------------------
# weights and inputs, from a seed alone


class _Draws:
    """Tensors in the order they are asked for; the same order gives the same tensors again."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.g, device=DEV) * std + mean).to(dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, generator=self.g, device=DEV) * (hi - lo) + lo


def _pieces(total, n, seed):
    """`total` tokens cut into `n` prompts of unequal lengths (each at least 1)."""
    if n == 1:
        return [total]
    w = np.random.RandomState(seed % (1 << 31)).uniform(0.6, 1.4, n)
    lens = np.maximum(1, (w / w.sum() * total).astype(int))
    lens[int(np.argmax(lens))] += total - int(lens.sum())
    return [int(x) for x in lens]


def _softplus_inverse(x):
    return torch.log(torch.expm1(x))


def _weights(case, d, dtype):
    """The tensors of a single part, by their local names."""
    kind, W = case["kind"], {}

    def mat(name, rows, cols, std=0.02):
        W[name] = d.normal(rows, cols, std=std, dtype=dtype)

    def vec(name, t):
        W[name] = t.to(dtype)
    if kind == "mlp":
        h, i = case["hidden"], case["inter"]
        mat("gate_proj.weight", i, h), mat("up_proj.weight", i, h), mat("down_proj.weight", h, i)
    elif kind == "attention":
        h = case["hidden"]
        mat("q_proj.weight", 4096, h), mat("k_proj.weight", 1024, h), mat("v_proj.weight", 1024, h), mat("o_proj.weight", h, 4096)
    elif kind == "moe":
        h, m = case["hidden"], _moe_sizes(case)
        mat("router", m["experts"], h)
        for e in range(m["experts"]):
            mat(f"e{e}.gate", m["ff"], h), mat(f"e{e}.up", m["ff"], h), mat(f"e{e}.down", h, m["ff"])
        if m["shared"]:
            mat("shared.gate", m["shared"], h), mat("shared.up", m["shared"], h), mat("shared.down", h, m["shared"])
        vec("router.b" if m["part"] == "moe" else "correction", d.normal(m["experts"], std=0.02))
    elif kind == "delta":
        G, H, D = case["kv_heads"], 32, 128
        mat("q", G * D, 4096), mat("k", G * D, 4096), mat("v", H * D, 4096), mat("g", H * D, 4096), mat("o", 4096, H * D)
        mat("b", H, 4096), mat("a", H, 4096)
        for n, c in (("q", G * D), ("k", G * D), ("v", H * D)):
            mat(n + ".conv", c, 4, std=0.5)
        vec("A_log", torch.log(d.uniform(1.0, 16.0, H)))
        vec("dt_bias", _softplus_inverse(torch.exp(d.uniform(math.log(1e-3), math.log(1e-1), H))))
        vec("norm", d.normal(D, std=0.02, mean=1.0))
    elif kind == "wkv":
        h, H, D, L = case["hidden"], 64, 64, 64
        for n in "rkvgw":
            vec("mu." + n, d.uniform(0.0, 1.0, h))
        for n in "rkvg":
            mat(n, H * D, h)
        mat("w1", L, h), mat("w2", H * D, L, std=0.1), mat("o", h, H * D)
        vec("w0", d.uniform(-6.0, -1.0, H * D)), vec("u", d.normal(H, D, std=0.5)), vec("norm", d.normal(H * D, std=0.02, mean=1.0))
    elif kind == "scan":
        h, C, N, R = case["hidden"], 8192, 16, 256
        mat("in", 2 * C, h), mat("conv", C, 4, std=0.5), mat("x", R + 2 * N, C), mat("dt", C, R, std=R ** -0.5), mat("o", h, C)
        vec("conv.b", d.normal(C, std=0.02))
        vec("dt.b", _softplus_inverse(torch.exp(d.uniform(math.log(1e-3), math.log(1e-1), C))))
        vec("A_log", torch.log(torch.arange(1, N + 1, device=DEV, dtype=torch.float32)).expand(C, N))
        vec("D", d.normal(C, std=0.02, mean=1.0))
    elif kind == "latent":
        h, H, D, R, rank = 4096, 32, 128, 64, 512
        mat("q", H * (D + R), h), mat("dkv", rank + R, h), mat("uk", H * D, rank, std=0.04), mat("uv", H * D, rank, std=0.04)
        mat("o", h, H * D), mat("g", H, h), vec("dkv.norm", d.normal(rank, std=0.02, mean=1.0))
    return {n: t.contiguous() for n, t in W.items()}


def _moe_sizes(case):
    if case["router"] == "softmax":
        return {"part": "moe", "experts": 16, "top": 2, "ff": 768, "shared": 2048}
    return {"part": "grouped_moe", "experts": 16, "top": 4, "ff": 896, "shared": 0, "groups": 4, "keep": 2, "scale": 2.5}


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _lens(case, seed):
    """Prompt lengths of a part's step (latent steps: cached positions per conversation)."""
    if case["kind"] in ("mlp", "moe"):
        return [case["tokens"]]
    if case["kind"] == "latent":
        w = np.random.RandomState(seed % (1 << 31)).uniform(0.5, 1.0, case["batch"])
        return [max(1, int(x * (case["context"] - 1))) for x in w]
    return _pieces(case["tokens"], case["batch"], seed)


# ---------------------------------------------------------------------------------------
# parts: what a program that assembles layers itself has in hand


def _part(case):
    """(category, kind, parameters) of the part under test."""
    kind = case["kind"]
    if kind == "mlp":
        return "ffn", "swiglu", {"hidden_size": case["hidden"], "intermediate_size": case["inter"]}
    if kind == "moe":
        m = _moe_sizes(case)
        p = {"hidden_size": case["hidden"], "experts": m["experts"], "top": m["top"], "expert_ff": m["ff"]}
        if m["shared"]:
            p["shared_ff"] = m["shared"]
        if m["part"] == "grouped_moe":
            p.update(identity=0, groups=m["groups"], keep=m["keep"], activation="silu", score="sigmoid", group_score="top2_sum",
                     weight_eps=1e-20, route_scale=m["scale"])
        return "ffn", m["part"], p
    if kind == "attention":
        return "mixer", "attention", {"hidden_size": case["hidden"], "heads": 32, "kv_heads": 8, "head_dim": 128,
                                      "window": case["window"] or None, "scale": 128 ** -0.5,
                                      "position": ("rope", {"theta": 10000.0, "rotary_dim": 128, "pairing": "half"})}
    if kind == "delta":
        return "mixer", "gated_delta", {"hidden_size": 4096, "heads": 32, "kv_heads": case["kv_heads"], "dim": 128, "vdim": 128,
                                        "conv": 4, "eps": 1e-5}
    if kind == "wkv":
        return "mixer", "wkv", {"hidden_size": case["hidden"], "heads": 64, "dim": 64, "decay_rank": 64, "eps": 1e-5}
    if kind == "scan":
        return "mixer", "selective_scan", {"hidden_size": case["hidden"], "inner": 8192, "state": 16, "dt_rank": 256, "conv": 4}
    return "mixer", "latent_attention", {"hidden_size": 4096, "heads": 32, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512,
                                         "q_rank": None, "scale": 192 ** -0.5, "sink": False, "gate": "head", "eps": 1e-5,
                                         "position": ("rope", {"theta": 10000.0, "rotary_dim": 64, "pairing": "interleaved"})}


def _context(rt, kind, q_lens, pos0, slots):
    from inference_engine_rust_b200.csrc import bindings as B
    from inference_engine_rust_b200.parts import StepContext
    n = len(q_lens)
    cu = np.concatenate([[0], np.cumsum(q_lens)])
    seqs = np.repeat(np.arange(n), q_lens)
    cu, slot, seq, pos = (torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV) for a in (cu, slots, seqs, pos0))
    view = B.BatchView(cu_q=cu.data_ptr(), slot_ids=slot.data_ptr(), tok_seq=seq.data_ptr(), pos0=pos.data_ptr(), n_seqs=n,
                       n_tokens=int(sum(q_lens)))
    ctx = StepContext(kind=kind, batch=view, n_tokens=int(sum(q_lens)), n_seqs=n, q_lens=list(q_lens), pos0=list(pos0),
                      slots=list(slots), stream=B.stream_ptr(), rt=rt, slot_ids_dev=slot, pos0_dev=pos, cu_q_dev=cu)
    return ctx, seq


def _prepare_part(case, seed):
    from inference_engine_rust_b200.cache import Cache
    from inference_engine_rust_b200.config.specs import PartSpec
    from inference_engine_rust_b200.parts import Runtime, Workspace, part_class
    d, dt, lens = _Draws(seed), _dtype(case), _lens(case, seed)
    rt = Runtime(dtype=dt, device=torch.device(DEV))
    category, kind, params = _part(case)
    if "position" in params:
        params["position"] = PartSpec(*params["position"])
    part = part_class(category, kind)(PartSpec(kind, params), rt)
    part.load(_weights(case, d, dt))
    step = case["kind"] == "latent"
    T, H = (len(lens) if step else sum(lens)), params["hidden_size"]
    s = {"part": part, "rt": rt, "x": d.normal(T, H, dtype=dt), "residual": torch.empty((T, H), dtype=torch.float32, device=DEV)}
    if category == "ffn":
        s["ctx"], s["keep"] = _context(rt, "prompt" if T > 64 else "decode", lens if T > 64 else [1] * T, [0] * (1 if T > 64 else T),
                                       list(range(1 if T > 64 else T)))
        return s
    longest = max(lens) + 1
    pages = sum(-(-(n + 1) // PAGE) for n in lens)
    cache = Cache({0: part.cache_request()}, max_tokens=pages * PAGE, max_seq_len=-(-longest // PAGE) * PAGE, max_sequences=len(lens),
                  dtype=dt, device=DEV)
    slots = [cache.open_sequence() for _ in lens]
    for slot, n in zip(slots, lens):
        cache.reserve(slot, n + 1)
    cache.upload()
    s["cache"], s["view"] = cache, cache.layer_view(0)
    if step:        # the conversations so far, eight at a time
        for a in range(0, len(lens), 8):
            some = lens[a:a + 8]
            hist = d.normal(sum(some), H, dtype=dt)
            ctx, keep = _context(rt, "prompt", some, [0] * len(some), slots[a:a + 8])
            part.forward(hist, torch.zeros((sum(some), H), dtype=torch.float32, device=DEV), ctx, s["view"], True)
        torch.cuda.synchronize()
        rt.workspace = Workspace(rt.device)
        s["ctx"], s["keep"] = _context(rt, "decode", [1] * T, lens, slots)
    else:
        s["ctx"], s["keep"] = _context(rt, "prompt", lens, [0] * len(lens), slots)
    return s


def _run_part(s):
    r = s["residual"].zero_()
    if "view" not in s:
        s["part"].forward(s["x"], r, s["ctx"])
        return [r]
    part, view = s["part"], s["view"]
    recurrent = hasattr(part, "s_floats")
    if recurrent:
        view.state.zero_()          # the slots' earlier conversations are over
    part.forward(s["x"], r, s["ctx"], view, True)
    return [r, view.state[:, :part.s_floats]] if recurrent else [r]


# ---------------------------------------------------------------------------------------
# whole conversations


LAYERS, HEADS, KV_HEADS, HEAD, INTER, EPS, THETA = 2, 32, 8, 128, 14336, 1e-5, 10000.0


def _turn_config(case):
    return {"architectures": ["MistralForCausalLM"], "model_type": "mistral", "hidden_act": "silu", "tie_word_embeddings": False,
            "bos_token_id": 1, "eos_token_id": 2, "num_hidden_layers": LAYERS, "hidden_size": case["hidden"],
            "num_attention_heads": HEADS, "num_key_value_heads": KV_HEADS, "head_dim": HEAD, "intermediate_size": INTER,
            "vocab_size": case["vocab"], "rope_theta": THETA, "sliding_window": case["window"] or None, "rms_norm_eps": EPS,
            "max_position_embeddings": 32768}


class _Tensors:
    """A source of named tensors, where a folder of weights would stand."""

    def __init__(self, tensors):
        self.tensors = tensors

    def names(self):
        return list(self.tensors)

    def describe(self, name):
        return "BF16", tuple(self.tensors[name].shape)

    def get(self, name):
        return self.tensors[name]


def _turn_weights(case, d):
    h, dt, W = case["hidden"], torch.bfloat16, {}
    W["model.embed_tokens.weight"] = d.normal(case["vocab"], h, dtype=dt)
    W["lm_head.weight"] = d.normal(case["vocab"], h, std=0.02, dtype=dt)
    W["model.norm.weight"] = d.normal(h, std=0.02, mean=1.0, dtype=dt)
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        for n, r, c in (("self_attn.q_proj", HEADS * HEAD, h), ("self_attn.k_proj", KV_HEADS * HEAD, h),
                        ("self_attn.v_proj", KV_HEADS * HEAD, h), ("self_attn.o_proj", h, HEADS * HEAD),
                        ("mlp.gate_proj", INTER, h), ("mlp.up_proj", INTER, h), ("mlp.down_proj", h, INTER)):
            W[p + n + ".weight"] = d.normal(r, c, std=0.02, dtype=dt)
        for n in ("input_layernorm", "post_attention_layernorm"):
            W[p + n + ".weight"] = d.normal(h, std=0.02, mean=1.0, dtype=dt)
    return W


def _turn_tokens(case, seed):
    """Prompts, and the token each conversation goes on with at every step (as another model, or a user, dictates)."""
    r = np.random.RandomState(seed % (1 << 31))
    n = case["batch"]
    lens = [case["prompt"]] if n == 1 else [max(1, int(x)) for x in r.uniform(0.8, 1.0, n) * case["prompt"]]
    lens[0] = case["prompt"]
    return [r.randint(0, case["vocab"], k).tolist() for k in lens], [r.randint(0, case["vocab"], n).tolist() for _ in range(case["steps"])]


def _prepare_turn(case, seed):
    from inference_engine_rust_b200 import LoadedModel, Model, config_from_dict, spec_of
    from inference_engine_rust_b200.parts import Runtime
    config = config_from_dict(_turn_config(case))
    model = Model(spec_of(config), Runtime(dtype=torch.bfloat16, device=torch.device(DEV)))
    model.load(_Tensors(_turn_weights(case, _Draws(seed))))
    prompts, forced = _turn_tokens(case, seed)
    room = sum(-(-(len(p) + case["steps"]) // PAGE) * PAGE for p in prompts)
    session = LoadedModel(config, model).session(max_tokens=room, max_sequences=len(prompts),
                                                 max_seq_len=-(-(case["prompt"] + case["steps"]) // PAGE) * PAGE)
    s = {"session": session, "prompts": prompts, "forced": forced}
    for _ in range(2):              # a server answers its first requests while it starts
        _run_turn(s)
    return s


def _run_turn(s):
    session = s["session"]
    out = [session.prefill(s["prompts"])]
    for tokens in s["forced"]:
        out.append(session.decode_tokens(tokens))
    session.reset()
    return out


# ---------------------------------------------------------------------------------------


def prepare(case, seed):
    return _prepare_turn(case, seed) if case["kind"] == "turn" else _prepare_part(case, seed)


def run(state):
    return _run_turn(state) if "session" in state else _run_part(state)


def _seen(n, window):
    """(query, key) pairs of a prompt of n tokens."""
    w = min(n, window) if window else n
    return w * (w + 1) / 2 + (n - w) * w


def work(case):
    """Bytes and operations of one pass: weights once per step, inputs, outputs, caches and states once."""
    kind, e = case["kind"], 4 if case.get("dtype") == "float32" else 2
    if kind == "turn":
        h, prompts = case["hidden"], [len(p) for p in _turn_tokens(case, 0)[0]]
        layer = h * (2 * HEADS + 2 * KV_HEADS) * HEAD + 3 * h * INTER
        head, n, steps, T = case["vocab"] * h, case["batch"], case["steps"], sum(prompts)
        kv = 2 * KV_HEADS * HEAD * 2 * LAYERS
        reach = case["window"] or 1 << 30
        cached = sum(min(p + k + 1, reach) for p in prompts for k in range(steps))
        pairs = sum(_seen(p, case["window"]) for p in prompts) + cached
        return {"bytes": (1 + steps) * (2 * (LAYERS * layer + head) + 4 * n * case["vocab"]) + kv * (T + n * steps + cached),
                "flops": 2 * LAYERS * layer * (T + n * steps) + 2 * head * n * (1 + steps) + 4 * LAYERS * HEADS * HEAD * pairs}
    if kind == "latent":
        lens, (H, D, R, rank) = _lens(case, 0), (32, 128, 64, 512)
        w = 4096 * (H * (D + R) + rank + R + H + H * D) + 2 * H * D * rank
        n, cached = len(lens), sum(x + 1 for x in lens)
        return {"bytes": 2 * w + 2 * (rank + R) * cached + n * 4096 * 6,
                "flops": 2 * w * n + 2 * H * (2 * rank + R) * cached}
    T = case["tokens"]
    h = case.get("hidden", 4096)
    if kind == "mlp":
        w = 3 * h * case["inter"]
        return {"bytes": e * w + T * h * (e + 4), "flops": 2 * w * T}
    if kind == "moe":
        m = _moe_sizes(case)
        one = 3 * h * m["ff"]
        touched = min(m["experts"], T * m["top"])
        shared = 3 * h * m["shared"]
        return {"bytes": 2 * (touched * one + shared + m["experts"] * h) + T * h * 6,
                "flops": 2 * T * (m["top"] * one + shared + m["experts"] * h)}
    lens = _lens(case, 0)
    if kind == "attention":
        w = h * (4096 + 2048 + 4096)
        return {"bytes": 2 * w + T * (h * 6 + 2 * 2048), "flops": 2 * w * T + 4 * 4096 * sum(_seen(n, case["window"]) for n in lens)}
    if kind == "delta":
        w = 4096 * (2 * case["kv_heads"] * 128 + 3 * 4096 + 64)
        state = 32 * 128 * 128
        return {"bytes": 2 * w + T * 4096 * 6 + 8 * len(lens) * state, "flops": 2 * w * T + 8 * T * state}
    if kind == "wkv":
        w, state = h * (5 * 4096 + 64) + 4096 * 64, 64 * 64 * 64
        return {"bytes": 2 * w + T * h * 6 + 8 * len(lens) * state, "flops": 2 * w * T + 7 * T * state}
    C, N, R = 8192, 16, 256
    w = 3 * C * h + C * (2 * R + 2 * N)
    return {"bytes": 2 * w + T * h * 6 + 8 * len(lens) * C * N, "flops": 2 * w * T + 6 * T * C * N}


def tolerance(case):
    # about four times what was seen between the present results and the 64-bit ones (mlp 0.0017, moe 0.0023, latent
    # 0.0035, attention 0.0054, recurrent mixers 0.0059, two whole layers and the head up to 0.0088, 32-bit runs 2.8e-6)
    if case["kind"] == "turn":
        return {"rel": 3.5e-2}
    if case.get("dtype") == "float32":
        return {"rel": 1.2e-5}
    return {"rel": {"mlp": 8e-3, "moe": 1e-2, "latent": 1.5e-2}.get(case["kind"], 2.4e-2)}


# ---------------------------------------------------------------------------------------
# the same results in 64 bits


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _mm(x, w):
    """x . w^T, the weight widened a run of rows at a time."""
    return torch.cat([x @ w[i:i + 4096].double().t() for i in range(0, w.shape[0], 4096)], dim=-1)


def _rotate(x, pos, theta, neighbours=False):
    """x [T, heads, d] at positions pos [T], all d numbers turned."""
    d = x.shape[-1]
    ang = pos.double()[:, None] * theta ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float64) / d)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    if neighbours:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _causal(q, k, v, scale, window):
    """One sequence: q [T, H, d], k and v [T, G, d]."""
    T, H, _ = q.shape
    i = torch.arange(T, device=DEV)
    out = torch.empty_like(q)
    for a in range(0, T, 512):
        rows = i[a:a + 512, None]
        hidden = (i[None] > rows) | ((i[None] <= rows - window) if window else False)
        for g in range(k.shape[1]):
            heads = slice(g * (H // k.shape[1]), (g + 1) * (H // k.shape[1]))
            s = torch.einsum("thd,sd->hts", q[a:a + 512, heads], k[:, g]) * scale
            out[a:a + 512, heads] = torch.einsum("hts,sd->thd", torch.softmax(s.masked_fill(hidden, -math.inf), -1), v[:, g])
    return out.reshape(T, -1)


def _gqa(x, q, k, v, o, lens, window):
    T = x.shape[0]
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens])
    qs = _rotate(_mm(x, q).view(T, -1, HEAD), pos, THETA)
    ks = _rotate(_mm(x, k).view(T, -1, HEAD), pos, THETA)
    vs = _mm(x, v).view(T, -1, HEAD)
    outs, a = [], 0
    for n in lens:
        outs.append(_causal(qs[a:a + n], ks[a:a + n], vs[a:a + n], HEAD ** -0.5, window))
        a += n
    return _mm(torch.cat(outs), o)


def _gated(x, gate, up, down):
    out = torch.empty(x.shape, dtype=torch.float64, device=DEV)
    for a in range(0, x.shape[0], 4096):
        b = x[a:a + 4096]
        out[a:a + 4096] = _mm(F.silu(_mm(b, gate)) * _mm(b, up), down)
    return out


def _exact_turn(case, seed):
    W = _turn_weights(case, _Draws(seed))
    prompts, forced = _turn_tokens(case, seed)
    n, steps = case["batch"], case["steps"]
    full = [p + [forced[k][i] for k in range(steps)] for i, p in enumerate(prompts)]
    lens = [len(f) for f in full]
    x = W["model.embed_tokens.weight"][torch.tensor(sum(full, []), device=DEV)].double()
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        xn = _rms(x, EPS) * W[p + "input_layernorm.weight"].double()
        x = x + _gqa(xn, *(W[p + f"self_attn.{m}_proj.weight"] for m in "qkvo"), lens, case["window"])
        xn = _rms(x, EPS) * W[p + "post_attention_layernorm.weight"].double()
        x = x + _gated(xn, *(W[p + f"mlp.{m}_proj.weight"] for m in ("gate", "up", "down")))
    ends = np.cumsum(lens) - steps - 1
    rows = torch.tensor(np.concatenate([ends + k for k in range(steps + 1)]), device=DEV)
    logits = _mm(_rms(x[rows], EPS) * W["model.norm.weight"].double(), W["lm_head.weight"])
    return list(logits.view(steps + 1, n, -1))


def _exact_moe(case, x, W):
    m = _moe_sizes(case)
    z = _mm(x, W["router"])
    if m["part"] == "moe":
        val, idx = torch.topk(z + W["router.b"].double(), m["top"], dim=-1)
        wt = torch.softmax(val, dim=-1)
    else:
        s = torch.sigmoid(z)
        choice = s + W["correction"].double()
        runs = choice.view(-1, m["groups"], m["experts"] // m["groups"])
        kept = torch.topk(torch.topk(runs, 2, dim=-1).values.sum(-1), m["keep"], dim=-1).indices
        mask = torch.zeros(runs.shape[:2], dtype=torch.bool, device=DEV).scatter_(1, kept, True)
        idx = torch.topk(runs.masked_fill(~mask[..., None], -math.inf).flatten(1), m["top"], dim=-1).indices
        wt = torch.gather(s, 1, idx)
        wt = wt / wt.sum(-1, keepdim=True) * m["scale"]
    out = torch.zeros_like(x)
    for e in range(m["experts"]):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        if t.numel():
            out[t] += wt[t, j, None] * _gated(x[t], W[f"e{e}.gate"], W[f"e{e}.up"], W[f"e{e}.down"])
    return out + _gated(x, W["shared.gate"], W["shared.up"], W["shared.down"]) if m["shared"] else out


def _conv(x, taps):
    """Causal convolution per channel of one sequence [T, C], the last tap the current token's."""
    K = taps.shape[1]
    pad = torch.cat([torch.zeros((K - 1, x.shape[1]), dtype=x.dtype, device=DEV), x])
    return sum(pad[j:j + x.shape[0]] * taps[:, j].double() for j in range(K))


def _exact_delta(case, x, W, lens):
    G, H, D = case["kv_heads"], 32, 128
    raw = {n: _mm(x, W[n]) for n in "qkvg"}
    beta = torch.sigmoid(_mm(x, W["b"]))
    decay = torch.exp(-torch.exp(W["A_log"].double()) * F.softplus(_mm(x, W["a"]) + W["dt_bias"].double()))
    outs, states, a = [], [], 0
    for n in lens:
        q, k, v = (F.silu(_conv(raw[m][a:a + n], W[m + ".conv"])).view(n, -1, D) for m in "qkv")
        q = (q / torch.sqrt(q.square().sum(-1, keepdim=True) + 1e-6) * D ** -0.5).repeat_interleave(H // G, dim=1)
        k = (k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
        S = torch.zeros((H, D, D), dtype=torch.float64, device=DEV)
        o = torch.empty((n, H, D), dtype=torch.float64, device=DEV)
        for t in range(n):
            S *= decay[a + t, :, None, None]
            u = beta[a + t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S += k[t][:, :, None] * u[:, None]
            o[t] = torch.einsum("hdv,hd->hv", S, q[t])
        outs.append(o)
        states.append(S.flatten())
        a += n
    o = (_rms(torch.cat(outs), 1e-5) * W["norm"].double()).flatten(1) * F.silu(raw["g"])
    return [_mm(o, W["o"]), torch.stack(states)]


def _exact_wkv(case, x, W, lens):
    H = D = 64
    starts = np.cumsum([0] + lens[:-1])
    prev = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
    prev[torch.tensor(starts, device=DEV)] = 0
    mixed = {m: x + (prev - x) * W["mu." + m].double() for m in "rkvgw"}
    r, k, v = (_mm(mixed[m], W[m]).view(-1, H, D) for m in "rkv")
    decay = torch.exp(-torch.exp(_mm(torch.tanh(_mm(mixed["w"], W["w1"])), W["w2"]) + W["w0"].double())).view(-1, H, D)
    u, o, states = W["u"].double(), torch.empty_like(r), []
    for a, n in zip(starts, lens):
        S = torch.zeros((H, D, D), dtype=torch.float64, device=DEV)
        for t in range(a, a + n):
            kv = k[t][:, :, None] * v[t][:, None]
            o[t] = torch.einsum("hdv,hd->hv", S + u[:, :, None] * kv, r[t])
            S = S * decay[t][:, :, None] + kv
        states.append(S.flatten())
    y = _rms(o, 1e-5).flatten(1) * W["norm"].double() * F.silu(_mm(mixed["g"], W["g"]))
    return [_mm(y, W["o"]), torch.stack(states)]


def _exact_scan(case, x, W, lens):
    C, N, R = 8192, 16, 256
    xz = _mm(x, W["in"])
    A = -torch.exp(W["A_log"].double())
    ys, states, a = [], [], 0
    for n in lens:
        u = F.silu(_conv(xz[a:a + n, :C], W["conv"]) + W["conv.b"].double())
        p = _mm(u, W["x"])
        dt = F.softplus(_mm(p[:, :R], W["dt"]) + W["dt.b"].double())
        S = torch.zeros((C, N), dtype=torch.float64, device=DEV)
        y = torch.empty_like(u)
        for t in range(n):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * p[t, R:R + N]
            y[t] = S @ p[t, R + N:] + W["D"].double() * u[t]
        ys.append(y)
        states.append(S.flatten())
        a += n
    return [_mm(torch.cat(ys) * F.silu(xz[:, C:]), W["o"]), torch.stack(states)]


def _exact_latent(case, x, W, lens, d):
    H, D, R, rank = 32, 128, 64, 512
    n = len(lens)

    def row(h, pos):
        """The cached row [latent | rotated key part] of each token."""
        down = _mm(h, W["dkv"])
        c = _rms(down[:, :rank], 1e-5) * W["dkv.norm"].double()
        return torch.cat([c, _rotate(down[:, None, rank:], pos, 10000.0, neighbours=True)[:, 0]], dim=-1)
    pos = torch.tensor(lens, device=DEV)
    q = _mm(x, W["q"]).view(n, H, D + R)
    uk, uv = W["uk"].double().view(H, D, rank), W["uv"].double().view(H, D, rank)
    q = torch.cat([torch.einsum("bhd,hdr->bhr", q[..., :D], uk), _rotate(q[..., D:], pos, 10000.0, neighbours=True)], dim=-1)
    own, out = row(x, pos), torch.empty((n, H, D), dtype=torch.float64, device=DEV)
    for a in range(0, n, 8):
        some = lens[a:a + 8]
        hist, at = d.normal(sum(some), 4096, dtype=torch.bfloat16).double(), 0
        for j, m in enumerate(some):
            rows = torch.cat([row(hist[at:at + m], torch.arange(m, device=DEV)), own[a + j:a + j + 1]])
            w = torch.softmax(q[a + j] @ rows.t() * (D + R) ** -0.5, dim=-1)
            out[a + j] = torch.einsum("hr,hdr->hd", w @ rows[:, :rank], uv)
            at += m
    gate = torch.sigmoid(_mm(x, W["g"]))
    return [_mm((out * gate[:, :, None]).flatten(1), W["o"])]


def exact(case, seed):
    kind = case["kind"]
    if kind == "turn":
        return _exact_turn(case, seed)
    d, lens = _Draws(seed), _lens(case, seed)
    W = _weights(case, d, _dtype(case))
    T = len(lens) if kind == "latent" else sum(lens)
    x = d.normal(T, case.get("hidden", 4096), dtype=_dtype(case)).double()
    if kind == "mlp":
        return [_gated(x, W["gate_proj.weight"], W["up_proj.weight"], W["down_proj.weight"])]
    if kind == "moe":
        return [_exact_moe(case, x, W)]
    if kind == "attention":
        return [_gqa(x, *(W[f"{m}_proj.weight"] for m in "qkvo"), lens, case["window"])]
    if kind == "latent":
        return _exact_latent(case, x, W, lens, d)
    return {"delta": _exact_delta, "wkv": _exact_wkv, "scan": _exact_scan}[kind](case, x, W, lens)
