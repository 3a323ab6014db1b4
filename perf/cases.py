"""What this engine is timed on: its layers and its decode steps, over the sizes that they serve.

Most cases are single layers as an engine's step runs them: a mixer or a feed-forward of ``distie_b200.parts`` on the
step's rows, and the norm that adds its output to the residual.  Two are whole decode steps through
``ModelRunner.step``, which return logits.  Sizes are those of the 1.5B, 7B and 14B layer shapes that ``bench.py`` uses,
of its hybrid designs at the same widths, and of the tests; lengths are ragged.

``exact`` recomputes a case in 64 bits from the same seed with plain tensor operations.
"""

from __future__ import annotations

import math

import torch

DEVICE = "cuda:0"
PAGE = 16
VOCAB = 32000  # of the decode steps

#: Layer shapes: width, feed-forward, heads, kv heads (heads of 128).
SHAPES = {
    "1.5b": (1536, 8960, 12, 2),
    "7b": (3584, 18944, 28, 4),
    "14b": (5120, 13824, 40, 8),
}


# -- the cases ------------------------------------------------------------------
def listed():
    return [
        # A whole prompt through an attention layer: the ordinary prefill step of the dense decoder.
        {"name": "attention_prompt", "path": "attention", "dtype": "bf16", "shape": "1.5b", "head_dim": 128, "tokens": 2048,
         "requests": 1, "past": 0},
        # Portions of three requests behind long pasts, odd lengths: chunked prefill in a busy batch.
        {"name": "attention_portions", "path": "attention", "dtype": "bf16", "shape": "7b", "head_dim": 128, "tokens": 1733,
         "requests": 3, "past": 7001},
        # The true 32-bit engine on prompts: what parity replays run.
        {"name": "attention_float32", "path": "attention", "dtype": "f32", "shape": "1.5b", "head_dim": 128, "tokens": 777,
         "requests": 2, "past": 0},
        # The dense feed-forward of a step that mixes a few portions.
        {"name": "feed_forward", "path": "mlp", "shape": "1.5b", "tokens": 1000},
        # The delta rule on one long prompt.
        {"name": "delta_prompt", "path": "delta", "shape": "1.5b", "dim": 128, "tokens": 2048, "requests": 1},
        # State-space duality on a ragged batch of portions.
        {"name": "ssd_portions", "path": "ssd", "shape": "1.5b", "dim": 128, "tokens": 1777, "requests": 3},
        # The matrix memory with exponential gates, an odd prompt.
        {"name": "memory_prompt", "path": "memory", "form": "exp_gate", "shape": "1.5b", "dim": 128, "tokens": 1531, "requests": 1},
        # A selective scan over twice the width.
        {"name": "scan_prompt", "path": "scan", "shape": "1.5b", "tokens": 1024, "requests": 1},
        # Attention through a latent on one prompt.
        {"name": "latent_prompt", "path": "latent", "shape": "1.5b", "tokens": 2048, "requests": 1, "past": 0},
        # Routed experts beside a shared one, a portion of odd length.
        {"name": "routed_portion", "path": "routed", "shape": "1.5b", "tokens": 1001},
        # One decode step of the dense decoder at batch 8: the step a server spends its time in.
        {"name": "decode_dense", "path": "decode", "model": "dense", "shape": "1.5b", "layers": 4, "batch": 8, "past": 1024},
        # The smallest call: one token of one request through the hybrid decoder.
        {"name": "decode_hybrid", "path": "decode", "model": "hybrid", "shape": "1.5b", "layers": 2, "batch": 1, "past": 300},
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _draw_once(rng):
    path = rng.choice(["attention", "attention", "float32", "mlp", "delta", "ssd", "memory", "scan", "latent", "routed", "decode", "decode"])
    shape = rng.choice(["1.5b", "1.5b", "7b", "14b"])
    if path in ("delta", "ssd", "memory", "scan", "latent", "routed") and shape == "14b":
        shape = "7b"  # the hybrid designs are measured at these two widths
    if path == "attention":
        return {"path": "attention", "dtype": "bf16", "shape": shape, "head_dim": rng.choice([128, 128, 64]),
                "tokens": _spread(rng, 130, 4096), "requests": rng.choice([1, 1, 2, 5]), "past": rng.choice([0, 0, _spread(rng, 50, 9000)])}
    if path == "float32":
        return {"path": "attention", "dtype": "f32", "shape": "1.5b", "head_dim": rng.choice([128, 64, 32]),
                "tokens": _spread(rng, 70, 1100), "requests": rng.choice([1, 2, 3]), "past": rng.choice([0, _spread(rng, 20, 1000)])}
    if path == "mlp":
        return {"path": "mlp", "shape": shape, "tokens": _spread(rng, 70, 3000)}
    if path in ("delta", "ssd"):
        return {"path": path, "shape": shape, "dim": rng.choice([128, 128, 64, 96]), "tokens": _spread(rng, 130, 4096),
                "requests": rng.choice([1, 1, 2, 4])}
    if path == "memory":
        return {"path": "memory", "form": rng.choice(["exp_gate", "exp_gate", "decay", "retention"]), "shape": shape,
                "dim": rng.choice([128, 128, 64, 96]), "tokens": _spread(rng, 130, 4096), "requests": rng.choice([1, 1, 2, 4])}
    if path == "scan":
        return {"path": "scan", "shape": shape, "tokens": _spread(rng, 130, 3000), "requests": rng.choice([1, 1, 2, 4])}
    if path == "latent":
        return {"path": "latent", "shape": shape, "tokens": _spread(rng, 130, 3000), "requests": rng.choice([1, 1, 2, 4]),
                "past": rng.choice([0, _spread(rng, 50, 4000)])}
    if path == "routed":
        return {"path": "routed", "shape": shape, "tokens": _spread(rng, 130, 3000)}
    model = rng.choice(["dense", "hybrid"])
    return {"path": "decode", "model": model, "shape": rng.choice(["1.5b", "7b"]), "layers": rng.choice([2, 4]) if model == "dense" else 2,
            "batch": _spread(rng, 1, 48), "past": _spread(rng, 40, 3000)}


def draw(rng):
    most = max(_cost(case) for case in listed())
    while True:
        case = _draw_once(rng)
        if _cost(case) <= most and case.get("tokens", 4096) >= 8 * case.get("requests", 1):
            return case


def _cost(case):
    """About the seconds of a pass on a well used machine, to compare cases with."""
    need = work(case)
    return need["bytes"] / 4e12 + need["flops"] / (3e13 if case.get("dtype") == "f32" else 6e14)


def _lengths(case):
    """How the case's tokens are shared out among its requests: uneven, every request at least two."""
    count, total = case.get("requests", 1), case["tokens"]
    weights = [1.0 + 0.7 * ((5 * i + 2) % 4) for i in range(count)]
    lengths = [max(2, int(total * w / sum(weights))) for w in weights]
    lengths[0] += total - sum(lengths)
    return lengths


def _pasts(case):
    return [max(0, case.get("past", 0) - 37 * i) for i in range(case.get("requests", 1))]


# -- inputs from a seed ---------------------------------------------------------
class _Source:
    """Tensors from a seed, rounded to what a checkpoint in 16 bits holds; the same in ``prepare`` and ``exact``."""

    def __init__(self, seed, dtype=torch.bfloat16):
        self.generator = torch.Generator(device=DEVICE).manual_seed(int(seed) * 7919 + 11)
        self.dtype = dtype

    def normal(self, *shape, std=1.0, mean=0.0):
        return torch.randn(*shape, generator=self.generator, device=DEVICE) * std + mean

    def uniform(self, low, high, *shape):
        return torch.rand(*shape, generator=self.generator, device=DEVICE) * (high - low) + low

    def typed(self, *shape, std=1.0):
        return self.normal(*shape, std=std).to(self.dtype)

    def matrix(self, rows, columns, gain=1.0):
        return self.typed(rows, columns, std=gain / columns**0.5)

    def norm(self, n):
        return 1.0 + self.normal(n, std=0.1)


def _rates(source, heads):
    """Decays as such layers are trained from: rates of 1 to 16, steps of 0.001 to 0.1 before the input's share."""
    step = torch.exp(source.uniform(math.log(1e-3), math.log(1e-1), heads))
    return torch.log(source.uniform(1.0, 16.0, heads)), step + torch.log(-torch.expm1(-step))


def _sizes(case):
    width, ff, heads, kv = SHAPES[case["shape"]]
    dim = case.get("head_dim", 128)
    if dim != 128:  # the same columns in more, smaller heads
        heads, kv = heads * 128 // dim, kv * 128 // dim
    return width, ff, heads, kv, dim


def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.bfloat16


def _part(case):
    """(registry kind, params) of the case's layer."""
    path = case["path"]
    width, ff, heads, kv, dim = _sizes(case)
    if path == "attention":
        return "gqa_attention", {"num_heads": heads, "num_kv_heads": kv, "head_dim": dim, "qkv_bias": True, "out_bias": False,
                                 "window": None, "position": ("rotary", {"head_dim": dim, "theta": 1e6})}
    if path == "mlp":
        return "swiglu", {"intermediate_size": ff, "names": ("gate", "up", "down")}
    d = case.get("dim", 128)
    if path == "delta":
        return "gated_delta_rule", {"heads": heads, "groups": heads, "key_dim": d, "value_dim": d, "taps": 4, "eps": 1e-5}
    if path == "ssd":
        return "mamba2", {"heads": 2 * width // 128, "value_dim": 128, "state": d, "groups": 2, "norm_groups": 2, "taps": 4, "eps": 1e-5}
    if path == "memory":
        if case["form"] == "exp_gate":
            return "exp_gate_memory", {"heads": heads, "key_dim": d, "value_dim": d, "gate_cap": 15.0, "eps": 1e-6}
        decay = [1.0 - 2.0 ** -(2 + 6 * h / max(1, heads - 1)) for h in range(heads)]
        prm = {"heads": heads, "key_dim": d, "value_dim": d, "decay": decay, "eps": 1e-6}
        if case["form"] == "retention":
            prm.update(activation="none", position=("rotary", {"head_dim": d, "theta": 1e4}), key_scale=d**-0.5, norm="head", gate="silu")
        return "decay_attention", prm
    if path == "scan":
        return "selective_scan", {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "taps": 4}
    if path == "latent":
        return "latent_attention", {"num_heads": heads, "head_dim": 128, "rot_dim": 64, "value_dim": 128, "kv_rank": 512,
                                    "q_rank": width // 2, "scale": 192**-0.5, "eps": 1e-6, "own_latent": True, "sink": True,
                                    "gate": "head_sigmoid", "position": ("rotary", {"head_dim": 64, "theta": 1e6})}
    return "routed_swiglu", {"experts": 16, "top": 3, "intermediate_size": ff // 4, "shared_size": ff // 4}


def _tensors(case, source):
    """The layer's checkpoint tensors by name."""
    kind, prm = _part(case)
    width = _sizes(case)[0]
    w = {}
    if kind == "gqa_attention":
        q, k = prm["num_heads"] * prm["head_dim"], prm["num_kv_heads"] * prm["head_dim"]
        for name, rows in (("q", q), ("k", k), ("v", k)):
            w[f"{name}_proj.weight"] = source.matrix(rows, width, 1.5)
            w[f"{name}_proj.bias"] = source.normal(rows, std=0.3)
        w["o_proj.weight"] = source.matrix(width, q)
    elif kind == "swiglu":
        ff = prm["intermediate_size"]
        w = {"gate": source.matrix(ff, width, 1.5), "up": source.matrix(ff, width, 1.5), "down": source.matrix(width, ff)}
    elif kind == "gated_delta_rule":
        n, heads = prm["heads"] * prm["key_dim"], prm["heads"]
        for name in ("q", "k", "v"):
            w[name], w[name + ".conv"] = source.matrix(n, width, 1.5), source.normal(n, 4, std=0.4)
        w["b"], w["a"] = source.matrix(heads, width), source.matrix(heads, width)
        w["A_log"], w["dt_bias"] = _rates(source, heads)
        w["norm"], w["g"], w["o"] = source.norm(prm["value_dim"]), source.matrix(n, width), source.matrix(width, n)
    elif kind == "mamba2":
        inner, gn, heads = prm["heads"] * prm["value_dim"], prm["groups"] * prm["state"], prm["heads"]
        w["in"] = source.matrix(2 * inner + 2 * gn + heads, width)
        w["conv"], w["conv.b"] = source.normal(inner + 2 * gn, 4, std=0.4), source.normal(inner + 2 * gn, std=0.1)
        w["A_log"], w["dt_bias"] = _rates(source, heads)
        w["D"], w["norm"], w["o"] = source.norm(heads), source.norm(inner), source.matrix(width, inner)
    elif kind == "exp_gate_memory":
        n, heads = prm["heads"] * prm["key_dim"], prm["heads"]
        for name in ("q", "k", "v", "g"):
            w[name] = source.matrix(n, width)
        w["i"], w["f"] = source.matrix(heads, width, 0.5), source.matrix(heads, width, 0.5)
        w["i.b"], w["f.b"] = source.normal(heads, std=1.0), source.uniform(3.0, 6.0, heads)
        w["norm"], w["o"] = source.norm(n), source.matrix(width, n)
    elif kind == "decay_attention":
        n = prm["heads"] * prm["key_dim"]
        for name in ("q", "k", "v", "g"):
            w[name] = source.matrix(n, width)
        w["o"] = source.matrix(width, n)
        if case["form"] == "decay":
            w["norm"] = source.norm(n)
    elif kind == "selective_scan":
        inner, state, rank = prm["inner"], prm["state"], prm["dt_rank"]
        w["in"], w["conv"], w["conv.b"] = source.matrix(2 * inner, width), source.normal(inner, 4, std=0.4), source.normal(inner, std=0.1)
        w["x"], w["dt"] = source.matrix(rank + 2 * state, inner, 1.5), source.matrix(inner, rank, 0.5)
        w["dt.b"] = _rates(source, inner)[1]
        w["A_log"] = torch.log(torch.arange(1, state + 1, device=DEVICE, dtype=torch.float32)).expand(inner, state).contiguous()
        w["D"], w["o"] = source.norm(inner), source.matrix(width, inner)
    elif kind == "latent_attention":
        heads, dim, rot, rank, q_rank = prm["num_heads"], prm["head_dim"], prm["rot_dim"], prm["kv_rank"], prm["q_rank"]
        w = {"dq": source.matrix(q_rank, width), "dq.norm": source.norm(q_rank), "uq": source.matrix(heads * (dim + rot), q_rank, 1.3),
             "dkv": source.matrix(rank + rot, width), "dkv.norm": source.norm(rank), "uk": source.matrix(heads * dim, rank),
             "uv": source.matrix(heads * prm["value_dim"], rank), "sink": source.normal(heads), "g": source.matrix(heads, width),
             "o": source.matrix(width, heads * prm["value_dim"])}
    else:
        ff = prm["intermediate_size"]
        for name in [f"e{e}" for e in range(prm["experts"])] + ["shared"]:
            w[name + ".gate"], w[name + ".up"] = source.matrix(ff, width, 1.5), source.matrix(ff, width, 1.5)
            w[name + ".down"] = source.matrix(width, ff)
        w["router"] = source.matrix(prm["experts"], width)
    return w


def _states(case, source):
    """What the requests' earlier tokens left: state tensors by name, ``[requests, ...]``."""
    kind, prm = _part(case)
    b = case.get("requests", 1)
    if kind == "gated_delta_rule":
        h, dk, dv = prm["heads"], prm["key_dim"], prm["value_dim"]
        return {"matrix": source.normal(b, h, dv, dk, std=0.2), "conv": source.normal(b, 3, h * (2 * dk + dv))}
    if kind == "mamba2":
        h, n, dv = prm["heads"], prm["state"], prm["value_dim"]
        return {"matrix": source.normal(b, h, dv, n, std=0.2), "conv": source.normal(b, 3, h * dv + 2 * prm["groups"] * n)}
    if kind == "exp_gate_memory":
        h, d = prm["heads"], prm["key_dim"]
        return {"matrix": source.normal(b, h, d + 1, d, std=0.2), "max": source.uniform(0.0, 1.0, b, h)}
    if kind == "decay_attention":
        return {"matrix": source.normal(b, prm["heads"], prm["value_dim"], prm["key_dim"], std=0.2)}
    if kind == "selective_scan":
        return {"channels": source.normal(b, prm["state"], prm["inner"], std=0.2), "conv": source.normal(b, 3, prm["inner"])}
    return {}


def _cached(case, source):
    """Keys and values of the tokens before the step, per request ``[kv heads, past, size]`` (or the latents' rows)."""
    kind, prm = _part(case)
    if kind == "gqa_attention":
        shape = lambda n: (prm["num_kv_heads"], n, prm["head_dim"])  # noqa: E731
        return [(source.typed(*shape(n)), source.typed(*shape(n))) for n in _pasts(case)]
    if kind == "latent_attention":
        return [(source.typed(1, n, prm["kv_rank"] + prm["rot_dim"]), None) for n in _pasts(case)]
    return []


def _table(case):
    """Block tables: every request's pages, scattered over the pool.  (table, pages)"""
    need = [-(-(p + n) // PAGE) for p, n in zip(_pasts(case), _lengths(case))]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(sum(need)))
    table = torch.full((len(need), max(need)), -1, dtype=torch.int32)
    at = 0
    for row, n in enumerate(need):
        table[row, :n] = order[at : at + n].to(torch.int32)
        at += n
    return table, sum(need)


def _paged(rows, table, row, pages):
    """Writes ``rows [kv heads, n, size]`` as positions 0.. of the request in ``row`` of the table into ``pages``."""
    n = rows.shape[1]
    at = torch.arange(n)
    page = table[row][at // PAGE].long().to(pages.device)
    pages[page, :, (at % PAGE).to(pages.device)] = rows.transpose(0, 1).to(pages.dtype)


def _inputs(case, seed):
    source = _Source(seed, _dtype(case))
    width = _sizes(case)[0]
    made = {"tensors": _tensors(case, source), "x": source.typed(case["tokens"], width), "states": _states(case, source),
            "cached": _cached(case, source), "residual": source.normal(case["tokens"], width, std=2.0), "weight": source.norm(width)}
    return made


# -- one layer ------------------------------------------------------------------
class _Layer:
    """A layer's part, the rows of a step and what the requests' earlier tokens left in caches and states."""


def _layer_state(case, seed):
    from distie_b200.config.model_spec import PartSpec
    from distie_b200.engine.batch import BatchEntry, StepStaging, lay_out
    from distie_b200.kernels import KvSlot, make_kernels
    from distie_b200.parts.base import FEED_FORWARDS, MIXERS, NORMS, BuildContext, SeqSlice, build_part
    from distie_b200.weights.loader import open_weights

    made = _inputs(case, seed)
    kind, prm = _part(case)
    prm = dict(prm)
    if "position" in prm:
        prm["position"] = PartSpec(*prm["position"])
    width, dtype = _sizes(case)[0], _dtype(case)
    registry = FEED_FORWARDS if case["path"] in ("mlp", "routed") else MIXERS
    spec = PartSpec(kind, prm, "layer.")
    # Behind a routed feed-forward the norm adds up a weighted sum of slices, as in the designs that have one.
    norm = PartSpec("rmsnorm", {"eps": 1e-6, "exact": kind == "routed_swiglu"}, "next.")
    specs = registry.get(kind).tensor_specs(spec, width) + NORMS.get("rmsnorm").tensor_specs(norm, width)
    kernels = make_kernels(dtype, DEVICE)
    tensors = {"layer." + name: t for name, t in made["tensors"].items()} | {"next.weight": made["weight"]}
    ctx = BuildContext(kernels, width, open_weights(tensors, specs, (), dtype, DEVICE))
    s = _Layer()
    s.part, s.norm = build_part(registry, spec, ctx), build_part(NORMS, norm, ctx)
    s.x, s.residual, s.dtype = made["x"], made["residual"], dtype
    s.out = torch.empty(case["tokens"], width, dtype=dtype, device=DEVICE)
    lengths, pasts = (_lengths(case), _pasts(case)) if "requests" in case else ([case["tokens"]], [0])
    s.layout = lay_out([BatchEntry(i, [0] * n, p) for i, (n, p) in enumerate(zip(lengths, pasts))])
    s.staging = StepStaging(8 * case["tokens"], torch.device(DEVICE))
    s.staging.upload(s.layout)
    s.seqs = s.layout.seqs
    assert all(isinstance(q, SeqSlice) for q in s.seqs)
    s.state = {n: t.clone() for n, t in made["states"].items()} or None
    s.kv = None
    if made["cached"]:
        table, pages = _table(case)
        k0, v0 = made["cached"][0]
        k = torch.zeros(pages, k0.shape[0], PAGE, k0.shape[2], dtype=dtype, device=DEVICE)
        v = torch.zeros_like(k) if v0 is not None else k[..., : prm["kv_rank"]]
        for row, (old_k, old_v) in enumerate(made["cached"]):
            _paged(old_k, table, row, k)
            if old_v is not None:
                _paged(old_v, table, row, v)
        s.kv = KvSlot(k, v, table.to(DEVICE), PAGE, pages)
    return s


@torch.inference_mode()
def _run_layer(s):
    from distie_b200.engine.batch import views
    from distie_b200.parts.base import LayerRun

    step, _ = views(s.staging.device_buffer, s.layout)  # a step's tensors, as the engine makes them for its layers
    delta = s.part.forward(s.x, LayerRun(step=step, seqs=s.seqs, kv=s.kv, state=s.state))
    s.norm.apply(delta, s.residual, s.out)
    outputs = {"out": s.out, "residual": s.residual}
    if s.kv is not None:
        outputs["keys"] = s.kv.k
        if s.kv.v.data_ptr() != s.kv.k.data_ptr():
            outputs["values"] = s.kv.v
    if s.state is not None:
        outputs |= {"state " + name: t for name, t in s.state.items()}
    return outputs


# -- a decode step --------------------------------------------------------------
def _decode_config(case):
    width, ff, heads, kv = SHAPES[case["shape"]]
    if case["model"] == "dense":
        return {"architectures": ["Qwen2ForCausalLM"], "num_hidden_layers": case["layers"], "hidden_size": width,
                "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": 128, "intermediate_size": ff, "vocab_size": VOCAB,
                "rope_theta": 1e6, "rms_norm_eps": 1e-6, "tie_word_embeddings": True, "max_position_embeddings": 8192}
    mlp = {"kind": "dense", "ff": ff}
    parallel = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128**-0.5, "mask": {"size": 1024}},
        "right": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "conv": 4}, "left_scale": 0.5, "right_scale": 0.5}}
    mamba = {"type": "mamba2", "mlp": mlp,
             "mixer": {"heads": 2 * width // 128, "vdim": 128, "state": 128, "groups": 2, "norm_groups": 2, "conv": 4}}
    return {"architecture": "Zelasun", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "layers": [parallel, mamba]}


def _decode_inputs(case, seed):
    """(weights by name, token ids, per-layer caches [(k, v)] of [batch, kv, past, 128], states by slot and name)"""
    source = _Source(seed)
    width, ff, heads, kv = SHAPES[case["shape"]]
    b, past = case["batch"], case["past"]
    w, caches, states = {}, [], {}

    def feed_forward(prefix, names):
        for name, (rows, columns) in zip(names, ((ff, width), (ff, width), (width, ff))):
            w[prefix + name] = source.matrix(rows, columns, 1.5)

    def cache():
        caches.append((source.typed(b, kv, past, 128), source.typed(b, kv, past, 128)))

    if case["model"] == "dense":
        w["model.embed_tokens.weight"] = source.typed(VOCAB, width, std=0.05)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            for name, rows in (("q", heads * 128), ("k", kv * 128), ("v", kv * 128)):
                w[f"{p}self_attn.{name}_proj.weight"] = source.matrix(rows, width, 1.5)
                w[f"{p}self_attn.{name}_proj.bias"] = source.normal(rows, std=0.3)
            w[p + "self_attn.o_proj.weight"] = source.matrix(width, heads * 128)
            feed_forward(p + "mlp.", ("gate_proj.weight", "up_proj.weight", "down_proj.weight"))
            w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = source.norm(width), source.norm(width)
            cache()
        w["model.norm.weight"] = source.norm(width)
    else:
        w["embed"] = source.typed(VOCAB, width, std=0.05)
        for i in range(2):
            w[f"l{i}.norm1"], w[f"l{i}.norm1.b"] = source.norm(width), source.normal(width, std=0.1)
            feed_forward(f"l{i}.mlp.", ("gate", "up", "down"))
        p = "l0.mix.left."
        for name, rows in (("q", heads * 128), ("k", kv * 128), ("v", kv * 128), ("g", heads)):
            w[p + name] = source.matrix(rows, width, 1.5)
        w[p + "o"] = source.matrix(width, heads * 128)
        cache()
        for prefix, part, index in (("l0.mix.right.", _hybrid_delta(case), 0), ("l1.mix.", _hybrid_ssd(case), 1)):
            made = _delta_tensors(part, width, source) if index == 0 else _tensors({"path": "ssd", "shape": case["shape"], "dim": 128}, source)
            w |= {prefix + name: t for name, t in made.items()}
            h, dv, dk, channels = part
            states[index] = {"matrix": source.normal(b, h, dv, dk, std=0.2), "conv": source.normal(b, 3, channels)}
        w["final.norm"], w["final.norm.b"] = source.norm(width), source.normal(width, std=0.1)
    ids = torch.randint(0, VOCAB, (b,), generator=source.generator, device=DEVICE)
    return w, ids, caches, states


def _hybrid_delta(case):
    """(heads, value size, key size, convolved channels); the keys of a few groups serve all heads"""
    _, _, heads, kv = SHAPES[case["shape"]]
    return heads, 128, 128, (heads + 2 * kv) * 128


def _hybrid_ssd(case):
    width = SHAPES[case["shape"]][0]
    return 2 * width // 128, 128, 128, 2 * width + 512


def _delta_tensors(part, width, source):
    heads, dv, dk, channels = part
    groups = (channels - heads * dv) // (2 * dk)
    w = {}
    for name, rows in (("q", groups * dk), ("k", groups * dk), ("v", heads * dv)):
        w[name], w[name + ".conv"] = source.matrix(rows, width, 1.5), source.normal(rows, 4, std=0.4)
    w["b"], w["a"] = source.matrix(heads, width), source.matrix(heads, width)
    w["A_log"], w["dt_bias"] = _rates(source, heads)
    w["norm"], w["g"], w["o"] = source.norm(dv), source.matrix(heads * dv, width), source.matrix(width, heads * dv)
    return w


class _Decode:
    """An engine behind its requests' prompts, and the tokens of the next step."""


def _decode_state(case, seed):
    from distie_b200.config import EngineConfig, architecture_of
    from distie_b200.engine.batch import BatchEntry
    from distie_b200.engine.engine import Engine
    from distie_b200.kernels import make_kernels

    weights, ids, caches, states = _decode_inputs(case, seed)
    raw = _decode_config(case)
    arch = architecture_of(raw)
    b, past = case["batch"], case["past"]
    pages = b * -(-(past + 1) // PAGE)
    config = EngineConfig(num_blocks=pages, page_size=PAGE, max_seqs=b, token_budget=256, max_model_len=4096,
                          dtype="bfloat16", decode_graphs=True, device=DEVICE)
    s = _Decode()
    s.engine = Engine.assemble(arch, arch.config_cls.from_dict(raw), weights, make_kernels(torch.bfloat16, DEVICE), config)
    cache = s.engine.cache
    seats = [cache.open_seat() for _ in range(b)]
    for seat in seats:
        assert cache.grow(seat, past + 1)
    cache.upload_tables(seats)
    s.entries = [BatchEntry(seat, [int(t)], past, (0,)) for seat, t in zip(seats, ids.tolist())]
    table = cache.kv_slot(0).block_table.cpu()
    for slot, (k, v) in enumerate(caches):
        kv = cache.kv_slot(slot)
        for row, seat in enumerate(seats):
            _paged(k[row], table, seat, kv.k)
            _paged(v[row], table, seat, kv.v)
    s.states, s.rows = [], torch.tensor(seats, device=DEVICE)
    s.engine.runner.step(s.entries)  # a server's steps replay a captured one
    for slot, named in states.items():
        held = cache.state_slot(slot)
        for name, value in named.items():
            own = "right." + name if "right." + name in held else name
            held[own][s.rows] = value
            s.states.append(held[own][: b])
    torch.cuda.synchronize()
    return s


def _run_decode(s):
    logits = s.engine.runner.step(s.entries)
    return {"logits": logits} | {f"state {i}": t for i, t in enumerate(s.states)}


# -- the interface --------------------------------------------------------------
def prepare(case, seed):
    return _decode_state(case, seed) if case["path"] == "decode" else _layer_state(case, seed)


def run(state):
    return _run_decode(state) if isinstance(state, _Decode) else _run_layer(state)


def work(case):
    """Bytes: every weight, input, cached row and state read once, outputs and moved states written once.  Operations: the
    products, and for a matrix state the fewest per token (its decay, the write and the read-out)."""
    if case["path"] == "decode":
        width, ff, heads, kv = SHAPES[case["shape"]]
        b, past = case["batch"], case["past"]
        seen = past if case["model"] == "dense" else past % 1024 + 1
        layer = 3 * width * ff
        attention = (2 * heads + 2 * kv) * 128 * width
        if case["model"] == "dense":
            weights, rows, state = case["layers"] * (layer + attention), case["layers"] * seen, 0
        else:
            h, dv, dk, channels = _hybrid_ssd(case)
            ssd = (2 * h * dv + 512 + h + h * dv) * width
            delta = ((3 * heads + 2 * kv) * 128 + 2 * heads) * width
            weights, rows, state = 2 * layer + attention + heads * width + ssd + delta, seen, (h + heads) * dv * dk
        weights += VOCAB * width
        kv_numbers = 2 * kv * 128 * rows * b
        return {"bytes": 2.0 * (weights + kv_numbers) + 8.0 * state * b + 4.0 * VOCAB * b,
                "flops": 2.0 * weights * b + 2.0 * kv_numbers * heads / kv + 6.0 * state * b}
    kind, prm = _part(case)
    width, tokens = _sizes(case)[0], case["tokens"]
    element = 4 if case.get("dtype") == "f32" else 2
    lengths, pasts = (_lengths(case), _pasts(case)) if "requests" in case else ([tokens], [0])
    b, pairs = len(lengths), sum(n * p + n * (n + 1) / 2 for n, p in zip(lengths, pasts))
    held = sum(pasts) + tokens
    rows = tokens * width * (2 * element + 8)  # the input, the normed output and the residual, read and written
    if kind == "gqa_attention":
        h, k, d = prm["num_heads"], prm["num_kv_heads"], prm["head_dim"]
        weights = width * d * (2 * h + 2 * k)
        return {"bytes": rows + element * (weights + 2.0 * k * d * held), "flops": 2.0 * weights * tokens + 4.0 * h * d * pairs}
    if kind == "swiglu":
        weights = 3 * width * prm["intermediate_size"]
        return {"bytes": rows + 2.0 * weights, "flops": 2.0 * weights * tokens}
    if kind == "latent_attention":
        h, d, r, v, c, q = (prm[n] for n in ("num_heads", "head_dim", "rot_dim", "value_dim", "kv_rank", "q_rank"))
        weights = width * (q + c + r + h + h * v) + q * h * (d + r)
        up = c * h * (d + v)
        return {"bytes": rows + 2.0 * (weights + up + (c + r) * held),
                "flops": 2.0 * (weights * tokens + up * held) + 2.0 * h * (d + r + v) * pairs}
    if kind == "routed_swiglu":
        ff, experts, top = prm["intermediate_size"], prm["experts"], prm["top"]
        return {"bytes": rows + 2.0 * (3 * width * ff * (experts + 1) + width * experts),
                "flops": 2.0 * tokens * (3 * width * ff * (top + 1) + width * experts)}
    if kind == "gated_delta_rule":
        h, dk, dv = prm["heads"], prm["key_dim"], prm["value_dim"]
        weights, state, per_token = width * h * (2 * dk + 3 * dv + 2), h * dk * dv, 7
    elif kind == "mamba2":
        h, dk, dv = prm["heads"], prm["state"], prm["value_dim"]
        weights, state, per_token = width * (3 * h * dv + 2 * prm["groups"] * dk + h), h * dk * dv, 5
    elif kind == "selective_scan":
        inner, n, rank = prm["inner"], prm["state"], prm["dt_rank"]
        weights, state, per_token = width * 3 * inner + inner * (2 * rank + 2 * n), inner * n, 6
    else:
        h, dk, dv = prm["heads"], prm["key_dim"], prm["value_dim"]
        weights, state, per_token = width * h * (2 * dk + 3 * dv), h * dk * dv, 5
    return {"bytes": rows + 2.0 * weights + 8.0 * state * b, "flops": 2.0 * weights * tokens + per_token * state * tokens}


def tolerance(case):
    if case.get("dtype") == "f32":  # 0.7e-6 to 1.6e-6 off the exact values
        return {"rel": 1e-5}
    if case["path"] == "decode":  # several layers in bfloat16 with logits behind them: 0.005 to 0.013 off the exact ones
        return {"rel": 0.03}
    return {"rel": 0.01}  # one layer: 0.0017 to 0.0026 off the exact values


# -- the same in 64 bits ----------------------------------------------------------
def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x, eps, weight=None):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _rotate(x, positions, theta):
    """x [T, heads, d], the two halves of a head turned by the position's angles."""
    d = x.shape[-1]
    freq = 1.0 / (theta ** (torch.arange(0, d, 2, dtype=torch.float32) / d)).to(DEVICE).double()
    angle = positions.double()[:, None] * freq
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., : d // 2], x[..., d // 2 :]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, past, scale, sink=None):
    """q [T, heads, d] at positions past.., k and v [kv, past + T, d] -> [T, heads, dv]"""
    heads, group = q.shape[1], q.shape[1] // k.shape[0]
    out = torch.empty(q.shape[0], heads, v.shape[-1], dtype=torch.float64, device=DEVICE)
    rows = max(1, int(2e8 // (heads * k.shape[1])))
    for at in range(0, q.shape[0], rows):
        part = q[at : at + rows]
        n = part.shape[0]
        qg = part.view(n, k.shape[0], group, -1)
        score = torch.einsum("tkgd,kjd->kgtj", qg, k) * scale
        last = past + at + torch.arange(n, device=DEVICE)
        score.masked_fill_(torch.arange(k.shape[1], device=DEVICE)[None, :] > last[:, None], -math.inf)
        if sink is not None:
            extra = sink.view(k.shape[0], group, 1, 1).expand(-1, -1, n, 1)
            p = torch.softmax(torch.cat([score, extra], -1), -1)[..., :-1]
        else:
            p = torch.softmax(score, -1)
        out[at : at + rows] = torch.einsum("kgtj,kjd->tkgd", p, v).reshape(n, heads, -1)
    return out


def _convolved(x, held, weight, bias=None):
    """x [T, C] behind the held inputs [taps - 1, C] -> (silu of the convolution, the inputs to hold)"""
    taps = weight.shape[1]
    full = torch.cat([held, x])
    y = sum(full[j : j + x.shape[0]] * weight[:, j] for j in range(taps))
    return _silu(y if bias is None else y + bias), full[full.shape[0] - (taps - 1) :]


def _delta_walk(q, k, v, g, beta, S):
    """q, k [T, h, dk], v [T, h, dv], g, beta [T, h], S [h, dv, dk]"""
    out = []
    for t in range(q.shape[0]):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]))
        S = S + u[:, :, None] * k[t][:, None, :]
        out.append(torch.einsum("hvk,hk->hv", S, q[t]))
    return torch.stack(out), S


def _plain_walk(q, k, v, g, S):
    out = []
    for t in range(q.shape[0]):
        S = S * g[t, :, None, None] + v[t][:, :, None] * k[t][:, None, :]
        out.append(torch.einsum("hvk,hk->hv", S, q[t]))
    return torch.stack(out), S


def _delta_mixer(w, prm, x, state):
    h, groups, dk, dv, eps = prm["heads"], prm["groups"], prm["key_dim"], prm["value_dim"], prm["eps"]
    mixed, held = _convolved(torch.cat([x @ w[n].t() for n in "qkv"], -1), state["conv"], torch.cat([w[n + ".conv"] for n in "qkv"]))
    q, k, v = mixed.split([groups * dk, groups * dk, h * dv], -1)
    unit = lambda y: (y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(h // groups, 1)  # noqa: E731
    q, k = unit(q.view(-1, groups, dk)) * dk**-0.5, unit(k.view(-1, groups, dk))
    g = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].t() + w["dt_bias"]))
    read, S = _delta_walk(q, k, v.view(-1, h, dv), g, torch.sigmoid(x @ w["b"].t()), state["matrix"])
    out = _rms(read, eps, w["norm"]).reshape(-1, h * dv) * _silu(x @ w["g"].t())
    return out @ w["o"].t(), {"matrix": S, "conv": held}


def _ssd_mixer(w, prm, x, state):
    h, n, dv, groups, eps = prm["heads"], prm["state"], prm["value_dim"], prm["groups"], prm["eps"]
    inner, gn = h * dv, groups * n
    z, xbc, dt = (x @ w["in"].t()).split([inner, inner + 2 * gn, h], -1)
    mixed, held = _convolved(xbc, state["conv"], w["conv"], w["conv.b"])
    v, B, C = mixed.split([inner, gn, gn], -1)
    dt = torch.nn.functional.softplus(dt + w["dt_bias"])
    wide = lambda y: y.reshape(-1, groups, n).repeat_interleave(h // groups, 1)  # noqa: E731
    v = v.reshape(-1, h, dv)
    read, S = _plain_walk(wide(C), wide(B), v * dt[:, :, None], torch.exp(-torch.exp(w["A_log"]) * dt), state["matrix"])
    y = (read + w["D"][None, :, None] * v).reshape(-1, inner) * _silu(z)
    y = _rms(y.view(-1, prm["norm_groups"], inner // prm["norm_groups"]), eps).reshape(-1, inner) * w["norm"]
    return y @ w["o"].t(), {"matrix": S, "conv": held}


def _memory_mixer(case, w, prm, x, state):
    h, dk, dv, eps = prm["heads"], prm["key_dim"], prm["value_dim"], prm["eps"]
    q, k, v = ((x @ w[n].t()).view(-1, h, dk) for n in "qkv")
    z = x @ w["g"].t()
    if case["form"] == "exp_gate":
        cap = prm["gate_cap"]
        i = cap * torch.tanh((x @ w["i"].t() + w["i.b"]) / cap)
        f = torch.nn.functional.logsigmoid(cap * torch.tanh((x @ w["f"].t() + w["f.b"]) / cap))
        m, keep, take, floor = state["max"], [], [], []
        for t in range(x.shape[0]):
            ahead = torch.maximum(f[t] + m, i[t])
            keep.append(torch.exp(f[t] + m - ahead))
            take.append(torch.exp(i[t] - ahead))
            floor.append(torch.exp(-ahead))
            m = ahead
        v1 = torch.cat([v, torch.ones_like(v[..., :1])], -1) * torch.stack(take)[:, :, None]
        read, S = _plain_walk(q * dk**-0.5, k, v1, torch.stack(keep), state["matrix"])
        out = read[..., :dv] / (torch.maximum(read[..., dv].abs(), torch.stack(floor)) + 1e-6)[..., None]
        out = _rms(out, eps).reshape(-1, h * dv) * w["norm"] * torch.sigmoid(z)
        return out @ w["o"].t(), {"matrix": S, "max": m}
    g = torch.tensor(prm["decay"], dtype=torch.float32, device=DEVICE).double().expand(x.shape[0], h)
    if case["form"] == "decay":
        read, S = _plain_walk(_silu(q), _silu(k), _silu(v), g, state["matrix"])
        out = _rms(read.reshape(-1, h * dv), eps, w["norm"]) * torch.sigmoid(z)
    else:
        at = torch.arange(x.shape[0], device=DEVICE)
        read, S = _plain_walk(_rotate(q, at, 1e4), _rotate(k, at, 1e4) * prm["key_scale"], v, g, state["matrix"])
        out = _rms(read, eps).reshape(-1, h * dv) * _silu(z)
    return out @ w["o"].t(), {"matrix": S}


def _scan_mixer(w, prm, x, state):
    inner, n, rank = prm["inner"], prm["state"], prm["dt_rank"]
    y, z = (x @ w["in"].t()).split([inner, inner], -1)
    y, held = _convolved(y, state["conv"], w["conv"], w["conv.b"])
    low, B, C = (y @ w["x"].t()).split([rank, n, n], -1)
    dt = torch.nn.functional.softplus(low @ w["dt"].t() + w["dt.b"])
    rate, S, out = -torch.exp(w["A_log"]).t(), state["channels"], []
    for t in range(x.shape[0]):
        S = torch.exp(dt[t] * rate) * S + (dt[t] * y[t]) * B[t][:, None]
        out.append((S * C[t][:, None]).sum(0))
    out = (torch.stack(out) + w["D"] * y) * _silu(z)
    return out @ w["o"].t(), {"channels": S, "conv": held}


def _swiglu(x, gate, up, down):
    return (_silu(x @ gate.t()) * (x @ up.t())) @ down.t()


def _routed(w, prm, x):
    top, ids = torch.sigmoid(x @ w["router"].t()).topk(prm["top"], -1)
    out = _swiglu(x, w["shared.gate"], w["shared.up"], w["shared.down"])
    for e in range(prm["experts"]):
        token, slot = (ids == e).nonzero(as_tuple=True)
        if token.numel():
            out[token] += _swiglu(x[token] * top[token, slot][:, None], w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"])
    return out


def _exact_layer(case, seed):
    made = _inputs(case, seed)
    w = {name: t.double() for name, t in made["tensors"].items()}
    x, states = made["x"].double(), {n: t.double() for n, t in made["states"].items()}
    kind, prm = _part(case)
    ends = {}
    if kind in ("swiglu", "routed_swiglu"):
        delta = _swiglu(x, w["gate"], w["up"], w["down"]) if kind == "swiglu" else _routed(w, prm, x)
    else:
        pieces, moved, at = [], [], 0
        table = pages_k = pages_v = None
        if made["cached"]:
            table, pages = _table(case)
            k0, v0 = made["cached"][0]
            pages_k = torch.zeros(pages, k0.shape[0], PAGE, k0.shape[2], dtype=torch.float64, device=DEVICE)
            pages_v = torch.zeros_like(pages_k) if v0 is not None else None
        for row, (n, past) in enumerate(zip(_lengths(case), _pasts(case))):
            xs, at = x[at : at + n], at + n
            state = {name: t[row] for name, t in states.items()}
            position = torch.arange(past, past + n, device=DEVICE)
            if kind == "gqa_attention":
                h, kv, d = prm["num_heads"], prm["num_kv_heads"], prm["head_dim"]
                q, k, v = ((xs @ w[f"{c}_proj.weight"].t() + w[f"{c}_proj.bias"]).view(n, -1, d) for c in "qkv")
                q, k = _rotate(q, position, 1e6), _rotate(k, position, 1e6)
                keys, values = (torch.cat([made["cached"][row][i].double(), y.transpose(0, 1)], 1) for i, y in ((0, k), (1, v)))
                _paged(keys, table, row, pages_k)
                _paged(values, table, row, pages_v)
                y = _attend(q, keys, values, past, d**-0.5).reshape(n, h * d) @ w["o_proj.weight"].t()
            elif kind == "latent_attention":
                h, d, r, c = prm["num_heads"], prm["head_dim"], prm["rot_dim"], prm["kv_rank"]
                q = (_rms(xs @ w["dq"].t(), prm["eps"], w["dq.norm"]) @ w["uq"].t()).view(n, h, d + r)
                q = torch.cat([q[..., :d], _rotate(q[..., d:], position, 1e6)], -1)
                low = xs @ w["dkv"].t()
                new = torch.cat([_rms(low[:, :c], prm["eps"], w["dkv.norm"]), _rotate(low[:, None, c:], position, 1e6)[:, 0]], -1)
                stored = torch.cat([made["cached"][row][0].double(), new[None]], 1)
                _paged(stored, table, row, pages_k)
                latent, part = stored[0, :, :c], stored[0, :, c:]
                keys = torch.cat([(latent @ w["uk"].t()).view(-1, h, d), part[:, None].expand(-1, h, -1)], -1).transpose(0, 1)
                values = (latent @ w["uv"].t()).view(-1, h, prm["value_dim"]).transpose(0, 1)
                mix = _attend(q, keys, values, past, prm["scale"], w["sink"]) * torch.sigmoid(xs @ w["g"].t())[..., None]
                y = mix.reshape(n, -1) @ w["o"].t()
            elif kind == "gated_delta_rule":
                y, state = _delta_mixer(w, prm, xs, state)
            elif kind == "mamba2":
                y, state = _ssd_mixer(w, prm, xs, state)
            elif kind == "selective_scan":
                y, state = _scan_mixer(w, prm, xs, state)
            else:
                y, state = _memory_mixer(case, w, prm, xs, state)
            pieces.append(y)
            moved.append(state)
        delta = torch.cat(pieces)
        if pages_k is not None:
            ends["keys"] = pages_k
            if pages_v is not None:
                ends["values"] = pages_v
        ends |= {"state " + name: torch.stack([m[name] for m in moved]) for name in states}
    residual = made["residual"].double() + delta
    return {"out": _rms(residual, 1e-6, made["weight"].double()), "residual": residual} | ends


def _exact_decode(case, seed):
    weights, ids, caches, states = _decode_inputs(case, seed)
    w = {name: t.double() for name, t in weights.items()}
    width, _, heads, kv = SHAPES[case["shape"]]
    b, past = case["batch"], case["past"]

    def attention(q, k, v, cache, first):
        out = []
        for row in range(b):
            keys, values = (torch.cat([c[row, :, first:].double(), y[row][:, None]], 1) for c, y in zip(cache, (k, v)))
            out.append(_attend(q[row : row + 1], keys, values, past - first, 128**-0.5))
        return torch.cat(out).reshape(b, heads * 128)

    ends = []
    if case["model"] == "dense":
        table = w["model.embed_tokens.weight"]
        x = table[ids]
        position = torch.full((b,), past, device=DEVICE)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            y = _rms(x, 1e-6, w[p + "input_layernorm.weight"])
            q, k, v = ((y @ w[f"{p}self_attn.{c}_proj.weight"].t() + w[f"{p}self_attn.{c}_proj.bias"]).view(b, -1, 128) for c in "qkv")
            mixed = attention(_rotate(q, position, 1e6), _rotate(k, position, 1e6), v, caches[i], 0)
            x = x + mixed @ w[p + "self_attn.o_proj.weight"].t()
            y = _rms(x, 1e-6, w[p + "post_attention_layernorm.weight"])
            x = x + _swiglu(y, *(w[f"{p}mlp.{c}_proj.weight"] for c in ("gate", "up", "down")))
        x = _rms(x, 1e-6, w["model.norm.weight"])
    else:
        table = w["embed"]
        x = table[ids]
        norm = lambda y, name: torch.nn.functional.layer_norm(y, (width,), w[name], w[name + ".b"], 1e-5)  # noqa: E731
        moved = {0: [], 1: []}
        y = norm(x, "l0.norm1")
        p = "l0.mix.left."
        q, k, v = ((y @ w[p + c].t()).view(b, -1, 128) for c in "qkv")
        mixed = attention(q, k, v, caches[0], past // 1024 * 1024)
        mixed = (mixed.view(b, heads, 128) * torch.sigmoid(y @ w[p + "g"].t())[..., None]).reshape(b, -1) @ w[p + "o"].t()
        prm = {"heads": heads, "groups": kv, "key_dim": 128, "value_dim": 128, "eps": 1e-5}
        own = {n[len("l0.mix.right.") :]: t for n, t in w.items() if n.startswith("l0.mix.right.")}
        delta = []
        for row in range(b):
            out, state = _delta_mixer(own, prm, y[row : row + 1], {n: t[row].double() for n, t in states[0].items()})
            delta.append(out)
            moved[0].append(state)
        x = x + 0.5 * mixed + 0.5 * torch.cat(delta) + _swiglu(y, *(w["l0.mlp." + c] for c in ("gate", "up", "down")))
        y = norm(x, "l1.norm1")
        own = {n[len("l1.mix.") :]: t for n, t in w.items() if n.startswith("l1.mix.")}
        prm, ssd = _part({"path": "ssd", "shape": case["shape"], "dim": 128})[1], []
        for row in range(b):
            out, state = _ssd_mixer(own, prm, y[row : row + 1], {n: t[row].double() for n, t in states[1].items()})
            ssd.append(out)
            moved[1].append(state)
        x = x + torch.cat(ssd) + _swiglu(y, *(w["l1.mlp." + c] for c in ("gate", "up", "down")))
        x = norm(x, "final.norm")
        ends = [torch.stack([m[name] for m in moved[i]]) for i in (0, 1) for name in ("matrix", "conv")]
    return {"logits": x @ table.t()} | {f"state {i}": t for i, t in enumerate(ends)}


@torch.inference_mode()
def exact(case, seed):
    return _exact_decode(case, seed) if case["path"] == "decode" else _exact_layer(case, seed)
