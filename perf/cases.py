"""Work that programs built on this engine have it do, as cases that can be timed and checked.

A case is one pass through a public entry point: a decode step of a whole model replayed from its CUDA graph (DecodeGraphs), a whole
pre-norm layer, or one mixer or feed-forward built from its PartSpec (mini_inference_b200.parts), on a batch that the engine's own
builder and cache manager made.  Layer sizes are those of Qwen3-4B and of the "2k" sizes at which the other designs are measured
(mini_inference_b200/cli/microbench.py); weights, inputs and the cache's contents are drawn from the seed.  `exact` states every case
once more in plain torch, in 64 bits.

kind             what it stands for in use
qwen3_step       a decode step of a served Qwen3: batch 1 (an interactive user; latency and launches count) up to 64, ragged contexts
qwen3_layer      a prompt step's layer: one long prompt, several ragged ones, portions of a chunked prefill that see earlier keys,
                 decoded tokens riding along; bfloat16, and float32 (the engine's true float32 path)
attention        softmax attention of the other designs: rotated and normed heads (Kofutar), blocks of positions with a sink
                 (Namesun), distance slopes with values that are the keys (Megovik)
latent           attention over one compressed row per token (Naditar, Kofutar, Megovik)
lightning        matrix state with one constant decay per head (Naditar; Namesun's retention is the same recurrence)
channel_delta    delta rule with a decay per head and key channel (Naditar)
selective_scan   selective state-space scan (Nununex)
experts          routed experts with a shared one (Namesun, Megovik, Nununex)
naditar_step     a decode step of a served design with recurrent states and latent attention
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

PAGE = 16
DEV = "cuda:0"
QWEN3_4B = dict(hidden=2560, heads=32, kv_heads=8, dim=128, inter=9728)
W2K = 2048                       # the width of the other designs' "2k" sizes
EPS = 1e-6
STEP_LAYERS = 4


# ---------------------------------------------------------------- the cases
def _entries(text):
    """"pos0:n,pos0:n,..": per request the tokens it already holds and those that this step feeds."""
    return [tuple(int(v) for v in e.split(":")) for e in text.split(",")]


def listed():
    return [
        # an interactive user's decode step: every kernel is small, launches and fixed costs count
        dict(name="qwen3_step_b1", kind="qwen3_step", batch=1, context=4096, vocab=32768, dtype="bfloat16"),
        # eight users at contexts around 4,096 (the engine's headline decode workload)
        dict(name="qwen3_step_b8", kind="qwen3_step", batch=8, context=4096, vocab=32768, dtype="bfloat16"),
        # a full token budget of prompt work: the end of a chunked prompt, whole shorter prompts, decoded tokens riding along
        dict(name="qwen3_layer_mixed", kind="qwen3_layer", entries="2048:1999,0:1517,0:571,4000:1,1203:1", dtype="bfloat16"),
        # the true float32 path, as checks and replays use it
        dict(name="qwen3_layer_f32", kind="qwen3_layer", entries="0:500,77:1", dtype="float32"),
        dict(name="attention_rotated", kind="attention", form="rotated", entries="0:2048", dtype="bfloat16"),
        dict(name="attention_blocks_mixed", kind="attention", form="blocks", entries="0:1030,700:771,0:37,2000:1,3001:1", dtype="bfloat16"),
        dict(name="latent_prompts", kind="latent", entries="0:1500,512:548", dtype="bfloat16"),
        dict(name="lightning_2048", kind="lightning", entries="0:2048", dtype="bfloat16"),
        dict(name="channel_delta_mixed", kind="channel_delta", entries="0:1300,640:517,0:231", dtype="bfloat16"),
        dict(name="selective_scan_2048", kind="selective_scan", entries="0:2048", dtype="bfloat16"),
        dict(name="experts_2048", kind="experts", entries="0:2048", dtype="bfloat16"),
        # 64 users of a design with matrix states: 4 layers (two delta, one latent, one lightning), each with its feed-forward
        dict(name="naditar_step_b64", kind="naditar_step", batch=64, context=2048, vocab=16384, dtype="bfloat16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_entries(rng, total, requests=4):
    """A step of about `total` tokens: one to `requests` prompts or portions (some behind earlier tokens), a few decoded tokens."""
    n = rng.randint(1, requests)
    cuts = sorted(rng.randint(0, total) for _ in range(n - 1))
    lens = [max(2, b - a) for a, b in zip([0] + cuts, cuts + [total])]
    out = [f"{rng.choice([0, 0, rng.randint(1, 3000)])}:{m}" for m in lens]
    out += [f"{_log_int(rng, 16, 4000)}:1" for _ in range(rng.choice([0, 0, 1, 5]))]
    return ",".join(out)


def draw(rng):
    kind = rng.choice(["qwen3_step", "qwen3_layer", "qwen3_layer", "attention", "attention", "latent", "lightning", "channel_delta",
                       "selective_scan", "experts", "naditar_step"])
    if kind == "qwen3_step":
        batch = _log_int(rng, 1, 24)
        return dict(kind=kind, batch=batch, context=_log_int(rng, 64, 4096), vocab=32768, dtype="bfloat16")
    if kind == "naditar_step":
        return dict(kind=kind, batch=_log_int(rng, 1, 64), context=_log_int(rng, 64, 2048), vocab=16384, dtype="bfloat16")
    dtype = "float32" if rng.random() < 0.2 and kind in ("qwen3_layer", "attention", "lightning", "channel_delta") else "bfloat16"
    total = _log_int(rng, 48, 3000 if dtype == "bfloat16" else 400)
    case = dict(kind=kind, entries=_draw_entries(rng, total), dtype=dtype)
    if kind == "attention":
        case["form"] = rng.choice(["rotated", "blocks", "slopes"])
    return case


# ---------------------------------------------------------------- inputs, from the seed alone
def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


class _Draw:
    """Seeded values on the GPU in the case's dtype, in the order they are asked for."""

    def __init__(self, seed, dtype):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)
        self.dtype = dtype

    def normal(self, *shape, std=1.0, dtype=None):
        return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0.0, std, generator=self.g).to(dtype or self.dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=None):
        return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(lo, hi, generator=self.g).to(dtype or self.dtype)

    def ints(self, n, hi):
        return torch.randint(0, hi, (n,), generator=self.g, device=DEV)


def _pages(case, entries):
    """Per request its pages, as a cache that nobody used yet hands them out: page 0 is the null page, then one after the other."""
    out, nxt = [], 1
    for pos0, n in entries:
        k = -(-(pos0 + n) // PAGE)
        out.append(list(range(nxt, nxt + k)))
        nxt += k
    return out, nxt - 1


def _mixer_weights(kind, d, width=W2K, form=None):
    """Tensors of a mixer or feed-forward by the names its part declares.  Matrices as a trained model's initialisation has them."""
    m = lambda n, k, std=0.02: d.normal(n, k, std=std)          # noqa: E731
    if kind == "lightning":
        H, D, V = 16, 128, 128
        w = {"q": m(H * D, width), "k": m(H * D, width), "v": m(H * V, width), "g": m(H * V, width), "o": m(width, H * V),
             "norm": d.uniform(H * V, lo=0.5, hi=1.5)}
    elif kind == "channel_delta":
        H, KV, D, V, taps, rank = 16, 8, 128, 128, 4, 64
        w = {"q": m(KV * D, width), "k": m(KV * D, width), "v": m(H * V, width), "b": m(H, width),
             "a1": m(rank, width), "a2": m(H * D, rank, 0.1), "g1": m(rank, width), "g2": m(H * V, rank, 0.1), "o": m(width, H * V),
             "norm": d.uniform(V, lo=0.5, hi=1.5), "A_log": d.uniform(H, lo=0.0, hi=math.log(16.0))}
        for n, c in (("q", KV * D), ("k", KV * D), ("v", H * V)):
            w[n + ".conv"] = d.uniform(c, taps, lo=-0.5, hi=0.5)
        dt = torch.exp(d.uniform(H * D, lo=math.log(1e-3), hi=math.log(0.1), dtype=torch.float32))
        w["dt_bias"] = (dt + torch.log(-torch.expm1(-dt))).to(d.dtype)               # softplus(dt_bias) = dt
    elif kind == "selective_scan":
        I, N, R, taps = 4096, 16, 128, 4
        dt = torch.exp(d.uniform(I, lo=math.log(1e-3), hi=math.log(0.1), dtype=torch.float32))
        w = {"in": m(2 * I, width), "conv": d.uniform(I, taps, lo=-0.5, hi=0.5), "conv.b": d.uniform(I, lo=-0.5, hi=0.5), "x": m(R + 2 * N, I),
             "dt": d.uniform(I, R, lo=-R ** -0.5, hi=R ** -0.5), "dt.b": (dt + torch.log(-torch.expm1(-dt))).to(d.dtype),
             "A_log": torch.log(torch.arange(1, N + 1, device=DEV, dtype=torch.float32)).repeat(I, 1).to(d.dtype),
             "D": d.uniform(I, lo=0.5, hi=1.5), "o": m(width, I)}
    elif kind == "latent":
        H, D, R, V, C = 16, 64, 32, 64, 96
        w = {"q": m(H * (D + R), width), "dkv": m(C + R, width), "dkv.norm": d.uniform(C, lo=0.5, hi=1.5), "uk": m(H * D, C, C ** -0.5),
             "uv": m(H * V, C, C ** -0.5), "g": m(H, width), "o": m(width, H * V)}
    elif kind == "attention":
        H, KV, D = 16, 8, 128
        w = {"q": m(H * D, width), "k": m(KV * D, width), "o": m(width, H * D)}
        if form != "slopes":
            w["v"] = m(KV * D, width)
        if form != "blocks":
            w["q.norm"], w["k.norm"] = d.uniform(D, lo=0.5, hi=1.5), d.uniform(D, lo=0.5, hi=1.5)
    elif kind == "experts":
        E, Fe, S = 32, 1024, 2048
        w = {"router": m(E, width), "correction": d.normal(E, std=0.01)}
        for e in range(E):
            w.update({f"e{e}.gate": m(Fe, width), f"e{e}.up": m(Fe, width), f"e{e}.down": m(width, Fe)})
        w.update({"shared.gate": m(S, width), "shared.up": m(S, width), "shared.down": m(width, S)})
    return w


LIGHT_DECAY = tuple(1.0 - 2.0 ** -(2 + 6 * h / 16) for h in range(16))
DELTA_C = 2 * 8 * 128 + 16 * 128                  # channels that pass the delta rule's convolution
STATE_FLOATS = {"lightning": 16 * 128 * 128, "channel_delta": 16 * 128 * 128 + 3 * DELTA_C, "selective_scan": 4096 * 16 + 3 * 4096}


def _state_rows(kind, d, entries):
    """The fixed-size states of the requests [n, floats]: zero for a request that starts, else what earlier tokens may have left."""
    n = STATE_FLOATS[kind]
    matrix = {"lightning": n, "channel_delta": 16 * 128 * 128, "selective_scan": 4096 * 16}[kind]
    rows = torch.cat([d.normal(len(entries), matrix, std=0.3, dtype=torch.float32),
                      d.normal(len(entries), n - matrix, std=0.9, dtype=torch.float32).bfloat16().float()], dim=1)
    live = torch.tensor([pos0 > 0 for pos0, _ in entries], device=DEV)
    return rows * live[:, None]


def _part_inputs(case, seed):
    kind, d, entries = case["kind"], _Draw(seed, _dtype(case)), _entries(case["entries"])
    T = sum(n for _, n in entries)
    x = {"w": _mixer_weights(kind, d, form=case.get("form")), "h": d.normal(T, W2K)}
    _, pages = _pages(case, entries)
    if kind == "attention":                                     # normed keys, values as a projection leaves them
        x["k"], x["v"] = d.normal(pages + 1, 8, PAGE, 128), d.normal(pages + 1, 8, PAGE, 128, std=0.9)
    elif kind == "latent":
        x["k"] = d.normal(pages + 1, 1, PAGE, 128)
    elif kind in STATE_FLOATS:
        x["state"] = _state_rows(kind, d, entries)
    return x


def _qwen3_weights(d, layers, vocab=None, tied=True):
    z = QWEN3_4B
    hid, H, KV, D, I = z["hidden"], z["heads"], z["kv_heads"], z["dim"], z["inter"]
    w = {}
    if vocab:
        w["model.embed_tokens.weight"], w["model.norm.weight"] = d.normal(vocab, hid, std=0.02), d.uniform(hid, lo=0.5, hi=1.5)
    for i in range(layers):
        p = f"model.layers.{i}."
        for n, s in (("self_attn.q_proj", (H * D, hid)), ("self_attn.k_proj", (KV * D, hid)), ("self_attn.v_proj", (KV * D, hid)),
                     ("self_attn.o_proj", (hid, H * D)), ("mlp.gate_proj", (I, hid)), ("mlp.up_proj", (I, hid)), ("mlp.down_proj", (hid, I))):
            w[p + n + ".weight"] = d.normal(*s, std=0.02)
        for n, s in (("input_layernorm", hid), ("post_attention_layernorm", hid), ("self_attn.q_norm", D), ("self_attn.k_norm", D)):
            w[p + n + ".weight"] = d.uniform(s, lo=0.5, hi=1.5)
    return w


def _naditar_config(vocab):
    ff = {"kind": "dense", "ff": 8192}
    delta = {"type": "channel_delta", "mlp": ff, "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}}
    light = {"type": "lightning", "mlp": ff, "mixer": {"heads": 16, "dim": 128, "vdim": 128, "decay": list(LIGHT_DECAY)}}
    lat = {"type": "latent_attention", "mlp": ff, "mixer": {"heads": 16, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 96, "scale": 96 ** -0.5,
                                                            "rot": {"base": 1e6, "dims": 32}}}
    return {"architecture": "Naditar", "vocab": vocab, "width": W2K, "norm": {"eps": EPS}, "layers": [delta, delta, lat, light]}


NADITAR_KINDS = ("channel_delta", "channel_delta", "latent", "lightning")


def _step_positions(case):
    """Positions of the batch's next tokens: ragged contexts, the longest of the given length."""
    n, c = case["batch"], case["context"]
    return [max(1, c - 1 - (i * 613) % max(1, c // 3)) for i in range(n)]


def _step_inputs(case, seed):
    d, pos = _Draw(seed, _dtype(case)), _step_positions(case)
    entries = [(p, 1) for p in pos]
    _, pages = _pages(case, entries)
    x = {"tokens": d.ints(case["batch"], case["vocab"]).tolist(), "pos": pos, "entries": entries}
    if case["kind"] == "qwen3_step":
        x["w"] = _qwen3_weights(d, STEP_LAYERS, case["vocab"])
        x["k"] = [d.normal(pages + 1, 8, PAGE, 128) for _ in range(STEP_LAYERS)]
        x["v"] = [d.normal(pages + 1, 8, PAGE, 128, std=0.9) for _ in range(STEP_LAYERS)]
        return x
    w = {"embed": d.normal(case["vocab"], W2K, std=0.02), "head": d.normal(case["vocab"], W2K, std=0.02),
         "embed.norm": d.uniform(1, lo=0.5, hi=1.5), "final.norm": d.uniform(1, lo=0.5, hi=1.5)}
    for i, kind in enumerate(NADITAR_KINDS):
        w.update({f"l{i}.mix.{n}": t for n, t in _mixer_weights(kind, d).items()})
        w.update({f"l{i}.mlp.up": d.normal(8192, W2K, std=0.02), f"l{i}.mlp.down": d.normal(W2K, 8192, std=0.02),
                  f"l{i}.mlp.act": torch.tensor([0.9, 0.3, 0.1, 0.01], device=DEV).to(d.dtype),
                  f"l{i}.norm1": d.uniform(1, lo=0.5, hi=1.5), f"l{i}.norm2": d.uniform(1, lo=0.5, hi=1.5)})
    x["w"] = w
    x["k"] = d.normal(pages + 1, 1, PAGE, 128)
    x["state"] = {i: _state_rows(k, d, entries) for i, k in enumerate(NADITAR_KINDS) if k in STATE_FLOATS}
    return x


# ---------------------------------------------------------------- what a program keeps
def _specs(kind, form=None):
    from mini_inference_b200.config.spec import PartSpec
    none = PartSpec.of("none")
    if kind == "lightning":
        return PartSpec.of("lightning", hidden_size=W2K, num_heads=16, key_dim=128, value_dim=128, decay=LIGHT_DECAY, out_norm_eps=EPS), none
    if kind == "channel_delta":
        return PartSpec.of("channel_delta", hidden_size=W2K, num_heads=16, num_kv_heads=8, key_dim=128, value_dim=128, conv_taps=4,
                           out_norm_eps=EPS, unit_eps=1e-6, decay_rank=64, gate_rank=64), none
    if kind == "selective_scan":
        return PartSpec.of("selective_scan", hidden_size=W2K, inner=4096, state=16, dt_rank=128, conv_taps=4), none
    if kind == "latent":
        return (PartSpec.of("latent_attention", hidden_size=W2K, num_heads=16, nope_dim=64, rot_dim=32, value_dim=64, kv_rank=96,
                            scale=96 ** -0.5, latent_norm_eps=EPS), PartSpec.of("rotary_interleaved", dims=32, theta=1e6))
    if kind == "experts":
        return PartSpec.of("routed_experts", hidden_size=W2K, num_experts=32, top=4, groups=(8, 4), expert_size=1024, limit=7.0,
                           gate_slope=1.702, shared_size=2048, shared_limit=7.0), none
    base = dict(hidden_size=W2K, num_heads=16, num_kv_heads=8, key_dim=128, value_dim=128, unit_norm_eps=EPS)
    if form == "rotated":
        return (PartSpec.of("sink_attention", scale=128 ** -0.5, norm_weights=True, rotate=True, **base),
                PartSpec.of("rotary_half", dims=64, theta=1e6, factor=4.0))
    if form == "blocks":
        return PartSpec.of("sink_attention", scale=128 ** -0.5 * 8, block_size=1024, sink=True, **base), none
    return PartSpec.of("sink_attention", scale=128 ** -0.5, norm_weights=True, values="keys", q_temp=(0.1, 1024), slope_exponent=8.0, **base), none


def _admit(cache, entries):
    """The requests as a cache holds them before the step: their earlier tokens stored, pages for the new ones taken."""
    seqs = []
    for i, (pos0, n) in enumerate(entries):
        seq = cache.admit(i, pos0 + n)
        assert seq is not None and seq.slot == i + 1 and cache.ensure(seq, pos0 + n)
        seq.num_tokens = pos0
        seqs.append(seq)
    return seqs


def _step_context(ops, cache, hooks, entries, dtype):
    from mini_inference_b200.engine.batch import BatchBuilder, StepEntry
    from mini_inference_b200.parts.base import StepContext
    seqs = _admit(cache, entries)
    builder = BatchBuilder(cache, DEV, hooks, tile=getattr(ops, "prefill_tile", 64))
    builder.ops = ops
    batch = builder.build([StepEntry(s, [0] * n) for s, (_, n) in zip(seqs, entries)])
    batch.apply_table_updates(ops)
    return StepContext(ops, batch, dtype, torch.device(DEV))


def _prepare_part(case, seed):
    from mini_inference_b200.cache.manager import CacheManager
    from mini_inference_b200.ops import get_ops
    from mini_inference_b200.parts.base import build_part
    x, entries, dtype = _part_inputs(case, seed), _entries(case["entries"]), _dtype(case)
    ops, kind = get_ops(DEV), case["kind"]
    mixer_spec, position_spec = _specs(kind, case.get("form"))
    part = build_part("feed_forward" if kind == "experts" else "mixer", mixer_spec)
    part.load(x["w"], dtype, DEV)
    position = build_part("position", position_spec)
    if position_spec.kind != "none":
        position.load({}, dtype, DEV)
    hooks = {part.step_arrays_key: part.step_arrays} if part.step_arrays_key else {}
    need = None if kind == "experts" else part.cache_need()
    _, pages = _pages(case, entries)
    longest = max(p + n for p, n in entries)
    cache = CacheManager([need], PAGE, pages + 1, len(entries), -(-longest // PAGE) * PAGE, dtype=dtype, device=DEV)
    ctx = _step_context(ops, cache, hooks, entries, dtype)
    if kind == "experts":
        return dict(call=lambda: part.forward(x["h"], ctx))
    layer = cache.layer_caches[0]
    kept = []
    if layer.k is not None:
        layer.k[1:pages + 1].copy_(x["k"][1:])
        kept = [layer.k[1:pages + 1]]
        if layer.v is not None:
            layer.v[1:pages + 1].copy_(x["v"][1:])
            kept.append(layer.v[1:pages + 1])
    if "state" in x:
        layer.state[1:].copy_(x["state"])
        kept = [layer.state[1:]]
    return dict(call=lambda: (part.forward(x["h"], ctx, layer, position, True), *kept))


def _qwen3_config(layers, vocab):
    z = QWEN3_4B
    return {"architectures": ["Qwen3ForCausalLM"], "hidden_size": z["hidden"], "num_hidden_layers": layers, "num_attention_heads": z["heads"],
            "num_key_value_heads": z["kv_heads"], "head_dim": z["dim"], "intermediate_size": z["inter"], "vocab_size": vocab, "rope_theta": 1e6,
            "rms_norm_eps": EPS, "tie_word_embeddings": True, "max_position_embeddings": 40960}


def _layer_inputs(case, seed):
    d, entries = _Draw(seed, _dtype(case)), _entries(case["entries"])
    _, pages = _pages(case, entries)
    return {"w": _qwen3_weights(d, 1), "x": d.normal(sum(n for _, n in entries), QWEN3_4B["hidden"]),
            "k": d.normal(pages + 1, 8, PAGE, 128), "v": d.normal(pages + 1, 8, PAGE, 128, std=0.9)}


def _prepare_layer(case, seed):
    from mini_inference_b200.config.registry import resolve
    from mini_inference_b200.engine.factory import make_runner
    from mini_inference_b200.parts.base import StepContext
    from mini_inference_b200.engine.batch import StepEntry
    from mini_inference_b200.parts.model import DecoderModel
    x, entries, dtype = _layer_inputs(case, seed), _entries(case["entries"]), _dtype(case)
    cfg = _qwen3_config(1, 64)
    arch = resolve(cfg)
    model = DecoderModel(arch.build_spec(arch.config_class.from_dict(cfg)))
    tensors = dict(x["w"])
    for name, ws in model.weight_table():
        if name not in tensors:                                # embedding and last norm: not part of the layer
            tensors[name] = torch.zeros(ws.shape, dtype=dtype, device=DEV)
    model.load(tensors, dtype, DEV)
    _, pages = _pages(case, entries)
    longest = max(p + n for p, n in entries)
    runner = make_runner(model, PAGE, pages + 1, len(entries), -(-longest // PAGE) * PAGE)
    if dtype == torch.bfloat16:                                # as the engine does when it loads a model
        runner.ops.tune_many_rows(model.matrix_weights(), model.first_product_probes(runner.ops))
    seqs = _admit(runner.cache, entries)
    batch = runner.builder.build([StepEntry(s, [0] * n) for s, (_, n) in zip(seqs, entries)])
    batch.apply_table_updates(runner.ops)
    ctx = StepContext(runner.ops, batch, dtype, torch.device(DEV))
    layer, block = runner.cache.layer_caches[0], model.blocks[0]
    layer.k[1:pages + 1].copy_(x["k"][1:])
    layer.v[1:pages + 1].copy_(x["v"][1:])
    ctx.hints_ok = getattr(runner.ops, "takes_hints", False)

    def call():                                                # the layer rewrites the stream in place: a step's stream is fresh
        stream, delta = block.forward(x["x"].clone(), None, ctx, layer)
        return stream, delta, layer.k[1:pages + 1], layer.v[1:pages + 1]
    return dict(call=call, keep=(runner, seqs))


def _prepare_step(case, seed):
    from mini_inference_b200.engine.graphs import DecodeGraphs
    from mini_inference_b200.engine.llm import LLM
    x, B = _step_inputs(case, seed), case["batch"]
    cfg = _qwen3_config(STEP_LAYERS, case["vocab"]) if case["kind"] == "qwen3_step" else _naditar_config(case["vocab"])
    _, pages = _pages(case, x["entries"])
    longest = -(-(max(x["pos"]) + 1) // PAGE) * PAGE
    llm = LLM(None, random_config=cfg, random_seed=0, dtype=case["dtype"], device=DEV, kv_block_size=PAGE, kv_cache_tokens=(pages + 2) * PAGE,
              kv_watermark=0.0, max_num_seqs=B, max_model_len=longest, max_batched_tokens=4096, cuda_graphs=False)
    llm.model.load(dict(x["w"]), _dtype(case), DEV)
    llm.ops.tune_linear(llm.model.matrix_weights(), {tuple(llm.model.lm_head.shape): torch.float32},
                        deferrable=llm.model.deferrable_shapes(), gated=llm.model.gated_shapes())
    llm.graphs = DecodeGraphs(llm.runner, B, buckets=[B])
    llm.graphs.capture()
    seqs = _admit(llm.cache, x["entries"])
    caches, kept = llm.cache.layer_caches, []
    if case["kind"] == "qwen3_step":
        for i in range(STEP_LAYERS):
            for pool, values in ((caches[i].k, x["k"][i]), (caches[i].v, x["v"][i])):
                pool[1:pages + 1].copy_(values[1:])
                kept.append(pool[1:pages + 1])
    else:
        caches[2].k[1:pages + 1].copy_(x["k"][1:])
        kept = [caches[2].k[1:pages + 1]]
        for i, rows in x["state"].items():
            caches[i].state[1:].copy_(rows)
            kept.append(caches[i].state[1:])
    graphs, tokens = llm.graphs, x["tokens"]

    def call():                                                # a decode step: metadata to the device, one graph
        graphs.fill(B, seqs, tokens)
        graphs.replay(B)
        return (graphs.logits_out[B], *kept)
    return dict(call=call, keep=llm)


def prepare(case, seed):
    with torch.inference_mode():
        if case["kind"] in ("qwen3_step", "naditar_step"):
            return _prepare_step(case, seed)
        return _prepare_layer(case, seed) if case["kind"] == "qwen3_layer" else _prepare_part(case, seed)


def run(state):
    with torch.inference_mode():
        return state["call"]()


# ---------------------------------------------------------------- what a pass cannot do without
def _pairs(entries, block=None):
    total = 0
    for pos0, n in entries:
        if block is None:
            total += n * pos0 + n * (n + 1) // 2
        else:
            total += sum(p % block + 1 for p in range(pos0, pos0 + n))
    return total


def _part_work(kind, entries, es, form=None):
    """(bytes, operations) of one mixer or feed-forward of the 2k sizes: weights, input and output rows, cache and states once."""
    T, S = sum(n for _, n in entries), len(entries)
    keys = sum(p + n for p, n in entries)
    io = 2 * T * W2K * es
    if kind == "lightning":
        mats = W2K * (5 * 2048)
        return mats * es + io + 2 * S * STATE_FLOATS[kind] * 4, 2 * T * mats + T * 4 * 16 * 128 * 128
    if kind == "channel_delta":
        mats = W2K * (DELTA_C + 16 + 128) + 64 * 4096 + W2K * 2048
        return mats * es + io + 2 * S * STATE_FLOATS[kind] * 4, 2 * T * mats + T * 8 * 16 * 128 * 128
    if kind == "selective_scan":
        mats = W2K * 3 * 4096 + 4096 * 160 + 128 * 4096
        return mats * es + io + 2 * S * STATE_FLOATS[kind] * 4, 2 * T * mats + T * 6 * 4096 * 16
    if kind == "latent":
        mats = W2K * (16 * 96 + 128 + 16) + 2 * 16 * 64 * 96 + W2K * 1024
        return mats * es + io + keys * 128 * es + T * 128 * es, 2 * T * mats + 2 * 16 * (128 + 96) * _pairs(entries)
    if kind == "attention":
        mats = W2K * (2048 + 1024 * (1 if form == "slopes" else 2) + 2048)
        read = keys if form != "blocks" else sum(p + n - p // 1024 * 1024 for p, n in entries)
        return mats * es + io + (read + T) * 2 * 1024 * es, 2 * T * mats + 4 * 2048 * _pairs(entries, 1024 if form == "blocks" else None)
    used = min(32, 4 * T)
    return (used * 3 * 1024 + 3 * 2048) * W2K * es + io, 2 * T * W2K * (32 + 4 * 3 * 1024 + 3 * 2048)


def work(case):
    es = 4 if case["dtype"] == "float32" else 2
    z = QWEN3_4B
    layer = z["hidden"] * (z["heads"] + 2 * z["kv_heads"]) * z["dim"] + z["heads"] * z["dim"] * z["hidden"] + 3 * z["hidden"] * z["inter"]
    if case["kind"] == "qwen3_layer":
        e = _entries(case["entries"])
        T, keys = sum(n for _, n in e), sum(p + n for p, n in e)
        return {"bytes": layer * es + 3 * T * z["hidden"] * es + (keys + T) * 2 * 1024 * es,
                "flops": 2 * T * layer + 4 * 4096 * _pairs(e)}
    if case["kind"] == "qwen3_step":
        pos, B = _step_positions(case), case["batch"]
        keys = sum(pos) + B
        head = case["vocab"] * z["hidden"]
        return {"bytes": STEP_LAYERS * (layer * es + (keys + B) * 2 * 1024 * es) + head * es + B * case["vocab"] * 4,
                "flops": 2 * B * (STEP_LAYERS * layer + head) + STEP_LAYERS * 4 * 4096 * keys}
    if case["kind"] == "naditar_step":
        e, B = [(p, 1) for p in _step_positions(case)], case["batch"]
        parts = [_part_work(k, e, es) for k in NADITAR_KINDS]
        mlp, head = 2 * 8192 * W2K, case["vocab"] * W2K
        return {"bytes": sum(b for b, _ in parts) + (4 * mlp + head) * es + B * case["vocab"] * 4,
                "flops": sum(f for _, f in parts) + 2 * B * (4 * mlp + head)}
    b, f = _part_work(case["kind"], _entries(case["entries"]), es, case.get("form"))
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the error against 64 bits that the engine's kernels showed when this file was written: float32 3e-6 (sums of
    2,560 to 9,728 products), one bfloat16 layer or part 2e-3 to 6e-3 (each intermediate rounded to 8 bits; 1e-2 behind a norm of a
    long sum), four layers and a head 1.6e-2."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 3e-2} if case["kind"] in ("qwen3_step", "naditar_step") else {"rel": 2e-2}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def _rms(x, eps=EPS):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _turn(x, pos, dims, theta, factor=1.0, interleaved=False):
    """The first `dims` coordinates of x [T, heads, D] turned by their position."""
    f = (theta ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims) / factor).float().double()
    ang = pos.double()[:, None] * f[None, :]
    c, s = ang.cos()[:, None, :], ang.sin()[:, None, :]
    out = x.clone()
    if interleaved:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        out[..., 0:dims:2], out[..., 1:dims:2] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        out[..., :dims // 2], out[..., dims // 2:dims] = u * c - v * s, v * c + u * s
    return out


def _spans(entries):
    a = 0
    for i, (pos0, n) in enumerate(entries):
        yield i, a, a + n, pos0
        a += n


def _positions(entries):
    return torch.cat([torch.arange(p, p + n, device=DEV) for p, n in entries])


def _written(pool, rows, entries):
    """The pool [pages + 1, heads, PAGE, D] with the step's rows [T, heads, D] in their places, and per request its rows in order."""
    lists, _ = _pages(None, entries)
    pool, per = pool.clone(), []
    for i, a, b, pos0 in _spans(entries):
        idx = torch.arange(pos0, pos0 + b - a, device=DEV)
        table = torch.tensor(lists[i], device=DEV)
        pool[table[idx // PAGE], :, idx % PAGE, :] = rows[a:b]
        per.append(pool[table].transpose(1, 2).reshape(-1, pool.shape[1], pool.shape[3])[:pos0 + b - a])
    return pool, per


def _softmax_attention(q, keys, values, entries, scale, block=None, sink=False, slopes=None):
    """q [T, H, D]; per request keys / values [n, KV, D]."""
    T, H, _ = q.shape
    out = torch.empty(T, H, values[0].shape[2], dtype=torch.float64, device=DEV)
    for i, a, b, pos0 in _spans(entries):
        K, V = keys[i], values[i]
        G = H // K.shape[1]
        p, j = torch.arange(pos0, pos0 + b - a, device=DEV), torch.arange(K.shape[0], device=DEV)
        seen = j[None, :] <= p[:, None]
        if block:
            seen &= (j[None, :] // block) == (p[:, None] // block)
        for h in range(H):
            s = q[a:b, h] @ K[:, h // G].T * scale
            if slopes is not None:
                s = s - slopes[h] * (p[:, None] - j[None, :])
            s = s.masked_fill(~seen, float("-inf"))
            if sink:
                s = torch.cat([s, torch.zeros(b - a, 1, dtype=torch.float64, device=DEV)], dim=1)
            w = torch.softmax(s, dim=-1)
            out[a:b, h] = (w[:, :-1] if sink else w) @ V[:, h // G]
    return out


def _conv(x, weight, hist):
    """Causal convolution of x [T, C] behind hist [taps - 1, C]; (output, the last taps - 1 inputs)."""
    ext = torch.cat([hist, x], dim=0)
    taps = weight.shape[1]
    return sum(weight[:, j] * ext[j:j + x.shape[0]] for j in range(taps)), ext[ext.shape[0] - (taps - 1):]


def _exact_part(kind, w, h, x, entries, form=None):
    """(output rows, updated cache tensors ..) of one mixer or feed-forward, everything float64."""
    T = h.shape[0]
    lin = lambda a, n: a @ w[n].T                                # noqa: E731
    if kind == "lightning":
        H, D = 16, 128
        q, k, v = (F.silu(lin(h, n)).view(T, H, D) for n in "qkv")
        decay = torch.tensor(LIGHT_DECAY, dtype=torch.float32, device=DEV).double()[:, None, None]
        o, states = torch.empty(T, H, D, dtype=torch.float64, device=DEV), []
        for i, a, b, _ in _spans(entries):
            S = x["state"][i].view(H, D, D).clone()
            for t in range(a, b):
                S = decay * S + k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
            states.append(S.reshape(-1))
        rows = _rms(o.reshape(T, H * D)) * w["norm"] * torch.sigmoid(lin(h, "g"))
        return lin(rows, "o"), torch.stack(states)
    if kind == "channel_delta":
        H, KV, D, M = 16, 8, 128, 16 * 128 * 128
        p = torch.cat([lin(h, n) for n in "qkv"], dim=1)
        cw = torch.cat([w[n + ".conv"] for n in "qkv"], dim=0)
        beta = torch.sigmoid(lin(h, "b"))
        g = torch.exp(-torch.exp(w["A_log"])[None, :, None] * F.softplus(lin(lin(h, "a1"), "a2") + w["dt_bias"]).view(T, H, D))
        o, states = torch.empty(T, H, D, dtype=torch.float64, device=DEV), []
        for i, a, b, _ in _spans(entries):
            y, tail = _conv(p[a:b], cw, x["state"][i, M:].view(3, DELTA_C))
            y = F.silu(y)
            qk = y[:, :2 * KV * D].view(b - a, 2 * KV, D)
            qk = qk / torch.sqrt(qk.pow(2).sum(-1, keepdim=True) + 1e-6)
            q = (qk[:, :KV] * D ** -0.5).repeat_interleave(H // KV, dim=1)
            k = qk[:, KV:].repeat_interleave(H // KV, dim=1)
            v = y[:, 2 * KV * D:].view(b - a, H, D)
            S = x["state"][i, :M].view(H, D, D).clone()
            for t in range(b - a):
                S = g[a + t][:, :, None] * S
                u = beta[a + t][:, None] * (v[t] - torch.bmm(k[t][:, None, :], S)[:, 0])
                S = S + k[t][:, :, None] * u[:, None, :]
                o[a + t] = torch.bmm(q[t][:, None, :], S)[:, 0]
            states.append(torch.cat([S.reshape(-1), tail.reshape(-1)]))
        rows = _rms(o) * w["norm"] * torch.sigmoid(lin(lin(h, "g1"), "g2")).view(T, H, D)
        return lin(rows.reshape(T, H * D), "o"), torch.stack(states)
    if kind == "selective_scan":
        I, N, R = 4096, 16, 128
        xz = lin(h, "in")
        A = -torch.exp(w["A_log"])
        y, states = torch.empty(T, I, dtype=torch.float64, device=DEV), []
        for i, a, b, _ in _spans(entries):
            u, tail = _conv(xz[a:b, :I], w["conv"], x["state"][i, I * N:].view(3, I))
            u = F.silu(u + w["conv.b"])
            p = lin(u, "x")
            dt = F.softplus(lin(p[:, :R], "dt") + w["dt.b"])
            S = x["state"][i, :I * N].view(I, N).clone()
            for t in range(b - a):
                S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * p[t, R:R + N][None, :]
                y[a + t] = S @ p[t, R + N:] + w["D"] * u[t]
            states.append(torch.cat([S.reshape(-1), tail.reshape(-1)]))
        return lin(y * F.silu(xz[:, I:]), "o"), torch.stack(states)
    pos = _positions(entries)
    if kind == "latent":
        H, D, R, V, C = 16, 64, 32, 64, 96
        q = lin(h, "q").view(T, H, D + R)
        qr = _turn(q[..., D:], pos, R, 1e6, interleaved=True)
        dkv = lin(h, "dkv")
        row = torch.cat([_rms(dkv[:, :C]) * w["dkv.norm"], _turn(dkv[:, None, C:], pos, R, 1e6, interleaved=True)[:, 0]], dim=1)
        pool, per = _written(x["k"], row[:, None, :], entries)
        keys = [torch.cat([(c[:, 0, :C] @ w["uk"].T).view(-1, H, D), c[:, :, C:].expand(-1, H, -1)], dim=2) for c in per]
        values = [(c[:, 0, :C] @ w["uv"].T).view(-1, H, V) for c in per]
        o = _softmax_attention(torch.cat([q[..., :D], qr], dim=2), keys, values, entries, 96 ** -0.5)
        return lin((o * torch.sigmoid(lin(h, "g"))[:, :, None]).reshape(T, H * V), "o"), pool[1:]
    if kind == "attention":
        H, KV, D = 16, 8, 128
        q, k_raw = lin(h, "q").view(T, H, D), lin(h, "k").view(T, KV, D)
        v = k_raw if form == "slopes" else lin(h, "v").view(T, KV, D)
        q, k = _rms(q), _rms(k_raw)
        if form != "blocks":
            q, k = q * w["q.norm"], k * w["k.norm"]
        slopes = None
        if form == "rotated":
            q, k = _turn(q, pos, 64, 1e6, 4.0), _turn(k, pos, 64, 1e6, 4.0)
        if form == "slopes":
            q = q * (1.0 + 0.1 * torch.log(((pos + 1) // 1024 + 1).double()))[:, None, None]
            slopes = [2.0 ** (-8.0 * (i + 1) / H) for i in range(H)]
        kp, keys = _written(x["k"], k, entries)
        vp, values = _written(x["v"], v, entries)
        o = _softmax_attention(q, keys, values, entries, 128 ** -0.5 * (8 if form == "blocks" else 1), 1024 if form == "blocks" else None,
                               form == "blocks", slopes)
        return lin(o.reshape(T, H * D), "o"), kp[1:], vp[1:]
    s = torch.softmax(lin(h, "router"), dim=-1)
    choice = s + w["correction"]
    kept = choice.view(T, 8, 4).max(-1).values.topk(4, dim=-1).indices
    allowed = torch.zeros(T, 8, dtype=torch.bool, device=DEV).scatter_(1, kept, True).repeat_interleave(4, dim=1)
    chosen = choice.masked_fill(~allowed, float("-inf")).topk(4, dim=-1).indices

    def expert(rows, name):
        g, u = lin(rows, name + ".gate").clamp(max=7.0), lin(rows, name + ".up").clamp(-7.0, 7.0)
        return lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), name + ".down")
    out = expert(h, "shared")
    for e in range(32):
        t, _ = torch.where(chosen == e)
        out[t] += s[t, e][:, None] * expert(h[t], f"e{e}")
    return (out,)


def _exact_qwen3_layer(w, p, x, k, v, entries):
    """(stream behind the attention, the feed-forward's output, key pool, value pool)."""
    z, T = QWEN3_4B, x.shape[0]
    H, KV, D, pos = z["heads"], z["kv_heads"], z["dim"], _positions(entries)
    h = _rms(x) * w[p + "input_layernorm.weight"]
    q, kk, vv = ((h @ w[p + f"self_attn.{n}_proj.weight"].T).view(T, -1, D) for n in "qkv")
    q = _turn(_rms(q) * w[p + "self_attn.q_norm.weight"], pos, D, 1e6)
    kk = _turn(_rms(kk) * w[p + "self_attn.k_norm.weight"], pos, D, 1e6)
    kp, keys = _written(k, kk, entries)
    vp, values = _written(v, vv, entries)
    o = _softmax_attention(q, keys, values, entries, D ** -0.5)
    x = x + o.reshape(T, H * D) @ w[p + "self_attn.o_proj.weight"].T
    h = _rms(x) * w[p + "post_attention_layernorm.weight"]
    y = F.silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)
    return x, y @ w[p + "mlp.down_proj.weight"].T, kp, vp


def _double(v):
    if isinstance(v, torch.Tensor):
        return v.double()
    if isinstance(v, dict):
        return {k: _double(t) for k, t in v.items()}
    return [_double(t) for t in v] if isinstance(v, list) and v and isinstance(v[0], torch.Tensor) else v


def exact(case, seed):
    with torch.inference_mode():
        kind = case["kind"]
        if kind == "qwen3_layer":
            x, e = _double(_layer_inputs(case, seed)), _entries(case["entries"])
            s, y, kp, vp = _exact_qwen3_layer(x["w"], "model.layers.0.", x["x"], x["k"], x["v"], e)
            return s, y, kp[1:], vp[1:]
        if kind not in ("qwen3_step", "naditar_step"):
            x, e = _double(_part_inputs(case, seed)), _entries(case["entries"])
            out = _exact_part(kind, x["w"], x["h"], x, e, case.get("form"))
            return out[0] if kind == "experts" else out
        raw = _step_inputs(case, seed)
        e, tokens = raw["entries"], torch.tensor(raw["tokens"], device=DEV)
        x = _double(raw)
        w = x["w"]
        kept = []
        if kind == "qwen3_step":
            s = w["model.embed_tokens.weight"][tokens]
            for i in range(STEP_LAYERS):
                s, y, kp, vp = _exact_qwen3_layer(w, f"model.layers.{i}.", s, x["k"][i], x["v"][i], e)
                s = s + y
                kept += [kp[1:], vp[1:]]
            return (_rms(s) * w["model.norm.weight"] @ w["model.embed_tokens.weight"].T, *kept)
        s = _rms(w["embed"][tokens]) * w["embed.norm"]
        states = []
        for i, mixer in enumerate(NADITAR_KINDS):
            p = f"l{i}."
            mw = {n[len(p) + 4:]: t for n, t in w.items() if n.startswith(p + "mix.")}
            own = {"state": x["state"][i]} if mixer in STATE_FLOATS else {"k": x["k"]}
            y, after = _exact_part(mixer, mw, _rms(s) * w[p + "norm1"], own, e)
            if mixer == "latent":
                kept.append(after)
            else:
                states.append(after)
            s = s + y
            zed = (_rms(s) * w[p + "norm2"]) @ w[p + "mlp.up"].T
            a, b, c, d = (float(v) for v in w[p + "mlp.act"])
            s = s + (a * _rms(zed) + b * _rms(zed * zed) + c * _rms(zed ** 3) + d) @ w[p + "mlp.down"].T
        return (_rms(s) * w["final.norm"] @ w["head"].T, *kept, *states)
