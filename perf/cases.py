"""The work that programs have this engine do, as cases that can be timed and checked: whole steps of an LFM2 model, and
the layers of the designs it serves, each through the entry point that a program calls (StepRunner.run, DecoderModel.forward,
a part's or a block's forward()).

A step of decoding is captured once in a CUDA graph, as the engine does with its decode steps, and a pass replays it; a
step that brings prompt tokens is launched as it comes. Sizes are those of the shapes in cellm_b200/config/presets.py
("1.2b": width 2,048, "700m": width 1,536); portions, contexts and batches those of bench.py and bin/workload.

kinds:
  step            a whole LFM2 model: the logits of a prompt's last place, or of one decoded token per request
  attention       an LFM2 attention layer's mixer over its pages
  conv_layer      an LFM2 layer with a short convolution: norm, mixer, norm, feed-forward, on the 32-bit stream
  latent          Gonozen's latent attention: every earlier row, a rotated key part, an output gate
  latent_window   Gonozen's second form: queries through a latent, a window of 1,024 rows, a sink a head
  experts         Tufadra's mixture of experts (64 of which 6 are chosen, and a shared one)
  gated_experts   Gonozen's, with the clamped gate
  delta           Padadra's gated delta rule with its convolutions and norms
  parallel        Padadra's two mixers side by side: windowed attention with sinks, and HGRN2
"""
from __future__ import annotations

import math
import zlib

import torch

from cellm_b200.cache import CacheManager
from cellm_b200.config.presets import GONOZEN_SHAPES, LFM2_SHAPES, PADADRA_SHAPES, TUFADRA_SHAPES
from cellm_b200.config.registry import config_from_dict
from cellm_b200.engine import StepEntry, StepRunner
from cellm_b200.models.decoder import DecoderModel
from cellm_b200.ops._state import error_word
from cellm_b200.parts.base import CacheBinding, Residual, StepContext
from cellm_b200.parts.registry import part_class
from cellm_b200.weights.loader import expected_tensors

DEV = "cuda:0"
PAGE = 16
F64 = torch.float64


def listed():
    return [
        # one user's token after a short prompt: the smallest whole call, bound by launches and latency
        dict(name="step decode 1", kind="step", size="1.2b", dtype="bfloat16", requests=1, tokens=1, context=500, ragged=False),
        # the benchmark's prompt
        dict(name="step prompt 2048", kind="step", size="1.2b", dtype="bfloat16", requests=1, tokens=2048, context=0, ragged=False),
        # a late portion of the long-context workload (one long prompt in portions of 2,048 tokens)
        dict(name="attention portion at 8192", kind="attention", size="700m", dtype="bfloat16", requests=1, tokens=2048, context=8192, ragged=False),
        # the streams that decode beside it
        dict(name="attention decode 16", kind="attention", size="1.2b", dtype="bfloat16", requests=16, tokens=1, context=4096, ragged=True),
        # a step of the continuous scheduler with a few short prompts of odd lengths
        dict(name="conv layer 5 prompts", kind="conv_layer", size="1.2b", dtype="bfloat16", requests=5, tokens=61, context=0, ragged=True),
        # the true 32-bit path, which checks of exactness run on
        dict(name="attention float32", kind="attention", size="700m", dtype="float32", requests=3, tokens=71, context=100, ragged=True),
        # the decode batch of the benchmark on a compressed cache
        dict(name="latent decode 8", kind="latent", size="1.2b", dtype="bfloat16", requests=8, tokens=1, context=2048, ragged=False),
        # a prompt of odd length through the windowed form
        dict(name="latent window prompt", kind="latent_window", size="1.2b", dtype="bfloat16", requests=1, tokens=1537, context=0, ragged=False),
        # a prompt's tokens over all experts
        dict(name="experts prompt 2048", kind="experts", size="1.2b", dtype="bfloat16", requests=1, tokens=2048, context=0, ragged=False),
        # the decode batch: nearly every token meets experts of its own
        dict(name="gated experts decode 8", kind="gated_experts", size="1.2b", dtype="bfloat16", requests=8, tokens=1, context=0, ragged=False),
        # one prompt through a recurrence, which a single request walks alone
        dict(name="delta prompt 2048", kind="delta", size="1.2b", dtype="bfloat16", requests=1, tokens=2048, context=0, ragged=False),
        # two unequal prompts through attention and recurrence side by side
        dict(name="parallel 2 prompts", kind="parallel", size="700m", dtype="bfloat16", requests=2, tokens=700, context=0, ragged=True),
    ]


KINDS = ("step", "attention", "conv_layer", "latent", "latent_window", "experts", "gated_experts", "delta", "parallel")


def draw(rng):
    """One more case of the listed ranges: a kind, a size, and either a decode step (1 to 64 requests, contexts up to
    8,192) or prompt portions (17 to 2,048 tokens in one to six portions, some behind a context)."""
    kind = rng.choice(KINDS)
    size = rng.choice(("1.2b", "700m"))
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    dtype = "float32" if kind in ("attention", "conv_layer") and rng.random() < 0.2 else "bfloat16"
    if rng.random() < 0.4:
        requests, tokens = log(1, 64), 1
        context = log(128, 8192) if kind != "step" else log(64, 600)
        context = min(context, 65536 // requests)
        ragged = rng.random() < 0.5 and requests > 1
    else:
        total = log(17, 2048 if dtype == "bfloat16" else 512)
        requests = rng.choice((1, 1, 2, 3, 6))
        tokens = max(2, total // requests)
        ragged = requests > 1
        context = rng.choice((0, 0, log(16, 4096))) if kind in ("attention", "latent", "latent_window") else 0
    if kind == "step":
        requests = min(requests, 8)
    if kind in ("experts", "gated_experts"):
        context = 0
    return dict(kind=kind, size=size, dtype=dtype, requests=requests, tokens=tokens, context=context, ragged=ragged)


# ------------------------------------------------------------------------------------------------ shapes and inputs
def _config(case):
    """The config.json of a model that is that layer alone (the whole model for a step), and the place of its tensors."""
    kind, size = case["kind"], case["size"]
    if kind == "step":
        return dict(LFM2_SHAPES["lfm2-" + size])
    if kind in ("attention", "conv_layer"):
        return dict(LFM2_SHAPES["lfm2-" + size], num_hidden_layers=1, full_attn_idxs=[0] if kind == "attention" else [])
    shapes, wanted = {"latent": (GONOZEN_SHAPES, "latent_attention"), "latent_window": (GONOZEN_SHAPES, "latent_attention_2"),
                      "gated_experts": (GONOZEN_SHAPES, "latent_attention"), "experts": (TUFADRA_SHAPES, "attention"),
                      "delta": (PADADRA_SHAPES, "channel_delta"), "parallel": (PADADRA_SHAPES, "parallel")}[kind]
    config = dict(shapes[size][0])
    layer = dict(next(x for x in config["layers"] if x["type"] == wanted))
    if kind not in ("experts", "gated_experts"):
        layer.pop("mlp")
    config["layers"] = [layer]
    return config


def _spread(n, mean, ragged):
    """n lengths around `mean`, unequal if asked: the same for every seed."""
    if not ragged:
        return [mean] * n
    return [max(1, int(mean * (0.25 + 1.5 * ((0.37 + 0.618034 * i) % 1.0)))) for i in range(n)]


def _lengths(case):
    n = case["requests"]
    return (_spread(n, case["tokens"], case["ragged"] and case["tokens"] > 1),
            _spread(n, case["context"], case["ragged"]) if case["context"] else [0] * n)


def _random(seed, name, shape, std, dtype=torch.float32, mean=0.0):
    g = torch.Generator(device=DEV).manual_seed(zlib.crc32(("%d:%s" % (seed, name)).encode()))
    return (torch.randn(tuple(shape), generator=g, device=DEV, dtype=torch.float32) * std + mean).to(dtype)


# a table of unit rows, the size of the stream between a trained model's layers (with rows of 0.02 the layers' own roundings
# would be all that a whole model's logits show)
_STD = {"linear": 0.02, "embedding": 1.0, "conv_tap": 0.1, "bias": 0.02, "conv_tap_wide": 0.5, "sink": 1.0}


def _tensor(seed, name, spec, dtype):
    """A weight as the random-weights mode would fill it (its values here are made on the GPU)."""
    if spec.init in ("norm", "norm_offset"):
        return _random(seed, name, spec.shape, 0.05, dtype, 1.0 if spec.init == "norm" else 0.0)
    if spec.init == "unit_interval":
        return (0.05 + 0.6 * torch.sigmoid(_random(seed, name, spec.shape, 1.0))).to(dtype)
    if spec.init == "log_rate":
        return torch.log(0.5 + 3.5 * torch.sigmoid(_random(seed, name, spec.shape, 1.0))).to(dtype)
    std = 1.0 / max(1, spec.shape[-1]) ** 0.5 if spec.init == "linear_wide" else _STD[spec.init]
    return _random(seed, name, spec.shape, std, dtype)


def _dtype(case):
    return getattr(torch, case["dtype"])


def _inputs(case, seed):
    """(plan, file tensors by name) of the case."""
    cfg, plan = config_from_dict(_config(case))
    outside = ("embed", "head", "final.norm", "pos", "bigram", "model.embed", "model.embedding_norm")
    tensors = {}
    for name, spec in expected_tensors(plan).items():
        if case["kind"] != "step" and name.startswith(outside):
            continue                    # a layer alone has no table of tokens
        if case["kind"] in ("experts", "gated_experts") and "mlp." not in name or case["kind"] == "attention" and "feed_forward" in name:
            continue
        tensors[name] = _tensor(seed, name, spec, _dtype(case))
    return plan, tensors


def _context(case, dtype):
    """What a step tells every part: lengths, positions, slots; and one table of pages in a shuffled order."""
    lens, ctxs = _lengths(case)
    B, T = len(lens), sum(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ctx = StepContext(T=T, B=B, dtype=dtype, device=torch.device(DEV), token_ids=i32([0] * T),
                      positions=i32([c + j for n, c in zip(lens, ctxs) for j in range(n)]),
                      seq_of_token=i32([b for b, n in enumerate(lens) for _ in range(n)]), cu_seqlens=i32(cu), ctx_lens=i32(ctxs),
                      slot_ids=i32(list(range(B))), err=error_word(torch.device(DEV)), q_lens=lens, ctx_lens_host=ctxs,
                      max_q_len=max(lens), max_total_len=max(n + c for n, c in zip(lens, ctxs)))
    per = [-(-(n + c) // PAGE) for n, c in zip(lens, ctxs)]
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(7)).tolist()
    rows, at = [], 0
    for p in per:
        rows.append(order[at:at + p] + [-1] * (max(per) - p))
        at += p
    return ctx, i32(rows), sum(per)


def _bind(case, needs, seed, dtype, table, pages, slots, fresh):
    """A binding of filled pools and states for what the mixer keeps: unit-size rows behind a context, zero states before
    a sequence's first token."""
    from cellm_b200.parts.base import PagedKV
    one = []
    for i, need in enumerate(needs):
        if isinstance(need, PagedKV):
            shape = (pages, need.num_kv_heads, PAGE, need.head_dim)
            k = _random(seed, "keys%d" % i, shape, 1.0, dtype)
            v = _random(seed, "values%d" % i, shape[:3] + (need.value_dim or need.head_dim,), 1.0, dtype) if need.values else None
            one.append(CacheBinding(need=need, k=k, v=v, block_table=table, page_size=PAGE, num_pages=pages))
        else:
            state = _random(seed, "state%d" % i, (slots,) + tuple(need.shape), 0.0 if fresh else 0.1)
            one.append(CacheBinding(need=need, state=state, num_slots=slots))
    return one[0] if len(one) == 1 else CacheBinding(need=tuple(needs), parts=tuple(one))


def _caches(cache):
    """The tensors of a binding, in order."""
    return [t for b in (cache.parts or (cache,)) for t in (b.k, b.v, b.state) if t is not None]


def _mixer_input(case, seed, plan, T):
    return _random(seed, "x", (T, plan.hidden_size), 1.0, _dtype(case))


def _raw(case, seed):
    """Everything a layer's pass reads: plan, weights, step context, caches, input."""
    plan, w = _inputs(case, seed)
    ctx, table, pages = _context(case, _dtype(case))
    cache = None
    if case["kind"] not in ("experts", "gated_experts"):
        spec = plan.layers[0].mixer
        need = part_class("mixer", spec.kind).cache_need(spec.params)
        needs = list(need) if isinstance(need, tuple) else [need]
        cache = _bind(case, needs, seed, _dtype(case), table, pages, ctx.B, fresh=case["context"] == 0)
    return plan, w, ctx, cache, _mixer_input(case, seed, plan, ctx.T)


# ------------------------------------------------------------------------------------------------ a program's calls
def _part(family, spec, tensors, dtype):
    return part_class(family, spec.kind)(spec.params, {k: tensors[n] for k, n in spec.weights.items() if n in tensors}, dtype)


def _graph(call, keep):
    """`call` captured as the engine captures a decode step: one run to load its kernels, the states it moves on put
    back, then the capture."""
    saved = [t.clone() for t in keep]
    call()
    for t, s in zip(keep, saved):
        t.copy_(s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    return graph, out


def _prepare_step(case, seed):
    plan, tensors = _inputs(case, seed)
    model = DecoderModel(plan, tensors, _dtype(case), DEV)
    lens, ctxs = _lengths(case)
    pages = sum(-(-(n + c) // PAGE) for n, c in zip(lens, ctxs))
    cache = CacheManager(model.cache_needs(), [e.cache_of for e in plan.order], PAGE, pages, len(lens), _dtype(case), DEV)
    runner = StepRunner(model, cache)
    ids = _tokens(seed, lens, ctxs, plan.vocab_size)
    if case["tokens"] > 1:
        return {"case": case, "runner": runner, "ids": ids, "next": 0}
    entries = []
    for r, (c, row) in enumerate(zip(ctxs, ids)):
        cache.add(r)
        if c:
            runner.run([StepEntry(r, row[:c], [])])
        entries.append(StepEntry(r, row[c:], [0]))
    ctx, tables, rows, _ = runner.build_context(entries)
    bindings = cache.bindings(tables)
    graph, out = _graph(lambda: model.forward(ctx, bindings, rows), cache.states)
    return {"case": case, "graph": graph, "out": out, "keep": (model, cache, ctx, bindings, rows)}


def _tokens(seed, lens, ctxs, vocab):
    g = torch.Generator().manual_seed(seed + 1)
    return [torch.randint(0, vocab, (n + c,), generator=g).tolist() for n, c in zip(lens, ctxs)]


def prepare(case, seed):
    """The weights, caches and inputs of a case, and for a decode step its captured graph."""
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    plan, w, ctx, cache, x = _raw(case, seed)
    layer, dtype, kind = plan.layers[0], _dtype(case), case["kind"]
    s = {"case": case, "ctx": ctx, "cache": cache, "x": x}
    if kind in ("experts", "gated_experts"):
        s["part"] = _part("feed_forward", layer.feed_forward, w, dtype)
    else:
        s["part"] = _part("mixer", layer.mixer, w, dtype)
    if kind == "conv_layer":
        s["x"] = _random(seed, "stream", (ctx.T, plan.hidden_size), 1.0)
        s["part"] = part_class("block", layer.block)(_part("norm", layer.mixer_norm, w, dtype), s["part"],
                                                     _part("norm", layer.feed_forward_norm, w, dtype),
                                                     _part("feed_forward", layer.feed_forward, w, dtype))
    if case["tokens"] == 1:
        states = [b.state for b in (cache.parts or (cache,)) if b.state is not None] if cache is not None else []
        s["graph"], s["out"] = _graph(lambda: _call(s), states)
    return s


def _call(s):
    kind = s["case"]["kind"]
    if kind in ("experts", "gated_experts"):
        return s["part"].forward(s["x"], s["ctx"])
    if kind == "conv_layer":
        res = Residual(s["x"].clone())
        s["part"].forward(res, s["ctx"], s["cache"])
        return [res.flush()] + _caches(s["cache"])
    return [s["part"].forward(s["x"], s["ctx"], s["cache"])] + _caches(s["cache"])


def run(s):
    if "graph" in s:
        s["graph"].replay()
        return s["out"]
    if s["case"]["kind"] == "step":
        cache, ids = s["runner"].cache, s["ids"]
        first = s["next"]
        s["next"] += len(ids)
        for r in range(len(ids)):
            cache.add(first + r)
        logits = s["runner"].run([StepEntry(first + r, row, [len(row) - 1]) for r, row in enumerate(ids)])
        for r in range(len(ids)):
            cache.release(first + r)
        return logits
    return _call(s)


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    config, kind = _config(case), case["kind"]
    cfg, plan = config_from_dict(config)
    lens, ctxs = _lengths(case)
    T, el, H = sum(lens), torch.empty((), dtype=_dtype(case)).element_size(), plan.hidden_size
    window = 1024 if kind in ("latent_window", "parallel") else 1 << 40
    seen = [min(c, window) for c in ctxs]                                                  # rows of the cache that are read
    pairs = sum(min(c + j + 1, window) for n, c in zip(lens, ctxs) for j in range(n))      # (query, key) pairs a head
    nbytes, flops = 0.0, 0.0

    def matrix(rows, cols, tokens=T):
        nonlocal nbytes, flops
        nbytes += rows * cols * el
        flops += 2.0 * rows * cols * tokens

    def attention(nh, nkv, hd, cached=None):
        nonlocal nbytes, flops
        nbytes += 2 * nkv * hd * el * (sum(seen) + T)
        flops += 4.0 * nh * hd * pairs

    def lfm_attention():
        nh, nkv, hd = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"]
        matrix((nh + 2 * nkv) * hd, H)
        matrix(H, nh * hd)
        attention(nh, nkv, hd)

    def conv():
        nonlocal nbytes
        matrix(3 * H, H)
        matrix(H, H)
        nbytes += 2 * len(lens) * 2 * H * 4

    def stream(values, size):
        nonlocal nbytes
        nbytes += values * size
    ff = cfg.ff_dim if kind in ("step", "attention", "conv_layer") else 0
    if kind == "step":
        for i in range(config["num_hidden_layers"]):
            lfm_attention() if i in config["full_attn_idxs"] else conv()
            matrix(3 * ff, H)
        matrix(plan.vocab_size, H, len(lens))
        stream(len(lens) * plan.vocab_size, 4)
        return {"bytes": nbytes, "flops": flops}
    if kind == "conv_layer":
        conv()
        matrix(3 * ff, H)
        stream(2 * T * H, 4)
        return {"bytes": nbytes, "flops": flops}
    m = config.get("layers", [{}])[0].get("mixer", {})
    stream(2 * T * H, el)
    if kind == "attention":
        lfm_attention()
    elif kind in ("latent", "latent_window"):
        nh, d, r, vd, rank = m["heads"], m["dim"], m.get("rot_dim", 0), m["vdim"], m["kv_rank"]
        if kind == "latent":
            matrix(nh * (d + r) + nh, H)
        else:
            matrix(m["q_rank"], H)
            matrix(nh * (d + r), m["q_rank"])
        matrix(rank + r, H)
        matrix(nh * (d + vd), rank)
        matrix(H, nh * vd)
        stream((sum(seen) + T) * (rank + r), el)
        flops += 2.0 * nh * (d + r + vd) * pairs
    elif kind in ("experts", "gated_experts"):
        f = config["layers"][0]["mlp"]
        E, top, per = f["router"]["experts"], f["router"]["top"], (3 if kind == "gated_experts" else 2) * H
        nbytes += per * f["expert"]["ff"] * el * E * (1.0 - (1.0 - top / E) ** T)
        flops += 2.0 * per * f["expert"]["ff"] * top * T
        matrix(per, f["shared"]["ff"])
        matrix(E, H)
    elif kind == "delta":
        h, g, d, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        matrix(2 * g * d + h * vd + h, H)
        matrix(m["decay_rank"] + m["gate_rank"], H)
        matrix(h * d, m["decay_rank"])
        matrix(h * vd, m["gate_rank"])
        matrix(H, h * vd)
        stream(2 * len(lens) * h * d * vd, 4)
        flops += 8.0 * T * h * d * vd
    else:
        a, b = m["left"], m["right"]
        matrix((a["heads"] + 2 * a["kv_heads"]) * a["dim"], H)
        matrix(H, a["heads"] * a["dim"])
        attention(a["heads"], a["kv_heads"], a["dim"])
        matrix(b["heads"] * (2 * b["dim"] + b["vdim"]), H)
        matrix(H, b["heads"] * b["vdim"])
        stream(2 * len(lens) * b["heads"] * b["dim"] * b["vdim"], 4)
        flops += 6.0 * T * b["heads"] * b["dim"] * b["vdim"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the paths were measured to be off 64-bit results: 0.002 to 0.004 for a layer in 16 bits (every
    product's result is rounded to 8 bits), 0.01 for a whole model (limited to three times that), 5e-7 for the 32-bit path."""
    if case["dtype"] == "float32":
        return {"rel": 4e-6}
    return {"rel": 0.03} if case["kind"] == "step" else {"rel": 0.015}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _turn(x, positions, freqs, interleaved, amplitude=1.0):
    """x [T, heads, d]: pairs of its first 2 * len(freqs) entries turn by position * frequency."""
    n = freqs.numel()
    angle = positions.double()[:, None] * freqs[None, :]
    c, s = (amplitude * torch.cos(angle))[:, None], (amplitude * torch.sin(angle))[:, None]
    out = x.clone()
    at = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if interleaved else (slice(0, n), slice(n, 2 * n))
    u, v = x[..., at[0]], x[..., at[1]]
    out[..., at[0]], out[..., at[1]] = u * c - v * s, v * c + u * s
    return out


def _plain_freqs(base, dims):
    return float(base) ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEV) / dims)


def _by_wavelength(base, dims, sc):
    """Stretched frequencies, by how often a pair turns within the original length."""
    f = _plain_freqs(base, dims)
    if not sc:
        return f
    turns = sc["original"] / (2 * math.pi / f)
    share = ((turns - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
    return (1 - share) * f / sc["factor"] + share * f


def _by_place(base, dims, sc):
    """(stretched frequencies, by a pair's place; the factor of cosine and sine)."""
    f = _plain_freqs(base, dims)
    if not sc:
        return f, 1.0
    place = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    first, last = max(math.floor(place(sc["fast"])), 0), min(math.ceil(place(sc["slow"])), dims - 1)
    share = ((torch.arange(dims // 2, dtype=F64, device=DEV) - first) / max(last - first, 0.001)).clamp(0, 1)
    return f / sc["factor"] * share + f * (1 - share), 0.1 * math.log(sc["factor"]) + 1.0


def _each(ctx):
    """(entry, its tokens among the step's, its context)."""
    at = 0
    for b, (n, c) in enumerate(zip(ctx.q_lens, ctx.ctx_lens_host)):
        yield b, slice(at, at + n), c
        at += n


def _put(pool, table, b, first, rows):
    """rows [n, heads, width] into the pages of entry b from position `first` on."""
    at = torch.arange(first, first + rows.shape[0], device=DEV)
    pool[table[b].long()[at // PAGE], :, at % PAGE] = rows


def _take(pool, table, b, n):
    at = torch.arange(n, device=DEV)
    return pool[table[b].long()[at // PAGE], :, at % PAGE]


def _softmax_rows(q, k, v, scale, first, window=None, sinks=None):
    """q [n, heads, d] at positions first.. over k [m, groups, d], v [m, groups, e]."""
    n, nh, m = q.shape[0], q.shape[1], k.shape[0]
    back = (first + torch.arange(n, device=DEV))[:, None] - torch.arange(m, device=DEV)[None, :]
    hidden = (back < 0) | (back >= (window or 1 << 40))
    out = []
    for h in range(nh):
        g = h // (nh // k.shape[1])
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(hidden, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks[h].expand(n, 1)], dim=1)
        out.append(torch.softmax(s, dim=1)[:, :m] @ v[:, g])
    return torch.stack(out, dim=1)


def _exact_attention(x, w, p, config, ctx, table, pools):
    nh, nkv, hd, eps = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"], config["norm_eps"]
    f = _plain_freqs(config["rope_theta"], hd)
    q, k, v = ((x @ w[p + n].T).view(x.shape[0], -1, hd) for n in ("q_proj.weight", "k_proj.weight", "v_proj.weight"))
    q = _turn(_rms(q, eps, w[p + "q_layernorm.weight"]), ctx.positions, f, False)
    k = _turn(_rms(k, eps, w[p + "k_layernorm.weight"]), ctx.positions, f, False)
    out = torch.empty_like(q)
    for b, at, c in _each(ctx):
        _put(pools[0], table, b, c, k[at])
        _put(pools[1], table, b, c, v[at])
        n = c + q[at].shape[0]
        out[at] = _softmax_rows(q[at], _take(pools[0], table, b, n), _take(pools[1], table, b, n), hd ** -0.5, c)
    return out.reshape(x.shape[0], -1) @ w[p + "out_proj.weight"].T


def _exact_conv(x, w, p, ctx, state):
    H = x.shape[1]
    taps = w[p + "conv.weight"].reshape(H, -1)
    B, C, u = (x @ w[p + "in_proj.weight"].T).split(H, dim=1)
    y = _taps_over(B * u, taps, ctx, state)
    return (C * y) @ w[p + "out_proj.weight"].T


def _taps_over(u, taps, ctx, state):
    """A causal convolution of every entry's rows behind its state [slots, taps - 1, channels], which moves on."""
    n = taps.shape[1]
    y = torch.empty_like(u)
    for b, at, _ in _each(ctx):
        rows = torch.cat([state[b], u[at]])
        y[at] = sum(rows[j:j + rows.shape[0] - n + 1] * taps[:, j] for j in range(n))
        state[b] = rows[rows.shape[0] - n + 1:]
    return y


def _exact_swiglu(x, w, p):
    return (torch.nn.functional.silu(x @ w[p + "w1.weight"].T) * (x @ w[p + "w3.weight"].T)) @ w[p + "w2.weight"].T


def _exact_latent(x, w, config, ctx, table, pools, windowed):
    m, p, eps = config["layers"][0]["mixer"], "l0.mix.", config["norm"]["eps"]
    T, nh, d, r, vd, rank = x.shape[0], m["heads"], m["dim"], m.get("rot_dim", 0), m["vdim"], m["kv_rank"]
    q = (_rms(x @ w[p + "dq"].T, eps, w[p + "dq.norm"]) @ w[p + "uq"].T if windowed else x @ w[p + "q"].T).view(T, nh, d + r)
    down = x @ w[p + "dkv"].T
    rows = _rms(down[:, :rank], eps, w[p + "dkv.norm"])
    if r:
        f, amp = _by_place(m["rot"]["base"], m["rot"]["dims"], m["rot"].get("scaling"))
        turn = lambda v: _turn(v, ctx.positions, f, False, amp)
        q = torch.cat([q[..., :d], turn(q[..., d:])], dim=2)
        rows = torch.cat([rows, turn(down[:, None, rank:])[:, 0]], dim=1)
    out = torch.empty(T, nh, vd, dtype=F64, device=DEV)
    for b, at, c in _each(ctx):
        _put(pools[0], table, b, c, rows[at][:, None])
        kept = _take(pools[0], table, b, c + rows[at].shape[0])[:, 0]
        k = (kept[:, :rank] @ w[p + "uk"].T).view(-1, nh, d)
        if r:
            k = torch.cat([k, kept[:, None, rank:].expand(-1, nh, r)], dim=2)
        v = (kept[:, :rank] @ w[p + "uv"].T).view(-1, nh, vd)
        out[at] = _softmax_rows(q[at], k, v, m["scale"], c, m["mask"]["size"] if windowed else None, w[p + "sink"] if windowed else None)
    if not windowed:
        out = out * torch.sigmoid(x @ w[p + "g"].T)[:, :, None]
    return out.reshape(T, -1) @ w[p + "o"].T


def _best(values, n):
    """True at the n largest of every row (the first of equal ones)."""
    order = torch.sort(values, dim=1, descending=True, stable=True).indices[:, :n]
    return torch.zeros_like(values, dtype=torch.bool).scatter_(1, order, True)


def _exact_experts(x, w, config, gated):
    f, p = config["layers"][0]["mlp"], "l0.mlp."
    r, T = f["router"], x.shape[0]
    z = x @ w[p + "router"].double().T
    s = torch.softmax(z, 1) if gated else torch.sigmoid(z)
    c = s if gated else s + w[p + "correction"].double()
    n = r["groups"]["count"]
    runs = c.view(T, n, -1)
    score = runs.amax(-1) if gated else runs.sort(-1, descending=True).values[..., :2].sum(-1)
    c = c.masked_fill(~_best(score, r["groups"]["keep"]).repeat_interleave(r["experts"] // n, dim=1), -math.inf)
    chosen = _best(c, r["top"])
    weight = torch.where(chosen, s, torch.zeros_like(s))
    weight = weight / (weight.sum(1, keepdim=True) + 1e-20) * r.get("scale", 1.0)

    def expert(h, q, limit):
        if not gated:
            return torch.nn.functional.gelu(h @ w[q + "up"].double().T) @ w[q + "down"].double().T
        g, u = (h @ w[q + "gate"].double().T).clamp(max=limit), (h @ w[q + "up"].double().T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[q + "down"].double().T
    out = expert(x, p + "shared.", f["shared"].get("limit"))
    if not gated:
        out = out * torch.sigmoid(x @ w[p + "shared.sg"].double().T)
    for e in range(r["experts"]):
        rows = chosen[:, e].nonzero()[:, 0]
        if rows.numel():
            out[rows] += weight[rows, e, None] * expert(x[rows], p + "e%d." % e, f["expert"].get("limit"))
    return out


def _exact_delta(x, w, config, ctx, states):
    m, p, eps = config["layers"][0]["mixer"], "l0.mix.", config["norm"]["eps"]
    T, h, g, d, vd = x.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    u = torch.cat([x @ w[p + n].T for n in ("q", "k", "v")], dim=1)
    u = torch.nn.functional.silu(_taps_over(u, torch.cat([w[p + n + ".conv"] for n in ("q", "k", "v")]), ctx, states[0]))
    q, k, v = u[:, :g * d].view(T, g, d), u[:, g * d:2 * g * d].view(T, g, d), u[:, 2 * g * d:].view(T, h, vd)
    unit = lambda a: (a / torch.sqrt((a * a).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(h // g, dim=1)
    q, k = unit(q) * d ** -0.5, unit(k)
    beta = torch.sigmoid(x @ w[p + "b"].T)
    a = (x @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "dt_bias"]
    decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * torch.nn.functional.softplus(a).view(T, h, d))
    out = torch.empty(T, h, vd, dtype=F64, device=DEV)
    for b, at, _ in _each(ctx):
        S = states[1][b]
        for t in range(at.start, at.stop):
            S = decay[t][:, :, None] * S
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None]
            out[t] = torch.einsum("hdv,hd->hv", S, q[t])
        states[1][b] = S
    gate = torch.sigmoid((x @ w[p + "g1"].T) @ w[p + "g2"].T).view(T, h, vd)
    return (_rms(out, eps, w[p + "norm"]) * gate).reshape(T, -1) @ w[p + "o"].T


def _exact_parallel(x, w, config, ctx, table, caches):
    m, eps = config["layers"][0]["mixer"], config["norm"]["eps"]
    a, r, T = m["left"], m["right"], x.shape[0]
    # what the binding holds, in the mixer's order: keys, values, the convolutions' rows; the recurrence's state
    keys, values, conv, state = caches
    p, widths = "l0.mix.left.", [a["heads"] * a["dim"], a["kv_heads"] * a["dim"], a["kv_heads"] * a["vdim"]]
    u = torch.cat([x @ w[p + n].T + w[p + n + ".b"] for n in ("q", "k", "v")], dim=1)
    q, k, v = _taps_over(u, torch.cat([w[p + n + ".conv"] for n in ("q", "k", "v")]), ctx, conv).split(widths, dim=1)
    q = _rms(q, eps, w[p + "q.norm"]).view(T, -1, a["dim"])
    k = _rms(k, eps, w[p + "k.norm"]).view(T, -1, a["dim"])
    f, fv = _by_wavelength(a["rot"]["base"], a["rot"]["dims"], a["rot"].get("scaling")), _plain_freqs(a["rot"]["base"], a["vdim"])
    q, k = _turn(q, ctx.positions, f, True), _turn(k, ctx.positions, f, True)
    v = _turn(v.reshape(T, -1, a["vdim"]), ctx.positions, fv, True)
    o = torch.empty(T, a["heads"], a["vdim"], dtype=F64, device=DEV)
    for b, at, c in _each(ctx):
        _put(keys, table, b, c, k[at])
        _put(values, table, b, c, v[at])
        n = c + k[at].shape[0]
        o[at] = _softmax_rows(q[at], _take(keys, table, b, n), _take(values, table, b, n), a["scale"], c, a["mask"]["size"], w[p + "sink"])
    left = _turn(o, ctx.positions, -fv, True).reshape(T, -1) @ w[p + "o"].T
    p, h, d, vd = "l0.mix.right.", r["heads"], r["dim"], r["vdim"]
    q = torch.nn.functional.silu(x @ w[p + "q"].T).view(T, h, d)
    v = (x @ w[p + "v"].T).view(T, h, vd)
    low = w[p + "lower"]
    f = (low + (1 - low) * torch.sigmoid(x @ w[p + "f"].T + w[p + "f.b"])).view(T, h, d)
    o = torch.empty(T, h, vd, dtype=F64, device=DEV)
    for b, at, _ in _each(ctx):
        S = state[b]
        for t in range(at.start, at.stop):
            S = f[t][:, :, None] * S + (1 - f[t])[:, :, None] * v[t][:, None]
            o[t] = torch.einsum("hdv,hd->hv", S, q[t])
        state[b] = S
    right = _rms(o, eps, w[p + "norm"]).reshape(T, -1) @ w[p + "o"].T
    return 0.5 * (_rms(left, eps, w["l0.mix.left.out"]) + _rms(right, eps, w["l0.mix.right.out"]))


def _exact_step(case, seed):
    """Every request's whole sequence through the model, the last place's logits."""
    plan, tensors = _inputs(case, seed)
    config = _config(case)
    lens, ctxs = _lengths(case)
    whole, table, pages = _context(dict(case, requests=1, tokens=1, context=0, ragged=False), _dtype(case))
    logits = []
    for row in _tokens(seed, lens, ctxs, plan.vocab_size):
        T, nkv, hd = len(row), config["num_key_value_heads"], config["head_dim"]
        whole.q_lens, whole.ctx_lens_host, whole.positions = [T], [0], torch.arange(T, device=DEV)
        table = torch.arange(-(-T // PAGE), device=DEV)[None]
        x = tensors["model.embed_tokens.weight"][torch.tensor(row, device=DEV)].double()
        for i in range(config["num_hidden_layers"]):
            p = "model.layers.%d." % i
            w = {n: t.double() for n, t in tensors.items() if n.startswith(p)}
            y = _rms(x, config["norm_eps"], w[p + "operator_norm.weight"])
            if i in config["full_attn_idxs"]:
                pools = [torch.zeros(table.shape[1], nkv, PAGE, hd, dtype=F64, device=DEV) for _ in range(2)]
                x = x + _exact_attention(y, w, p + "self_attn.", config, whole, table, pools)
            else:
                x = x + _exact_conv(y, w, p + "conv.", whole, torch.zeros(1, config["conv_L_cache"] - 1, x.shape[1], dtype=F64, device=DEV))
            x = x + _exact_swiglu(_rms(x, config["norm_eps"], w[p + "ffn_norm.weight"]), w, p + "feed_forward.")
        last = _rms(x[-1:], config["norm_eps"], tensors["model.embedding_norm.weight"].double())
        logits.append(last @ tensors["model.embed_tokens.weight"].double().T)
    return torch.cat(logits)


def exact(case, seed):
    kind, config = case["kind"], _config(case)
    if kind == "step":
        return _exact_step(case, seed)
    plan, w, ctx, cache, x = _raw(case, seed)
    if kind in ("experts", "gated_experts"):
        return _exact_experts(x.double(), w, config, kind == "gated_experts")
    w, x = {n: t.double() for n, t in w.items()}, x.double()
    caches = [t.double() for t in _caches(cache)]
    table = next((b.block_table for b in (cache.parts or (cache,)) if b.block_table is not None), None)
    if kind == "attention":
        y = _exact_attention(x, w, "model.layers.0.self_attn.", config, ctx, table, caches)
    elif kind == "conv_layer":
        p, eps = "model.layers.0.", config["norm_eps"]
        x = _random(seed, "stream", (ctx.T, plan.hidden_size), 1.0).double()
        y = x + _exact_conv(_rms(x, eps, w[p + "operator_norm.weight"]), w, p + "conv.", ctx, caches[0])
        y = y + _exact_swiglu(_rms(y, eps, w[p + "ffn_norm.weight"]), w, p + "feed_forward.")
    elif kind in ("latent", "latent_window"):
        y = _exact_latent(x, w, config, ctx, table, caches, kind == "latent_window")
    elif kind == "delta":
        y = _exact_delta(x, w, config, ctx, caches)
    else:
        y = _exact_parallel(x, w, config, ctx, table, caches)
    return [y] + caches
