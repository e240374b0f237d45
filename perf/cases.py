"""Performance cases: the work that users of this framework have it do, through its public entry points.

Four families, each over a range of sizes:

* ``layer``: a decode step of one paged decoder layer, ``BlockTopkDecoderLayer`` (block top-k attention) or
  ``DecoderLayer`` (dense attention), replayed from the CUDA graph that ``make_graphed`` returns.  The shapes are those of
  the repository's configurations: one KV-head shard of Qwen3-8B or Qwen3-32B, and the small fp32 layer.
* ``prompt``: new tokens of one or several sequences written into the paged cache and attended (``ops.append_tokens`` and
  ``ops.prefill_attention``): whole prompts, and portions on top of what the cache holds.
* ``gifetar``, ``munadra``: the two models with free layer sizes, a prompt (whole or in portions, logits at the places
  asked for) and a decode step of a batch (one captured step, as the engine replays it).  Gifetar with two attention
  layers, Munadra with a recurrent layer, a dense feed-forward and a latent-attention layer.
* ``experts``: the mixture-of-experts feed-forward of either model on the embedded tokens of a step, between the two row
  kernels around it.  It stands by itself because a router's near ties would otherwise hang on the roundings of all
  layers in front of it, and two correct results could differ in whole rows.

Every input comes from a seed; the random weights have the models' usual scales, caches hold N(0, 1) values.
"""
import math
import random

import numpy as np
import torch

import kinetics_b200 as kb
from kinetics_b200 import layer_ops, ops
from kinetics_b200.gifetar import Gifetar
from kinetics_b200.munadra import Munadra

PAGE, HEAD = 16, 128            # the paged decoder layers: tokens of a page, columns of a head
VOCAB = 32768                   # the models' vocabulary in this repository's benchmark
PLACES = 64                     # places of a prompt whose logits are asked for
CHUNK = 64                      # sequences whose cache is made at once

# The models' sizes: the two of the repository's benchmark and a small one.
SIZES = {
    "w1024": dict(width=1024, heads=8, kv_heads=2, blocks=4, experts=16, top=4, ff=512),
    "w2048": dict(width=2048, heads=16, kv_heads=4, blocks=8, experts=64, top=8, ff=768),
    "w4096": dict(width=4096, heads=32, kv_heads=8, blocks=16, experts=32, top=4, ff=2048),
}
DIM, VDIM, SOFTCAP, DIFF, MULT = 64, 128, 30.0, 0.3, 0.3                     # Gifetar's constants
NOPE, ROT, RANK, TAPS, CAP, DENSE = 128, 64, 512, 4, 30.0, 3                # Munadra's
LIMIT, SLOPE, SHIFT = 7.0, 1.702, 1.0                                       # and of its experts' gated activation
BASE, STRETCH = 1e5, dict(factor=4.0, original=4096, fast=32.0, slow=1.0)
EPS = 1e-6


def listed():
    layer = lambda name, **kw: dict(dict(name=name, family="layer", topk=0, ragged=False, dtype="bfloat16"), **kw)
    return [
        # the smallest step there is: four sequences, fp32, one KV head; its time is launches and latency
        layer("step fp32 b4", model="cfg1", tp=1, batch=4, context=2048, topk=16, dtype="float32"),
        # a served batch of moderate contexts on one of eight tensor-parallel ranks
        layer("step b256 8k", model="Qwen3-8B", tp=8, batch=256, context=8192, topk=64),
        # ragged contexts of a continuous batch, eight query heads per KV head, fragmented page table
        layer("step ragged b1024 g8", model="Qwen3-32B", tp=8, batch=1024, context=16384, topk=64, ragged=True),
        # the throughput shape: a large batch of long contexts
        layer("step b2048 32k", model="Qwen3-8B", tp=8, batch=2048, context=32768, topk=128),
        # a long prompt of the 8B shape at once
        dict(name="prompt 8k", family="prompt", sequences=1, new=8192, history=0, heads=32, kv_heads=8),
        # ragged portions of several prompts on top of what their caches hold
        dict(name="portions 6x700", family="prompt", sequences=6, new=700, history=5000, heads=16, kv_heads=8),
        # a long prompt of the differential-attention model
        dict(name="gifetar prompt 8k", family="gifetar", size="w2048", phase="prompt", tokens=8192, portion=0),
        # its decode step at the benchmark's batch
        dict(name="gifetar decode b64", family="gifetar", size="w2048", phase="decode", batch=64, context=8192, ragged=False),
        # a long prompt of the latent-attention and recurrence model, the largest work here
        dict(name="munadra prompt 8k", family="munadra", size="w4096", phase="prompt", tokens=8192, portion=0),
        # its decode step at a continuous batch's ragged contexts
        dict(name="munadra decode b128", family="munadra", size="w4096", phase="decode", batch=128, context=4096, ragged=True),
        # the experts of a long prompt: every expert has a thousand rows
        dict(name="experts 8k", family="experts", size="w2048", style="gifetar", phase="prompt", tokens=8192),
        # the experts of a decode step: a few rows each, so their weights are the time
        dict(name="experts b64", family="experts", size="w4096", style="munadra", phase="decode", tokens=64),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(("layer", "layer", "prompt", "gifetar", "munadra", "experts", "experts"))
    if family == "layer":
        context = _spread(rng, 300, 32768)
        case = dict(family=family, model=rng.choice(("Qwen3-8B", "Qwen3-8B", "Qwen3-32B")), tp=rng.choice((4, 8, 8)),
                    ragged=rng.random() < 0.5, dtype="bfloat16", context=context, topk=0)
        top = 2048 * 32768 if rng.random() < 0.7 else 512 * 8192             # the second: dense
        case["batch"] = _spread(rng, 3, min(2048, max(4, top * (case["tp"] // 4) // (2 * context))))
        if top == 2048 * 32768:
            case["topk"] = _spread(rng, 8, 160)
        if rng.random() < 0.15:                                              # the fp32 form, at small sizes
            case.update(model="cfg1", tp=1, dtype="float32", batch=rng.randint(1, 16), context=min(context, 4096))
        return case
    if family == "prompt":
        heads, kv_heads = rng.choice(((32, 8), (16, 8), (8, 1), (8, 8)))
        sequences = rng.randint(1, 8)
        new = _spread(rng, 17, 8192 // sequences)
        return dict(family=family, sequences=sequences, new=new, history=rng.choice((0, _spread(rng, 30, 8192 // sequences))),
                    heads=heads, kv_heads=kv_heads)
    size = rng.choice(tuple(SIZES))
    if family == "experts":
        phase = rng.choice(("prompt", "decode"))
        tokens = _spread(rng, 65, 8192) if phase == "prompt" else _spread(rng, 1, 256)
        return dict(family=family, size=size, style=rng.choice(("gifetar", "munadra")), phase=phase, tokens=tokens)
    if rng.random() < 0.5:
        tokens = _spread(rng, 65, 4096 if size == "w4096" else 8192)
        return dict(family=family, size=size, phase="prompt", tokens=tokens, portion=rng.choice((0, 0, max(64, tokens // 3))))
    context = _spread(rng, 150, 16384)
    return dict(family=family, size=size, phase="decode", context=context, ragged=rng.random() < 0.5,
                batch=_spread(rng, 1, max(2, min(128, 128 * 4096 // context))))


# ---------------------------------------------------------------- inputs, from the seed alone
class _Source:
    """Random tensors on the GPU; `part` names an independent stream of the seed."""

    def __init__(self, seed, part=0):
        self.g = torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + part) % (1 << 62))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        t = torch.empty(*shape, dtype=dtype, device="cuda").normal_(generator=self.g)
        return t if std == 1.0 and mean == 0.0 else t.mul_(std).add_(mean)

    def tokens(self, *shape):
        return torch.randint(0, VOCAB, shape, generator=self.g, device="cuda")


def _contexts(case):
    """Tokens that each sequence's cache holds in front of the step: a property of the case, the same for every seed."""
    n, top = case["batch"], case["context"]
    if not case["ragged"]:
        return [top] * n
    r = random.Random(n * 100003 + top)
    low = max(1, top // 16)
    return [r.randint(low, top) for _ in range(n)]


# ---- paged decoder layers
def _layer_dtype(case):
    return getattr(torch, case["dtype"])


def _layer_sizes(case):
    c = kb.get_config(case["model"])
    return c, c.num_attention_heads // case["tp"], c.num_key_value_heads // case["tp"], c.intermediate_size // case["tp"]


def _layer_contexts(case):
    lens = _contexts(case)
    return lens if case["ragged"] else [n // PAGE * PAGE for n in lens]


def _layer_inputs(case, seed):
    """(weights by parameter name, hidden states)."""
    c, hq, hkv, inter = _layer_sizes(case)
    s, dtype, H = _Source(seed), _layer_dtype(case), c.hidden_size
    rows = {"wqkv.weight": ((hq + 2 * hkv) * HEAD, H), "wo.weight": (H, hq * HEAD), "up_proj.weight": (inter, H),
            "gate_proj.weight": (inter, H), "down_proj.weight": (H, inter)}
    w = {name: s.normal(*shape, std=0.02, dtype=dtype) for name, shape in rows.items()}
    w["wqkv.bias"] = s.normal((hq + 2 * hkv) * HEAD, std=0.02, dtype=dtype)
    for name, n in (("qnorm_weight", HEAD), ("knorm_weight", HEAD), ("input_layernorm_weight", H),
                    ("post_attention_layernorm_weight", H)):
        w[name] = s.normal(n, std=0.1, mean=1.0, dtype=dtype)
    return w, s.normal(case["batch"], 1, H, dtype=dtype)


def _layer_pages(case, seed, chunk, pages):
    """The pages [pages, 2, PAGE, kv heads, HEAD] of one chunk of sequences, in the order of their page lists."""
    return _Source(seed, 1 + chunk).normal(pages, 2, PAGE, _layer_sizes(case)[2], HEAD, dtype=_layer_dtype(case))


def _prepare_layer(case, seed):
    config = _layer_sizes(case)[0]
    lens, dtype = _layer_contexts(case), _layer_dtype(case)
    most = (max(lens) // PAGE + 1) * PAGE
    kw = dict(config=config, world_size=case["tp"], batch_size=case["batch"], prefix_len=max(lens), max_len=most,
              page_size=PAGE, device="cuda", dtype=dtype)
    if case["ragged"]:
        kw.update(context_lens=lens, page_table="random")
    kv = torch.zeros(most // PAGE * case["batch"], 2, PAGE, _layer_sizes(case)[2], HEAD, dtype=dtype, device="cuda")
    if case["topk"]:
        layer = kb.BlockTopkDecoderLayer(topk_page=case["topk"], kv_cache=kv, **kw)
    else:
        layer = kb.DecoderLayer(kv_cache=kv, **kw)
    weights, hidden = _layer_inputs(case, seed)
    layer.eval().to("cuda", dtype=dtype)
    with torch.no_grad():
        for name, p in layer.named_parameters():
            p.copy_(weights[name])
    starts = np.concatenate(([0], np.cumsum([n // PAGE + 1 for n in lens])))
    for c in range(0, case["batch"], CHUNK):
        a, b = int(starts[c]), int(starts[min(c + CHUNK, case["batch"])])
        kv[layer.paged_kv_indices[a:b].long()] = _layer_pages(case, seed, c, b - a)
    if case["topk"]:
        layer.rebuild_summaries()
    _, out, graph = layer.make_graphed(hidden)
    return dict(layer=layer, graph=graph, out=out)


def _run_layer(state):
    state["graph"].replay()
    return {"hidden": state["out"], **({"pages": state["layer"].topk_page_indices} if hasattr(state["layer"], "topk_page") else {})}


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _exact_layer(case, seed):
    c, hq, hkv, _ = _layer_sizes(case)
    w, hidden = _layer_inputs(case, seed)
    w = {k: v.double() for k, v in w.items()}
    x = hidden.double().view(case["batch"], -1)
    qkv = _rms(x, w["input_layernorm_weight"], c.rms_norm_eps) @ w["wqkv.weight"].t() + w["wqkv.bias"]
    q, k, v = (t.reshape(case["batch"], -1, HEAD) for t in qkv.split((hq * HEAD, hkv * HEAD, hkv * HEAD), dim=1))
    q, k = _rms(q, w["qnorm_weight"], c.rms_norm_eps), _rms(k, w["knorm_weight"], c.rms_norm_eps)
    lens, out = _layer_contexts(case), torch.empty(case["batch"], hq, HEAD, dtype=torch.float64, device="cuda")
    for first in range(0, case["batch"], CHUNK):
        rows = range(first, min(first + CHUNK, case["batch"]))
        counts = [lens[b] // PAGE + 1 for b in rows]
        for b, mine in zip(rows, _layer_pages(case, seed, first, sum(counts)).split(counts)):
            at = lens[b] % PAGE
            keep = torch.arange(len(mine) - 1, device="cuda").expand(hkv, -1)
            qb = q[b].view(hkv, -1, HEAD)
            if case["topk"] and case["topk"] < len(mine) - 1:                # page summary: the mean key, in the cache's type
                mean = mine[:-1, 0].double().mean(1).to(mine.dtype).double()
                score = torch.einsum("hd,phd->hp", qb.mean(1), mean)
                keep = score.topk(case["topk"], dim=1).indices
            last = mine[-1].double()
            last[0, at], last[1, at] = k[b], v[b]
            for h in range(hkv):
                kk, vv = (torch.cat((mine[keep[h], i, :, h].double().reshape(-1, HEAD), last[i, :at + 1, h])) for i in (0, 1))
                out[b].view(hkv, -1, HEAD)[h] = torch.softmax(qb[h] @ kk.t() / math.sqrt(HEAD), dim=1) @ vv
    x = x + out.view(case["batch"], -1) @ w["wo.weight"].t()
    h = _rms(x, w["post_attention_layernorm_weight"], c.rms_norm_eps)
    gate = h @ w["gate_proj.weight"].t()
    y = x + (gate * torch.sigmoid(gate) * (h @ w["up_proj.weight"].t())) @ w["down_proj.weight"].t()
    return {"hidden": y.view(case["batch"], 1, -1), **({"pages": None} if case["topk"] else {})}


def _work_layer(case):
    c, hq, hkv, inter = _layer_sizes(case)
    size, B, H = 4 if case["dtype"] == "float32" else 2, case["batch"], c.hidden_size
    weights = H * HEAD * (2 * hq + 2 * hkv) + 3 * H * inter
    scored = attended = 0
    for n in _layer_contexts(case):
        full = n // PAGE
        if case["topk"] and case["topk"] < full:
            scored, full = scored + full, case["topk"]
        attended += full * PAGE + n % PAGE + 1
    return {"bytes": size * (weights + 2 * B * H + hkv * HEAD * (scored + 2 * attended)),
            "flops": 2 * B * weights + 2 * hkv * HEAD * scored + 4 * hq * HEAD * attended}


# ---- prompts over the paged cache
def _prompt_lengths(case):
    """(new tokens, tokens held before) of every sequence, around the case's sizes."""
    r, n = random.Random(case["new"] * 100003 + case["history"]), case["sequences"]
    if n == 1:
        return [(case["new"], case["history"])]
    near = lambda v: r.randint(max(1, v // 2), v + v // 2) if v else 0
    return [(near(case["new"]), near(case["history"])) for _ in range(n)]


def _prompt_inputs(case, seed):
    """(q, k, v of the new tokens, keys and values held before), packed by sequence."""
    s, hkv = _Source(seed), case["kv_heads"]
    new, held = (sum(v) for v in zip(*_prompt_lengths(case)))
    return s.normal(new, case["heads"], HEAD), s.normal(new, hkv, HEAD), s.normal(new, hkv, HEAD), s.normal(held, 2, hkv, HEAD)


def _prepare_prompt(case, seed):
    lengths, hkv = _prompt_lengths(case), case["kv_heads"]
    q, k, v, held = _prompt_inputs(case, seed)
    pages = [(n + h + PAGE - 1) // PAGE for n, h in lengths]
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    total = sum(pages)
    table = torch.randperm(total, generator=_Source(seed, 1).g, device="cuda").int()
    indptr = i32([0] + np.cumsum(pages).tolist())
    last = i32([(n + h - 1) % PAGE + 1 for n, h in lengths])
    cache = torch.zeros(total, 2, PAGE, hkv, HEAD, dtype=torch.bfloat16, device="cuda")
    summaries = torch.zeros(len(lengths), hkv, max(pages), HEAD, dtype=torch.bfloat16, device="cuda")
    held_indptr = i32([0] + np.cumsum([h for _, h in lengths]).tolist())
    if held.shape[0]:                                                        # what earlier portions left in the cache
        before = [(h + PAGE - 1) // PAGE for _, h in lengths]
        cut = torch.cat([table[a:a + n] for a, n in zip(indptr.tolist(), before)])
        ops.append_tokens(held[:, 0].contiguous(), held[:, 1].contiguous(), held_indptr, cache, summaries, cut,
                          i32([0] + np.cumsum(before).tolist()), i32([(h - 1) % PAGE + 1 if h else 0 for _, h in lengths]))
    new = [n for n, _ in lengths]
    return dict(q=q, k=k, v=v, indptr=i32([0] + np.cumsum(new).tolist()), most=max(new), cache=cache, summaries=summaries,
                table=(table, indptr, last))


def _run_prompt(s):
    ops.append_tokens(s["k"], s["v"], s["indptr"], s["cache"], s["summaries"], *s["table"])
    return {"out": ops.prefill_attention(s["q"], s["indptr"], s["most"], s["cache"], *s["table"]), "summaries": s["summaries"]}


def _exact_prompt(case, seed):
    lengths, hkv, group = _prompt_lengths(case), case["kv_heads"], case["heads"] // case["kv_heads"]
    q, k, v, held = _prompt_inputs(case, seed)
    out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    most = max((n + h + PAGE - 1) // PAGE for n, h in lengths)
    summaries = torch.zeros(len(lengths), hkv, most, HEAD, dtype=torch.float64, device="cuda")
    new, held = [n for n, _ in lengths], held.split([h for _, h in lengths])
    for b, (qb, kb_, vb, ob) in enumerate(zip(q.split(new), k.split(new), v.split(new), out.split(new))):
        kk, vv = torch.cat((held[b][:, 0], kb_)).double(), torch.cat((held[b][:, 1], vb)).double()
        total = kk.shape[0]
        full = torch.cat((kk, kk.new_zeros(-total % PAGE, hkv, HEAD))).view(-1, PAGE, hkv, HEAD).sum(1)
        fill = torch.full((full.shape[0], 1, 1), float(PAGE), dtype=torch.float64, device="cuda")
        fill[-1] = (total - 1) % PAGE + 1
        summaries[b, :, :full.shape[0]] = (full / fill).transpose(0, 1)
        for h in range(case["heads"]):
            ob[:, h] = _causal(qb[:, h].double() / math.sqrt(HEAD), kk[:, h // group], vv[:, h // group])
    return {"out": out, "summaries": summaries}


def _causal(q, k, v, cap=0.0, sink=None, step=2048):
    """softmax(q k^T) v of the newest rows q [n, d] over k [total, d], each row up to its own key; cap: soft cap of the
    scores; sink: exp(sink) joins the denominators."""
    out = torch.empty(q.shape[0], v.shape[1], dtype=q.dtype, device=q.device)
    first = k.shape[0] - q.shape[0]
    for a in range(0, q.shape[0], step):
        b = min(a + step, q.shape[0])
        seen = first + b
        s = q[a:b] @ k[:seen].t()
        s = cap * torch.tanh(s / cap) if cap else s
        at = torch.arange(seen, device=q.device)
        s = s.masked_fill(at[None] > first + torch.arange(a, b, device=q.device)[:, None], -math.inf)
        if sink is not None:
            s = torch.cat((s, sink.expand(b - a, 1)), dim=1)
        out[a:b] = torch.softmax(s, dim=1)[:, :seen] @ v[:seen]
    return out


def _work_prompt(case):
    lengths = _prompt_lengths(case)
    pairs = sum(n * h + n * (n + 1) // 2 for n, h in lengths)
    new, seen = sum(n for n, _ in lengths), sum(n + h for n, h in lengths)
    rows = 2 * new * case["heads"] + 2 * new * case["kv_heads"] + 2 * seen * case["kv_heads"]
    return {"bytes": 2 * HEAD * rows, "flops": 4 * HEAD * case["heads"] * pairs}


# ---- the models: configuration and weights under the checkpoint's names
def _model_config(case):
    z = SIZES[case["size"]]
    raw = {"vocab": VOCAB, "width": z["width"], "norm": {"eps": EPS}}
    if case["family"] == "gifetar":
        mixer = {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": DIM, "vdim": VDIM, "scale": DIM ** -0.5,
                 "softcap": SOFTCAP, "diff": DIFF, "q_temp": {"coef": 0.1, "every": 2048}}
        return dict(raw, residual_mult=MULT, layers=[{"type": "attention", "mixer": mixer, "mlp": None}] * 2)
    rec = {"width": z["width"], "blocks": z["blocks"], "conv": TAPS}
    lat = {"heads": z["heads"], "dim": NOPE, "rot_dim": ROT, "vdim": VDIM, "kv_rank": RANK, "scale": (NOPE + ROT) ** -0.5,
           "rot": {"base": BASE, "dims": ROT, "scaling": STRETCH}}
    return dict(raw, embedding={"scale": 1.0}, logit_scale=1.0, logit_softcap=CAP,
                layers=[{"type": "rglru", "mixer": rec, "mlp": {"kind": "dense", "ff": DENSE * z["width"]}},
                        {"type": "latent_attention", "mixer": lat, "mlp": None}])


def _model_weights(case, seed):
    z, s, W = SIZES[case["size"]], _Source(seed), {}
    C, H, gifetar = z["width"], z["heads"], case["family"] == "gifetar"

    def put(name, *shape, std=None, mean=0.0):
        W[name] = s.normal(*shape, std=shape[-1] ** -0.5 if std is None else std, mean=mean)

    def norm(name):
        put(name, C, std=0.1, mean=1.0 if gifetar else 0.0)
        if gifetar:
            put(name + ".b", C, std=0.1)

    put("embed", VOCAB, C, std=1.0)
    norm("final.norm")
    for i in range(2):
        p, m = f"l{i}.", f"l{i}.mix."
        for n in ("norm1", "norm1b") if gifetar else ("norm1", "norm2")[:2 - i]:
            norm(p + n)
        if gifetar:
            for n, rows in (("q", H * 2 * DIM), ("k", z["kv_heads"] * 2 * DIM), ("v", z["kv_heads"] * VDIM)):
                put(m + n, rows, C)
                put(f"{m}{n}.b", rows, std=0.1)
            for n in ("lq1", "lk1", "lq2", "lk2"):
                put(m + n, DIM, std=0.1)
            put(m + "o", C, H * VDIM)
        elif i == 0:
            for b in ("y", "x"):
                put(m + b, C, C)
                put(f"{m}{b}.b", C, std=0.1)
            put(m + "conv", C, TAPS)
            put(m + "conv.b", C, std=0.1)
            for r in ("ra", "ri"):
                put(m + r, z["blocks"], C // z["blocks"], C // z["blocks"])
                put(f"{m}{r}.b", C, std=0.5)
            put(m + "lam", C, std=1.5, mean=-4.0)
            put(m + "o", C, C)
            put(p + "mlp.gate", DENSE * C, C)
            put(p + "mlp.up", DENSE * C, C)
            put(p + "mlp.down", C, DENSE * C)
        else:
            put(m + "q", H * (NOPE + ROT), C)
            put(m + "dkv", RANK + ROT, C)
            put(m + "dkv.norm", RANK, std=0.1, mean=1.0)
            put(m + "uk", H * NOPE, RANK)
            put(m + "uv", H * VDIM, RANK)
            put(m + "sink", H, std=1.0)
            put(m + "g", H, C)
            put(m + "o", C, H * VDIM)
    return W


def _model_tokens(case, seed):
    return _Source(seed, 1).tokens(1, case["tokens"]) if case["phase"] == "prompt" else _Source(seed, 1).tokens(case["batch"], 1)


def _model_cache(case, seed, layer, pages, page):
    """What the pages of one layer hold in front of a decode step, in the order of the sequences' page lists: (keys, values)
    of Gifetar, (latent rows,) of Munadra."""
    s, kv_heads = _Source(seed, 2 + layer), SIZES[case["size"]]["kv_heads"]
    if case["family"] == "gifetar":
        return s.normal(pages, kv_heads * 2, page, DIM), s.normal(pages, kv_heads, page, VDIM)
    return (s.normal(pages, 1, page, RANK + ROT),)


def _model_recurrence(case, seed):
    """Munadra's state and the newest inputs of its convolution, per sequence."""
    s, C = _Source(seed, 2), SIZES[case["size"]]["width"]
    return s.normal(case["batch"], C, dtype=torch.float32), s.normal(case["batch"], TAPS, C)


def _wanted(case):
    """The places of a prompt's last portion whose logits are asked for."""
    n = case["tokens"] % case["portion"] or case["portion"] if case["portion"] else case["tokens"]
    return [n - 1 - i * n // PLACES for i in range(PLACES)][::-1] if n >= PLACES else list(range(n))


def _prepare_model(case, seed):
    kind = Gifetar if case["family"] == "gifetar" else Munadra
    model = kind(kind.from_config(_model_config(case)), _model_weights(case, seed), "cuda")
    ids = _model_tokens(case, seed)
    if case["phase"] == "prompt":
        n, portion = case["tokens"], case["portion"] or case["tokens"]
        at = torch.arange(n, device="cuda")[None]
        cuts = [(a, min(a + portion, n)) for a in range(0, n, portion)]
        return dict(case=case, model=model, kv=model.new_cache(1, n + 64), slot=torch.tensor([0], device="cuda"),
                    parts=[(ids[:, a:b], at[:, a:b]) for a, b in cuts], rows=_wanted(case))
    B, lens = case["batch"], _contexts(case)
    kv, slots = model.new_cache(B, max(lens) + 64), list(range(B))
    kv.assume_filled(dict(enumerate(lens)), headroom=8)
    kv.prepare_step(slots)
    pages = kv.pool.export(slots)[0].long().cuda()
    for i in range(2):
        if kv.k_pages[i] is not None:
            for whole, mine in zip((kv.k_pages[i], kv.v_pages[i]), _model_cache(case, seed, i, len(pages), kv.page_size)):
                whole[pages] = mine
    at, batch_idx = torch.tensor(lens, device="cuda")[:, None], torch.arange(B, device="cuda")
    step = lambda: model.inference(ids, at, batch_idx, kv)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        logits = step()
    kv.end_step()
    states = [s for s in kv.states if s is not None]
    if states:
        state, ring = _model_recurrence(case, seed)
        states[0].copy_(state)
        kv.rings[0].copy_(ring)
    return dict(case=case, model=model, kv=kv, graph=graph, logits=logits, states=states, ids=ids, at=at, batch_idx=batch_idx)


def _run_model(s):
    if s["case"]["phase"] == "decode":
        s["graph"].replay()
        return {"logits": s["logits"], "states": s["states"]}
    model, kv, n = s["model"], s["kv"], s["case"]["tokens"]
    kv.clear_cache(0)
    kv.admit(0, n, n)
    kv.begin_step([0])
    logits = None
    for i, (ids, at) in enumerate(s["parts"]):
        logits = model.inference(ids, at, s["slot"], kv, rows=s["rows"] if i + 1 == len(s["parts"]) else [])
    return {"logits": logits, "states": [t for t in kv.states if t is not None]}


def _work_model(case):
    z = SIZES[case["size"]]
    C, H, gifetar = z["width"], z["heads"], case["family"] == "gifetar"
    if case["phase"] == "prompt":
        rows, seen = case["tokens"], 0
        pairs, asked = rows * (rows + 1) // 2, len(_wanted(case))
    else:
        rows, seen = case["batch"], sum(_contexts(case))
        pairs, asked = seen + rows, rows
    if gifetar:
        weights = 2 * C * (H + z["kv_heads"]) * (2 * DIM + VDIM)
    else:
        weights = 3 * C * C + 2 * C * C // z["blocks"] + 3 * DENSE * C * C + C * (H * (NOPE + ROT + VDIM + 1) + RANK + ROT) + \
            H * (NOPE + VDIM) * RANK
    if gifetar:
        cache, products = 2 * z["kv_heads"] * (2 * DIM + VDIM), 2 * 4 * H * (DIM + VDIM) * pairs
    else:
        cache = RANK + ROT
        products = 2 * H * pairs * (NOPE + ROT + VDIM if case["phase"] == "prompt" else 2 * RANK + ROT)
    state = 0 if gifetar else C * (2 * 4 + TAPS * 2) * (rows if case["phase"] == "decode" else 1)
    return {"bytes": 2 * (weights + VOCAB * C) + 2 * cache * (seen + rows) + 4 * asked * VOCAB + 2 * rows * C + state,
            "flops": 2 * rows * weights + 2 * asked * VOCAB * C + products}


# ---- the models in 64 bits
def _exact_model(case, seed):
    """Both models as their formulas give them; logits of the asked places, and Munadra's state behind the step."""
    W, gifetar = _model_weights(case, seed), case["family"] == "gifetar"
    w = lambda name: W[name].double()
    ids = _model_tokens(case, seed)
    prompt = case["phase"] == "prompt"
    lens = [0] if prompt else _contexts(case)
    at = torch.arange(ids.numel(), device="cuda") if prompt else torch.tensor(lens, device="cuda")
    x, states = w("embed")[ids.reshape(-1)], []

    def norm(x, name):
        if gifetar:
            x = x - x.mean(-1, keepdim=True)
        y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
        return y * w(name) + w(name + ".b") if gifetar else y * (1 + w(name))

    for i in range(2):
        p = f"l{i}."
        h = norm(x, p + "norm1") if gifetar else x
        if gifetar:
            y = _exact_differential(case, seed, i, h, w, p + "mix.", at, lens)
        elif i == 0:
            y, state = _exact_recurrence(case, seed, h, w, p + "mix.", at)
            states.append(state)
        else:
            y = _exact_latent(case, seed, i, h, w, p + "mix.", at, lens)
        x = x + (MULT * norm(y, p + "norm1b") if gifetar else norm(y, p + "norm1"))
        if p + "mlp.gate" in W:
            g = x @ w(p + "mlp.gate").t()
            y = (g * torch.sigmoid(g) * (x @ w(p + "mlp.up").t())) @ w(p + "mlp.down").t()
            x = x + norm(y, p + "norm2")
    h = norm(x, "final.norm")
    if prompt:
        wanted = _wanted(case)
        first = case["tokens"] - (case["tokens"] % case["portion"] or case["portion"] if case["portion"] else case["tokens"])
        h = h[[first + r for r in wanted]]
    logits = h @ w("embed").t()
    logits = logits if gifetar else CAP * torch.tanh(logits / CAP)
    return {"logits": logits[None] if prompt else logits[:, None], "states": states}


def _held(case, seed, i, lens):
    """The cached rows of every sequence of a decode step, one after the other: lists of [heads, tokens, columns]."""
    page = 64
    counts = [(n + 1 + page - 1) // page for n in lens]
    for parts in zip(*(t.split(counts) for t in _model_cache(case, seed, i, sum(counts), page))):
        yield [t.transpose(0, 1).reshape(t.shape[1], -1, t.shape[3]).double() for t in parts]


def _exact_differential(case, seed, i, h, w, m, at, lens):
    z = SIZES[case["size"]]
    H, G = z["heads"], z["kv_heads"]
    q, k, v = (h @ w(m + n).t() + w(f"{m}{n}.b") for n in ("q", "k", "v"))
    temp = 1 + 0.1 * torch.log(torch.floor((at.double() + 1) / 2048) + 1)
    q = q.view(-1, H, 2, DIM) * (temp * DIM ** -0.5).view(-1, 1, 1, 1)
    k, v = k.view(-1, G, 2, DIM), v.view(-1, G, VDIM)
    lam = torch.exp((w(m + "lq1") * w(m + "lk1")).sum()) - torch.exp((w(m + "lq2") * w(m + "lk2")).sum()) + DIFF
    out = torch.empty(h.shape[0], H, VDIM, dtype=torch.float64, device="cuda")
    if case["phase"] == "prompt":
        for j in range(H):
            g = j // (H // G)
            a, b = (_causal(q[:, j, n], k[:, g, n], v[:, g], cap=SOFTCAP) for n in (0, 1))
            out[:, j] = a - lam * b
    else:
        for r, (kk, vv) in enumerate(_held(case, seed, i, lens)):
            n = lens[r]
            kk = torch.cat((kk.view(G, 2, -1, DIM)[:, :, :n], k[r, :, :, None]), dim=2)
            vv = torch.cat((vv[:, :n], v[r, :, None]), dim=1)
            s = torch.einsum("gjmd,gmtd->gjmt", q[r].view(G, -1, 2, DIM), kk)
            a = torch.einsum("gjmt,gtd->gjmd", torch.softmax(SOFTCAP * torch.tanh(s / SOFTCAP), -1), vv)
            out[r] = (a[:, :, 0] - lam * a[:, :, 1]).reshape(H, VDIM)
    out = out / torch.sqrt((out * out).mean(-1, keepdim=True) + EPS) * (1 - DIFF)
    return out.reshape(-1, H * VDIM) @ w(m + "o").t()


def _turned(x, at):
    """Rotary positions on the pairs (2 i, 2 i + 1) of the last dimension, stretched for long contexts."""
    pair = lambda turns: ROT * math.log(STRETCH["original"] / (2 * math.pi * turns)) / (2 * math.log(BASE))
    lo, hi = max(math.floor(pair(STRETCH["fast"])), 0), min(math.ceil(pair(STRETCH["slow"])), ROT - 1)
    i = torch.arange(ROT // 2, dtype=torch.float64, device="cuda")
    f, ramp = BASE ** (-2 * i / ROT), ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    a = at.double().view(-1, *([1] * (x.dim() - 1))) * (f * (1 - ramp) + f / STRETCH["factor"] * ramp)
    amplitude = 0.1 * math.log(STRETCH["factor"]) + 1
    u, v, c, s = x[..., 0::2], x[..., 1::2], torch.cos(a) * amplitude, torch.sin(a) * amplitude
    return torch.stack((u * c - v * s, v * c + u * s), -1).flatten(-2)


def _exact_latent(case, seed, i, h, w, m, at, lens):
    H, scale = SIZES[case["size"]]["heads"], (NOPE + ROT) ** -0.5
    q = (h @ w(m + "q").t()).view(-1, H, NOPE + ROT)
    kv = h @ w(m + "dkv").t()
    c = _rms(kv[:, :RANK], w(m + "dkv.norm"), EPS)
    q, q_rot, k_rot = q[..., :NOPE], _turned(q[..., NOPE:], at), _turned(kv[:, RANK:], at)
    uk, uv, sink = w(m + "uk").view(H, NOPE, RANK), w(m + "uv").view(H, VDIM, RANK), w(m + "sink")
    out = torch.empty(h.shape[0], H, VDIM, dtype=torch.float64, device="cuda")
    if case["phase"] == "prompt":
        for j in range(H):
            keys = torch.cat((c @ uk[j].t(), k_rot), 1)
            out[:, j] = _causal(torch.cat((q[:, j], q_rot[:, j]), 1) * scale, keys, c @ uv[j].t(), sink=sink[j])
    else:
        wide = torch.cat((torch.einsum("rhd,hdc->rhc", q, uk), q_rot), 2) * scale
        for r, (rows,) in enumerate(_held(case, seed, i, lens)):
            rows = torch.cat((rows[0, :lens[r]], torch.cat((c[r], k_rot[r]))[None]))
            s = torch.cat((wide[r] @ rows.t(), sink[:, None]), 1)
            out[r] = torch.einsum("hc,hvc->hv", torch.softmax(s, 1)[:, :-1] @ rows[:, :RANK], uv)
    out = out * torch.sigmoid(h @ w(m + "g").t())[..., None]
    return out.reshape(-1, H * VDIM) @ w(m + "o").t()


def _exact_recurrence(case, seed, h, w, m, at):
    z = SIZES[case["size"]]
    C, n = z["width"], z["blocks"]
    y, x = (h @ w(m + b).t() + w(f"{m}{b}.b") for b in ("y", "x"))
    y = 0.5 * y * (1 + torch.tanh(math.sqrt(2 / math.pi) * (y + 0.044715 * y ** 3)))
    taps = w(m + "conv")
    if case["phase"] == "prompt":
        state = torch.zeros(1, C, dtype=torch.float64, device="cuda")
        back = [torch.cat((x.new_zeros(j, C), x[:x.shape[0] - j])) for j in range(TAPS)]
    else:
        state, ring = (t.double() for t in _model_recurrence(case, seed))
        rows = torch.arange(x.shape[0], device="cuda")
        back = [x] + [torch.where((at >= j)[:, None], ring[rows, (at - j) % TAPS], 0) for j in range(1, TAPS)]
    u = sum(taps[:, TAPS - 1 - j] * back[j] for j in range(TAPS)) + w(m + "conv.b")
    gate = lambda r: torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(-1, n, C // n), w(m + r)).reshape(-1, C) + w(f"{m}{r}.b"))
    log_a = -8 * gate("ra") * torch.log1p(torch.exp(w(m + "lam")))
    a, fresh = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * gate("ri") * u
    if case["phase"] == "prompt":
        every = torch.empty_like(u)
        for t in range(u.shape[0]):
            torch.addcmul(fresh[t], a[t], state[0], out=every[t])
            state = every[t:t + 1]
        state, s = state.clone(), every
    else:
        s = state = a * state + fresh
    return (s * y) @ w(m + "o").t(), state


# ---- the experts of a layer
def _experts_inputs(case, seed):
    """(weights, token ids): the embedding, the norms around the experts, their router and their matrices, as the models
    keep them."""
    z, s, W = SIZES[case["size"]], _Source(seed), {}
    C, E, F, gifetar = z["width"], z["experts"], z["ff"], case["style"] == "gifetar"
    f32 = lambda *shape, **kw: s.normal(*shape, dtype=torch.float32, **kw)
    W["embed"] = s.normal(VOCAB, C)
    W["gate_up"], W["down"] = s.normal(E, F, 2, C, std=C ** -0.5), s.normal(E, C, F, std=F ** -0.5)
    W["router"], W["router_b"] = s.normal(E, C, std=C ** -0.5), f32(E, std=0.1) if gifetar else None
    norm = lambda: (f32(C, std=0.1, mean=1.0), f32(C, std=0.1) if gifetar else None)
    W["pre"], W["post"], W["after"] = norm() if gifetar else None, norm(), norm()
    return W, s.tokens(case["tokens"])


def _experts_spec(case):
    z, gifetar = SIZES[case["size"]], case["style"] == "gifetar"
    gate = layer_ops.SILU if gifetar else layer_ops.GateSpec(LIMIT, SLOPE, SHIFT)
    return layer_ops.MoeSpec(z["experts"], z["top"], z["width"], z["ff"], score_all=not gifetar, gate=gate)


def _prepare_experts(case, seed):
    W, ids = _experts_inputs(case, seed)
    rows, C, E = case["tokens"], SIZES[case["size"]]["width"], SIZES[case["size"]]["experts"]
    s = dict(W, spec=_experts_spec(case), ids=ids, mult=MULT if case["style"] == "gifetar" else 1.0,
             center=case["style"] == "gifetar", x=torch.empty(rows, C, dtype=torch.float32, device="cuda"),
             h=torch.empty(rows, C, dtype=torch.bfloat16, device="cuda"),
             counts=torch.zeros(E, dtype=torch.int32, device="cuda"), status=ops.new_status("cuda"))
    if case["phase"] == "decode":
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _experts_step(s)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _experts_step(s)
        s["graph"] = graph
    return s


def _experts_step(s):
    """The launches of a layer between its mixer and the next one, on the embedded tokens."""
    x, h, spec = s["x"], s["h"], s["spec"]
    row = lambda **kw: layer_ops.residual_norm(x, h, spec.width, EPS, center=s["center"], status=s["status"], **kw)
    row(tokens=s["ids"], embed=s["embed"], pre=s["pre"], zero=s["counts"])
    routing = layer_ops.moe_route(h, s["router"], s["router_b"], spec, s["counts"])
    y = layer_ops.moe_experts(h, s["gate_up"], s["down"], routing, spec, status=s["status"])
    row(y=y, parts=spec.top, post=s["post"], mult=s["mult"], pre=s["after"])


def _run_experts(s):
    if "graph" in s:
        s["graph"].replay()
    else:
        _experts_step(s)
    return {"stream": s["x"], "next": s["h"]}


def _exact_experts(case, seed):
    W, ids = _experts_inputs(case, seed)
    z, gifetar = SIZES[case["size"]], case["style"] == "gifetar"

    def norm(x, weight):
        x = x - x.mean(-1, keepdim=True) if gifetar else x
        y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * weight[0].double()
        return y + weight[1].double() if gifetar else y
    x = W["embed"][ids].double()
    h = (norm(x, W["pre"]) if gifetar else x).to(torch.bfloat16).double()    # the experts' input is kept in bf16
    scores = h @ W["router"].double().t() + (W["router_b"].double() if gifetar else 0)
    best, chosen = scores.topk(z["top"], dim=1)
    share = torch.softmax(best, 1) if gifetar else torch.softmax(scores, 1).gather(1, chosen)
    y = torch.zeros_like(h)
    for e in range(z["experts"]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        g, u = (h[rows] @ W["gate_up"][e, :, i].double().t() for i in (0, 1))
        if gifetar:
            a = g * torch.sigmoid(g) * u
        else:
            g, u = g.clamp(max=LIMIT), u.clamp(-LIMIT, LIMIT)
            a = g * torch.sigmoid(SLOPE * g) * (u + SHIFT)
        y.index_add_(0, rows, share[rows, place, None] * (a @ W["down"][e].double().t()))
    x = x + (MULT if gifetar else 1.0) * norm(y, W["post"])
    return {"stream": x, "next": norm(x, W["after"])}


def _work_experts(case):
    z, rows = SIZES[case["size"]], case["tokens"]
    C, E, T, F = z["width"], z["experts"], z["top"], z["ff"]
    used = E * (1 - (1 - T / E) ** rows)                                     # experts that some row uses
    return {"bytes": 2 * (used * 3 * C * F + E * C) + rows * C * (2 + 4 + 2), "flops": 2 * rows * (3 * T * C * F + E * C)}


# ---------------------------------------------------------------- what a measuring program calls
_FAMILIES = {"layer": (_prepare_layer, _run_layer, _exact_layer, _work_layer),
             "prompt": (_prepare_prompt, _run_prompt, _exact_prompt, _work_prompt),
             "gifetar": (_prepare_model, _run_model, _exact_model, _work_model),
             "munadra": (_prepare_model, _run_model, _exact_model, _work_model),
             "experts": (_prepare_experts, _run_experts, _exact_experts, _work_experts)}


def prepare(case, seed):
    return dict(_FAMILIES[case["family"]][0](case, seed), family=case["family"])


def run(state):
    return _FAMILIES[state["family"]][1](state)


def exact(case, seed):
    with torch.no_grad():
        return _FAMILIES[case["family"]][2](case, seed)


def work(case):
    return _FAMILIES[case["family"]][3](case)


def tolerance(case):
    """About four times what the path differs by from 64 bits, or from its own sums in another order.  A layer's output is
    its residual plus small terms, in bf16 the rounding of the type; a page whose score ties with another's may change
    with a rounding of the query, as an expert may with a rounding of its input (then by a row, hence the `max`)."""
    if case["family"] == "layer":
        return {"rel": 1e-6, "differ": 1e-3} if case["dtype"] == "float32" else {"rel": 1e-2, "max": 0.2, "differ": 1e-2}
    return {"prompt": {"rel": 8e-3, "max": 0.1}, "experts": {"rel": 1e-2, "max": 0.8}, "gifetar": {"rel": 8e-3, "max": 0.05},
            "munadra": {"rel": 3e-2, "max": 0.4}}[case["family"]]
