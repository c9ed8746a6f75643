"""What the speed of this engine is measured on: steps of whole models through ``Engine.step``.

A case is a model (a preset of ``shiso_llm_b200/config/presets``, random weights), a compute type and
one of three kinds of pass:

* ``decode``  - every one of ``seqs`` running requests, whose contexts start between ``low`` and
  ``high`` tokens, brings its next token: one step.  The requests stay and grow from pass to pass.
* ``prompt``  - ``seqs`` new requests of ``low`` to ``high`` tokens are read in one step and end;
  logits are wanted at the last ``want`` tokens of each (1: the next token; more: scoring).
* ``portions`` - one prompt of ``long`` tokens is read in portions of ``portion`` tokens while
  ``seqs`` running requests bring a token beside each portion.

Tokens are uniform over the vocabulary and given from outside (so that a rounding that changes a
pick changes no later input); weights are drawn as ``shiso_llm_b200.weights`` draws them.  ``layers`` runs a preset's first layers only, as bench.py's option of that name does.

Of the designs with routed experts those stand here, at the size and depth, at which two correct
implementations agree: a router decides between close scores in every layer, and a rounding that
falls the other way is another expert.  Two cuts of one prompt differ by 0.3 % of the logits' norm with
povilorn-350m (2 to 5 % with povilorn-1b), by 1 % with Zetavik's first six layers (3 % with all), and
by 5 to 12 % with Nodepel and Raketar, which share their expert, product and attention kernels with these.
"""

from __future__ import annotations

import json
import math

import numpy as np
import torch

F64 = torch.float64
CTX = 4096  # most tokens of a running request


def _case(name, kind, preset, seqs, low, high, want=1, dtype="bfloat16", long=0, portion=0, layers=0):
    case = {"kind": kind, "preset": preset, "layers": layers, "dtype": dtype, "seqs": seqs, "low": low, "high": high,
            "want": want, "long": long, "portion": portion}
    return case if name is None else {"name": name, **case}


def listed():
    return [
        # one user's chat with the smallest model: a step is latency and launches
        _case("chat-350m", "decode", "lfm2-350m", 1, 200, 200),
        # the headline of bench.py: eight requests behind prompts of 2,048 tokens
        _case("decode-1.2b-b8", "decode", "lfm2-1.2b", 8, 2048, 2048),
        # a full server: 64 requests of all lengths
        _case("decode-1.2b-b64", "decode", "lfm2-1.2b", 64, 100, 1500),
        # the headline's prompt: the tensor cores' share of the work
        _case("prompt-1.2b", "prompt", "lfm2-1.2b", 1, 2048, 2048),
        # a step of continuous batching as the 350M serving workload of bench.py has them: a few short prompts
        _case("prompts-350m-ragged", "prompt", "lfm2-350m", 3, 83, 259),
        # bench.py's mixed workload: a long prompt in portions beside running streams (the largest case)
        _case("portions-1.2b-beside-32", "portions", "lfm2-1.2b", 32, 300, 700, long=8192, portion=1024),
        # the true 32-bit type, as used to check a checkpoint
        _case("prompt-350m-float32", "prompt", "lfm2-350m", 1, 300, 300, dtype="float32"),
        # windowed and chunked attention, an odd prompt that ends inside a chunk
        _case("prompt-volalorn-1b", "prompt", "volalorn-1b", 1, 1501, 1501),
        # several streams, data-dependent decays, pooled blocks: prompts beyond the window of 1,024
        _case("prompt-filulix-1b", "prompt", "filulix-1b", 1, 2000, 2000),
        # routed experts, latent attention, lightning and Mamba-2: scoring the ends of four prompts
        _case("score-zetavik-1b", "prompt", "zetavik-1b", 4, 400, 600, want=16, layers=6),
        # routed experts and latent attention, a prompt of full length
        _case("prompt-povilorn-350m", "prompt", "povilorn-350m", 1, 2048, 2048),
        # the same design serving eight requests
        _case("decode-povilorn-350m-b8", "decode", "povilorn-350m", 8, 900, 2048),
    ]


def draw(rng):
    def between(a, b):  # spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["decode", "decode", "prompt", "prompt", "prompt", "portions"])
    if kind == "decode":
        preset = rng.choice(["lfm2-350m", "lfm2-1.2b", "volalorn-350m", "volalorn-1b", "povilorn-350m", "filulix-350m"])
        low = between(16, 1900)
        return _case(None, kind, preset, between(1, 64), low, between(low, 2048))
    if kind == "prompt":
        preset, dtype = rng.choice([("lfm2-350m", "bfloat16"), ("lfm2-1.2b", "bfloat16"), ("volalorn-1b", "bfloat16"),
                                    ("volalorn-350m", "bfloat16"), ("filulix-350m", "bfloat16"), ("zetavik-1b", "bfloat16"),
                                    ("povilorn-350m", "bfloat16"), ("lfm2-350m", "float32")])
        zetavik = preset == "zetavik-1b"
        # (float32 for checks of short texts; single rows of Zetavik that change experts need others beside them)
        rows = between(640 if zetavik else 24, 256 if dtype == "float32" else 2048)
        seqs = min(between(1, 8), rows // 24)
        if seqs == 1:
            low = high = rows
        else:  # lengths evenly spread around rows / seqs
            low = max(20, int(rows / seqs * rng.uniform(0.3, 0.9)))
            high = 2 * (rows // seqs) - low
        return _case(None, kind, preset, seqs, low, max(low, high), want=16 if zetavik else 1, dtype=dtype,
                     layers=6 if zetavik else 0)
    portion = rng.choice([256, 512, 1024])
    return _case(None, kind, rng.choice(["lfm2-350m", "lfm2-1.2b"]), between(2, 32), 100, between(100, 700),
                 long=between(2 * portion, 6000), portion=portion)


# --------------------------------------------------------------------------- inputs


def _document(case):
    from shiso_llm_b200.cli import preset_path

    with open(preset_path(case["preset"])) as f:
        document = json.load(f)
    if case["layers"]:
        document["layers"] = document["layers"][: case["layers"]]
    return document


def _model(case, device):
    """The plan of the case's model and the specs of its tensors."""
    from shiso_llm_b200.config import plan_from_document
    from shiso_llm_b200.kernels import ops
    from shiso_llm_b200.parts import BuildEnv, Model

    _, _, plan = plan_from_document(_document(case))
    model = Model(plan, BuildEnv(dtype=getattr(torch, case["dtype"]), device=device, ops=ops))
    return plan, model


def _tensors(case, seed, model, device):
    from shiso_llm_b200.weights import random_device_tensors

    return random_device_tensors(model.tensor_specs(), seed, getattr(torch, case["dtype"]), device)


def _lengths(case):
    n = case["seqs"]
    return [case["low"] + ((case["high"] - case["low"]) * i) // max(1, n - 1) for i in range(n)]


def _token_lists(case, seed, vocab):
    """Per request its tokens (for a running one all it can ever bring), then the long prompt's."""
    rng = np.random.RandomState(seed % (2**31) + 17)
    counts = _lengths(case) if case["kind"] == "prompt" else [CTX] * case["seqs"]
    return [rng.randint(0, vocab, n).tolist() for n in counts], rng.randint(0, vocab, case["long"]).tolist()


def prepare(case, seed):
    from shiso_llm_b200 import Engine, EngineOptions

    device = torch.device("cuda:0")
    plan, model = _model(case, device)
    lists, long = _token_lists(case, seed, plan.vocab_size)
    rows = sum(len(t) for t in lists) if case["kind"] == "prompt" else max(2048, case["portion"] + case["seqs"])
    ctx = max(CTX, len(long) + 16)
    running = 0 if case["kind"] == "prompt" else case["seqs"]
    seqs = case["seqs"] + (1 if long else 0)
    options = EngineOptions(dtype=case["dtype"], ctx=ctx, page_size=16, kv_cache_tokens=ctx + running * CTX + rows,
                            max_num_seqs=max(2, seqs), max_num_batched_tokens=rows)
    engine = Engine.from_plan(plan, _tensors(case, seed, model, device), options)
    state = {"case": case, "engine": engine, "lists": lists, "long": long, "at": None, "turn": 0}
    if running:
        _read_contexts(state)
    for _ in range(2):  # as a server warms up: a step's shape is captured when it comes again
        run(state, warm=True)
    return state


def _read_contexts(state):
    """Every running request's first tokens, a request a step."""
    from shiso_llm_b200 import StepEntry

    case, engine = state["case"], state["engine"]
    for i, n in enumerate(_lengths(case)):
        engine.step([StepEntry(("r", i), state["lists"][i][:n], [])])
    state["at"] = _lengths(case)


def _next_tokens(state):
    """One entry per running request; one that has filled its context starts over."""
    from shiso_llm_b200 import StepEntry

    if max(state["at"]) >= CTX - 1:
        for i in range(state["case"]["seqs"]):
            state["engine"].finish(("r", i))
        _read_contexts(state)
    entries = [StepEntry(("r", i), [tokens[at]], [0]) for i, (tokens, at) in enumerate(zip(state["lists"], state["at"]))]
    state["at"] = [at + 1 for at in state["at"]]
    return entries


def _last(count, want):
    return list(range(max(0, count - want), count))


def run(state, warm=False):
    from shiso_llm_b200 import StepEntry

    case, engine = state["case"], state["engine"]
    state["turn"] += 1
    if case["kind"] == "decode":
        return engine.step(_next_tokens(state))
    if case["kind"] == "prompt":
        entries = [StepEntry((state["turn"], i), tokens, _last(len(tokens), case["want"])) for i, tokens in enumerate(state["lists"])]
        logits = engine.step(entries)
        for e in entries:
            engine.finish(e.request)
        return logits
    out, long, portion = [], state["long"], case["portion"]
    request = (state["turn"], "long")
    if warm:
        long = long[: 2 * portion]
    for at in range(0, len(long), portion):
        part = long[at : at + portion]
        # (the prompt's portion comes last: its row is the last one of the logits)
        entries = _next_tokens(state) + [StepEntry(request, part, [len(part) - 1] if at + portion >= len(long) else [])]
        out.append(engine.step(entries).clone())  # the next portion's step writes over the logits
    engine.finish(request)
    return out


# --------------------------------------------------------------------------- what a pass cannot do without


def _mixers(spec):
    """The mixers of a layer: itself, or its branches."""
    if "branches" in spec.params:
        return [m for part, _ in spec.params["branches"] for m in _mixers(part)]
    return [spec]


def work(case):
    from shiso_llm_b200.parts.base import PagedKV
    from shiso_llm_b200.weights.spec import MATRIX

    plan, model = _model(case, torch.device("cpu"))
    itemsize = 4 if case["dtype"] == "float32" else 2
    lengths = _lengths(case)
    if case["kind"] == "decode":
        spans = [(n + 2, n + 3) for n in lengths]  # positions of the rows of the first pass
        steps = 1
        wanted = len(lengths)
    elif case["kind"] == "prompt":
        spans = [(0, n) for n in lengths]
        steps, wanted = 1, sum(min(n, case["want"]) for n in lengths)
    else:
        steps = -(-case["long"] // case["portion"])
        spans = [(n + 4, n + 4 + steps) for n in lengths] + [(0, case["long"])]
        wanted = steps * len(lengths) + 1
    rows = sum(b - a for a, b in spans)
    specs = {s.name: s for s in model.tensor_specs()}
    size = {n: int(np.prod(s.shape)) for n, s in specs.items()}
    table = plan.embedding.params["tensor"]
    vocab, width = plan.vocab_size, plan.hidden_size
    bytes_, flops = 0.0, 2.0 * wanted * vocab * width
    bytes_ += steps * vocab * width * itemsize + wanted * vocab * 4 + rows * width * itemsize
    seen = set()
    runs = [plan.layers[o.layer] for o in plan.order]
    for layer, entry in zip(runs, model.cache_needs()):
        ff = layer.feed_forward
        names = {v for part in [layer.mixer, ff] + _mixers(layer.mixer) for v in part.params.values() if isinstance(v, str) and v in specs}
        names |= {v for part in [layer.mixer, ff] for d in part.params.values() if isinstance(d, dict) for v in d.values() if isinstance(v, str) and v in specs}
        experts = ff.params.get("expert_names") or ()
        per_step = rows / steps
        for e in experts:
            for n in e.values():
                share = ff.params["top"] / ff.params["experts"]
                if n not in seen:
                    bytes_ += steps * size[n] * itemsize * (1 - (1 - share) ** per_step)
                seen.add(n)
                flops += 2.0 * rows * size[n] * share
        shared = ff.params.get("shared_names") or ff.params.get("shared") or {}
        names |= {v for v in (shared.values() if isinstance(shared, dict) else ()) if isinstance(v, str) and v in specs}
        for n in names - {table}:
            matrix = specs[n].role == MATRIX
            if n not in seen:
                bytes_ += steps * size[n] * (itemsize if matrix else 4)
            seen.add(n)
            if matrix:
                flops += 2.0 * rows * size[n]
        needs = [x for x in (entry if isinstance(entry, tuple) else (entry,)) if x is not None]
        window = next((x.window for x in needs if isinstance(x, PagedKV) and x.window), None)
        for x in needs:
            if isinstance(x, PagedKV):
                row = (x.num_kv_heads * x.head_dim + x.value_heads * x.value_dim) * (x.dtype.itemsize if x.dtype else itemsize)
                for a, b in spans:  # rows of the cache are read once and the new ones written
                    bytes_ += (min(b, x.window or b) + (b - a)) * row / x.every
            else:
                bytes_ += 2 * steps * len(spans) * x.nbytes
        for m in _mixers(layer.mixer):
            p = m.params
            if "num_heads" not in p:
                continue
            dim = p.get("state") or p.get("head_dim") or width // p["num_heads"]
            dim, value = dim + (p.get("rot_dim") or 0), p.get("v_head_dim") or dim
            if any(isinstance(x, PagedKV) for x in needs) and m.kind not in ("retention",):
                pairs = sum(sum(min(i + 1, window or i + 1) for i in range(a, b)) for a, b in spans)
                flops += 2.0 * pairs * p["num_heads"] * (dim + value)
            else:
                flops += 4.0 * rows * p["num_heads"] * dim * value
    return {"bytes": float(bytes_), "flops": float(flops)}


def tolerance(case):
    """Measured between two cuts of one prompt (one portion, two, single tokens), which take other
    kernels: 2.0 to 2.3 % of the logits' norm for the LFM2 models, 1.1 to 1.6 % for Filulix, 0.6 % for
    Volalorn, 0.3 % for povilorn-350m and 0.8 to 1.2 % for six layers of Zetavik (single rows, whose
    routing changes, up to 5 %); in 32 bits 7e-6 of the 64-bit result."""
    if case["dtype"] == "float32":
        return {"rel": 3e-5, "max": 1e-3}
    return {"rel": 0.03, "max": 0.99}


# --------------------------------------------------------------------------- the same in 64 bits


def exact(case, seed):
    device = torch.device("cuda:0")
    plan, model = _model(case, device)
    tensors = _tensors(case, seed, model, device)
    lists, long = _token_lists(case, seed, plan.vocab_size)
    doc = _document(case)
    family = doc.get("architecture", "Lfm2")
    forward = {"Lfm2": _lfm2, "Zetavik": _zetavik, "Povilorn": _povilorn, "Filulix": _filulix, "Volalorn": _volalorn}[family]

    def w(name):
        return tensors[name].to(F64)

    def logits(tokens, rows):
        return forward(doc, w, torch.tensor(tokens, device=device), torch.tensor(rows, device=device))

    lengths = _lengths(case)
    if case["kind"] == "decode":  # prepare() has brought two tokens behind the contexts
        return torch.cat([logits(t[: n + 3], [n + 2]) for t, n in zip(lists, lengths)])
    if case["kind"] == "prompt":
        return torch.cat([logits(t, _last(len(t), case["want"])) for t in lists])
    steps = -(-len(long) // case["portion"])
    warm = 2 * min(2, steps)
    streams = [logits(t[: n + warm + steps], list(range(n + warm, n + warm + steps))) for t, n in zip(lists, lengths)]
    out = [torch.stack([s[i] for s in streams]) for i in range(steps)]
    out[-1] = torch.cat([out[-1], logits(long, [len(long) - 1])])
    return out


def _rms(x, eps, weight=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _layer_norm(x, eps, weight):
    x = x - x.mean(-1, keepdim=True)
    return _rms(x, eps, weight)


def _silu(x):
    return x * torch.sigmoid(x)


def _ladder(rot):
    """Frequencies of the rotation's pairs and the factor on cosine and sine."""
    dims, base = rot["dims"], float(rot["base"])
    i = torch.arange(dims // 2, dtype=F64)
    f = base ** (-2.0 * i / dims)
    s = rot.get("scaling")
    if s is None:
        return f, 1.0

    def pair(turns):
        return dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    lo, hi = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _rotate(x, rot, neighbours=False):
    """``x[T, heads, D]``, row t at position t; pairs are halves of the first ``dims`` entries, or neighbours."""
    f, factor = _ladder(rot)
    dims = rot["dims"]
    angle = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * f.to(x.device)[None, :]
    cos, sin = (torch.cos(angle) * factor)[:, None], (torch.sin(angle) * factor)[:, None]
    if neighbours:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        turned = torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2)
    else:
        u, v = x[..., : dims // 2], x[..., dims // 2 : dims]
        turned = torch.cat([u * cos - v * sin, v * cos + u * sin], -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _causal(T, device, window=None, keep=0, chunk=None):
    i, j = torch.arange(T, device=device)[:, None], torch.arange(T, device=device)[None, :]
    seen = j <= i
    if window is not None:
        seen &= (i - j < window) | (j < keep)
    return seen if chunk is None else seen & (i // chunk == j // chunk)


def _attend(q, k, v, scale, seen):
    """Softmax attention ``[T, H, D]`` over ``[T, G, D]``, a head at a time."""
    out, group = [], q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        scores = (q[:, h] @ k[:, h // group].T * scale).masked_fill(~seen, -math.inf)
        out.append(torch.softmax(scores, -1) @ v[:, h // group])
    return torch.stack(out, 1)


def _walk(r, k, v, decay, bonus=None):
    """``S <- decay S + k v^T`` token by token, ``o = S^T r``; with ``bonus`` the output sees the
    state before the token plus ``bonus k v^T``.  ``decay[T, H, dk or 1]``; ``r``, ``k`` ``[T, H, dk]``."""
    T, H, dk = k.shape
    state = torch.zeros(H, dk, v.shape[-1], dtype=F64, device=k.device)
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=k.device)
    for t in range(T):
        kv = k[t, :, :, None] * v[t, :, None, :]
        after = decay[t, :, :, None] * state + kv
        seen = after if bonus is None else state + bonus[:, :, None] * kv
        out[t] = (r[t, :, None, :] @ seen)[:, 0]
        state = after
    return out


def _lfm2(doc, w, tokens, rows):
    eps, heads, groups = doc["norm_eps"], doc["num_attention_heads"], doc["num_key_value_heads"]
    T = tokens.shape[0]
    x = w("model.embed_tokens.weight")[tokens]
    seen = _causal(T, x.device)
    for i, kind in enumerate(doc["layer_types"]):
        p = f"model.layers.{i}"
        h = _rms(x, eps, w(f"{p}.operator_norm.weight"))
        if kind == "conv":
            b, c, u = (h @ w(f"{p}.conv.in_proj.weight").T).chunk(3, -1)
            taps = w(f"{p}.conv.conv.weight").reshape(u.shape[1], -1)
            L = taps.shape[1]
            padded = torch.cat([torch.zeros(L - 1, u.shape[1], dtype=F64, device=u.device), b * u])
            y = c * sum(taps[:, j] * padded[j : j + T] for j in range(L))
            y = y @ w(f"{p}.conv.out_proj.weight").T
        else:
            a = f"{p}.self_attn"
            rot = {"dims": x.shape[1] // heads, "base": doc["rope_theta"]}
            q, k, v = ((h @ w(f"{a}.{n}_proj.weight").T).view(T, m, -1) for n, m in (("q", heads), ("k", groups), ("v", groups)))
            q = _rotate(_rms(q, eps, w(f"{a}.q_layernorm.weight")), rot)
            k = _rotate(_rms(k, eps, w(f"{a}.k_layernorm.weight")), rot)
            y = _attend(q, k, v, q.shape[-1] ** -0.5, seen).reshape(T, -1) @ w(f"{a}.out_proj.weight").T
        x = x + y
        h = _rms(x, eps, w(f"{p}.ffn_norm.weight"))
        f = f"{p}.feed_forward"
        x = x + (_silu(h @ w(f"{f}.w1.weight").T) * (h @ w(f"{f}.w3.weight").T)) @ w(f"{f}.w2.weight").T
    return _rms(x[rows], eps, w("model.embedding_norm.weight")) @ w("model.embed_tokens.weight").T


def _chosen(choice, r):
    """Which experts each row takes: the best ``top`` among the experts of the groups with the best members."""
    T, E = choice.shape
    groups = r.get("groups") or {"count": 1, "keep": 1}
    best = choice.view(T, groups["count"], -1).max(-1).values
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(groups["keep"], -1).indices, True)
    masked = choice.masked_fill(~kept.repeat_interleave(E // groups["count"], 1), -math.inf)
    return torch.zeros_like(choice, dtype=torch.bool).scatter_(1, masked.topk(r["top"], -1).indices, True)


def _routed(mlp, h, weights, chosen, expert, prefix):
    out = torch.zeros_like(h)
    for e in range(mlp["router"]["experts"]):
        rows = chosen[:, e].nonzero().flatten()
        if rows.numel():
            out[rows] += weights[rows, e : e + 1] * expert(f"{prefix}.e{e}", h[rows])
    return out


def _latent(w, p, m, h, eps, neighbours):
    T, H, dim, rank = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
    if "q_rank" in m:
        q = _rms(h @ w(f"{p}.dq").T, eps, w(f"{p}.dq.norm")) @ w(f"{p}.uq").T
    else:
        q = h @ w(f"{p}.q").T
    q = q.view(T, H, dim + m["rot_dim"])
    down = h @ w(f"{p}.dkv").T
    c = _rms(down[:, :rank], eps, w(f"{p}.dkv.norm"))
    shared = _rotate(down[:, None, rank:], m["rot"], neighbours).expand(T, H, -1)
    q = torch.cat([q[..., :dim], _rotate(q[..., dim:], m["rot"], neighbours)], -1)
    k = torch.cat([(c @ w(f"{p}.uk").T).view(T, H, dim), shared], -1)
    return _attend(q, k, (c @ w(f"{p}.uv").T).view(T, H, -1), m["scale"], _causal(T, h.device))


def _zetavik(doc, w, tokens, rows):
    eps, T = doc["norm"]["eps"], tokens.shape[0]
    x = w("embed")[tokens]

    def expert(p, h):
        return (_silu(h @ w(f"{p}.gate").T) * (h @ w(f"{p}.up").T)) @ w(f"{p}.down").T

    for i, layer in enumerate(doc["layers"]):
        h, p, m = _layer_norm(x, eps, w(f"l{i}.norm1")), f"l{i}.mix", layer["mixer"]
        if layer["type"] == "latent_attention":
            y = _latent(w, p, m, h, eps, False) * torch.sigmoid(h @ w(f"{p}.g").T)[:, :, None]
            y = y.reshape(T, -1)
        elif layer["type"] == "lightning":
            q, k, v = (_silu(h @ w(f"{p}.{n}").T).view(T, m["heads"], -1) for n in "qkv")
            decay = torch.tensor(m["decay"], dtype=F64, device=h.device)[None, :, None].expand(T, -1, 1)
            y = _rms(_walk(q, k, v, decay).reshape(T, -1), eps, w(f"{p}.norm")) * torch.sigmoid(h @ w(f"{p}.g").T)
        else:
            H, N, G = m["heads"], m["state"], m["groups"]
            inner = H * m["vdim"]
            z, xbc, dt = (h @ w(f"{p}.in").T).split([inner, inner + 2 * G * N, H], -1)
            taps = w(f"{p}.conv")
            L = taps.shape[1]
            padded = torch.cat([torch.zeros(L - 1, xbc.shape[1], dtype=F64, device=h.device), xbc])
            xbc = _silu(sum(padded[j : j + T] * taps[:, j] for j in range(L)) + w(f"{p}.conv.b"))
            u, B, C = xbc.split([inner, G * N, G * N], -1)
            u = u.view(T, H, -1)
            B, C = (a.view(T, G, N).repeat_interleave(H // G, 1) for a in (B, C))
            dt = torch.nn.functional.softplus(dt + w(f"{p}.dt_bias"))
            decay = torch.exp(-torch.exp(w(f"{p}.A_log")) * dt)[:, :, None]
            y = _walk(C, B * dt[:, :, None], u, decay) + w(f"{p}.D")[:, None] * u
            y = (y.reshape(T, inner) * _silu(z)).view(T, m["norm_groups"], -1)
            y = _rms(y, eps).reshape(T, inner) * w(f"{p}.norm")
        y = y @ w(f"{p}.o").T
        f, mlp = f"l{i}.mlp", layer["mlp"]
        if mlp["kind"] == "dense":
            y = y + torch.relu(h @ w(f"{f}.up").T) ** 2 @ w(f"{f}.down").T
        else:
            scores = torch.softmax(h @ w(f"{f}.router").T, -1)
            chosen = _chosen(scores, mlp["router"])
            y = y + _routed(mlp, h, scores * mlp["router"]["scale"], chosen, expert, f) + expert(f"{f}.shared", h)
        x = x + y
    return _layer_norm(x[rows], eps, w("final.norm")) @ w("embed").T


def _povilorn(doc, w, tokens, rows):
    eps, T = doc["norm"]["eps"], tokens.shape[0]
    first = w("embed")[tokens] * doc["embedding"]["scale"]
    loop, n = doc["loop"], len(doc["layers"])
    order = [(i, None) for i in range(loop["start"])]
    for t in range(loop["times"]):
        order += [(i, t if i == loop["start"] else None) for i in range(loop["start"], loop["stop"])]
    order += [(i, None) for i in range(loop["stop"], n)]

    def squash(x, name):
        return torch.tanh(w(f"{name}.alpha") * x) * w(name) + w(f"{name}.b")

    def expert(limit):
        def of(p, h):
            g = (h @ w(f"{p}.gate").T).clamp(max=limit)
            u = (h @ w(f"{p}.up").T).clamp(-limit, limit)
            return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(f"{p}.down").T
        return of

    x = first
    for i, begins in order:
        layer = doc["layers"][i]
        if begins is not None:
            x = x + (first if begins > 0 else 0.0) + w("loop.step")[begins]
        h, p, m = squash(x, f"l{i}.norm1"), f"l{i}.mix", layer["mixer"]
        if layer["type"] == "attention":
            q, k = (h @ w(f"{p}.{a}").T + w(f"{p}.{a}.b") for a in "qk")
            v = k.view(T, m["kv_heads"], -1)
            q, k = _rms(q, eps, w(f"{p}.q.norm")), _rms(k, eps, w(f"{p}.k.norm"))
            if m.get("q_temp") is not None:
                pos = torch.arange(T, dtype=F64, device=h.device)
                q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1.0) / m["q_temp"]["every"]) + 1.0))[:, None]
            y = _attend(q.view(T, m["heads"], -1), k.view_as(v), v, m["scale"], _causal(T, h.device))
            y = y.reshape(T, -1) * torch.sigmoid(h @ w(f"{p}.g").T)
        else:
            y = _latent(w, p, m, h, eps, True).reshape(T, -1)
        x = x + y @ w(f"{p}.o").T
        f, mlp = f"l{i}.mlp", layer["mlp"]
        h = squash(x, f"l{i}.norm2")
        if mlp["kind"] == "dense":
            x = x + (torch.nn.functional.gelu(h @ w(f"{f}.gate").T, approximate="tanh") * (h @ w(f"{f}.up").T)) @ w(f"{f}.down").T
            continue
        scores = torch.softmax(h @ w(f"{f}.router").T, -1)
        chosen = _chosen(scores + w(f"{f}.correction"), mlp["router"])
        picked = scores * chosen
        weights = picked / (picked.sum(-1, keepdim=True) + 1e-20)
        y = _routed(mlp, h, weights, chosen, expert(mlp["expert"]["limit"]), f)
        y = y + weights[:, mlp["router"]["experts"] :].sum(-1, keepdim=True) * h  # identity experts
        x = x + y + torch.sigmoid(h @ w(f"{f}.shared.sg").T) * expert(mlp["shared"]["limit"])(f"{f}.shared", h)
    return squash(x[rows], "final.norm") @ w("head").T


def _filulix(doc, w, tokens, rows):
    eps, T = doc["norm"]["eps"], tokens.shape[0]
    emb = doc["embedding"]
    big = emb["bigram"]
    before = torch.cat([tokens[:1], tokens[:-1]])
    pairs = (before * big["mul_prev"] + tokens * big["mul_cur"]) % big["buckets"]
    pairs[0] = big["buckets"]
    x = w("embed")[tokens] * emb["scale"] + w("bigram")[pairs]
    lanes = x[None].repeat(doc["streams"], 1, 1)

    def norm(x, name):
        return _rms(x, eps, 1.0 + w(name))

    def wkv(p, m, h):
        prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        r, k, v, g, z = (h + (prev - h) * w(f"{p}.mu.{c}") for c in "rkvgw")
        r, k, v = ((a @ w(f"{p}.{c}").T).view(T, m["heads"], -1) for a, c in ((r, "r"), (k, "k"), (v, "v")))
        z = torch.tanh(z @ w(f"{p}.w1").T) @ w(f"{p}.w2").T + w(f"{p}.w0")
        y = _walk(r, k, v, torch.exp(-torch.exp(z)).view_as(r), w(f"{p}.u").view(m["heads"], -1))
        return (_rms(y, eps).reshape(T, -1) * w(f"{p}.norm") * _silu(g @ w(f"{p}.g").T)) @ w(f"{p}.o").T

    def parallel(p, m, h):
        a = m["left"]
        q, k, v = ((h @ w(f"{p}.left.{c}").T).view(T, n, -1) for c, n in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])))
        window, pool = a["mask"]["size"], a["mask"]["pool"]
        blocks = T // pool
        k, v = (torch.cat([b[: blocks * pool].view(blocks, pool, *b.shape[1:]).mean(1), b]) for b in (k, v))
        i = torch.arange(T, device=h.device)[:, None]
        ends = torch.arange(blocks, device=h.device)[None, :] * pool + pool - 1
        seen = torch.cat([ends <= i - window, _causal(T, h.device, window)], 1)
        left = _attend(q, k, v, a["scale"], seen).reshape(T, -1) @ w(f"{p}.left.o").T
        a = m["right"]
        q, k, v = ((h @ w(f"{p}.right.{c}").T).view(T, a["heads"], -1) for c in "qkv")
        if a.get("rot") is not None:
            q, k = _rotate(q, a["rot"]), _rotate(k, a["rot"])
        decay = torch.tensor(a["decay"], dtype=F64, device=h.device)[None, :, None].expand(T, -1, 1)
        y = _rms(_walk(q, k * a["dim"] ** -0.5, v, decay), eps).reshape(T, -1)
        right = (y * _silu(h @ w(f"{p}.right.g").T)) @ w(f"{p}.right.o").T
        return m["left_scale"] * left + m["right_scale"] * right

    def dense(p, _, h):
        return (_silu(h @ w(f"{p}.gate").T) * (h @ w(f"{p}.up").T)) @ w(f"{p}.down").T

    for i, layer in enumerate(doc["layers"]):
        for q, part, of, spec in ((1, "mix", wkv if layer["type"] == "wkv" else parallel, layer["mixer"]), (2, "mlp", dense, None)):
            u = torch.einsum("s,std->td", w(f"l{i}.hc{q}.in"), lanes)
            y = of(f"l{i}.{part}", spec, norm(u, f"l{i}.norm{q}"))
            lanes = torch.einsum("sr,std->rtd", w(f"l{i}.hc{q}.mix"), lanes) + w(f"l{i}.hc{q}.out")[:, None, None] * y[None]
    return norm(lanes.sum(0)[rows], "final.norm") @ w("head").T


def _volalorn(doc, w, tokens, rows):
    eps, T = doc["norm"]["eps"], tokens.shape[0]
    x = w("embed")[tokens]
    for i, layer in enumerate(doc["layers"]):
        p, m, a = f"l{i}.mix", layer["mixer"], layer["mixer"]["mask"]
        heads = (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"]))
        if layer["type"] == "attention_2":
            q, k, v = ((x @ w(f"{p}.{c}").T + w(f"{p}.{c}.b")).view(T, n, -1) for c, n in heads)
            q, k = (_rotate(_rms(b, eps, w(f"{p}.{c}.norm")), m["rot"]) for b, c in ((q, "q"), (k, "k")))
            y = _attend(q, k, v, m["scale"], _causal(T, x.device, a["size"], a.get("keep_first", 0)))
        else:
            q, k, v = ((x @ w(f"{p}.{c}").T).view(T, n, -1) for c, n in heads)
            q, k = (_rms(_rotate(b, m["rot"]), eps) for b in (q, k))
            seen, bias, out = _causal(T, x.device, chunk=a["size"]), w(f"{p}.pb"), []
            for h in range(m["heads"]):
                g = h * m["kv_heads"] // m["heads"]
                s = q[:, h] @ k[:, g].T * m["scale"]
                if m.get("softcap") is not None:
                    s = m["softcap"] * torch.tanh(s / m["softcap"])
                out.append((torch.sigmoid(s + bias[h]) * seen) @ v[:, g])
            y = torch.stack(out, 1) * torch.sigmoid(x @ w(f"{p}.g").T)[:, :, None]
        x = x + _rms(y.reshape(T, -1) @ w(f"{p}.o").T, eps, w(f"l{i}.norm1").reshape(()))
        z, c = x @ w(f"l{i}.mlp.up").T, w(f"l{i}.mlp.act")
        z = c[0] * _rms(z, eps) + c[1] * _rms(z * z, eps) + c[2] * _rms(z * z * z, eps) + c[3]
        x = x + _rms(z @ w(f"l{i}.mlp.down").T, eps, w(f"l{i}.norm2").reshape(()))
    return _rms(x[rows], eps, w("final.norm").reshape(())) @ w("head").T * doc.get("logit_scale", 1.0)
