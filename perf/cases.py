"""What this framework is timed on: the work its users have it do, through the engine that ``EngineBuilder`` gives them.

Three kinds of pass, each over the sizes, weight formats and cache formats that are served:

* ``decode``: one step of the live sequences (``step_batch``, what the scheduler calls for every token): one chat alone, a
  few, a full server of 64.
* ``prompt``: a whole prompt to its first token (``open_sequence``): what a user waits for before the answer begins.
* ``verify``: the drafted tokens of speculative decoding, checked in one pass (``verify_logits``).

Models have the widths, heads and block formats of the 1.7B, 4B and 8B shapes of ``bench.py``, with a quarter of their depth
and of their vocabulary: a pass then has the parts of a whole model's in the same proportion at a quarter of the time, and
three states fit the card beside one another.  Embedding and head are tied, so the most likely next token is the last one
by a wide margin: greedy and sampled tokens do not hang on the last digits, and a decode step can be repeated.

The cached context of a decode step is drawn directly: normalised keys and values are close to unit normal, whatever text they
come from.  Weights are the same for every seed (a program keeps its model); prompts, tokens and contexts follow the seed.
"""
import math
import os
import tempfile

import numpy as np
import torch

from oxibonsai_b200.core import GgufWriter
from oxibonsai_b200.runtime import EngineBuilder

DEV = "cuda:0"
HEAD_DIM, PAGE, EPS, ROPE_BASE, EMBD_STD = 128, 64, 1e-6, 1e6, 0.25
VOCAB = 151936 // 4
MODELS = {
    "1.7b": dict(hidden=2048, inter=6144, layers=28 // 4, heads=16, kv_heads=8),
    "4b": dict(hidden=2560, inter=9728, layers=36 // 4, heads=32, kv_heads=8),
    "8b": dict(hidden=4096, inter=12288, layers=36 // 4, heads=32, kv_heads=8),
}
# GGUF type id, weights and bytes of a block
FORMATS = {"q1": (41, 128, 18), "tq2": (42, 128, 34), "q4_0": (2, 32, 18), "q8_0": (8, 32, 34), "q4_k": (12, 256, 144), "q6_k": (14, 256, 210)}
PACKED = ("q1", "tq2")
KV_BYTES = {"f16": HEAD_DIM * 2, "q8": HEAD_DIM + 4, "q4": HEAD_DIM // 2 + 4}


def _case(name, do, model, weights, kv, streams=1, shortest=0, context=0, tokens=1, preset="greedy"):
    c = dict(do=do, model=model, weights=weights, kv=kv, streams=streams, shortest=shortest or context, context=context, tokens=tokens, preset=preset)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest model and hardly any context: launches and latency
        _case("decode 1 1.7B start of a chat", "decode", "1.7b", "tq2", "f16", context=24),
        # the headline of bench.py: one stream at 4096 tokens
        _case("decode 1 8B 4096", "decode", "8b", "tq2", "f16", context=4096),
        # one reader of a long document on a 1-bit model, INT8 cache
        _case("decode 1 4B 1-bit q8 20000", "decode", "4b", "q1", "q8", context=20001),
        # a handful of chats, ragged
        _case("decode 5 8B 1-bit 90-700", "decode", "8b", "q1", "f16", streams=5, shortest=90, context=700, preset="balanced"),
        # a half-full server with the densest cache format
        _case("decode 24 4B q4 100-1500", "decode", "4b", "tq2", "q4", streams=24, shortest=100, context=1500, preset="balanced"),
        # the serving benchmark: 64 streams, prompts of 128 to 2048 tokens, INT8 cache, Balanced preset
        _case("decode 64 4B q8 128-2048", "decode", "4b", "tq2", "q8", streams=64, shortest=128, context=2048, preset="balanced"),
        # bench.py's aggregate: 64 streams at 1024 tokens
        _case("decode 64 8B 1024", "decode", "8b", "tq2", "f16", streams=64, context=1024),
        # a draft of eight tokens checked at a long context
        _case("verify 9 8B 4096", "verify", "8b", "tq2", "f16", context=4096, tokens=9),
        # an ordinary prompt of odd length into the INT8 cache
        _case("prompt 777 4B q8", "prompt", "4b", "tq2", "q8", tokens=777),
        # the longest prompt that is one chunk: time to first token of bench.py
        _case("prompt 4096 8B", "prompt", "8b", "tq2", "f16", tokens=4096),
        # checkpoints in the common block formats, which are used as stored
        _case("decode 1 8B q4_k 300", "decode", "8b", "q4_k", "f16", context=300),
        _case("prompt 500 4B q8_0", "prompt", "4b", "q8_0", "f16", tokens=500),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode one", "decode few", "decode many", "decode many", "prompt", "prompt", "verify", "blocks decode", "blocks prompt"])
    model, weights, kv = rng.choice(list(MODELS)), rng.choice(PACKED), rng.choice(["f16", "f16", "q8", "q8", "q4"])
    preset = rng.choice(["greedy", "balanced"])
    if kind == "decode one":
        return _case("", "decode", model, weights, kv, context=_log(rng, 16, 24000), preset=preset)
    if kind in ("decode few", "decode many"):
        streams = _log(rng, 2, 12) if kind == "decode few" else rng.randint(13, 64)
        context = _log(rng, 64, 2048 if streams > 12 else 4096)
        return _case("", "decode", model, weights, kv, streams=streams, shortest=rng.randint(max(16, context // 16), context), context=context, preset=preset)
    if kind == "prompt":
        return _case("", "prompt", model, weights, kv, tokens=_log(rng, 17, 4096), preset=preset)
    if kind == "verify":
        return _case("", "verify", model, weights, kv, context=_log(rng, 64, 8192), tokens=rng.randint(2, 9))
    weights = rng.choice([f for f in FORMATS if f not in PACKED])
    if kind == "blocks decode":
        context = _log(rng, 20, 500)
        streams = _log(rng, 1, 8)
        return _case("", "decode", model, weights, kv, streams=streams, shortest=rng.randint(max(18, context // 4), max(18, context)), context=max(18, context), preset=preset)
    return _case("", "prompt", model, weights, kv, tokens=_log(rng, 18, 1000), preset=preset)


def _lengths(case):
    """Context length of every stream: evenly spread between shortest and longest, neighbours not alike."""
    n, lo, hi = case["streams"], case["shortest"], case["context"]
    spread = [hi - (hi - lo) * i // max(1, n - 1) for i in range(n)]
    step = next(s for s in range(max(1, int(n * 0.382)), n + 2) if math.gcd(s, n) == 1)
    return [spread[i * step % n] for i in range(n)]


# ---- the checkpoint ---------------------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _matrices(case):
    """(name, rows, columns, root mean square of a weight) of one layer."""
    m = MODELS[case["model"]]
    h, i, qd, kvd = m["hidden"], m["inter"], m["heads"] * HEAD_DIM, m["kv_heads"] * HEAD_DIM
    return [("attn_q", qd, h, h ** -0.5), ("attn_k", kvd, h, h ** -0.5), ("attn_v", kvd, h, h ** -0.5), ("attn_output", h, qd, 0.25 * qd ** -0.5),
            ("ffn_gate", i, h, h ** -0.5), ("ffn_up", i, h, h ** -0.5), ("ffn_down", h, i, 0.4 * i ** -0.5)]


def _half_bytes(x):
    return x.half().contiguous().view(torch.uint8).reshape(*x.shape, 2)


def _blocks(fmt, layer, index, rows, cols, rms):
    """The blocks of one matrix as bytes [rows, blocks, bytes of a block]."""
    _, per, nbytes = FORMATS[fmt]
    g, nb = _gen(1000 * layer + index + 7), cols // per
    b = torch.randint(0, 256, (rows, nb, nbytes), dtype=torch.uint8, device=DEV, generator=g)
    d = 1 + 0.1 * torch.randn((rows, nb), device=DEV, generator=g)
    if fmt == "tq2":
        for j in range(4):                      # codes 0, 1, 2 for -1, 0, +1
            c = torch.randint(0, 3, (rows, nb, 32), dtype=torch.uint8, device=DEV, generator=g)
            b[..., :32] = c if j == 0 else b[..., :32] | (c << (2 * j))
        b[..., 32:] = _half_bytes(d * rms * 1.5 ** 0.5)
    elif fmt == "q1":
        b[..., :2] = _half_bytes(d * rms)
    elif fmt == "q4_0":
        b[..., :2] = _half_bytes(d * rms / 4.6)
    elif fmt == "q8_0":
        b[..., :2] = _half_bytes(d * rms / 74)
    elif fmt == "q4_k":                         # eight scales of six bits, minima of 7.5 steps each: no mean
        sc = torch.randint(32, 64, (rows, nb, 8), dtype=torch.uint8, device=DEV, generator=g)
        lo, hi = sc & 15, sc >> 4
        low = lo[..., 0::2] | (lo[..., 1::2] << 4)
        b[..., 4:8], b[..., 8:12] = low, low
        for half in range(2):
            q = hi[..., 4 * half:4 * half + 4]
            b[..., 12 + half] = b[..., 14 + half] = q[..., 0] | (q[..., 1] << 2) | (q[..., 2] << 4) | (q[..., 3] << 6)
        d = (d * rms / (48 * 4.6)).half().float()
        b[..., :2], b[..., 2:4] = _half_bytes(d), _half_bytes(d * 7.5)
    else:                                       # q6_k
        sign = torch.randint(0, 2, (rows, nb, 16), device=DEV, generator=g) * 2 - 1
        sc = torch.randint(32, 128, (rows, nb, 16), device=DEV, generator=g) * sign
        b[..., 192:208] = sc.to(torch.int8).view(torch.uint8)
        b[..., 208:] = _half_bytes(d * rms / (84 * 18.5))
    return b


def _bits(b, width):
    """Unpacks bytes [..., n] into values of `width` bits, lowest first: [..., n * 8 / width]."""
    s = torch.arange(0, 8, width, dtype=torch.uint8, device=b.device)
    return ((b[..., None] >> s) & ((1 << width) - 1)).flatten(-2)


def _dequantize(fmt, b):
    """The matrix that the blocks stand for, in 64 bits [rows, columns]."""
    half = lambda lo: b[..., lo:lo + 2].contiguous().view(torch.float16).double()  # noqa: E731
    if fmt == "tq2":
        w = (_bits(b[..., :32], 2).double() - 1) * half(32)
    elif fmt == "q1":
        w = (_bits(b[..., 2:], 1).double() * 2 - 1) * half(0)
    elif fmt == "q4_0":
        w = (_bits(b[..., 2:], 4).double() - 8) * half(0)
    elif fmt == "q8_0":
        w = b[..., 2:].contiguous().view(torch.int8).double() * half(0)
    elif fmt == "q4_k":
        def six(at, high):
            return (_bits(b[..., 4 + at:8 + at], 4) | (_bits(b[..., 12 + high:14 + high], 2) << 4)).double()
        w = (_bits(b[..., 16:], 4).double().unflatten(-1, (8, 32)) * (half(0) * six(0, 0))[..., None] - (half(2) * six(4, 2))[..., None]).flatten(-2)
    else:
        q = (_bits(b[..., :128], 4) | (_bits(b[..., 128:192], 2) << 4)).double() - 32
        sc = b[..., 192:208].contiguous().view(torch.int8).double() * half(208)
        w = (q.unflatten(-1, (16, 16)) * sc[..., None]).flatten(-2)
    return w.flatten(-2)


def _embedding(case):
    return (EMBD_STD * torch.randn((VOCAB, MODELS[case["model"]]["hidden"]), device=DEV, generator=_gen(3))).half()


def _checkpoint(case):
    """Path of the model's GGUF file; written on first use."""
    m, fmt = MODELS[case["model"]], case["weights"]
    folder = os.path.join(tempfile.gettempdir(), "oxibonsai_cases_%d" % os.getuid())
    path = os.path.join(folder, "%s_%s_v1.gguf" % (case["model"], fmt))
    if os.path.exists(path):
        return path
    os.makedirs(folder, exist_ok=True)
    w = GgufWriter()
    w.add("general.architecture", "qwen3").add("general.name", "%s %s, a quarter" % (case["model"], fmt))
    for key, value in (("embedding_length", m["hidden"]), ("block_count", m["layers"]), ("attention.head_count", m["heads"]),
                       ("attention.head_count_kv", m["kv_heads"]), ("attention.key_length", HEAD_DIM), ("feed_forward_length", m["inter"]),
                       ("vocab_size", VOCAB), ("context_length", 65536), ("attention.layer_norm_rms_epsilon", EPS), ("rope.freq_base", ROPE_BASE)):
        w.add("qwen3." + key, value)

    def ones(name, n):
        w.add_tensor(name + ".weight", (n,), 0, np.ones(n, dtype=np.float32))

    w.add_tensor("token_embd.weight", (m["hidden"], VOCAB), 1, _embedding(case).cpu().numpy())
    ones("output_norm", m["hidden"])
    for layer in range(m["layers"]):
        p = "blk.%d." % layer
        for name, n in (("attn_norm", m["hidden"]), ("ffn_norm", m["hidden"]), ("attn_q_norm", HEAD_DIM), ("attn_k_norm", HEAD_DIM)):
            ones(p + name, n)
        for index, (name, rows, cols, rms) in enumerate(_matrices(case)):
            w.add_tensor(p + name + ".weight", (cols, rows), FORMATS[fmt][0], _blocks(fmt, layer, index, rows, cols, rms).cpu().numpy())
    part = "%s.%d" % (path, os.getpid())
    w.write(part)
    os.replace(part, path)
    return path


# ---- the cached context ------------------------------------------------------------------------------------------------------------

def _context_rows(case, seed, layer, pages):
    """Cached keys and values of one layer as the cache holds them: [(codes or rows, scales or None)] for K and V."""
    m, g, out = MODELS[case["model"]], _gen(int(seed) * 131 + layer * 7 + 1), []
    for _ in range(2):
        x = torch.randn((pages, m["kv_heads"], PAGE, HEAD_DIM), device=DEV, generator=g)
        if case["kv"] == "f16":
            out.append((x.half(), None))
            continue
        top = 127 if case["kv"] == "q8" else 7
        scale = x.abs().amax(-1) / top
        q = (x / scale[..., None]).round().clamp(-top, top).to(torch.int8)
        if case["kv"] == "q4":
            n = (q + 8).to(torch.uint8)
            q = n[..., 0::2] | (n[..., 1::2] << 4)
        out.append((q, scale))
    return out


def _read_rows(case, rows):
    """The values that the cached rows stand for, in 64 bits."""
    q, scale = rows
    if scale is None:
        return q.double()
    v = _bits(q, 4).double() - 8 if case["kv"] == "q4" else q.double()
    return v * scale.double()[..., None]


def _tokens(case, seed):
    """A case's own tokens: the last one of every stream, a prompt, or drafted tokens."""
    g = _gen(int(seed) * 17 + 5)
    n = case["streams"] if case["do"] == "decode" else case["tokens"]
    return torch.randint(0, VOCAB, (n,), device=DEV, generator=g, dtype=torch.int32)


def _prompts(case, seed):
    """Decoding from block formats: the prompts that fill the cache through the engine, one per stream."""
    g = _gen(int(seed) * 19 + 11)
    return [torch.randint(0, VOCAB, (n,), device=DEV, generator=g, dtype=torch.int32).tolist() for n in _lengths(case)]


def _pages(n):
    return -(-n // PAGE)


# ---- what is timed -------------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    blocks, do = case["weights"] not in PACKED, case["do"]
    lengths = _lengths(case) if do != "prompt" else [0]
    fed = 1 if do == "decode" else case["tokens"] + (do == "prompt")
    totals = [n + fed for n in lengths]
    pages = None if blocks else sum(_pages(n) for n in totals)
    eng = (EngineBuilder().model_path(_checkpoint(case)).preset(case["preset"]).max_seq_len(-(-max(totals) // PAGE) * PAGE)
           .max_batch(case["streams"]).kv_cache(case["kv"], pages=pages).build())
    state = dict(do=do, engine=eng, kv=case["kv"], logits=eng._eng.logits if blocks else eng.runner.logits)
    if do == "prompt":
        prompt = _tokens(case, seed).tolist()
        return dict(state, prompt=prompt, blocks=blocks, total=len(prompt) + 1)
    if do == "decode" and blocks:
        for slot, prompt in enumerate(_prompts(case, seed)):
            eng.begin_sequence(prompt, len(prompt) + 1, slot)
            eng.prefill(prompt, slot, 0)
            eng.finish_sequence(prompt, slot)
        eng.step_batch(lengths)
        return dict(state, positions=lengths)
    tokens = _tokens(case, seed)
    # the last token of a stream is fed again before the timed step: it is sampled once more, and the sampler leaves it to the step
    last = tokens.tolist()
    for slot, n in enumerate(lengths):
        eng.begin_sequence([last[slot]] * n, totals[slot], slot)
    for layer in range(MODELS[case["model"]]["layers"]):
        for (rows, scale), pool, scales in zip(_context_rows(case, seed, layer, pages), (eng.kv.k, eng.kv.v), (eng.kv.k_scale, eng.kv.v_scale)):
            pool[layer].copy_(rows)
            if scale is not None:
                scales[layer].copy_(scale)
    if do == "verify":
        eng.runner.verify_logits(tokens, 0, lengths[0])
        return dict(state, tokens=tokens, position=lengths[0])
    for slot, n in enumerate(lengths):
        eng.prefill([last[slot]], slot, n - 1)
        eng.finish_sequence([last[slot]] * n, slot)
    eng.step_batch(lengths)
    return dict(state, positions=lengths)


def run(state):
    eng = state["engine"]
    if state["do"] == "decode":
        return {"tokens": np.array(eng.step_batch(state["positions"])), "logits": state["logits"]}
    if state["do"] == "verify":
        return {"logits": eng.runner.verify_logits(state["tokens"], 0, state["position"])}
    if state["blocks"]:
        eng.begin_sequence(state["prompt"], state["total"], 0)
        eng.prefill(state["prompt"], 0, 0)
        return {"token": eng.finish_sequence(state["prompt"], 0), "logits": state["logits"]}
    out = {"token": eng.open_sequence(state["prompt"], state["total"], 0), "logits": state["logits"]}
    if state["kv"] == "f16":
        out.update(keys=eng.kv.k, values=eng.kv.v)       # the cache that the prompt leaves behind
    return out


def _sizes(case):
    """(rows that pass the layers, rows that pass the head, [(context, fed)] of every stream)."""
    if case["do"] == "decode":
        return case["streams"], case["streams"], [(n, 1) for n in _lengths(case)]
    if case["do"] == "verify":
        return case["tokens"], case["tokens"], [(case["context"], case["tokens"])]
    return case["tokens"], 1, [(0, case["tokens"])]


def work(case):
    """Weights and head once, the cached rows once, the rows that are added, the logits; products of all rows, causal attention."""
    m, (_, per, nbytes) = MODELS[case["model"]], FORMATS[case["weights"]]
    rows, heads_rows, streams = _sizes(case)
    weights = m["layers"] * sum(r * c for _, r, c, _ in _matrices(case))
    row_bytes = 2 * m["layers"] * m["kv_heads"] * KV_BYTES[case["kv"]]
    pairs = sum(fed * n + fed * (fed + 1) // 2 for n, fed in streams)
    return {"bytes": weights // per * nbytes + 2 * VOCAB * m["hidden"] + sum(n + fed for n, fed in streams) * row_bytes + 4 * heads_rows * VOCAB,
            "flops": 2 * weights * rows + 2 * VOCAB * m["hidden"] * heads_rows + 4 * m["layers"] * m["heads"] * HEAD_DIM * pairs}


def tolerance(case):
    """Four times what the logits are off the 64-bit ones: f16 operands of the tensor cores and f16 cache rows 0.0002 (one stream) to
    0.0009, INT8 rows up to 0.0024, INT4 rows up to 0.0053."""
    return {"rel": {"f16": 0.004, "q8": 0.008, "q4": 0.02}[case["kv"]]}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------------------

def _rms(x):
    return x / (x.square().mean(-1, keepdim=True) + EPS).sqrt()


def _rotate(x, positions):
    """Rotary positions, halves paired; the angles are 32-bit products, as the model format defines them."""
    freq = torch.tensor([1.0 / np.float32(ROPE_BASE) ** np.float32(2 * i / HEAD_DIM) for i in range(HEAD_DIM // 2)], dtype=torch.float32, device=DEV)
    a = (positions.float()[:, None] * freq).double()
    c, s = a.cos()[:, None], a.sin()[:, None]
    lo, hi = x[..., :HEAD_DIM // 2], x[..., HEAD_DIM // 2:]
    return torch.cat([lo * c - hi * s, lo * s + hi * c], -1)


def _forward(case, streams, rows_of):
    """Logits-ready rows of every token in `streams` [(tokens, first position)] and the keys and values they add;
    rows_of(layer) gives [(K, V)] per stream, [context, kv heads, 128] each, or None."""
    m, kept = MODELS[case["model"]], []
    heads, kvh = m["heads"], m["kv_heads"]
    embd = _embedding(case)
    h = torch.cat([embd[t.long()] for t, _ in streams]).double()
    pos = torch.cat([torch.arange(p, p + len(t), device=DEV) for t, p in streams])
    for layer in range(m["layers"]):
        w = [_dequantize(case["weights"], _blocks(case["weights"], layer, i, r, c, rms)) for i, (_, r, c, rms) in enumerate(_matrices(case))]
        x = _rms(h)
        q = _rotate(_rms((x @ w[0].T).unflatten(-1, (heads, HEAD_DIM))), pos)
        k = _rotate(_rms((x @ w[1].T).unflatten(-1, (kvh, HEAD_DIM))), pos)
        v = (x @ w[2].T).unflatten(-1, (kvh, HEAD_DIM))
        kept.append((k, v))
        out, at, before = torch.empty_like(q), 0, rows_of(layer)
        for i, (t, p) in enumerate(streams):
            s = slice(at, at + len(t))
            at += len(t)
            ks, vs = (k[s], v[s]) if before is None else (torch.cat([before[i][0], k[s]]), torch.cat([before[i][1], v[s]]))
            for g in range(kvh):
                qg = q[s, g * heads // kvh:(g + 1) * heads // kvh].transpose(0, 1)
                score = qg @ ks[:, g].T / HEAD_DIM ** 0.5
                score.masked_fill_(torch.arange(ks.shape[0], device=DEV)[None] > pos[s, None], -math.inf)
                out[s, g * heads // kvh:(g + 1) * heads // kvh] = (score.softmax(-1) @ vs[:, g]).transpose(0, 1)
        h = h + out.flatten(1) @ w[3].T
        x = _rms(h)
        h = h + (torch.nn.functional.silu(x @ w[4].T) * (x @ w[5].T)) @ w[6].T
    return _rms(h), kept, embd


def exact(case, seed):
    if case["do"] == "prompt":
        tokens = _tokens(case, seed)
        h, kept, embd = _forward(case, [(tokens, 0)], lambda layer: None)
        out = {"token": None, "logits": h[-1:] @ embd.double().T}
        if case["weights"] in PACKED and case["kv"] == "f16":
            pages = _pages(len(tokens) + 1)

            def paged(rows):
                full = torch.zeros((pages * PAGE, *rows.shape[1:]), dtype=rows.dtype, device=DEV)
                full[:len(tokens)] = rows
                return full.unflatten(0, (pages, PAGE)).transpose(1, 2)

            out.update(keys=torch.stack([paged(k) for k, _ in kept]), values=torch.stack([paged(v) for _, v in kept]))
        return out
    lengths = _lengths(case)
    if case["weights"] not in PACKED:
        streams = [(torch.tensor(p + p[-1:], device=DEV), 0) for p in _prompts(case, seed)]
        h, _, embd = _forward(case, streams, lambda layer: None)
        ends = torch.tensor([len(t) for t, _ in streams], device=DEV).cumsum(0) - 1
        return {"tokens": None, "logits": h[ends] @ embd.double().T}
    tokens = _tokens(case, seed)
    verify = case["do"] == "verify"
    fed = case["tokens"] if verify else 1
    pages = [_pages(n + fed) for n in lengths]
    known = [n if verify else n - 1 for n in lengths]       # rows drawn; a decode step's last row is the token's own

    def rows_of(layer):
        k, v = (_read_rows(case, r) for r in _context_rows(case, seed, layer, sum(pages)))
        out, at = [], 0
        for n, count in zip(known, pages):                  # the pool hands its pages out in order
            out.append(tuple(x[at:at + count].transpose(1, 2).flatten(0, 1)[:n] for x in (k, v)))
            at += count
        return out

    if verify:
        h, _, embd = _forward(case, [(tokens, known[0])], rows_of)
        return {"logits": h @ embd.double().T}
    h, _, embd = _forward(case, [(t.repeat(2), n) for t, n in zip(tokens, known)], rows_of)
    return {"tokens": None, "logits": h[1::2] @ embd.double().T}
