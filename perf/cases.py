"""The work whose speed is measured: what a program that uses this engine has it do, at sizes of this repository's benchmark.

Two forms of it.  A `step` is one step of the engine over a model of a few layers with its output head, as generation runs it: single
tokens of live requests replayed from captured graphs, or prompt portions beside them by the native runner.  The others are single
layers as the seven architectures are assembled from: embedding, a block of one mixer (or a feed-forward), and the norm that reads the
stream next, called the way a model's walk calls them.  `sampling` picks tokens from logits.

Every tensor is a function of (seed, its name), so `exact` can state the same computation in 64 bits without the package.
"""
from __future__ import annotations

import hashlib
import math

import torch

from kestrel_llm_b200.cache.manager import CacheManager
from kestrel_llm_b200.config import EngineOptions, Qwen3Config
from kestrel_llm_b200.config.registry import resolve_architecture
from kestrel_llm_b200.engine import Engine, Entry, StepBatch
from kestrel_llm_b200.parts import (ChannelDeltaMixer, ForgetGateRecurrence, GatedMLP, GatedWindowAttention, GroupedQueryAttention,
                                    LatentAttention, ParallelMixers, PreNormBlock, RemovalDeltaMixer, RMSNorm, RotaryHalf,
                                    RotaryInterleaved, RoutedExperts, TokenEmbedding)
from kestrel_llm_b200.sampling import SamplingParams
from kestrel_llm_b200.sampling.sampler import Sampler

DEV = "cuda:0"
EPS = 1e-6
PAGE = 16
ROWS = 8192             # rows of a single layer's token table
STEP_LAYERS = 4         # layers of the models that take whole steps
STEP = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=STEP_LAYERS, hidden_size=4096, num_attention_heads=32,
            num_key_value_heads=8, head_dim=128, intermediate_size=12288, vocab_size=151936, rope_theta=1000000.0, rms_norm_eps=EPS,
            tie_word_embeddings=False, attention_bias=False, max_position_embeddings=40960, hidden_act="silu")
# the two layer sizes of the benchmark's workloads
SIZES = {"a": dict(width=2048, heads=16, kv=4, window=1024, ff=6144, q_rank=768, rank=64, experts=32, e_ff=768),
         "b": dict(width=4096, heads=32, kv=8, window=2048, ff=12288, q_rank=1536, rank=128, experts=64, e_ff=1024)}
HEAD = 128              # head size
KEEP = 4                # first tokens that a window keeps
TOP = 4                 # experts of a token
LATENT, LATENT_ROT = 192, 64
R_DIM = 64              # key channels of a forget-gate head
TAPS = 4
THETA = {"dense": 1000000.0, "latent": 10000.0, "parallel": 500000.0}
DECAY_RATE = math.exp(-0.5)


def listed():
    return [
        # one user generating: a single token behind about a thousand, bound by the weights' bytes and by latency
        dict(name="decode_one", kind="step", decode=1, portion=0, context=1000),
        # the headline serving load: eight requests at contexts up to 4,096
        dict(name="decode_eight", kind="step", decode=8, portion=0, context=4096),
        # continuous batching: a prompt portion beside requests that decode
        dict(name="mixed_step", kind="step", decode=12, portion=500, context=1500),
        # a layer of the dense decoder over a whole prompt
        dict(name="dense_prompt", kind="dense", size="b", dtype="bfloat16", tokens=2048, requests=1, context=0),
        # the same layer on the true 32-bit path, which replays and checks run on, with two ragged prompts
        dict(name="dense_float32", kind="dense", size="a", dtype="float32", tokens=411, requests=2, context=0),
        # window attention that keeps a request's first tokens, gated per head, over a whole prompt
        dict(name="window_prompt", kind="window", size="a", dtype="bfloat16", tokens=2048, requests=1, context=0),
        # gated delta rule with a decay per key channel over two prompts
        dict(name="delta_prompts", kind="delta", size="a", dtype="bfloat16", tokens=1777, requests=2, context=0),
        # routed experts over a prompt portion
        dict(name="experts_portion", kind="experts", size="a", dtype="bfloat16", tokens=1000, requests=1, context=0),
        # attention over cached latents with a rotated part: a later portion of a long prompt
        dict(name="latent_portion", kind="latent", size="a", dtype="bfloat16", tokens=1024, requests=1, context=2000),
        # attention with a learned softmax term beside a forget-gate recurrence
        dict(name="parallel_prompt", kind="parallel", size="a", dtype="bfloat16", tokens=2048, requests=1, context=0),
        # generalised delta rule: a few tokens of three requests that go on, where launches count
        dict(name="removal_portions", kind="removal", size="a", dtype="bfloat16", tokens=700, requests=3, context=300),
        # picking the next tokens of sixteen requests with all filters
        dict(name="sampling", kind="sampling", rows=16, vocab=151936, top_k=50, top_p=0.9, min_p=0.02),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["step", "step", "dense", "window", "delta", "experts", "latent", "parallel", "removal", "sampling"])
    if kind == "step":
        portion = rng.choice([0, spread(2, 1024)])
        return dict(kind=kind, decode=spread(1, 8) if not portion else rng.randint(0, 12), portion=portion, context=spread(16, 4096))
    if kind == "sampling":
        return dict(kind=kind, rows=spread(1, 16), vocab=rng.choice([32000, 64000, 151936]), top_k=rng.choice([0, 20, 50]),
                    top_p=rng.choice([1.0, 0.9, 0.95]), min_p=rng.choice([0.0, 0.02]))
    dtype = "float32" if kind == "dense" and rng.random() < 0.3 else "bfloat16"
    size = rng.choice(["a", "a", "b"]) if dtype == "bfloat16" else "a"
    tokens = spread(1, 400 if dtype == "float32" else 1024 if size == "b" else 2048)
    return dict(kind=kind, size=size, dtype=dtype, tokens=tokens, requests=min(tokens, rng.randint(1, 4)),
                context=rng.choice([0, spread(16, 3000)]))


# ---- numbers from (seed, name) -----------------------------------------------------------------

def _tensor(seed, name, shape, mean=0.0, std=1.0):
    """Normal numbers on the device (standard deviation 0: uniform in [0, 1)), float32."""
    gen = torch.Generator(device=DEV).manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    t = torch.empty(tuple(shape), dtype=torch.float32, device=DEV)
    return t.normal_(mean, std, generator=gen) if std else t.uniform_(0.0, 1.0, generator=gen)


def _weight(seed, name, shape, dtype):
    """A weight by its checkpoint name, as it is stored: matrices and biases N(0, 0.02), norm weights around one, and what sets a
    recurrence's memory as a trained model has it (hundreds of tokens)."""
    last = name.rsplit(".", 1)[-1]
    if "norm" in last:
        mean, std = 1.0, 0.02
    elif last in ("dt_bias", "w0"):
        mean, std = -1.0, 1.0
    elif last == "A_log":
        mean, std = -0.5, 0.5
    elif name.endswith("f.b"):
        mean, std = 2.0, 1.0
    elif last == "lower":
        mean, std = 0.0, 0.0
    elif last == "conv":
        mean, std = 0.0, 0.5
    elif last == "o":               # heads that average over many keys: the mixer's result is of the stream's size
        mean, std = 0.0, 0.1
    else:
        mean, std = 0.0, 0.02
    return _tensor(seed, name, shape, mean, std).to(dtype)


def _fill(parts, seed, dtype):
    for part in parts:
        for slot in part.weight_slots():
            slot.dest.copy_(_weight(seed, slot.name, slot.dest.shape, dtype))


def _ids(seed, n, vocab):
    gen = torch.Generator().manual_seed(seed * 7919 + 11)
    return torch.randint(0, vocab, (n,), generator=gen)


def _portions(case):
    """(tokens, context) of every request: unequal portions that add up, unequal contexts up to the case's."""
    if case["kind"] == "step":
        ctx, n = case["context"], case["decode"]
        out = [(1, ctx - (ctx * i) // (3 * max(1, n))) for i in range(n)]
        if case["portion"] > 1:
            out.append((case["portion"], ctx // 2))
        elif case["portion"] == 1:
            out.append((1, ctx // 2))
        return out
    n, T, ctx = case["requests"], case["tokens"], case["context"]
    edges = [T * i * (i + 1) // (n * (n + 1)) for i in range(n + 1)]
    for i in range(1, n + 1):                       # every request has a token
        edges[i] = max(edges[i], edges[i - 1] + 1)
    for i in range(n, 0, -1):
        edges[i] = min(edges[i], T - (n - i))
    return [(edges[i + 1] - edges[i], ctx - (ctx * i) // (2 * n)) for i in range(n)]


def _context(seed, layer, rid, length, heads, dim, dtype):
    """Keys (or values) that earlier steps left in the cache."""
    return _tensor(seed, f"cache.{layer}.{rid}", (length, heads, dim)).to(dtype)


def _fill_pages(plane, pages, rows):
    """rows [n, heads, dim] into the pages of a request (those the window has given back are -1)."""
    n, heads, dim = rows.shape
    full = torch.zeros((len(pages) * PAGE, heads, dim), dtype=rows.dtype, device=rows.device)
    full[:n] = rows[:len(pages) * PAGE]
    paged = full.view(len(pages), PAGE, heads, dim).permute(0, 2, 1, 3)
    at = torch.tensor(pages, device=rows.device)
    plane[at[at >= 0]] = paged[at >= 0]


# ---- prepare and run ---------------------------------------------------------------------------

class _State:
    pass


def _layer_parts(case, dtype):
    """(embedding, block or feed-forward, the norm that reads the stream next)."""
    z, kind = SIZES[case["size"]], case["kind"]
    W, H, G = z["width"], z["heads"], z["kv"]
    if kind == "experts":
        ffn = RoutedExperts(W, z["e_ff"], z["experts"], TOP, 7.0, dtype, DEV, "mlp.")
        return TokenEmbedding(ROWS, W, dtype, DEV, "embed"), ffn, RMSNorm(W, EPS, DEV, "after.norm")
    norm2 = ffn = None
    if kind == "dense":
        mixer = GroupedQueryAttention(W, H, G, HEAD, dtype, DEV, "mix.", RotaryHalf(HEAD, THETA["dense"], DEV), qk_norm_eps=EPS)
        norm2, ffn = RMSNorm(W, EPS, DEV, "second.norm"), GatedMLP(W, z["ff"], dtype, DEV, "mlp.")
    elif kind == "window":
        mixer = GatedWindowAttention(W, H, G, HEAD, HEAD, dtype, DEV, "mix.", HEAD ** -0.5, EPS, window=z["window"], keep_first=KEEP)
    elif kind == "delta":
        mixer = ChannelDeltaMixer(W, H, G, HEAD, HEAD, TAPS, z["rank"], z["rank"], EPS, dtype, DEV, "mix.")
    elif kind == "latent":
        mixer = LatentAttention(W, H, HEAD, HEAD, z["q_rank"], LATENT, dtype, DEV, "mix.", (HEAD + LATENT_ROT) ** -0.5, EPS, head_gate=False,
                                element_gate=True, rot_dim=LATENT_ROT,
                                position=RotaryInterleaved(LATENT_ROT, THETA["latent"], DEV, rotary_dim=LATENT_ROT))
    elif kind == "parallel":
        left = GatedWindowAttention(W, H, G, HEAD, HEAD, dtype, DEV, "mix.left.", HEAD ** -0.5, EPS, head_gate=False, bias=True, out_bias=False,
                                    qk_norm=None, weighting="softmax_sink", head_sink=True,
                                    position=RotaryInterleaved(HEAD, THETA["parallel"], DEV, rotary_dim=HEAD // 2))
        right = ForgetGateRecurrence(W, H, R_DIM, HEAD, EPS, dtype, DEV, "mix.right.")
        mixer = ParallelMixers(left, right, W, EPS, DEV, "mix.", names=("left.norm", "right.norm2"))
    else:
        mixer = RemovalDeltaMixer(W, H, HEAD, z["rank"], DECAY_RATE, EPS, dtype, DEV, "mix.")
    block = PreNormBlock(RMSNorm(W, EPS, DEV, "first.norm"), mixer, norm2, ffn, dtype)
    return TokenEmbedding(ROWS, W, dtype, DEV, "embed"), block, RMSNorm(W, EPS, DEV, "after.norm")


def _prepare_step(case, seed):
    s = _State()
    portions = _portions(case)
    cfg = Qwen3Config.from_dict(dict(STEP))
    model = resolve_architecture(cfg.architecture).build(cfg, torch.bfloat16, DEV)
    _fill([model], seed, torch.bfloat16)
    longest = max(n + c for n, c in portions) + PAGE
    s.engine = Engine(model, EngineOptions(dtype="bfloat16", page_size=PAGE, batch_max=16, max_model_len=longest,
                                           max_tokens=sum(n + c + PAGE for n, c in portions), max_step_tokens=2048, prefill_batch=2048))
    cache = s.engine.cache
    cache.shuffle_free(seed)
    ids = _ids(seed, sum(n for n, _ in portions), cfg.vocab_size).tolist()
    s.entries, at = [], 0
    for rid, (n, ctx) in enumerate(portions):
        s.engine.admit(rid)
        cache.reserve(rid, ctx)
        cache.commit(rid, ctx)
        for i in range(STEP_LAYERS):
            pages = cache.block_table(rid, 0)
            _fill_pages(cache.k[i], pages, _context(seed, f"k{i}", rid, ctx, cfg.num_key_value_heads, HEAD, torch.bfloat16))
            _fill_pages(cache.v[i], pages, _context(seed, f"v{i}", rid, ctx, cfg.num_key_value_heads, HEAD, torch.bfloat16))
        cache.reserve(rid, n)
        s.entries.append(Entry(rid, ids[at:at + n], (n - 1,)))
        at += n
    s.decode_only = all(n == 1 for n, _ in portions)
    _run_step(s)                    # a program warms up at its start: captured graphs, workspaces
    return s


def _run_step(s):
    # what Engine.step launches, without the commit that would lengthen the requests, so that a pass can be repeated
    engine = s.engine
    logits = engine.graphs.run(s.entries)[0] if s.decode_only else engine.runner.step(s.entries, engine.vocab_size)
    return {"logits": logits, "k": engine.cache.k[-1], "v": engine.cache.v[-1]}


def _prepare_layer(case, seed):
    s = _State()
    dtype = getattr(torch, case["dtype"])
    s.dtype, s.kind = dtype, case["kind"]
    s.embedding, s.layer, s.after = _layer_parts(case, dtype)
    parts = [s.embedding, s.layer, s.after]
    _fill(parts, seed, dtype)
    portions = _portions(case)
    spec = s.layer.cache_spec() if case["kind"] != "experts" else None
    pages = sum((n + c + PAGE) // PAGE + 1 for n, c in portions)
    cache = CacheManager([spec], dtype, torch.device(DEV), PAGE, pages, len(portions), max(n + c for n, c in portions) + PAGE)
    cache.shuffle_free(seed)
    s.cache = cache.layer(0)
    s.manager = cache
    ids = _ids(seed, sum(n for n, _ in portions), ROWS).tolist()
    entries, at = [], 0
    for rid, (n, ctx) in enumerate(portions):
        cache.admit(rid)
        cache.reserve(rid, ctx)
        cache.commit(rid, ctx)
        if s.cache.k is not None and ctx:
            table = cache.block_table(rid, 0)
            heads, dim = s.cache.k.shape[1], s.cache.k.shape[3]
            _fill_pages(s.cache.k, table, _context(seed, "k0", rid, ctx, heads, dim, dtype))
            if s.cache.v is not s.cache.k:
                _fill_pages(s.cache.v, table, _context(seed, "v0", rid, ctx, heads, s.cache.v.shape[3], dtype))
        if s.cache.state is not None and ctx:
            s.cache.state[cache.slot(rid)] = _tensor(seed, f"state.{rid}", (s.cache.state.shape[1],), 0.0, 0.3)
        cache.reserve(rid, n)
        entries.append(Entry(rid, ids[at:at + n], (n - 1,)))
        at += n
    s.before = s.cache.state.clone() if s.cache.state is not None else None
    s.slots = [cache.slot(rid) for rid in range(len(portions))]
    s.batch = StepBatch(entries, cache, torch.device(DEV))      # the step's description, which all of its layers share
    if case["kind"] == "experts":                               # a feed-forward is handed normed activations
        s.h = _tensor(seed, "h", (at, s.embedding.width)).to(dtype)
    return s


def _run_layer(s):
    x = s.embedding.forward(s.batch.token_ids)
    if s.kind == "experts":
        return {"y": s.after.add_forward(x, s.layer.forward(s.h, s.batch), s.dtype), "x": x}
    if s.before is not None:
        s.cache.state.copy_(s.before)                           # the requests' states as the steps before left them
    x, pending = s.layer.forward(x, None, s.batch, s.cache)
    out = {"y": s.after.add_forward(x, pending, s.dtype), "x": x}
    if s.cache.k is not None:
        out["k"] = s.cache.k
    if s.cache.state is not None:
        out["state"] = [s.cache.state[slot] for slot in s.slots]
    return out


def prepare(case, seed):
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    if case["kind"] != "sampling":
        return _prepare_layer(case, seed)
    s = _State()
    s.kind, n = "sampling", case["rows"]
    s.logits = _tensor(seed, "logits", (n, case["vocab"]), 0.0, 2.5)
    s.sampler = Sampler(DEV)
    s.params = [SamplingParams(temperature=0.7 + 0.02 * i, top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"]) for i in range(n)]
    s.seeds, s.indices = [seed + i for i in range(n)], [5 + i for i in range(n)]
    return s


def run(state):
    if hasattr(state, "engine"):
        return _run_step(state)
    if state.kind == "sampling":
        return state.sampler.sample(state.logits, state.params, state.seeds, state.indices)
    return _run_layer(state)


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "sampling":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 0.0}
    portions = _portions(case)
    T = sum(n for n, _ in portions)
    pairs = sum(n * c + n * (n + 1) / 2 for n, c in portions)      # (query, key) pairs of causal attention
    keys = sum(n + c for n, c in portions)
    if kind == "step":
        W, H, G, ff, V = 4096, 32, 8, 12288, STEP["vocab_size"]
        layer = W * HEAD * (2 * H + 2 * G) + 3 * W * ff
        rows = len(portions)
        return {"bytes": 2.0 * STEP_LAYERS * (layer + 2 * keys * G * HEAD) + 2.0 * V * W + 4.0 * rows * V,
                "flops": 2.0 * T * STEP_LAYERS * layer + 4.0 * STEP_LAYERS * H * HEAD * pairs + 2.0 * rows * V * W}
    z = SIZES[case["size"]]
    W, H, G, e = z["width"], z["heads"], z["kv"], 4 if case["dtype"] == "float32" else 2
    nbytes, flops = T * W * (2.0 * e + 4.0), 0.0                   # table rows in, the stream and its norm out
    if kind == "experts":
        share = 1.0 - (1.0 - TOP / z["experts"]) ** T
        per = 3 * W * z["e_ff"]
        return {"bytes": nbytes + T * W * e + e * (z["experts"] * share * per + W * z["experts"]), "flops": 2.0 * T * (TOP * per + W * z["experts"])}
    if kind == "dense":
        weights = W * HEAD * (2 * H + 2 * G) + 3 * W * z["ff"]
        nbytes += 2 * e * keys * G * HEAD
        flops += 4.0 * H * HEAD * pairs
    elif kind == "window":
        weights = W * HEAD * (2 * H + 2 * G) + W * H
        seen = sum(sum(min(c + i + 1, z["window"] + KEEP) for i in range(n)) for n, c in portions)
        nbytes += 2 * e * sum(n + min(c, z["window"] + KEEP) for n, c in portions) * G * HEAD
        flops += 4.0 * H * HEAD * seen
    elif kind == "delta":
        cols = HEAD * (2 * G + H)
        weights = W * (cols + H + 2 * z["rank"]) + 2 * z["rank"] * H * HEAD + H * HEAD * W
        nbytes += 8.0 * len(portions) * (H * HEAD * HEAD + (TAPS - 1) * cols)
        flops += T * 7.0 * H * HEAD * HEAD
    elif kind == "latent":
        row = LATENT + LATENT_ROT
        weights = W * (z["q_rank"] + row + H * HEAD) + z["q_rank"] * H * row + 2 * H * HEAD * LATENT + H * HEAD * W
        nbytes += e * keys * row
        flops += 2.0 * H * (row + LATENT) * pairs
    elif kind == "parallel":
        weights = W * HEAD * (2 * H + 2 * G) + W * H * (2 * R_DIM + 2 * HEAD)
        nbytes += 2 * e * keys * G * HEAD + 8.0 * len(portions) * H * R_DIM * HEAD
        flops += 4.0 * H * HEAD * pairs + T * 5.0 * H * R_DIM * HEAD
    else:
        weights = W * (5 * H * HEAD + z["rank"]) + z["rank"] * H * HEAD + H * HEAD * W
        nbytes += 8.0 * len(portions) * H * HEAD * HEAD
        flops += T * 9.0 * H * HEAD * HEAD
    return {"bytes": nbytes + e * weights, "flops": flops + 2.0 * T * weights}


def tolerance(case):
    if case["kind"] == "sampling":
        return "exact"
    if case.get("dtype") == "float32":
        return {"rel": 5e-6, "max": 1e-3}          # 1.1e-6 from 64 bits
    return {"rel": 1e-2, "max": 0.3}               # 2e-3 to 3e-3 from 64 bits: operands and results in 16 bits


# ---- the same in 64 bits -------------------------------------------------------------------------

def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, first, dims, theta, half):
    """x [T, heads, d]: the first ``dims`` dimensions turned by position, pairs (j, j + dims / 2) or (2j, 2j + 1)."""
    n = dims // 2
    freq = theta ** (-torch.arange(n, dtype=torch.float64, device=x.device) / n)
    ang = (first + torch.arange(x.shape[0], dtype=torch.float64, device=x.device))[:, None] * freq
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    out = x.clone()
    a, b = (slice(0, n), slice(n, dims)) if half else (slice(0, dims, 2), slice(1, dims, 2))
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _attend(q, k, v, scale, first, window=0, keep=0, sink=None):
    """Causal softmax attention of queries at positions first.. over keys at positions 0..; query head h on key head h G / H."""
    T, H, _ = q.shape
    L, G = k.shape[:2]
    i = first + torch.arange(T, device=q.device)[:, None]
    j = torch.arange(L, device=q.device)[None]
    hidden = j > i
    if window:
        hidden |= (i - j >= window) & (j >= keep)
    out = []
    for h in range(H):
        g = h * G // H
        s = ((q[:, h] @ k[:, g].T) * scale).masked_fill(hidden, -math.inf)
        top = s.max(1, keepdim=True).values
        top = top if sink is None else torch.maximum(top, sink[h])
        p = torch.exp(s - top)
        total = p.sum(1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[h] - top))
        out.append((p @ v[:, g]) / total)
    return torch.stack(out, 1)


def _conv(x, taps, tail):
    """Causal filter per channel, x [T, C], taps [C, n], tail [n - 1, C] the inputs before x."""
    full, T = torch.cat([tail, x]), x.shape[0]
    return sum(full[j:j + T] * taps[:, j] for j in range(taps.shape[1])), full[T:]


def _scan(S, steps, T):
    """S [H, d, dv] through T tokens: steps(S, t) -> (S, read-out [H, dv])."""
    out = []
    for t in range(T):
        S, o = steps(S, t)
        out.append(o)
    return S, torch.stack(out)


def _dense_attention(h, w, p, H, G, first, past):
    T = h.shape[0]
    q = _rms((h @ w(p + "q_proj.weight", H * HEAD).T).view(T, H, HEAD)) * w(p + "q_norm.weight", HEAD, 0)
    k = _rms((h @ w(p + "k_proj.weight", G * HEAD).T).view(T, G, HEAD)) * w(p + "k_norm.weight", HEAD, 0)
    v = (h @ w(p + "v_proj.weight", G * HEAD).T).view(T, G, HEAD)
    q, k = _rotate(q, first, HEAD, THETA["dense"], True), _rotate(k, first, HEAD, THETA["dense"], True)
    a = _attend(q, torch.cat([past[0], k]), torch.cat([past[1], v]), HEAD ** -0.5, first)
    return a.reshape(T, H * HEAD) @ w(p + "o_proj.weight", h.shape[1], H * HEAD).T


def _dense_mlp(h, w, p, ff):
    act = _silu(h @ w(p + "gate_proj.weight", ff).T) * (h @ w(p + "up_proj.weight", ff).T)
    return act @ w(p + "down_proj.weight", h.shape[1], ff).T


def _mixer(case, z, h, w, first, past, state):
    """y and the state afterwards."""
    kind, W, H, G, T = case["kind"], z["width"], z["heads"], z["kv"], h.shape[0]
    if kind == "dense":
        return _dense_attention(h, w, "mix.", H, G, first, past), None
    if kind == "window":
        q, k = _rms((h @ w("mix.q", H * HEAD).T).view(T, H, HEAD)), _rms((h @ w("mix.k", G * HEAD).T).view(T, G, HEAD))
        v = (h @ w("mix.v", G * HEAD).T).view(T, G, HEAD)
        a = _attend(q, torch.cat([past[0], k]), torch.cat([past[1], v]), HEAD ** -0.5, first, z["window"], KEEP)
        a = a * torch.sigmoid(h @ w("mix.g", H).T)[:, :, None]
        return a.reshape(T, H * HEAD) @ w("mix.o", W, H * HEAD).T, None
    if kind == "latent":
        row = HEAD + LATENT_ROT
        cq = _rms(h @ w("mix.dq", z["q_rank"]).T) * w("mix.dq.norm", z["q_rank"], 0)
        q = (cq @ w("mix.uq", H * row, z["q_rank"]).T).view(T, H, row)
        kv = h @ w("mix.dkv", LATENT + LATENT_ROT).T
        c = _rms(kv[:, :LATENT]) * w("mix.dkv.norm", LATENT, 0)
        turned = _rotate(torch.cat([q[..., HEAD:], kv[:, None, LATENT:]], 1), first, LATENT_ROT, THETA["latent"], False)
        rows = torch.cat([past[0][:, 0], torch.cat([c, turned[:, H]], 1)])
        k = (rows[:, :LATENT] @ w("mix.uk", H * HEAD, LATENT).T).view(-1, H, HEAD)
        k = torch.cat([k, rows[:, None, LATENT:].expand(-1, H, -1)], 2)
        v = (rows[:, :LATENT] @ w("mix.uv", H * HEAD, LATENT).T).view(-1, H, HEAD)
        a = _attend(torch.cat([q[..., :HEAD], turned[:, :H]], 2), k, v, row ** -0.5, first).reshape(T, H * HEAD)
        return (a * torch.sigmoid(h @ w("mix.g", H * HEAD).T)) @ w("mix.o", W, H * HEAD).T, None
    if kind == "delta":
        C, size = HEAD * (2 * G + H), H * HEAD * HEAD
        x = torch.cat([h @ w("mix.q", G * HEAD).T, h @ w("mix.k", G * HEAD).T, h @ w("mix.v", H * HEAD).T], 1)
        taps = torch.cat([w("mix.q.conv", G * HEAD, TAPS), w("mix.k.conv", G * HEAD, TAPS), w("mix.v.conv", H * HEAD, TAPS)])
        x, tail = _conv(x, taps, state[size:].view(TAPS - 1, C))
        q, k, v = (t.view(T, -1, HEAD) for t in _silu(x).split([G * HEAD, G * HEAD, H * HEAD], 1))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(H // G, 1) for t in (q * HEAD ** -0.5, k))
        beta = torch.sigmoid(h @ w("mix.b", H).T)
        a = (h @ w("mix.a1", z["rank"]).T) @ w("mix.a2", H * HEAD, z["rank"]).T + w("mix.dt_bias", H * HEAD, 0)
        decay = torch.exp(-torch.exp(w("mix.A_log", H, 0))[:, None] * torch.nn.functional.softplus(a, threshold=700.0).view(T, H, HEAD))

        def token(S, t):
            S = decay[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            return S, torch.einsum("hdv,hd->hv", S, q[t])
        S, o = _scan(state[:size].view(H, HEAD, HEAD), token, T)
        o = _rms(o) * w("mix.norm", HEAD, 0)
        o = o.reshape(T, H * HEAD) * torch.sigmoid((h @ w("mix.g1", z["rank"]).T) @ w("mix.g2", H * HEAD, z["rank"]).T)
        return o @ w("mix.o", W, H * HEAD).T, torch.cat([S.reshape(-1), tail.reshape(-1)])
    if kind == "parallel":
        def proj(p, n):
            return h @ w(p, n).T + w(p + ".b", n, 0)
        q, k, v = (proj("mix.left." + s, n * HEAD).view(T, n, HEAD) for s, n in (("q", H), ("k", G), ("v", G)))
        q, k = (_rotate(t, first, HEAD // 2, THETA["parallel"], False) for t in (q, k))
        a = _attend(q, torch.cat([past[0], k]), torch.cat([past[1], v]), HEAD ** -0.5, first, sink=w("mix.left.sink", H, 0))
        left = a.reshape(T, H * HEAD) @ w("mix.left.o", W, H * HEAD).T
        r = _silu(h @ w("mix.right.q", H * R_DIM).T).view(T, H, R_DIM)
        low = w("mix.right.lower", H * R_DIM, 0)
        f = (low + (1.0 - low) * torch.sigmoid(proj("mix.right.f", H * R_DIM))).view(T, H, R_DIM)
        u = (h @ w("mix.right.v", H * HEAD).T).view(T, H, HEAD)

        def token(S, t):
            S = f[t][:, :, None] * S + (1.0 - f[t])[:, :, None] * u[t][:, None, :]
            return S, torch.einsum("hdv,hd->hv", S, r[t])
        S, o = _scan(state.view(H, R_DIM, HEAD), token, T)
        right = (_rms(o) * w("mix.right.norm", HEAD, 0)).reshape(T, H * HEAD) @ w("mix.right.o", W, H * HEAD).T
        return 0.5 * (_rms(left) * w("mix.left.norm", W, 0) + _rms(right) * w("mix.right.norm2", W, 0)), S.reshape(-1)
    r, k, v, a, g = (h @ w("mix." + n, H * HEAD).T for n in "rkvag")
    wz = torch.tanh(h @ w("mix.w1", z["rank"]).T) @ w("mix.w2", H * HEAD, z["rank"]).T
    decay = torch.exp(-DECAY_RATE * torch.sigmoid(wz + w("mix.w0", H * HEAD, 0))).view(T, H, HEAD)
    a = torch.sigmoid(a + w("mix.a.b", H * HEAD, 0)).view(T, H, HEAD)
    r, k, v = (t.view(T, H, HEAD) for t in (r, k, v))
    unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)

    def token(S, t):
        held = torch.einsum("hdv,hd->hv", S, unit[t])
        S = decay[t][:, :, None] * S - (a[t] * unit[t])[:, :, None] * held[:, None, :] + k[t][:, :, None] * v[t][:, None, :]
        return S, torch.einsum("hdv,hd->hv", S, r[t])
    S, o = _scan(state.view(H, HEAD, HEAD), token, T)
    o = _rms(o).reshape(T, H * HEAD) * w("mix.norm", H * HEAD, 0) * torch.sigmoid(g)
    return o @ w("mix.o", W, H * HEAD).T, S.reshape(-1)


def _exact_step(case, seed):
    W, H, G, ff, V = 4096, 32, 8, 12288, STEP["vocab_size"]

    def w(name, rows, cols=W):
        return _weight(seed, name, (rows, cols) if cols else (rows,), torch.bfloat16).double()
    portions = _portions(case)
    ids = _ids(seed, sum(n for n, _ in portions), V).to(DEV)
    x = w("model.embed_tokens.weight", V)[ids]
    for i in range(STEP_LAYERS):
        p, at, parts = f"model.layers.{i}.", 0, []
        h = _rms(x) * w(p + "input_layernorm.weight", W, 0)
        for rid, (n, ctx) in enumerate(portions):
            past = [_context(seed, f"{c}{i}", rid, ctx, G, HEAD, torch.bfloat16).double() for c in "kv"]
            parts.append(_dense_attention(h[at:at + n], w, p + "self_attn.", H, G, ctx, past))
            at += n
        x = x + torch.cat(parts)
        x = x + _dense_mlp(_rms(x) * w(p + "post_attention_layernorm.weight", W, 0), w, p + "mlp.", ff)
    last = torch.tensor([n for n, _ in portions], device=x.device).cumsum(0) - 1
    logits = (_rms(x[last]) * w("model.norm.weight", W, 0)) @ w("lm_head.weight", V).T
    return {"logits": logits, "k": None, "v": None}


def exact(case, seed):
    if case["kind"] == "sampling":
        return None
    if case["kind"] == "step":
        return _exact_step(case, seed)
    z, kind, dtype = SIZES[case["size"]], case["kind"], getattr(torch, case["dtype"])
    W = z["width"]

    def w(name, rows, cols=W):
        return _weight(seed, name, (rows, cols) if cols else (rows,), dtype).double()
    portions = _portions(case)
    T = sum(n for n, _ in portions)
    x = w("embed", ROWS)[_ids(seed, T, ROWS).to(DEV)]
    if kind == "experts":
        h = _tensor(seed, "h", (T, W)).to(dtype).double()
        best = torch.topk(h @ w("mlp.router", z["experts"]).T + w("mlp.router.b", z["experts"], 0), TOP, dim=1)
        share, y = torch.softmax(best.values, 1), torch.zeros_like(h)
        for e in range(z["experts"]):
            rows, slot = torch.nonzero(best.indices == e, as_tuple=True)
            g = (h[rows] @ w(f"mlp.e{e}.gate", z["e_ff"]).T).clamp(max=7.0)
            u = (h[rows] @ w(f"mlp.e{e}.up", z["e_ff"]).T).clamp(-7.0, 7.0)
            y[rows] += share[rows, slot][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(f"mlp.e{e}.down", W, z["e_ff"]).T)
        x = x + y
        return {"y": _rms(x) * w("after.norm", W, 0), "x": x}
    heads, dim = (1, LATENT + LATENT_ROT) if kind == "latent" else (z["kv"], HEAD)
    size = {"delta": z["heads"] * HEAD * HEAD + (TAPS - 1) * HEAD * (2 * z["kv"] + z["heads"]), "parallel": z["heads"] * R_DIM * HEAD,
            "removal": z["heads"] * HEAD * HEAD}.get(kind, 0)
    h, at, ys, states = _rms(x) * w("first.norm", W, 0), 0, [], []
    for rid, (n, ctx) in enumerate(portions):
        past = [_context(seed, f"{c}0", rid, ctx, heads, dim, dtype).double() for c in "kv"]
        state = _tensor(seed, f"state.{rid}", (size,), 0.0, 0.3).double() if ctx else torch.zeros(size, dtype=torch.float64, device=DEV)
        y, state = _mixer(case, z, h[at:at + n], w, ctx, past, state)
        ys.append(y)
        states.append(state)
        at += n
    x = x + torch.cat(ys)
    if kind == "dense":
        x = x + _dense_mlp(_rms(x) * w("second.norm", W, 0), w, "mlp.", z["ff"])
    out = {"y": _rms(x) * w("after.norm", W, 0), "x": x}
    if kind not in ("delta", "removal"):
        out["k"] = None
    if size:
        out["state"] = states
    return out
