"""The work that users of this framework have it do, as cases that can be timed and checked.

A case goes through the public Python entry points (`B200TransformerHandler`, `B200MatVec`, `PagedKvCache`):

  decode     one step for `batch` requests, token ids in, logits out (`forward_batch`): what a serving loop does per token.  The
             contexts of the requests differ: between half of `ctx` and `ctx` cached positions, one request has all of them
  prefill    `tokens` prompt positions of one request after `start` cached ones, with the logits of `want` of them
             (`prefill_logits`): 1 place to start generating, more to score a text or to replay a trace
  matvec     one product with a resident quantised matrix, host vector in and out (`B200MatVec.sgemv`): what Juno's own layers
             call when they keep the model on the host side
  attention  decode attention over paged FP16 keys and values for `batch` requests, host in and out (`PagedKvCache.attention`)

Models are random, with the sizes of this repository's benchmarks: the TinyLlama and Llama-3-8B architectures, the 8B layer shapes
with 4 layers, and the Vosotar and Desilorn stacks beside them.  A process that serves requests holds one model for all of them: the
last model that was asked for stays loaded, and a state is a set of requests of its own (other token ids, other contexts).

Quantised weights have the spread of trained ones: zero mean, standard deviation 1 / sqrt(columns), a scale per sub-block.
"""
from __future__ import annotations

import gc
import math
import shutil
import tempfile

import numpy as np
import torch

F32, Q8_0, Q4_K, Q6_K = 0, 8, 12, 14
TYPES = {"q8_0": Q8_0, "q4_k": Q4_K, "q6_k": Q6_K}
BYTES_PER_WEIGHT = {F32: 4.0, Q8_0: 34 / 32, Q4_K: 144 / 256, Q6_K: 210 / 256}
MAX_CTX = 2112

# hidden, layers, heads, key/value heads, feed-forward, vocabulary, eps, rotation base, most requests at a time
LLAMA = {"tinyllama": (2048, 22, 32, 4, 5632, 32000, 1e-5, 10000.0, 256),
         "llama3-8b": (4096, 32, 32, 8, 14336, 128256, 1e-5, 500000.0, 40),
         "llama3-8b-4layer": (4096, 4, 32, 8, 14336, 32000, 1e-5, 500000.0, 256)}
# width, heads, feed-forward, rank of the queries, rank of keys and values, layers; heads of 128, vocabulary of 32000
STACK = {"small": (2048, 16, 8192, 768, 512, 8), "medium": (4096, 32, 14336, 1536, 512, 4)}
STACK_VOCAB, STACK_KV_HEADS, STREAMS, STACK_EPS = 32000, 8, 4, 1e-6


def listed():
    return [
        # the smallest call: one projection of a small model, all latency
        {"name": "matvec-q4k-2048x2048-b1", "kind": "matvec", "type": "q4_k", "rows": 2048, "cols": 2048, "batch": 1},
        # a chat with the small model: launches and latency
        {"name": "decode-tinyllama-b1", "kind": "decode", "model": "tinyllama", "quant": "q4_k_m", "batch": 1, "ctx": 150},
        # a short prompt in the 8-bit format, odd length
        {"name": "prefill-tinyllama-q8-333", "kind": "prefill", "model": "tinyllama", "quant": "q8_0", "tokens": 333, "start": 0, "want": 1},
        # the benchmark's own step: one request at 2048 positions
        {"name": "decode-8b-b1", "kind": "decode", "model": "llama3-8b", "quant": "q4_k_m", "batch": 1, "ctx": 2048},
        # a few requests together
        {"name": "decode-8b-b6", "kind": "decode", "model": "llama3-8b", "quant": "q4_k_m", "batch": 6, "ctx": 1024},
        # a loaded server: many requests in a step
        {"name": "decode-8b-4layer-b48", "kind": "decode", "model": "llama3-8b-4layer", "quant": "q4_k_m", "batch": 48, "ctx": 1500},
        # a long prompt: the largest case
        {"name": "prefill-8b-2048", "kind": "prefill", "model": "llama3-8b", "quant": "q4_k_m", "tokens": 2048, "start": 0, "want": 1},
        # the attention operator alone, long contexts
        {"name": "attention-b8-4096", "kind": "attention", "heads": 32, "kv_heads": 8, "dim": 128, "batch": 8, "ctx": 4096},
        # layer stacks with BF16 weights: a batch of requests, a prompt that is scored, a single request, a prompt's next part
        {"name": "decode-vosotar-medium-b24", "kind": "decode", "model": "vosotar", "quant": "medium", "batch": 24, "ctx": 1000},
        {"name": "prefill-vosotar-small-1000", "kind": "prefill", "model": "vosotar", "quant": "small", "tokens": 1000, "start": 0, "want": 8},
        {"name": "decode-desilorn-medium-b2", "kind": "decode", "model": "desilorn", "quant": "medium", "batch": 2, "ctx": 1500},
        {"name": "prefill-desilorn-medium-1500", "kind": "prefill", "model": "desilorn", "quant": "medium", "tokens": 1500, "start": 500, "want": 1},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model, quant, most = rng.choice([("tinyllama", "q4_k_m", 32), ("tinyllama", "q8_0", 32), ("llama3-8b", "q4_k_m", 8), ("llama3-8b-4layer", "q4_k_m", 64),
                                     ("vosotar", "small", 64), ("vosotar", "medium", 64), ("desilorn", "small", 64), ("desilorn", "medium", 64)])
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "prefill", "matvec", "attention"])
    if kind == "matvec":
        cols = 256 * size(4, 56)
        return {"kind": kind, "type": rng.choice(["q4_k", "q6_k", "q8_0"]), "rows": size(200, 28672), "cols": cols, "batch": size(1, 8)}
    if kind == "attention":
        heads, kv_heads, dim = rng.choice([(32, 8, 128), (32, 4, 64), (64, 8, 128)])
        batch = size(1, 32)
        return {"kind": kind, "heads": heads, "kv_heads": kv_heads, "dim": dim, "batch": batch, "ctx": min(size(64, 8192), 65536 // batch)}
    if kind == "decode":
        return {"kind": kind, "model": model, "quant": quant, "batch": size(1, most), "ctx": size(16, 2048)}
    tokens = size(9, 2000)
    start = 0 if model == "vosotar" or rng.random() < 0.5 else size(1, 2100 - tokens)
    return {"kind": kind, "model": model, "quant": quant, "tokens": tokens, "start": start, "want": min(tokens, rng.choice([1, 1, 1, 5]))}


# ── what a request holds ──────────────────────────────────────────────────────────────────────────────────────────────────────

def _vocab(case):
    return LLAMA[case["model"]][5] if case["model"] in LLAMA else STACK_VOCAB


def _lengths(case, seed):
    """Cached positions of each request of a decode step."""
    r = np.random.default_rng([seed, 1])
    n = r.integers(max(1, case["ctx"] // 2), case["ctx"] + 1, case["batch"])
    n[0] = case["ctx"]
    return [int(v) for v in n]


def _tokens(case, seed):
    """Per request: the cached token ids, then the ids that a pass feeds."""
    r = np.random.default_rng([seed, 2])
    if case["kind"] == "decode":
        return [(r.integers(0, _vocab(case), n), r.integers(0, _vocab(case), 1)) for n in _lengths(case, seed)]
    return [(r.integers(0, _vocab(case), case["start"]), r.integers(0, _vocab(case), case["tokens"]))]


def _places(case):
    """Places of a prompt whose logits are wanted: the last one, and others spread before it."""
    return [case["tokens"] * (i + 1) // case["want"] - 1 for i in range(case["want"])]


# ── quantised blocks ──────────────────────────────────────────────────────────────────────────────────────────────────────────

def _generator(*key):
    g = torch.Generator("cuda")
    g.manual_seed(int(np.random.SeedSequence([int(v) for v in key]).generate_state(1, np.uint64)[0] >> np.uint64(1)))
    return g


def _f16_bytes(v):
    return v.half().view(torch.uint8).view(-1, 2)


def _blocks(kind, rows, cols, g):
    """Raw row-major GGUF blocks, [blocks, bytes] uint8 on the GPU."""
    def ints(lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=torch.int32)

    n = rows * cols // (32 if kind == Q8_0 else 256)
    std, spread = cols ** -0.5, 0.5 + torch.rand(n, generator=g, device="cuda")
    if kind == Q8_0:
        return torch.cat([_f16_bytes(spread * std / 73.3), ints(-127, 128, n, 32).to(torch.int8).view(torch.uint8)], 1)
    if kind == Q4_K:
        d = spread * std / (4.61 * 41)
        sc = ints(16, 64, n, 8)
        mn = (sc + ints(-3, 4, n, 8)).clamp(0, 63)
        p = torch.empty((n, 12), dtype=torch.int32, device="cuda")
        p[:, 0:4] = sc[:, :4] | ((sc[:, 4:] >> 4) << 6)
        p[:, 4:8] = mn[:, :4] | ((mn[:, 4:] >> 4) << 6)
        p[:, 8:12] = (sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)
        return torch.cat([_f16_bytes(d), _f16_bytes(7.5 * d), p.to(torch.uint8), ints(0, 256, n, 128).to(torch.uint8)], 1)
    sc = ints(48, 128, n, 16) * (2 * ints(0, 2, n, 16) - 1)
    return torch.cat([ints(0, 256, n, 192).to(torch.uint8), sc.to(torch.int8).view(torch.uint8), _f16_bytes(spread * std / (18.5 * 91))], 1)


def _values(kind, blocks, rows, cols):
    """The blocks' values in 64 bits, [rows, cols]."""
    def f16(b):
        return b.contiguous().view(torch.float16).double()

    n = blocks.shape[0]
    if kind == Q8_0:
        return (f16(blocks[:, :2]) * blocks[:, 2:].contiguous().view(torch.int8).double()).view(rows, cols)
    if kind == Q4_K:
        p, q = blocks[:, 4:16].int(), blocks[:, 16:].view(n, 4, 1, 32)
        sc = torch.cat([p[:, :4] & 63, (p[:, 8:] & 15) | ((p[:, :4] >> 6) << 4)], 1).double() * f16(blocks[:, :2])
        mn = torch.cat([p[:, 4:8] & 63, (p[:, 8:] >> 4) | ((p[:, 4:8] >> 6) << 4)], 1).double() * f16(blocks[:, 2:4])
        w = torch.cat([q & 15, q >> 4], 2).double().view(n, 8, 32) * sc[:, :, None] - mn[:, :, None]
        return w.view(rows, cols)
    ql, qh = blocks[:, :128].view(n, 2, 2, 32), blocks[:, 128:192].view(n, 2, 1, 32)
    lo = torch.cat([ql & 15, ql >> 4], 2)  # [n, 2 halves, 4 quarters, 32]
    hi = torch.cat([(qh >> s) & 3 for s in (0, 2, 4, 6)], 2)
    q = (lo | (hi << 4)).double() - 32
    sc = blocks[:, 192:208].contiguous().view(torch.int8).double() * f16(blocks[:, 208:210])
    return (q.view(n, 16, 16) * sc[:, :, None]).view(rows, cols)


# ── LLaMA models ──────────────────────────────────────────────────────────────────────────────────────────────────────────────

# tensor kinds of the C ABI
EMBD, OUT_NORM, OUT, ATTN_NORM, FFN_NORM, WQ, WK, WV, WO, GATE, UP, DOWN = range(12)


def _llama_shape(model, kind):
    H, _, heads, kv, ff, V = LLAMA[model][:6]
    kd = H // heads * kv
    return {EMBD: (V, H), OUT: (V, H), WQ: (H, H), WK: (kd, H), WV: (kd, H), WO: (H, H), GATE: (ff, H), UP: (ff, H), DOWN: (H, ff)}.get(kind, (1, H))


def _llama_type(quant, kind):
    if kind in (OUT_NORM, ATTN_NORM, FFN_NORM):
        return F32
    return Q8_0 if quant == "q8_0" else Q6_K if kind in (WV, DOWN) else Q4_K


def _llama_tensor(model, quant, kind, layer):
    """(type, rows, cols, blocks on the GPU); a norm's weights as floats."""
    (rows, cols), t = _llama_shape(model, kind), _llama_type(quant, kind)
    g = _generator(7, sorted(LLAMA).index(model), t, kind, layer)
    if t == F32:
        return t, rows, cols, 1.0 + 0.2 * torch.randn(cols, generator=g, device="cuda")
    return t, rows, cols, _blocks(t, rows, cols, g)


def _llama_tensors(model, quant):
    for kind in (EMBD, OUT_NORM, OUT):
        yield (kind, 0) + _llama_tensor(model, quant, kind, 0)
    for layer in range(LLAMA[model][1]):
        for kind in range(ATTN_NORM, DOWN + 1):
            yield (kind, layer) + _llama_tensor(model, quant, kind, layer)


class _Model:
    """A loaded model: the handler that a program keeps for as long as it serves."""

    def __init__(self, model, quant):
        from juno_b200 import synth
        from juno_b200.handler import B200TransformerHandler
        self.names = 0
        if model in LLAMA:
            seqs = LLAMA[model][8]
            self.h = B200TransformerHandler(synth.Arch(*LLAMA[model][:8]), max_batch=64, max_seqs=seqs, max_ctx=MAX_CTX)
            self.h.load((k, l, t, r, c, b.cpu().numpy().view(np.uint8)) for k, l, t, r, c, b in _llama_tensors(model, quant))
            return
        folder = tempfile.mkdtemp(prefix="cases_")
        try:
            from juno_b200.safetensors_file import write_model_folder
            w = {k: v.view(torch.int16).cpu().numpy().view(np.uint16) for k, v in _stack_tensors(model, quant)}
            write_model_folder(folder, _stack_config(model, quant), w)
            self.h = B200TransformerHandler.open(folder, max_batch=64, max_seqs=256, max_ctx=MAX_CTX)
        finally:
            shutil.rmtree(folder, ignore_errors=True)

    def name(self):
        self.names += 1
        return "r%d" % self.names

    def __del__(self):
        if hasattr(self, "h"):
            self.h.release_gpu_resources()


_loaded = {}


def _model(case):
    key = (case["model"], case["quant"])
    if key not in _loaded:
        _loaded.clear()
        gc.collect()
        _loaded[key] = _Model(*key)
        torch.cuda.empty_cache()
    return _loaded[key]


# ── layer stacks ──────────────────────────────────────────────────────────────────────────────────────────────────────────────

def _stack_config(model, size):
    from juno_b200 import synth
    w, heads, ff, qr, kr, n = STACK[size]
    if model == "vosotar":
        one = dict(heads=heads, dim=128, vdim=128, q_rank=qr, kv_rank=kr, scale=128 ** -0.5, ff=ff)
        return synth.vosotar_config(w, STACK_VOCAB, [dict(one) for _ in range(n)])
    one = dict(heads=heads, kv_heads=STACK_KV_HEADS, dim=128, vdim=128, scale=128 ** -0.5, ff=ff)
    kinds = (dict(one, size=8192, rot=(500000.0, 128)), dict(one, size=4096, q_temp=(0.1, 1024)))
    return synth.desilorn_config(w, STACK_VOCAB, [dict(kinds[i % 2]) for i in range(n)], streams=STREAMS)


def _stack_shapes(model, size):
    """(name, shape, (mean, standard deviation)) of every tensor."""
    W, H, ff, qr, kr, n = STACK[size]
    near1, G, S = (1.0, 0.3), STACK_KV_HEADS, STREAMS

    def mat(name, rows, cols):
        return name, (rows, cols), (0.0, cols ** -0.5)

    if model == "vosotar":
        yield "embed", (STACK_VOCAB, W), (0.0, 1.0)
        yield "embed.norm", (), near1
        yield "final.norm", (), near1
        yield mat("head", STACK_VOCAB, W)
        for i in range(n):
            p = "l%d." % i
            yield p + "norm1", (), near1
            yield p + "norm1b", (), near1
            yield mat(p + "mix.dq", qr, W)
            yield p + "mix.dq.norm", (qr,), near1
            yield mat(p + "mix.uq", H * 128, qr)
            yield mat(p + "mix.dkv", kr, W)
            yield p + "mix.dkv.norm", (kr,), near1
            yield mat(p + "mix.uk", H * 128, kr)
            yield mat(p + "mix.uv", H * 128, kr)
            yield mat(p + "mix.g", H, W)
            yield mat(p + "mix.o", W, H * 128)
            yield p + "canon1", (W, 4), (0.0, 0.5)
            yield mat(p + "rg1", W, W)
            yield p + "rg1.b", (W,), (0.0, 0.5)
            yield p + "norm2", (), near1
            yield p + "norm2b", (), near1
            yield mat(p + "mlp.up", ff, W)
            yield mat(p + "mlp.down", W, ff)
            yield mat(p + "rg2", W, W)
            yield p + "rg2.b", (W,), (0.0, 0.5)
        return
    yield "embed", (STACK_VOCAB, W), (0.0, 1.0)
    yield "final.norm", (W,), (0.0, 0.3)
    for i in range(n):
        p = "l%d." % i
        yield p + "norm1", (W,), (0.0, 0.3)
        for name, rows in (("q", H * 128), ("k", G * 128), ("v", G * 128)):
            yield mat(p + "mix." + name, rows, W)
            yield p + "mix." + name + ".b", (rows,), (0.0, 0.3)
        if i % 2 == 0:
            yield p + "mix.q.norm", (128,), near1
            yield p + "mix.k.norm", (128,), near1
        else:
            yield p + "mix.sink", (H,), (0.0, 1.0)
        yield mat(p + "mix.o", W, H * 128)
        yield p + "norm2", (W,), (0.0, 0.3)
        yield mat(p + "mlp.gate", ff, W)
        yield mat(p + "mlp.up", ff, W)
        yield mat(p + "mlp.down", W, ff)
        for q in ("hc1.", "hc2."):
            yield p + q + "in", (S,), (1.0 / S, 0.2)
            yield p + q + "out", (S,), (0.7, 0.3)
            yield p + q + "mix", (S, S), (None, 0.15)  # near the identity


def _stack_tensors(model, size):
    """name, BF16 tensor on the GPU, in file order."""
    for i, (name, shape, (mean, std)) in enumerate(_stack_shapes(model, size)):
        v = torch.randn(shape, generator=_generator(11, model == "vosotar", size == "small", i), device="cuda") * std
        yield name, ((torch.eye(shape[0], device="cuda") if mean is None else mean) + v).bfloat16()


# ── prepare and run ───────────────────────────────────────────────────────────────────────────────────────────────────────────

class _Requests:
    """Requests of a model with their cached contexts; they leave it when the state goes."""

    def __init__(self, model, case, seed):
        self.m, self.kind, self.ids = model, case["kind"], []
        self.feed, self.positions = [], []
        for cached, feed in _tokens(case, seed):
            rid = model.name()
            self.ids.append(rid)
            if len(cached):
                model.h.prefill(rid, cached, 0)
            self.feed.append(feed if self.kind == "prefill" else [int(feed[0])])
            self.positions.append(len(cached))
        self.want = _places(case) if self.kind == "prefill" else None

    def __del__(self):
        for rid in getattr(self, "ids", ()):
            self.m.h.evict(rid)


class _MatVec:
    def __init__(self, case, seed):
        from juno_b200.matvec import B200MatVec
        self.kind, t = "matvec", TYPES[case["type"]]
        blocks, self.x = _matvec_inputs(case, seed)
        self.mv = B200MatVec()
        self.a = self.mv.upload_quantized(blocks.cpu().numpy(), t, case["rows"], case["cols"])
        self.x = self.x[0] if case["batch"] == 1 else self.x

    def __del__(self):
        if hasattr(self, "a"):
            self.a.close()


def _matvec_inputs(case, seed):
    g = _generator(3, seed)
    blocks = _blocks(TYPES[case["type"]], case["rows"], case["cols"], g)
    return blocks, torch.randn(case["batch"], case["cols"], generator=g, device="cuda").cpu().numpy()


class _Attention:
    def __init__(self, case, seed):
        from juno_b200.matvec import GpuContext, PagedKvCache
        self.kind, self.heads = "attention", case["heads"]
        lengths = _lengths(case, seed)
        self.pool = PagedKvCache(GpuContext.shared(0), 1, case["kv_heads"], case["dim"], sum((n + 15) // 16 for n in lengths))
        self.seqs = []
        for i, n in enumerate(lengths):
            k, v = _keys_values(case, seed, i, n)
            s = self.pool.new_sequence(n)
            self.pool.append(s, 0, 0, k.float().cpu().numpy(), v.float().cpu().numpy())
            self.seqs.append(s)
        self.q = _queries(case, seed).cpu().numpy()

    def __del__(self):
        if hasattr(self, "seqs"):
            for s in self.seqs:
                self.pool.free_sequence(s)
            self.pool.close()


def _keys_values(case, seed, i, n):
    """Values of the cache's own 16-bit type."""
    g = _generator(5, seed, i)
    return [torch.randn(n, case["kv_heads"] * case["dim"], generator=g, device="cuda").half() for _ in range(2)]


def _queries(case, seed):
    return torch.randn(case["batch"], case["heads"] * case["dim"], generator=_generator(6, seed), device="cuda")


def prepare(case, seed):
    if case["kind"] == "matvec":
        return _MatVec(case, seed)
    if case["kind"] == "attention":
        return _Attention(case, seed)
    return _Requests(_model(case), case, seed)


def run(s):
    if s.kind == "matvec":
        return s.mv.sgemv(s.a, s.x)
    if s.kind == "attention":
        return s.pool.attention(0, s.seqs, s.q, s.heads)
    if s.kind == "decode":
        return s.m.h.forward_batch(s.ids, s.feed, s.positions)
    return s.m.h.prefill_logits(s.ids[0], s.feed[0], s.positions[0], s.want)


# ── what a pass cannot do without ─────────────────────────────────────────────────────────────────────────────────────────────

def _layer_matrices(case):
    """(rows, cols, bytes of a weight) of every matrix of all layers, and of the output projection."""
    if case["model"] in LLAMA:
        out = _llama_shape(case["model"], OUT) + (BYTES_PER_WEIGHT[_llama_type(case["quant"], OUT)],)
        one = [_llama_shape(case["model"], k) + (BYTES_PER_WEIGHT[_llama_type(case["quant"], k)],) for k in range(WQ, DOWN + 1)]
        return one * LLAMA[case["model"]][1], out
    mats = [s for name, s, _ in _stack_shapes(case["model"], case["quant"]) if len(s) == 2 and name.startswith("l") and "hc" not in name]
    return [s + (2.0,) for s in mats], (STACK_VOCAB, STACK[case["quant"]][0], 2.0)


def _cache_and_attention(case, length):
    """Bytes of one cached position over all layers, and attention FLOPs of one query position over `length` keys."""
    if case["model"] in LLAMA:
        H, n, heads, kv = LLAMA[case["model"]][:4]
        return n * 2 * kv * (H // heads) * 2, n * 4 * H * length
    _, H, _, _, kr, n = STACK[case["quant"]]
    # latents are attended to by every head, or expanded to keys and values first: the cheaper of the two grows with 2 x 128 per head
    return n * (kr if case["model"] == "vosotar" else 2 * STACK_KV_HEADS * 128) * 2, n * 4 * H * 128 * length


def work(case):
    if case["kind"] == "matvec":
        r, c, b = case["rows"], case["cols"], case["batch"]
        return {"bytes": r * c * BYTES_PER_WEIGHT[TYPES[case["type"]]] + 4 * b * (r + c), "flops": 2 * b * r * c}
    if case["kind"] == "attention":
        n = sum(_lengths(case, 0))
        return {"bytes": n * case["kv_heads"] * case["dim"] * 4 + 8 * case["batch"] * case["heads"] * case["dim"], "flops": 4 * n * case["heads"] * case["dim"]}
    layers, (V, H, out_bytes) = _layer_matrices(case)
    per_pos, _ = _cache_and_attention(case, 1)
    if case["kind"] == "decode":
        rows, logits, lens = case["batch"], case["batch"], [n + 1 for n in _lengths(case, 0)]
    else:
        rows, logits = case["tokens"], case["want"]
        lens = [case["start"] + i + 1 for i in range(case["tokens"])]
    read = sum(lens) if case["kind"] == "decode" else case["start"] + case["tokens"]
    return {"bytes": sum(r * c * b for r, c, b in layers) + V * H * out_bytes + read * per_pos + rows * H * out_bytes + 4 * logits * V,
            "flops": sum(2 * r * c for r, c, _ in layers) * rows + 2 * V * H * logits + sum(_cache_and_attention(case, n)[1] for n in lens)}


def tolerance(case):
    # about four times the relative errors against 64 bits that were measured
    if case["kind"] in ("matvec", "attention"):
        return {"rel": 3e-6}  # 32-bit products and sums
    # 16-bit cache, products of 16-bit operands through all layers; Vosotar's norms after each sublayer pass more of it on
    return {"rel": 3e-2 if case["model"] == "vosotar" else 1.5e-2}


# ── the same in 64 bits ───────────────────────────────────────────────────────────────────────────────────────────────────────

def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "matvec":
            blocks, x = _matvec_inputs(case, seed)
            y = torch.from_numpy(x).cuda().double() @ _values(TYPES[case["type"]], blocks, case["rows"], case["cols"]).T
            return (y[0] if case["batch"] == 1 else y).cpu().numpy()
        if case["kind"] == "attention":
            return _exact_attention(case, seed)
        total = sum(len(a) + len(b) for a, b in _tokens(case, seed))
        layers, _ = _layer_matrices(case)
        if total * sum(2 * r * c for r, c, _ in layers) > 2.5e14:  # over about 20 seconds
            return None
        ids = [np.concatenate(t) for t in _tokens(case, seed)]
        keep = [[len(t) - 1] for t in ids] if case["kind"] == "decode" else [[case["start"] + p for p in _places(case)]]
        net = _exact_llama if case["model"] in LLAMA else _exact_vosotar if case["model"] == "vosotar" else _exact_desilorn
        return net(case, ids, keep).cpu().numpy()


def _exact_attention(case, seed):
    H, G, d = case["heads"], case["kv_heads"], case["dim"]
    q, out = _queries(case, seed).double(), []
    for i, n in enumerate(_lengths(case, seed)):
        k, v = (t.double().view(n, G, 1, d) for t in _keys_values(case, seed, i, n))
        s = (q[i].view(1, G, H // G, d) * k).sum(-1) * d ** -0.5
        out.append((s.softmax(0)[..., None] * v).sum(0).reshape(-1))
    return torch.stack(out).cpu().numpy()


def _mm(x, w):
    """x @ w.T a part of the rows at a time."""
    out = torch.empty((x.shape[0], w.shape[0]), dtype=torch.float64, device="cuda")
    for i in range(0, x.shape[0], 8192):
        torch.mm(x[i:i + 8192], w.T, out=out[i:i + 8192])
    return out


def _unit(x, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt()


def _positions(ids):
    return torch.cat([torch.arange(len(t), device="cuda") for t in ids]).double()


def _causal(q, k, v, ids, scale, bias=None, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv], requests side by side: causal attention inside each.  bias(i, j) is added to the
    scores [H, i, j]; sink [H]: one more term in the denominator."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty((q.shape[0], H, v.shape[2]), dtype=torch.float64, device="cuda")
    at = 0
    for t in ids:
        n = len(t)
        ks, vs = (x[at:at + n].repeat_interleave(H // G, 1).transpose(0, 1) for x in (k, v))
        for i0 in range(0, n, 512):
            i1 = min(n, i0 + 512)
            s = q[at + i0:at + i1].transpose(0, 1) @ ks[:, :i1].transpose(1, 2) * scale
            i, j = torch.arange(i0, i1, device="cuda")[:, None], torch.arange(i1, device="cuda")[None]
            if bias is not None:
                s = s + bias(i, j)
            s = s.masked_fill(j > i, -math.inf)
            if sink is not None:
                p = torch.cat([s, sink[:, None, None].expand(H, i1 - i0, 1)], 2).softmax(2)[..., :-1]
            else:
                p = s.softmax(2)
            out[at + i0:at + i1] = (p @ vs[:, :i1]).transpose(0, 1)
        at += n
    return out.reshape(q.shape[0], -1)


def _kept(x, ids, keep):
    rows, at = [], 0
    for t, k in zip(ids, keep):
        rows += [at + p for p in k]
        at += len(t)
    return x[torch.tensor(rows, device="cuda")]


def _exact_llama(case, ids, keep):
    model, quant = case["model"], case["quant"]
    H, n, heads, kv, _, _, eps, base, _ = LLAMA[model]
    d = H // heads

    def w(kind, layer=0):
        t, r, c, b = _llama_tensor(model, quant, kind, layer)
        return b.double() if t == F32 else _values(t, b, r, c)

    angle = _positions(ids)[:, None] * base ** (-2.0 * torch.arange(d // 2, device="cuda").double() / d)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(x):
        x = x.view(x.shape[0], -1, d // 2, 2)
        a, b = x[..., 0], x[..., 1]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(2)

    x = w(EMBD)[torch.from_numpy(np.concatenate(ids)).cuda()]
    for l in range(n):
        h = _unit(x, eps) * w(ATTN_NORM, l)
        q, k, v = turn(_mm(h, w(WQ, l))), turn(_mm(h, w(WK, l))), _mm(h, w(WV, l)).view(-1, kv, d)
        x = x + _mm(_causal(q, k, v, ids, d ** -0.5), w(WO, l))
        h = _unit(x, eps) * w(FFN_NORM, l)
        wg, wu, wd = w(GATE, l), w(UP, l), w(DOWN, l)
        for i in range(0, x.shape[0], 8192):
            x[i:i + 8192] += (torch.nn.functional.silu(h[i:i + 8192] @ wg.T) * (h[i:i + 8192] @ wu.T)) @ wd.T
    return _mm(_unit(_kept(x, ids, keep), eps) * w(OUT_NORM), w(OUT))


def _exact_vosotar(case, ids, keep):
    w = {k: v.double() for k, v in _stack_tensors("vosotar", case["quant"])}
    _, H, _, _, _, n = STACK[case["quant"]]
    eps = STACK_EPS
    x = _unit(w["embed"][torch.from_numpy(np.concatenate(ids)).cuda()], eps) * w["embed.norm"]
    at, starts = 0, []
    for t in ids:
        starts.append((at, at + len(t)))
        at += len(t)
    for i in range(n):
        p = "l%d." % i
        h = _unit(x, eps) * w[p + "norm1"]
        c = h.clone()
        for a, b in starts:
            for tap in range(4):
                back = 3 - tap
                if b - a > back:
                    c[a + back:b] += w[p + "canon1"][:, tap] * h[a:b - back]
        m = p + "mix."
        q = _mm(_unit(_mm(c, w[m + "dq"]), eps) * w[m + "dq.norm"], w[m + "uq"]).view(-1, H, 128)
        z = _unit(_mm(c, w[m + "dkv"]), eps) * w[m + "dkv.norm"]
        o = _causal(q, _mm(z, w[m + "uk"]).view(-1, H, 128), _mm(z, w[m + "uv"]).view(-1, H, 128), ids, 128 ** -0.5)
        o = (o.view(-1, H, 128) * _mm(c, w[m + "g"]).sigmoid()[..., None]).flatten(1)
        x = x + _unit(_mm(o, w[m + "o"]) * (_mm(h, w[p + "rg1"]) + w[p + "rg1.b"]).sigmoid(), eps) * w[p + "norm1b"]
        h = _unit(x, eps) * w[p + "norm2"]
        y = _mm(_mm(h, w[p + "mlp.up"]).relu().square(), w[p + "mlp.down"]) * (_mm(h, w[p + "rg2"]) + w[p + "rg2.b"]).sigmoid()
        x = x + _unit(y, eps) * w[p + "norm2b"]
    return _mm(_unit(_kept(x, ids, keep), eps) * w["final.norm"], w["head"])


def _exact_desilorn(case, ids, keep):
    w = {k: v.double() for k, v in _stack_tensors("desilorn", case["quant"])}
    _, H, _, _, _, n = STACK[case["quant"]]
    G, eps, pos = STACK_KV_HEADS, STACK_EPS, _positions(ids)
    e = w["embed"][torch.from_numpy(np.concatenate(ids)).cuda()]
    xs = [e] * STREAMS
    angle = pos[:, None] * 500000.0 ** (-2.0 * torch.arange(64, device="cuda").double() / 128)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, device="cuda").double() / H)

    def turn(x):
        a, b = x[..., :64], x[..., 64:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def mixer(h, p, window):
        m = p + "mix."
        q, k, v = ((_mm(h, w[m + s]) + w[m + s + ".b"]).view(-1, c, 128) for s, c in (("q", H), ("k", G), ("v", G)))
        if window:
            q = q * (1.0 + 0.1 * (((pos + 1) / 1024).floor() + 1.0).log())[:, None, None]
            o = _causal(q, k, v, ids, 128 ** -0.5, lambda i, j: -slopes[:, None, None] * (i - j), w[m + "sink"])
        else:
            q, k = turn(_unit(q, eps) * w[m + "q.norm"]), turn(_unit(k, eps) * w[m + "k.norm"])
            o = _causal(q, k, v, ids, 128 ** -0.5, None, torch.zeros(H, device="cuda").double())
        return _mm(o, w[m + "o"])

    def mlp(h, p):
        return _mm(torch.nn.functional.gelu(_mm(h, w[p + "mlp.gate"]), approximate="tanh") * _mm(h, w[p + "mlp.up"]), w[p + "mlp.down"])

    def connect(xs, p, norm, f):
        y = f(_unit(sum(a * x for a, x in zip(w[p + "in"], xs)), eps) * (1.0 + norm))
        return [sum(w[p + "mix"][s, t] * x for s, x in enumerate(xs)) + w[p + "out"][t] * y for t in range(len(xs))]

    for i in range(n):
        p = "l%d." % i
        xs = connect(xs, p + "hc1.", w[p + "norm1"], lambda h: mixer(h, p, i % 2 == 1))
        xs = connect(xs, p + "hc2.", w[p + "norm2"], lambda h: mlp(h, p))
    return _mm(_unit(_kept(sum(xs), ids, keep), eps) * (1.0 + w["final.norm"]), w["embed"])
