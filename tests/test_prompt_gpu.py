"""Prompts of the quantised layers that take the many-row path (FP16 rows of a whole pass on the row products, flash attention
over the pages), against the oracle fed token by token."""
import numpy as np
import pytest

from conftest import rel_err
from juno_b200 import synth
from modelutil import SMALL128, TINY

pytestmark = pytest.mark.gpu
# Weights, activations and pages are rounded to FP16 once each: at most 2^-11 of a value, so a product of two is off by less than
# 2^-10 of its rms; two or three layers of seven products add up to a few of these.
TOL = 4e-3
MAPS = {"q4_k_m": synth.q4_k_m_type, "q6_k": lambda k: synth.Q6_K, "q8_0": lambda k: synth.Q8_0}


def tame(tensors):
    """The random blocks with the spread of trained weights (zero mean, 1 / sqrt(columns)), so that rounding errors are not
    amplified from layer to layer: scales and minima kept, the block factors replaced."""
    for kind, layer, t, rows, cols, raw in tensors:
        raw = raw.copy()
        if t != synth.F32:
            std = cols ** -0.5
            b = raw.reshape(-1, synth.BLOCK_BYTES[t])
            if t == synth.Q4_K:  # value = d * scale * (q - 7.5): the minima repeat the scales
                sc = np.random.default_rng([kind, layer]).integers(8, 64, (len(b), 8), dtype=np.uint8)
                b[:, 4:16] = synth.pack_q4k_scales(sc, sc)
                d = np.full(len(b), std / (4.6 * 39))
                b[:, 2:4] = (7.5 * d).astype(np.float16).view(np.uint8).reshape(-1, 2)
                b[:, 0:2] = d.astype(np.float16).view(np.uint8).reshape(-1, 2)
            else:
                d = np.full(len(b), std / (18.5 * 73) if t == synth.Q6_K else std / 73).astype(np.float16)
                at = 208 if t == synth.Q6_K else 0
                b[:, at:at + 2] = d.view(np.uint8).reshape(-1, 2)
        yield kind, layer, t, rows, cols, raw


def build_pair(oracle, arch, seed, kv, max_ctx, max_batch, ctx, types, bias=False):
    from juno_b200.handler import B200TransformerHandler
    tensors = list(tame(synth.random_model(arch, seed, types, norm="random", qkv_bias=bias)))
    om = oracle.Model(arch.hidden, arch.n_layers, arch.n_heads, arch.n_kv_heads, arch.inter, arch.vocab, arch.rms_eps, arch.rope_theta,
                      kv_f16=kv == "f16", max_seq=max_ctx)
    for kind, layer, t, rows, cols, blocks in tensors:
        om.set_tensor(kind, layer, blocks, t, rows if kind not in (1, 3, 4) and kind < 12 else 1, cols)
    h = B200TransformerHandler(arch, ctx, max_batch=max_batch, max_seqs=2, max_ctx=max_ctx, kv_dtype=kv)
    return om, h.load(tensors)


@pytest.mark.parametrize("arch,types,max_batch,start,n,kv,bias", [
    (TINY, "q4_k_m", 64, 0, 65, "f16", False),       # one position more than the small passes take
    (TINY, "q8_0", 8, 0, 9, "f16", False),           # few rows; an MMA tile that is almost empty
    (TINY, "q6_k", 1, 0, 3, "f16", False),           # a model opened for one sequence
    (SMALL128, "q4_k_m", 64, 37, 131, "f16", False),  # starts inside a page, one row tile of 128 and three rows
    (SMALL128, "q6_k", 16, 64, 64, "f16", False),    # starts at a key tile, whole tiles
    (SMALL128, "q8_0", 32, 1, 63, "f16", True),      # attention biases
    (SMALL128, "q4_k_m", 8, 5, 90, "f32", False),    # FP32 pages
])
def test_many_row_prompt_matches_oracle(ctx, oracle, arch, types, max_batch, start, n, kv, bias):
    om, h = build_pair(oracle, arch, 51, kv, 256, max_batch, ctx, MAPS[types], bias)
    rng = np.random.default_rng(n)
    toks = rng.integers(0, arch.vocab, start + n).tolist()
    seq, refs = om.new_seq(), []
    for p, t in enumerate(toks):
        ref, hid = om.forward(seq, t, p, want_hidden=True)
        refs.append(ref)
    for p in range(start):
        h.forward_batch(["a"], [[toks[p]]], [p])
    want = [n - 1, 0, n // 2] if n < 60 else list(range(n - 1, -1, -5))  # out of order; more than the exact product takes
    got = h.prefill_logits("a", toks[start:], start, want)
    for row, w in zip(got, want):
        assert rel_err(row, refs[start + w]) < TOL, (w, rel_err(row, refs[start + w]))
    assert rel_err(h.last_hidden(1) if max_batch == 1 else h.last_hidden((n - 1) % min(max_batch, 64) + 1)[-1:], hid) < TOL
    # the cache it left: a decode step on top of it, and the same prompt again from its start
    nxt = int(np.argmax(refs[-1]))
    ref = om.forward(seq, nxt, start + n)
    assert rel_err(h.forward_batch(["a"], [[nxt]], [start + n])[0], ref) < TOL
    again = h.prefill("a", toks[start:], start, want_logits=True)
    assert rel_err(again, refs[-1]) < TOL and h.length("a") == start + n + 1
    h.release_gpu_resources()


def test_prompt_of_two_passes(ctx):
    """2,300 positions: a pass of 2,048 and one of 252, against the same prompt in portions of 64 (the small passes)."""
    from juno_b200.handler import B200TransformerHandler
    h = B200TransformerHandler(SMALL128, ctx, max_batch=64, max_seqs=2, max_ctx=2304)
    h.load(tame(synth.random_model(SMALL128, 52, norm="random")))
    toks = np.random.default_rng(1).integers(0, SMALL128.vocab, 2300)
    places = [0, 1000, 2047, 2048, 2299]
    got = h.prefill_logits("a", toks, 0, places)
    for p in range(0, 2300, 64):
        part = toks[p:p + 64]
        inside = [w - p for w in places if p <= w < p + 64]
        ref = h.prefill_logits("b", part, p, inside)
        for w, row in zip(inside, ref):
            assert rel_err(got[places.index(p + w)], row) < TOL, p + w
    h.release_gpu_resources()


@pytest.mark.parametrize("arch,n,start,at", [(TINY, 80, 0, 40), (TINY, 70, 7, 63), (SMALL128, 200, 0, 130), (SMALL128, 65, 3, 1)])
def test_values_beyond_fp16_stay_behind_their_position(ctx, arch, n, start, at):
    """One position whose first-layer values overflow FP16 (infinite in its page, NaN from the next layer on): the positions before it
    have the logits that they have without it, to the last bit."""
    from juno_b200.handler import B200TransformerHandler
    odd = arch.vocab - 1

    def tensors():
        for kind, layer, t, rows, cols, raw in tame(synth.random_model(arch, 53, MAPS["q8_0"], norm="ones")):
            if kind == 0:  # the first column of the embeddings: of the odd token alone, which has no other
                b = raw.reshape(rows, cols // 32, 34)
                b[:, 0, 2] = 0
                b[odd, :, 2:] = 0
                b[odd, 0, 2] = 127
            elif (kind, layer) == (7, 0):  # W_v reads it with a factor of 12,700
                b = raw.reshape(rows, cols // 32, 34)
                b[:, 0, :2] = np.full(1, 100, np.float16).view(np.uint8)
                b[:, 0, 2:] = 0
                b[:, 0, 2] = 127
            yield kind, layer, t, rows, cols, raw

    h = B200TransformerHandler(arch, ctx, max_batch=8, max_seqs=2, max_ctx=256)
    h.load(tensors())
    toks = np.random.default_rng(n).integers(0, odd, start + n)
    got = {}
    for name, tok in (("plain", toks[start + at]), ("odd", odd)):
        toks[start + at] = tok
        if start:
            h.prefill(name, toks[:start], 0)
        got[name] = h.prefill_logits(name, toks[start:], start, range(n))
    assert np.isfinite(got["plain"]).all() and not np.isfinite(got["odd"][at]).any()
    assert np.array_equal(got["odd"][:at], got["plain"][:at])
    h.release_gpu_resources()


# rows of a pass take 71 KB each, the FP16 matrices 67 MB: what is left decides how many positions go in one
@pytest.mark.parametrize("before,left_mb,passes", [(200, 40, 4), (0, 100, 8), (0, 60, None)])
def test_prompts_with_little_memory_left(ctx, before, left_mb, passes):
    """2,000 positions where memory is short: passes of as many rows as there is room for (not fewer than an earlier prompt had), or the
    small passes; and whole again when memory is back."""
    import torch
    from juno_b200.handler import B200TransformerHandler
    arch = synth.Arch(1024, 2, 16, 4, 8192, 512, 1e-5, 10000.0)
    toks = np.random.default_rng(4).integers(0, arch.vocab, 2000)
    places = [0, 700, 1999]

    def opened():
        h = B200TransformerHandler(arch, ctx, max_batch=64, max_seqs=2, max_ctx=2048)
        return h.load(tame(synth.random_model(arch, 54, MAPS["q8_0"], norm="random")))

    def launches(h):
        n = ctx.counters()["kernel_launches"]
        rows = h.prefill_logits("a", toks, 0, places)
        return rows, ctx.counters()["kernel_launches"] - n

    h = opened()
    h.prefill("a", toks[:60], 0)
    want, whole = launches(h)
    h.release_gpu_resources()
    h = opened()
    if before:
        h.prefill("a", toks[:before], 0)
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (left_mb << 20), dtype=torch.uint8, device="cuda")
    got, count = launches(h)
    del held
    torch.cuda.empty_cache()
    again, count_again = launches(h)
    h.release_gpu_resources()
    assert max(rel_err(g, w) for g, w in zip(got, want)) < TOL
    assert np.array_equal(again, want) and count_again == whole
    per_pass, logits, hidden = whole - 3, 2, 1
    if passes is None:
        assert count > 500  # 32 small passes
    else:
        assert count == passes * per_pass + 3 * logits + hidden, (count, whole)


def test_short_prompts_need_no_room_for_fp16_weights(ctx):
    """300 positions with room for their rows (36 MB), but not for FP16 rows of the weights (67 MB): one pass all the same; and where memory is back, a long prompt
    finds room for both, in place of the rows that are there."""
    import torch
    from juno_b200.handler import B200TransformerHandler
    arch = synth.Arch(1024, 2, 16, 4, 8192, 512, 1e-5, 10000.0)
    toks = np.random.default_rng(5).integers(0, arch.vocab, 900)

    def run(h, n, name):
        count = ctx.counters()["kernel_launches"]
        return h.prefill_logits(name, toks[:n], 0, [0, n - 1]), ctx.counters()["kernel_launches"] - count

    got = []
    for left_mb in (None, 45):
        h = B200TransformerHandler(arch, ctx, max_batch=64, max_seqs=2, max_ctx=1024)
        h.load(tame(synth.random_model(arch, 54, MAPS["q8_0"], norm="random")))
        h.prefill("a", toks[:60], 0)
        held = None
        if left_mb:
            torch.cuda.empty_cache()
            held = torch.empty(torch.cuda.mem_get_info()[0] - (left_mb << 20), dtype=torch.uint8, device="cuda")
        got.append(run(h, 300, "a"))
        del held
        torch.cuda.empty_cache()
        got.append(run(h, 900, "b"))
        h.release_gpu_resources()
    for (rows, count), (want, whole) in zip(got[2:], got[:2]):
        assert np.array_equal(rows, want) and count == whole


def test_profiled_bytes_of_the_products(ctx):
    """What the profile counts for the products of a prompt: 16-bit operands, FP32 results, one column per gate and up row."""
    from juno_b200.handler import B200TransformerHandler
    a, n = SMALL128, 100
    h = B200TransformerHandler(a, ctx, max_batch=64, max_seqs=1, max_ctx=128)
    h.load(synth.random_model(a, 55))
    ctx.profile(True)
    ctx.profile_read()
    h.prefill("a", np.arange(n), 0)
    got = ctx.profile_read()["gemm_rows"]
    ctx.profile(False)
    kv = a.hidden // a.n_heads * a.n_kv_heads
    shapes = [(a.hidden, a.hidden + 2 * kv, 1), (a.hidden, a.hidden, 1), (a.hidden, 2 * a.inter, 2), (a.inter, a.hidden, 1)]  # columns, rows, rows per result
    want = sum(2 * k * (n + rows) + 4 * n * rows // per for k, rows, per in shapes)
    assert got["launches"] == 4 * a.n_layers and got["algo_bytes"] == want * a.n_layers
    h.release_gpu_resources()
