"""Products of quantised matrices with FP16 rows: row tiles and rows of x that are missing, rows whose scales lie far apart, and prompts at
the edges of their passes."""
import numpy as np
import pytest

from conftest import rel_err
from juno_b200 import synth
from test_prompt_gpu import MAPS, TOL, tame

pytestmark = pytest.mark.gpu
TYPES = [synth.Q4_K, synth.Q6_K, synth.Q8_0]


@pytest.fixture(scope="module")
def mv(ctx):
    from juno_b200.matvec import B200MatVec
    return B200MatVec(ctx)


@pytest.fixture(scope="module")
def ctx():
    from juno_b200.matvec import GpuContext
    return GpuContext.shared(0)


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("rows,cols,batch", [(1, 256, 9), (15, 512, 16), (129, 256, 17), (2400, 768, 65), (20000, 256, 31), (1040, 9 * 256, 64)])
def test_ragged_products(mv, oracle, t, rows, cols, batch):
    rng = np.random.default_rng(31)
    raw = synth.random_blocks(rng, t, rows, cols)
    x = rng.standard_normal((batch, cols)).astype(np.float32)
    A = mv.upload_quantized(raw, t, rows, cols)
    y = mv.sgemv(A, x)
    assert rel_err(y, oracle.matvec(t, raw, x, rows, cols)) < 1e-3
    assert np.array_equal(mv.sgemv(A, x), y)
    A.close()


@pytest.mark.parametrize("t", TYPES)
def test_rows_of_very_different_scale(mv, oracle, t):
    """Every row, alike in itself, has a power of two of its own: factors from the smallest to the largest that FP16 blocks hold, a row of zeros, and one whose
    minima dwarf its scales (blocks of one row that differ: test_blocks_of_one_row_far_apart).  Scale, minimum, weight and activation are rounded to FP16 once each, so a product is off by less than
    4 * 2^-11 of the row's largest part of a weight (scale * q or minimum) times the sum of |x|."""
    rng = np.random.default_rng(32)
    rows, cols, batch = 40, 1024, 12
    raw = synth.random_blocks(rng, t, rows, cols).copy()
    b = raw.reshape(rows, -1, synth.BLOCK_BYTES[t])
    d = (2.0 ** np.linspace(-19, 7, rows)).astype(np.float16)
    d[5] = 0
    at = {synth.Q4_K: 0, synth.Q6_K: 208, synth.Q8_0: 0}[t]
    b[:, :, at:at + 2] = d.view(np.uint8).reshape(rows, 1, 2)
    part = d.astype(np.float64) * {synth.Q4_K: 63 * 15, synth.Q6_K: 128 * 32, synth.Q8_0: 128}[t]
    if t == synth.Q4_K:
        dmin = (d * np.float16(4)).astype(np.float16)
        dmin[9] = np.float16(d[9] * np.float32(2000))
        b[:, :, 2:4] = dmin.view(np.uint8).reshape(rows, 1, 2)
        part = np.maximum(part, 63 * dmin.astype(np.float64))
    x = rng.standard_normal((batch, cols)).astype(np.float32)
    A = mv.upload_quantized(raw.reshape(-1), t, rows, cols)
    y = mv.sgemv(A, x).astype(np.float64)
    ref = oracle.matvec(t, raw.reshape(-1), x, rows, cols).astype(np.float64)
    bound = 2.0 ** -9 * np.abs(x).sum(1)[:, None] * part[None, :]
    assert (np.abs(y - ref) <= bound).all()
    big = np.arange(rows) != 5
    err = np.linalg.norm((y - ref)[:, big], axis=0) / np.linalg.norm(ref[:, big], axis=0)
    assert err.max() < 1e-2, err  # no row has lost its digits to another's scale
    assert (y[:, 5] == 0).all() or t == synth.Q4_K
    A.close()


@pytest.mark.parametrize("quant", ["q4_k_m", "q8_0"])
@pytest.mark.parametrize("n", [65, 128, 129, 224, 225, 449, 512, 513])
def test_prompts_match_small_passes(ctx, quant, n):
    """Portions on both sides of every change of pass: two CTAs per SM or one, one to four passes over the weights, FP16 rows behind 512."""
    from juno_b200.handler import B200TransformerHandler
    arch = synth.Arch(1024, 2, 8, 4, 4352, 500, 1e-5, 10000.0)
    h = B200TransformerHandler(arch, ctx, max_batch=64, max_seqs=2, max_ctx=544)
    h.load(tame(synth.random_model(arch, 61, MAPS[quant], norm="random")))
    toks = np.random.default_rng(3).integers(0, arch.vocab, n)
    places = [0, n // 2, n - 1]
    got = h.prefill_logits("a", toks, 0, places)
    refs = {}
    for p in range(0, n, 48):
        inside = [w - p for w in places if p <= w < p + 48]
        for w, row in zip(inside, h.prefill_logits("b", toks[p:p + 48], p, inside)):
            refs[p + w] = row
    assert max(rel_err(g, refs[w]) for w, g in zip(places, got)) < TOL
    h.release_gpu_resources()


def far_apart(t, rows, cols, ratio, place, minimum=7.5, seed=33):
    """Blocks of alike rows, one super-block of each `ratio` times as large as the others."""
    rng = np.random.default_rng(seed)
    raw = synth.random_blocks(rng, t, rows, cols).copy()
    per = synth.BLOCK_ELEMS[t]
    b = raw.reshape(rows, cols // per, synth.BLOCK_BYTES[t])
    std = cols ** -0.5
    d = (0.5 + rng.random((rows, cols // per))) * {synth.Q4_K: std / (4.61 * 41), synth.Q6_K: std / (18.5 * 91), synth.Q8_0: std / 73.3}[t]
    d[:, place * 256 // per:(place + 1) * 256 // per] *= ratio
    d = d.astype(np.float16)
    at = {synth.Q4_K: 0, synth.Q6_K: 208, synth.Q8_0: 0}[t]
    b[:, :, at:at + 2] = d[..., None].view(np.uint8)
    if t == synth.Q4_K:
        b[:, :, 2:4] = (np.float16(minimum) * d)[..., None].view(np.uint8)
        sc = rng.integers(16, 64, (b.shape[0] * b.shape[1], 8), dtype=np.uint8)
        b[:, :, 4:16] = synth.pack_q4k_scales(sc, sc).reshape(b.shape[0], b.shape[1], 12)
    elif t == synth.Q6_K:
        sc = rng.integers(48, 128, b.shape[:2] + (16,)) * rng.choice([-1, 1], b.shape[:2] + (16,))
        b[:, :, 192:208] = sc.astype(np.int8).view(np.uint8)
    return raw.reshape(-1)


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("ratio", [1, 16, 64, 512, 4096])
@pytest.mark.parametrize("place", [0, 2, 5])
def test_blocks_of_one_row_far_apart(mv, oracle, t, ratio, place):
    """A large super-block takes no digits from the others of its row: the path's 1e-3 holds where the activation is zero on it, and each single weight
    is off by its own rounding.  Weights come out through activations of a single one: the sum has one term, and is exact.  A weight of a wide row is
    rounded once (2^-11 of it at most); of a quick one, scale, minimum and weight are (of Q4_K a weight is the difference of two parts)."""
    rows, cols, batch = 70, 6 * 256, 16
    raw = far_apart(t, rows, cols, ratio, place)
    rng = np.random.default_rng(ratio)
    x = rng.standard_normal((batch, cols)).astype(np.float32)
    x[::2, place * 256:(place + 1) * 256] = 0
    A = mv.upload_quantized(raw, t, rows, cols)
    y, ref = mv.sgemv(A, x), oracle.matvec(t, raw, x, rows, cols)
    for part in (slice(0, None, 2), slice(1, None, 2)):
        assert np.linalg.norm(y[part] - ref[part]) < 1e-3 * np.linalg.norm(ref[part])
    w = oracle.dequantize(t, raw, rows, cols).reshape(rows, cols).astype(np.float64)
    cols_of = rng.choice(cols, batch, replace=False)
    one = np.zeros((batch, cols), np.float32)
    one[np.arange(batch), cols_of] = 1
    got = mv.sgemv(A, one).astype(np.float64).T
    if ratio >= 512 and t != synth.Q8_0 or ratio > 512:
        assert (np.abs(got - w[:, cols_of]) <= 2.0 ** -11 * 1.001 * np.abs(w[:, cols_of]) + 2.0 ** -38 * np.abs(w).max()).all()
    A.close()


def round11(v):
    m, e = np.frexp(v)
    return np.ldexp(np.round(m * 2048.0) / 2048.0, e)


@pytest.mark.parametrize("t,minimum,ratio", [(synth.Q4_K, 7.5, 1), (synth.Q4_K, 0, 1), (synth.Q4_K, 4, 1), (synth.Q4_K, 15, 1), (synth.Q4_K, 4, 512),
                                             (synth.Q6_K, 0, 1), (synth.Q6_K, 0, 512), (synth.Q8_0, 0, 1), (synth.Q8_0, 0, 4096)])
def test_prompts_round_weights_once(ctx, oracle, t, minimum, ratio):
    """A prompt through one layer against the same in 64 bits with the gate and up weights rounded to 11 bits once.  The rest is made so that nothing else
    rounds, but for the FP16 rows of the down projection (stated too): activations of the feed-forward are plus or minus one, its down weights
    and the heads have few bits, the attention adds zero.  What is left: FP32 sums, and a few roundings of those rows that go the other way (the share of sums
    within 1e-6 of a tie, 0.2 %, times an ulp: 2e-5)."""
    from juno_b200.handler import B200TransformerHandler
    arch = synth.Arch(1024, 1, 8, 4, 4352, 512, 1e-12, 10000.0)
    H, ff, V, n = arch.hidden, arch.inter, arch.vocab, 70
    rng = np.random.default_rng(7)
    q8 = lambda rows, cols, d, q: np.concatenate([np.full((rows, cols // 32, 1), d, np.float16).view(np.uint8), q.astype(np.int8).reshape(rows, cols // 32, 32).view(np.uint8)],
                                                 2).reshape(-1)
    emb = rng.choice([-64, 64], (V, H))
    on = np.ones(H, np.float32)
    if ratio > 1:
        emb[:, :256] = 0
    on *= np.float32(np.sqrt((emb[0] != 0).mean()))
    down = rng.integers(-64, 65, (H, ff))
    head = rng.integers(-64, 65, (V, H))
    mats = {k: far_apart(t, ff, H, ratio, 0, minimum, k) for k in (synth.T_FFN_GATE, synth.T_FFN_UP)}
    plain = {synth.T_TOKEN_EMBD: (V, H, emb), synth.T_OUTPUT: (V, H, head), synth.T_ATTN_OUT: (H, H, np.zeros((H, H))), synth.T_FFN_DOWN: (H, ff, down),
             synth.T_ATTN_Q: (H, H, rng.integers(-64, 65, (H, H))), synth.T_ATTN_K: (H // 2, H, rng.integers(-64, 65, (H // 2, H))),
             synth.T_ATTN_V: (H // 2, H, rng.integers(-64, 65, (H // 2, H)))}

    def tensors():
        for k, (rows, cols, q) in plain.items():
            yield k, 0, synth.Q8_0, rows, cols, q8(rows, cols, 2.0 ** -6, q)
        for k, raw in mats.items():
            yield k, 0, t, ff, H, raw
        for k in (synth.T_OUTPUT_NORM, synth.T_ATTN_NORM, synth.T_FFN_NORM):
            yield k, 0, synth.F32, 1, H, on.view(np.uint8)

    toks = rng.integers(0, V, n)
    places = [0, 9, 23, 40, 41, 55, 68, 69]
    h = B200TransformerHandler(arch, ctx, max_batch=64, max_seqs=1, max_ctx=96).load(tensors())
    got = h.prefill_logits("a", toks, 0, places)
    h.release_gpu_resources()
    x = emb[toks[places]] / 64.0
    xn = np.round(x / np.sqrt((x * x).mean(1, keepdims=True)) * on)
    g, u = (xn @ round11(oracle.dequantize(t, mats[k], ff, H).reshape(ff, H).astype(np.float64)).T for k in (synth.T_FFN_GATE, synth.T_FFN_UP))
    res = x + round11(g / (1 + np.exp(-g)) * u) @ (down / 64.0).T
    ref = res / np.sqrt((res * res).mean(1, keepdims=True)) * on @ (head / 64.0).T
    err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    assert err < 6e-5, err


@pytest.mark.parametrize("cols", [16384, 16640, 28672, 32768, 33024])
def test_long_rows(mv, oracle, cols):
    """Rows of x on both sides of the widths that staging keeps in registers, one CTA per SM or two, and of those that it reads twice."""
    rng = np.random.default_rng(cols)
    raw = synth.random_blocks(rng, synth.Q4_K, 40, cols)
    x = rng.standard_normal((9, cols)).astype(np.float32) * (2.0 ** np.arange(-12, 15, 3, dtype=np.float32))[:, None]
    A = mv.upload_quantized(raw, synth.Q4_K, 40, cols)
    y, ref = mv.sgemv(A, x), oracle.matvec(synth.Q4_K, raw, x, 40, cols)
    assert max(rel_err(a, b) for a, b in zip(y, ref)) < 1e-3
    A.close()


@pytest.mark.parametrize("hidden", [16640, 33024])
def test_long_rows_with_norms_and_addends(ctx, oracle, hidden):
    """The same inside a model, whose rows are summed, stored and normed on their way to FP16: nine requests at their first position, the attention adds zero."""
    from juno_b200.handler import B200TransformerHandler
    arch = synth.Arch(hidden, 1, hidden // 128, hidden // 256, 256, 64, 1e-5, 10000.0)
    rng = np.random.default_rng(hidden)
    shapes = {k: synth.tensor_shape(arch, k) for k in (synth.T_TOKEN_EMBD, synth.T_OUTPUT, synth.T_ATTN_Q, synth.T_ATTN_K, synth.T_ATTN_V, synth.T_ATTN_OUT,
                                                       synth.T_FFN_GATE, synth.T_FFN_UP, synth.T_FFN_DOWN)}

    def tensors():
        for k, (rows, cols) in shapes.items():
            if k in (synth.T_ATTN_Q, synth.T_ATTN_K, synth.T_ATTN_V, synth.T_ATTN_OUT):
                yield k, 0, synth.Q4_K, rows, cols, np.zeros(rows * cols // 256 * 144, np.uint8)
            else:
                yield from tame([(k, 0, synth.Q8_0, rows, cols, synth.random_blocks(rng, synth.Q8_0, rows, cols))])
        for k in (synth.T_OUTPUT_NORM, synth.T_ATTN_NORM, synth.T_FFN_NORM):
            yield k, 0, synth.F32, 1, hidden, (1 + 0.3 * rng.standard_normal(hidden)).astype(np.float32).view(np.uint8)

    w = {(k, t): raw for k, _, t, _, _, raw in tensors()}
    h = B200TransformerHandler(arch, ctx, max_batch=16, max_seqs=16, max_ctx=16)
    h.load((k, 0, t, *(shapes[k] if t != synth.F32 else (1, hidden)), raw) for (k, t), raw in w.items())
    got = h.forward_batch(["r%d" % i for i in range(9)], [[5 * i] for i in range(9)], [0] * 9)
    h.release_gpu_resources()
    emb, head, gate, up, down = (oracle.dequantize(synth.Q8_0, w[k, synth.Q8_0], *shapes[k]).reshape(shapes[k]).astype(np.float64)
                                 for k in (synth.T_TOKEN_EMBD, synth.T_OUTPUT, synth.T_FFN_GATE, synth.T_FFN_UP, synth.T_FFN_DOWN))
    normed = lambda v, k: v / np.sqrt((v * v).mean(1, keepdims=True) + arch.rms_eps) * w[k, synth.F32].view(np.float32)
    x = emb[5 * np.arange(9)]
    g = normed(x, synth.T_FFN_NORM) @ gate.T
    x = x + g / (1 + np.exp(-g)) * (normed(x, synth.T_FFN_NORM) @ up.T) @ down.T
    ref = normed(x, synth.T_OUTPUT_NORM) @ head.T
    assert max(rel_err(a, b) for a, b in zip(got, ref)) < TOL
