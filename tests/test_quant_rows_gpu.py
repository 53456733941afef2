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
    """Every row has a power of two of its own: factors from the smallest to the largest that FP16 blocks hold, a row of zeros, and one whose
    minima dwarf its scales.  Scale, minimum, weight and activation are rounded to FP16 once each, so a product is off by less than
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
