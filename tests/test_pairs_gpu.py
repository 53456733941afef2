"""Products of many rows on pairs of SMs: the last rows and columns of a tile missing, every epilogue that such a product has, K tails, K
shared by two and four pairs - in prompts whose feed-forwards are wide enough to take them."""
import numpy as np
import pytest

import desilornutil
import vosotarutil
from conftest import rel_err
from juno_b200 import synth
from test_prompt_gpu import TOL, tame

pytestmark = pytest.mark.gpu
VOSOTAR = synth.vosotar_config(1000, 200, [vosotarutil.L(4, 64, 64, 64, 64, 4200)], taps=2)
WIDE = synth.vosotar_config(2100, 200, [vosotarutil.L(2, 64, 64, 64, 64, 4200)], taps=1)
DESILORN = synth.desilorn_config(1000, 200, [desilornutil.W(4, 2, 64, 64, 300, 2100)], streams=2)


@pytest.mark.parametrize("util,cfg", [(vosotarutil, VOSOTAR), (desilornutil, DESILORN)], ids=["vosotar", "desilorn"])
@pytest.mark.parametrize("n", [130, 300, 513, 700, 768])
def test_prompts_match_the_oracle(tmp_path, util, cfg, n):
    p = util.Pair(tmp_path, cfg, seed=41)
    toks = p.tokens(n, 5)
    h = p.open("default", max_ctx=1024)
    places = list(range(0, n, 37)) + [n - 1]
    util.check(h.prefill_logits("a", toks, 0, places), p.oracle(toks)[places], "default", f"{n} positions")
    h.release_gpu_resources()


def test_two_pairs_share_k(tmp_path):
    p = vosotarutil.Pair(tmp_path, WIDE, seed=42)
    toks = p.tokens(768, 6)
    h = p.open("default", max_ctx=1024)
    places = list(range(0, 768, 51)) + [767]
    vosotarutil.check(h.prefill_logits("a", toks, 0, places), p.oracle(toks)[places], "default")
    h.release_gpu_resources()


@pytest.mark.parametrize("types", [synth.q4_k_m_type, lambda k: synth.Q8_0], ids=["q4_k_m", "q8_0"])
def test_quantised_prompt_matches_small_passes(ctx, types):
    from juno_b200.handler import B200TransformerHandler
    arch = synth.Arch(1024, 2, 8, 4, 4352, 500, 1e-5, 10000.0)
    h = B200TransformerHandler(arch, ctx, max_batch=64, max_seqs=2, max_ctx=704)
    h.load(tame(synth.random_model(arch, 43, types, norm="random")))
    toks = np.random.default_rng(2).integers(0, arch.vocab, 700)
    got = h.prefill_logits("a", toks, 0, [0, 300, 511, 512, 699])
    refs = {}
    for p in range(0, 700, 64):
        inside = [w - p for w in (0, 300, 511, 512, 699) if p <= w < p + 64]
        for w, row in zip(inside, h.prefill_logits("b", toks[p:p + 64], p, inside)):
            refs[p + w] = row
    for w, row in zip((0, 300, 511, 512, 699), got):
        assert rel_err(row, refs[w]) < TOL, w
    h.release_gpu_resources()
