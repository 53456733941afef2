"""Products of few rows (decode batches and short portions of the layer stacks): row counts at the edges of the MMA's N, K split over
one to eight CTAs with remainders, row tiles that are partly empty - through whole models against their numpy statements."""
import pytest

import desilornutil
import vosotarutil
from juno_b200 import synth

pytestmark = pytest.mark.gpu
# widths 1100 and 520 are 18 and 9 stages of 64 columns, 2200 is 35: splits of 4, 2 and 8 with unequal parts
VOSOTAR = synth.vosotar_config(1100, 300, [vosotarutil.L(5, 72, 40, 520, 136, 2200)], taps=3)
DESILORN = synth.desilorn_config(1100, 300, [desilornutil.W(6, 2, 72, 40, 90, 2200), desilornutil.C(4, 4, 48, 64, 200, 200)], streams=3)


@pytest.mark.parametrize("util,cfg", [(vosotarutil, VOSOTAR), (desilornutil, DESILORN)], ids=["vosotar", "desilorn"])
def test_row_counts(tmp_path, util, cfg):
    p = util.Pair(tmp_path, cfg, seed=31)
    toks = p.tokens(129, 3)
    ref = p.oracle(toks)
    h = p.open("default", max_batch=40, max_seqs=60)
    for n in (9, 16, 17, 33, 64, 65, 97, 128, 129):
        util.check(h.prefill_logits(f"p{n}", toks[:n], 0, range(n)), ref[:n], "default", f"{n} positions")
    names = [f"d{i}" for i in range(35)]  # a decode batch: a different prefix each
    for i, r in enumerate(names):
        h.feed(r, toks[:i + 2])
    got = h.forward_batch(names, [[toks[i + 2]] for i in range(35)], [i + 2 for i in range(35)])
    util.check(got, ref[2:37], "default", "35 requests")
    h.release_gpu_resources()
