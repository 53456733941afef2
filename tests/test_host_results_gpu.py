"""Where the results of host calls live."""
import gc

import numpy as np
import pytest

import vosotarutil
from juno_b200 import synth

pytestmark = pytest.mark.gpu


def test_large_results_are_page_locked_and_outlive_their_call(tmp_path):
    """Results of a megabyte and more come from a bounded pool: an array keeps its values while others are made, blocks return when the
    last view is dropped, and when the pool is used up results are ordinary arrays."""
    p = vosotarutil.Pair(tmp_path, synth.vosotar_config(64, 40000, [vosotarutil.L(2, 16, 16, 16, 16, 32)], taps=1), seed=7)
    h = p.open("default", max_batch=16, max_seqs=16)
    names = [f"r{i}" for i in range(16)]
    for i, r in enumerate(names):
        h.feed(r, p.tokens(3, i))
    kept, copies = [], []
    for _ in range(50):  # 2.5 MB each: more than the pool holds
        kept.append(h.forward_batch(names, [[1]] * 16, [3] * 16))
        copies.append(kept[-1].copy())
    assert all(np.array_equal(a, b) for a, b in zip(kept, copies))
    row = kept[0][3]  # a view alone keeps its block
    del kept
    gc.collect()
    again = h.forward_batch(names, [[2]] * 16, [3] * 16)
    assert np.array_equal(row, copies[0][3]) and not np.array_equal(again, copies[0])
    h.release_gpu_resources()
    assert np.array_equal(row, copies[0][3])
