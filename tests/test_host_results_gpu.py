"""Where the results of host calls live."""
import ctypes as C
import gc

import numpy as np
import pytest

import vosotarutil
from juno_b200 import _lib, synth
from juno_b200.matvec import PINNED_FROM

pytestmark = pytest.mark.gpu
MB = 1 << 20
POOL = 96 * MB


def alloc(ctx, nbytes):
    p = C.c_void_p()
    rc = ctx._L.juno_host_alloc(ctx.handle, nbytes, C.byref(p))
    assert rc in (_lib.OK, _lib.ERR_OOM)
    return p.value if rc == _lib.OK else None


def pinned(a):
    """Does the array lie in a block of the pool?"""
    while isinstance(a, np.ndarray):
        a = a.base
    return a is not None


def test_pool_is_bounded_and_reuses_its_blocks(ctx):
    gc.collect()
    blocks = []
    while (p := alloc(ctx, 5 * MB)) is not None:
        blocks.append(p)
        assert len(blocks) * 5 * MB <= POOL
    assert len(blocks) > 10
    assert ctx._L.juno_host_free(blocks[3]) == _lib.OK
    assert ctx._L.juno_host_free(blocks[3]) == _lib.ERR_INVALID_ARG and ctx._L.juno_host_free(blocks[0] + 64) == _lib.ERR_INVALID_ARG
    assert alloc(ctx, 5 * MB - 100) == blocks[3]
    for p in blocks:
        assert ctx._L.juno_host_free(p) == _lib.OK


def test_pool_holds_two_results_of_a_full_batch(ctx):
    """72 rows of a vocabulary of 128,256 (35 MB): the result of a call and the one before it."""
    gc.collect()
    blocks = [alloc(ctx, 72 * 128256 * 4) for _ in range(2)]
    for p in blocks:
        assert p is not None and ctx._L.juno_host_free(p) == _lib.OK
    whole = alloc(ctx, POOL)  # all of it in one, the two are given back
    assert whole is not None and ctx._L.juno_host_free(whole) == _lib.OK


def test_refused_requests_leave_the_idle_blocks(ctx):
    """What an idle block holds is still there after a request that cannot be served (a new block is zeroed)."""
    gc.collect()
    p = alloc(ctx, 3 * MB)
    C.memset(p, 0x5A, 3 * MB)
    assert ctx._L.juno_host_free(p) == _lib.OK
    assert alloc(ctx, POOL + 1) is None and alloc(ctx, 1 << 40) is None
    again = alloc(ctx, 3 * MB)
    assert again == p and C.string_at(again, 3 * MB) == b"\x5a" * (3 * MB)
    assert ctx._L.juno_host_free(again) == _lib.OK


def test_results_from_the_threshold_on_are_page_locked(ctx):
    gc.collect()
    below, at = ctx.host_rows(1, PINNED_FROM // 4 - 1), ctx.host_rows(1, PINNED_FROM // 4)
    assert pinned(at) and not pinned(below) and at.flags.writeable and at.shape == (1, PINNED_FROM // 4)


def test_large_results_outlive_their_call(tmp_path):
    """An array keeps its values while others are made, its block returns when the last view of it is dropped, and when the pool is used
    up results are ordinary arrays."""
    p = vosotarutil.Pair(tmp_path, synth.vosotar_config(64, 40000, [vosotarutil.L(2, 16, 16, 16, 16, 32)], taps=1), seed=7)
    h = p.open("default", max_batch=16, max_seqs=16)
    names = [f"r{i}" for i in range(16)]
    for i, r in enumerate(names):
        h.feed(r, p.tokens(3, i))
    gc.collect()
    kept, copies = [], []
    for _ in range(50):  # 2.5 MB each: more than the pool holds
        kept.append(h.forward_batch(names, [[1]] * 16, [3] * 16))
        copies.append(kept[-1].copy())
    assert all(np.array_equal(a, b) for a, b in zip(kept, copies))
    assert pinned(kept[0]) and sum(a.nbytes for a in kept if pinned(a)) <= POOL and not pinned(kept[-1])
    row = kept[0][3]  # a view alone keeps its block
    del kept
    gc.collect()
    again = h.forward_batch(names, [[2]] * 16, [3] * 16)
    assert pinned(again) and np.array_equal(row, copies[0][3]) and not np.array_equal(again, copies[0])
    h.release_gpu_resources()
    assert np.array_equal(row, copies[0][3])
