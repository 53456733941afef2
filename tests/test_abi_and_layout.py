"""CPU checks of the product library: it loads and exports every symbol the header declares (and nothing else with
the juno_ prefix); the tile layout round-trips bit-exactly through a host build of the device index maps."""
import ctypes as C
import os
import re

import numpy as np
import pytest

from juno_b200 import _lib, synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    L = _lib.load()
    hdr = open(os.path.join(ROOT, "include", "juno_b200.h")).read()
    declared = set(re.findall(r"\b(juno_[a-z0-9_]+)\s*\(", hdr))
    assert len(declared) >= 30
    for name in declared:
        assert hasattr(L, name), name
    assert declared == set(_lib.SIGNATURES), declared ^ set(_lib.SIGNATURES)
    # no undeclared juno_* export (debug hooks do not belong in the product library)
    import subprocess
    out = subprocess.run(["nm", "-D", "--defined-only", _lib.LIB_PATH], capture_output=True, text=True).stdout
    exported = {ln.split()[-1] for ln in out.splitlines() if ln.split() and ln.split()[-1].startswith("juno_")}
    assert exported == declared, exported ^ declared


def test_cfg_struct_matches_header():
    assert C.sizeof(_lib.ModelCfg) == 4 * 15 + 128
    assert C.sizeof(_lib.Counters) == 40


def test_device_probe_fails_soft():
    n = C.c_int32(-1)
    assert _lib.load().juno_device_count(C.byref(n)) == _lib.OK and n.value >= 0
    if n.value == 0:  # no GPU: the context refuses loudly, there is no CPU fallback
        h = C.c_void_p()
        assert _lib.load().juno_ctx_create(0, C.byref(h)) == _lib.ERR_CUDA
        assert "no CPU fallback" in _lib.last_error()


def test_null_and_closed_handles_return_codes():
    L = _lib.load()
    assert L.juno_qmat_free(None) == _lib.ERR_INVALID_ARG
    assert L.juno_ctx_destroy(None) == _lib.ERR_INVALID_ARG
    assert L.juno_model_free(None) == _lib.ERR_INVALID_ARG
    assert L.juno_seq_free(None) == _lib.ERR_INVALID_ARG


@pytest.mark.parametrize("t", [synth.Q4_K, synth.Q6_K, synth.Q8_0])
@pytest.mark.parametrize("rows,cols", [(16, 256), (37, 512), (5, 1024)])
def test_tile_layout_round_trip_bit_exact(oracle, layout_host, t, rows, cols):
    L = layout_host
    raw = synth.random_blocks(np.random.default_rng(t), t, rows, cols)
    n = L.layout_tiled_bytes(t, rows, cols)
    assert n == ((rows + 15) // 16) * (cols // 256) * {12: 2368, 14: 3360, 8: 4352}[t]
    tiles = np.zeros(n, dtype=np.uint8)
    assert L.layout_repack(t, raw.ctypes.data, rows, cols, tiles.ctypes.data) == 0
    out = np.empty((rows, cols), dtype=np.float32)
    assert L.layout_dequant_tiled(t, tiles.ctypes.data, rows, cols, out.ctypes.data) == 0
    ref = oracle.dequantize(t, raw, rows, cols)
    assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))


def test_synthetic_block_distributions(oracle):
    rng = np.random.default_rng(0)
    raw = synth.random_blocks(rng, synth.Q4_K, 64, 1024).reshape(-1, 144)
    d = raw[:, 0:2].copy().view(np.float16).astype(np.float32)
    assert 1e-3 * 0.99 <= d.min() and d.max() <= 2e-2 * 1.01
    sc = np.array([[oracle.lib().jo_q4k_scale(np.ascontiguousarray(b[4:16]).ctypes.data, j) for j in range(8)] for b in raw[:50]])
    assert sc.min() >= 0 and sc.max() <= 63 and sc.max() > 40
    q8 = synth.random_blocks(rng, synth.Q8_0, 8, 256).reshape(-1, 34)[:, 2:].view(np.int8)
    assert q8.min() >= -127 and q8.max() <= 127


def test_tensor_shard_context_geometry():
    from juno_b200.handler import TensorShardContext
    c = TensorShardContext(num_heads=32, hidden_dim=4096, tensor_rank=3, tensor_world_size=8)
    assert (c.heads_per_node(), c.head_start(), c.head_end(), c.head_dim(), c.slice_dim()) == (4, 12, 16, 128, 512)
    with pytest.raises(ValueError):
        TensorShardContext(32, 4096, 8, 8)
    with pytest.raises(ValueError):
        TensorShardContext(31, 4096, 0, 1)


def test_gemv_work_split_covers_every_tile_once(layout_host):
    """The split of a fused dequant-GEMV launch over CTAs, chunks and warps (csrc/qsplit.cuh, the same functions the
    kernel calls, built for the host): every (row tile, block) exactly once, the request order of a warp equals its use
    order, the finisher reads exactly the partial-sum slots that were written, and the busiest warp carries at most one
    row tile's worth of rounding more than the mean."""
    import ctypes as C
    import random
    L = layout_host
    L.qsplit_check.restype = C.c_int
    L.qsplit_check.argtypes = [C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int)]
    # (row tiles, blocks of K, CTAs): the decode-step products of the 8B and 70B architectures on 148 SMs x 1 or 2 CTAs,
    # their tensor-parallel shards, and degenerate shapes
    cases = [(384, 16, 148), (256, 16, 256), (1792, 16, 296), (256, 56, 148), (8016, 16, 296), (640, 32, 148), (3584, 32, 296),
             (512, 112, 148), (896, 16, 296), (128, 8, 128), (1002, 16, 296), (64, 1, 64), (8016, 1, 296), (300, 16, 296),
             (1, 16, 1), (3, 2, 3), (17, 3, 4), (33, 5, 2), (5000, 7, 296)]
    rng = random.Random(1)
    cases += [(rt := rng.randint(1, 3000), rng.randint(1, 60), min(rng.choice([1, 2, 7, 148, 296]), rt)) for _ in range(200)]
    for rt, nb, grid in cases:
        busiest = C.c_int()
        assert L.qsplit_check(rt, nb, grid, C.byref(busiest)) == 0, (rt, nb, grid)
        per_cta = -(-rt // grid)  # row tiles of the busiest CTA
        chunks = -(-per_cta // 16)
        assert busiest.value <= -(-per_cta * nb // 16) + chunks, (rt, nb, grid, busiest.value)


@pytest.mark.parametrize("slots", [2, 3, 4, 6])
def test_rings_know_the_copies_that_are_in_flight(layout_host, slots):
    for n in range(1, 30):
        for fail in range(n + 1):
            assert layout_host.ring_check(n, slots, fail) == 0, (n, fail)


@pytest.mark.parametrize("t", [12, 14, 8])
def test_row_tiles_that_quick_unpacking_would_cost_digits_are_wide(layout_host, t):
    """The powers of two of a row and the choice between quick and wide unpacking (csrc/row_pow.cuh, as the device finds them).  Wherever a row stays quick, the
    weights of every super-block, however far below the largest, are off by at most a quarter more than scales, minima and weights rounded to 11 bits
    each, at their own size, would be; and rows whose super-blocks are alike do stay quick.  Wide, the largest weight lies in [2^12, 2^15) (the bound of it in the
    upper half) unless that would take digits from a row that FP16 holds as it is."""
    import ctypes as C
    L = layout_host
    L.row_pow_of.restype, L.row_pow_of.argtypes = C.c_uint32, [C.c_int, C.c_int, C.c_void_p, C.c_void_p]

    def r11(v):
        m, e = np.frexp(v)
        return np.ldexp(np.round(m * 2048.0) / 2048.0, e)

    def h(v):
        return np.asarray(v, np.float64).astype(np.float16).astype(np.float64)

    rng = np.random.default_rng(t)
    quick = 0
    for trial in range(300):
        n, spread = 16, float(rng.choice([1.0, 3.0])) if trial % 2 else 2.0 ** rng.uniform(0, 13)
        d = (2.0 ** rng.uniform(-17, -6) * spread ** rng.uniform(-1, 0, n)).astype(np.float16).astype(np.float64)
        if t == 12:
            sc, mn = rng.integers(16, 64, (n, 8)), rng.integers(0, 64, (n, 8))
            dm = h(d * rng.choice([0.0, 1.0, 7.5, 15.0]))
            q = rng.integers(0, 16, (n, 8, 32)).astype(np.float64)
            s, m = d[:, None] * sc, dm[:, None] * mn
            scales, factors = np.concatenate([sc, mn], 1).astype(np.uint8), np.concatenate([d, dm]).astype(np.float32)
        elif t == 14:
            sc = rng.integers(16, 128, (n, 16)) * rng.choice([-1, 1], (n, 16))
            q = rng.integers(-32, 32, (n, 16, 16)).astype(np.float64)
            s, m = d[:, None] * sc, np.zeros((n, 16))
            scales, factors = sc.astype(np.int8).view(np.uint8), d.astype(np.float32)
        else:
            q = rng.integers(-127, 128, (n, 1, 32)).astype(np.float64)
            s, m = d[:, None], np.zeros((n, 1))
            scales, factors = np.zeros(1, np.uint8), d.astype(np.float32)
        scales, factors = np.ascontiguousarray(scales), np.ascontiguousarray(factors)
        word = L.row_pow_of(t, n, factors.ctypes.data, scales.ctypes.data)
        p, wp, wide = (word & 255) - 64, (word >> 8 & 255) - 64, word >> 16
        w = s[..., None] * q - m[..., None]
        own = r11(r11(s)[..., None] * q - r11(m)[..., None])
        got = h(q * 2.0 ** -24 * h(s * 2.0 ** p)[..., None] - h(m * 2.0 ** (p - 24))[..., None]) * 2.0 ** (24 - p)
        axes = (1, 2)
        if not wide:
            quick += 1
            assert (np.sqrt(((got - w) ** 2).mean(axes)) <= 1.25 * np.sqrt(((own - w) ** 2).mean(axes)) + 1e-30).all(), (trial, spread)
        elif trial % 2:
            raise AssertionError("alike super-blocks, yet wide")
        most = np.abs(w).max() * 2.0 ** wp
        assert most < 2.0 ** 15 and (most >= 2.0 ** 12 or wp == 30)
    assert quick >= 150
    if t != 8:  # a lone sub-block 64 (Q4_K) or 128 (Q6_K) times and more below the bound of the row's scales
        small = np.full(256, 60, np.uint8)
        small[3] = 1
        one = np.full(32, 2.0 ** -10, np.float32)
        assert (L.row_pow_of(t, 16, (one * 1.01).ctypes.data, small.ctypes.data) >> 16) == 0
        one[:1] /= 4
        assert (L.row_pow_of(t, 16, one.ctypes.data, small.ctypes.data) >> 16) == 1
    zero = np.zeros(32, np.float32)
    assert L.row_pow_of(t, 16, zero.ctypes.data, np.zeros(256, np.uint8).ctypes.data) == 64 | 64 << 8
    inf = np.full(32, np.inf, np.float32)
    inf[1:] = 1.0
    assert L.row_pow_of(t, 16, inf.ctypes.data, np.full(256, 9, np.uint8).ctypes.data) & 0xFFFF == 64 | 64 << 8


@pytest.mark.parametrize("missing", [(), (8,), (5, 7, 8), (2, 3, 4, 5, 6, 7, 8), (1, 2, 3, 4, 5, 6, 7, 8)])
def test_quantised_products_skip_cluster_sizes_that_do_not_fit(layout_host, missing):
    """The choice of CTAs that share K (csrc/quant_split.cuh) where the device takes some cluster sizes only: another size that fits is taken, for any product;
    a cluster that shares K has one piece of at most eight row tiles of one column block, and the clusters' shares cover every row tile of every column block once."""
    import ctypes as C
    fit = (C.c_int * 9)(0, *[0 if s in missing else 148 // s for s in range(1, 9)])
    out = (C.c_int * 4)()
    for n in (1, 9, 64, 129, 224, 225, 500, 1000):
        for rt in (1, 2, 7, 64, 128, 160, 384, 1792, 8016):
            for nb in (1, 2, 8, 16, 56):
                for pair in (0, 1):
                    layout_host.quant_split_of(n, rt, nb, pair, fit, out)
                    N, blocks, splits, clusters = out
                    assert N % 16 == 0 and 16 <= N <= 224 and (blocks - 1) * N < n <= blocks * N
                    if len(missing) == 8:
                        assert splits == 0
                        continue
                    assert 1 <= splits <= nb and splits not in missing and 1 <= clusters <= fit[splits] * (1 + pair)
                    if splits > 1:
                        assert clusters % blocks == 0 and -(-rt * blocks // clusters) <= 8
                    most, least = C.c_int(), C.c_int()
                    assert layout_host.quant_walk_check(n, rt, nb, pair, fit, C.byref(most), C.byref(least)) == 0, (n, rt, nb, pair)
                    assert most.value - least.value <= 1


def test_even_shares_begin_where_a_division_would_put_them(layout_host):
    for n in list(range(1, 300)) + [512, 1000, 1024]:
        for total in (n, n + 1, 2 * n - 1, 384, 1792, 7168, 8016, 32064, 1000003):
            assert layout_host.even_shares_check(total, n), (total, n)
