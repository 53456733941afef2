"""Decode attention of contexts that one CTA takes alone: stored without a merge, with eight warps while there are few such CTAs and four
above; every ratio of query to key heads, empty warps, and batches in which only some contexts are that short."""
import pytest

from test_attn_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_heads,n_kv,hd,n", [(32, 8, 128, 1), (32, 8, 128, 18), (32, 8, 128, 19), (32, 4, 64, 74), (32, 4, 64, 75), (8, 8, 128, 3), (16, 8, 64, 5),
                                               (64, 8, 128, 2), (64, 8, 64, 40)])
def test_short_contexts(ctx, oracle, n_heads, n_kv, hd, n):
    lens = [[1, 16, 17, 31, 63, 64, 65, 127, 128, 129, 200, 255, 256][i * 5 % 13] for i in range(n)]
    _run(ctx, oracle, n_heads, n_kv, hd, lens, "f16")


def test_many_requests_with_long_contexts(ctx, oracle):
    _run(ctx, oracle, 8, 8, 128, [3, 700, 64, 1025] * 14, "f16")
