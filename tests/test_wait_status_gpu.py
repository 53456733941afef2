"""Waits that kernels gave up: reported once, by the call that they belong to."""
import ctypes as C

import numpy as np
import pytest

from juno_b200 import _lib, synth
from juno_b200._lib import JunoError
from modelutil import TINY

pytestmark = pytest.mark.gpu
TILE = 1 | 3 << 8 | 7 << 16  # a weight tile of warp 3, block 7


@pytest.mark.parametrize("batch", [1, 9])
def test_product_reports_its_failure_once(ctx, mv, wait_words, batch):
    A = mv.upload_quantized(synth.random_blocks(np.random.default_rng(1), synth.Q4_K, 64, 512), synth.Q4_K, 64, 512)
    x = np.ones((batch, 512), np.float32)
    want = mv.sgemv(A, x)
    wait_words[0] = TILE
    with pytest.raises(JunoError, match="warp 3 of block 7") as e:
        mv.sgemv(A, x)
    assert e.value.rc == _lib.ERR_TIMEOUT and wait_words[0] == 0
    assert np.array_equal(mv.sgemv(A, x), want)
    A.close()


def test_enqueued_product_is_reported_by_the_synchronisation(ctx, mv, wait_words):
    from juno_b200.handler import B200TransformerHandler
    import torch
    h = B200TransformerHandler(TINY, ctx, max_ctx=64)
    h.load(synth.random_model(TINY, 5))
    A = mv.upload_quantized(synth.random_blocks(np.random.default_rng(1), synth.Q4_K, 64, 512), synth.Q4_K, 64, 512)
    x, y = torch.ones(9, 512, device="cuda"), torch.empty(9, 64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(mv._L.juno_gemv_device(ctx.handle, A.handle, C.c_void_p(x.data_ptr()), 9, C.c_void_p(y.data_ptr()), None), "juno_gemv_device")
    wait_words[1] = TILE
    mv.sgemv(A, np.ones(512, np.float32))  # neither a product nor a model step answers for it
    h.forward_batch(["a"], [[1]], [0])
    with pytest.raises(JunoError) as e:
        ctx.synchronize()
    assert e.value.rc == _lib.ERR_TIMEOUT
    ctx.synchronize()
    wait_words[0] = TILE  # a step's own
    with pytest.raises(JunoError):
        h.forward_batch(["a"], [[1]], [1])
    h.forward_batch(["a"], [[1]], [1])
    A.close()
    h.release_gpu_resources()
