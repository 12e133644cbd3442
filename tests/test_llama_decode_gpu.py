"""One token of the Q8_0 Llama: the launches that hold several steps give the bits of the step-by-step forward, which a workspace without room for a second
residual gets.  (Both share the attention's sums, which are compared with 64 bits where the attention is tested alone.)"""
import ctypes as C

import numpy as np
import pytest

from bpd_substrate_b200 import llama
from tests.util import Dev

pytestmark = pytest.mark.gpu

VOCAB, ROWS = 1000, 300


def up64(n):
    return (n + 63) // 64 * 64


# heads, key heads, head size, feed-forward, fp16 cache, rotated dimensions, keys ahead, position.  Attention over a few keys, and split over CTAs: one to eight
# heads of a key head; the new row first, inside and last of a CTA's stretch, beyond what the query sees, and nowhere
CASES = [(8, 2, 32, 96, 1, 32, 70, 70), (16, 4, 64, 704, 1, 64, 5, 5), (16, 4, 64, 704, 1, 64, 64, 64), (16, 8, 64, 704, 0, 40, 199, 199), (4, 2, 64, 1024, 1, 64, 128, 128),
         (16, 2, 64, 1000 // 32 * 32, 1, 64, 255, 255), (8, 1, 128, 256, 0, 128, 130, 130), (4, 1, 128, 2016, 1, 0, 290, 290), (16, 4, 64, 704, 1, 64, 200, 64),
         (16, 4, 64, 704, 1, 64, 100, 250), (16, 4, 64, 704, 0, 64, 200, 0), (16, 4, 64, 704, 1, 64, 200, ROWS), (16, 4, 64, 704, 1, 64, 200, -1)]


@pytest.mark.parametrize("heads,kv_heads,dim,ff,f16,rope_dim,context,pos", CASES)
def test_token(lib, heads, kv_heads, dim, ff, f16, rope_dim, context, pos):
    E, row, layers = heads * dim, kv_heads * dim, 3
    cfg = llama.make_config(layers, heads, kv_heads, dim, ff, VOCAB, ROWS, rope_dim=rope_dim, kv_cache_f16=f16)
    dev = llama.DeviceLlama(llama.SyntheticLlama(cfg, seed=heads + context), lib)
    rng = np.random.default_rng(context)
    if context % 2:
        dev.weights.rope_freqs = dev._up((1 + rng.random(dim // 2)).astype(np.float32))
    cache = [rng.standard_normal((layers, ROWS, row)).astype(np.float16 if f16 else np.float32) for _ in range(2)]
    nx, n1, n2 = up64(E), up64(max(E, ff)), up64(max(E, ff))
    whole = lib.bpdq_llama_forward_workspace_bytes(C.byref(cfg), 1)
    results = []
    for size in (whole, 4 * (nx + n1 + 2 * n2) + 512):
        tok, p = Dev(lib, np.array([7], np.int32)), Dev(lib, np.array([pos], np.int32))
        k, v = Dev(lib, cache[0]), Dev(lib, cache[1])
        logits, out, ws = Dev(lib, nbytes=4 * VOCAB, fill=0xFF), Dev(lib, nbytes=8, fill=0xFF), Dev(lib, nbytes=size, fill=0xFF)
        assert lib.bpd_llama_forward_ws_cuda(tok.ptr, 1, C.byref(dev.weights), None, C.byref(cfg), p.ptr, context, k.ptr, v.ptr, logits.ptr, out.ptr, ws.ptr,
                                             size, dev.stream) == 0
        assert lib.bpdq_stream_sync(dev.stream) == 0
        word = lib.bpdq_device_error_word()
        assert word == (0 if 0 <= pos < ROWS else 20)
        if word:
            lib.bpdq_clear_status()
        results.append((logits.read(np.uint32), out.read(np.int64), k.read(np.uint8), v.read(np.uint8)))
    for a, b in zip(*results):
        assert np.array_equal(a, b)
    dev.close()


def test_tiles_that_leave_no_room_for_the_vector(lib):
    """Weight tiles as large as bpdq_set_tuning lets them be: a launch of several steps also holds its vector in shared memory, where 6144 numbers then do not
    fit beside them."""
    lib.bpdq_set_tuning(27000, 2, 0, 16, -1)
    try:
        test_token(lib, 48, 8, 128, 256, 1, 128, 70, 70)
    finally:
        lib.bpdq_set_tuning(8192, 2, 0, 16, -1)     # the library's defaults
