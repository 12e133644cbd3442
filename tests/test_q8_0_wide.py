"""Q8_0 products of many tokens with fp16 operands (gemm_q8_0_wide.cu): the scalar reference bit for bit, like the narrow kernel's."""
import ctypes as C

import numpy as np
import pytest

from bpd_substrate_b200 import llama, synth
from tests.test_q8_0_tiles import tiles_matmul
from tests.util import Dev, assert_bits_equal

pytestmark = pytest.mark.gpu

# sizes that take the wide kernel: rows that fill the narrow one's waves badly (N * M), at tokens around the edges of its tiles, rows below
# and beyond a row tile, K of one block and of a number of blocks that leaves a stage, and a set of accumulators, partly filled
SHAPES = [(64, 14400, 32), (40, 14336, 96), (129, 9600, 64), (257, 9580, 32), (300, 6000, 96), (640, 3300, 160), (1000, 2500, 96), (1000, 4096, 64), (333, 6100, 32),
          (480, 4600, 32)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_product_is_the_scalar_reference_bit_for_bit(lib, oracle, M, N, K):
    rng = np.random.default_rng(M * 7 + N + K)
    W = synth.q8_0_matrix(N, K, rng).reshape(N, K // 32, 34)
    X = synth.activations(K, rng, rows=M)
    W[0, 0, 2:], X[0, :32] = 0x80, -3.0                      # -128 against -127: the largest sum of a block
    W[1, 0, :2] = np.frombuffer(np.float16(3e-7).tobytes(), np.uint8)      # scales below fp16's normal numbers, on both sides
    X[1, :32] *= 1e-6
    X[2, :32] = 0.0
    assert_bits_equal(tiles_matmul(lib, W.reshape(-1), X, M, N, K), oracle.qmatmul_q8_0(W.reshape(-1), X, M, N, K).reshape(M, N))


def test_forward_in_a_workspace_of_the_narrow_kernel(lib):
    """A caller's scratch that holds only the narrow kernel's activations is still enough, and gives the same bits: q/k/v and gate/up
    as one launch against one launch each."""
    n = 300
    cfg = llama.make_config(2, 8, 2, 32, 704, 500, n)
    model = llama.SyntheticLlama(cfg, seed=5)
    toks, pos = np.random.default_rng(1).integers(0, 500, n).astype(np.int32), np.arange(n, dtype=np.int32)
    tiles = -(-n // 128) * 80 * 128 - -(-n // 64) * 36 * 64
    results = []
    for less in (0, (704 // 32) * tiles):
        dev = llama.DeviceLlama(model, lib)
        try:
            dev.retile()
            d_tok, d_pos, logits, out = Dev(lib, toks), Dev(lib, pos), Dev(lib, nbytes=4 * n * 500, fill=0xFF), Dev(lib, nbytes=8 * n)
            size = lib.bpdq_llama_forward_workspace_bytes(C.byref(dev.cfg), n) - less
            ws = Dev(lib, nbytes=size, fill=0xEE)
            assert lib.bpd_llama_forward_ws_cuda(d_tok.ptr, n, C.byref(dev.weights), C.byref(dev.tiles), C.byref(dev.cfg), d_pos.ptr, 0, dev.d_k,
                                                 dev.d_v, logits.ptr, out.ptr, ws.ptr, size, dev.stream) == 0
            assert lib.bpdq_stream_sync(dev.stream) == 0
            assert lib.bpdq_last_status() == 0
            results.append((logits.read(np.uint32), out.read(np.int64)))
        finally:
            dev.close()
    assert np.array_equal(results[0][0], results[1][0]) and np.array_equal(results[0][1], results[1][1])
