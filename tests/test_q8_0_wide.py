"""Q8_0 products of many tokens with fp16 operands (gemm_q8_0_wide.cu): the scalar reference bit for bit, like the narrow kernel's."""
import ctypes as C

import numpy as np
import pytest

from bpd_substrate_b200 import capi, llama, synth
from tests.test_q8_0_tiles import tiles_matmul
from tests.util import Dev, assert_bits_equal

# sizes that take the wide kernel (129 tokens of 9600 rows do not: two waves of either): rows that fill the narrow one's waves badly (N * M), at tokens around the edges of its tiles, rows below
# and beyond a row tile, K of one block and of a number of blocks that leaves a stage, and a set of accumulators, partly filled
SHAPES = [(64, 14400, 32), (40, 14336, 96), (129, 9600, 64), (257, 9580, 32), (300, 6000, 96), (640, 3300, 160), (1000, 2500, 96), (1000, 4096, 64), (333, 6100, 32),
          (480, 4600, 32)]


def test_these_sizes_take_it():
    """On 148 SMs, which are assumed where there is no device.  (Tiles of 32 tokens pay where several matrices share a launch: the forward below.)"""
    width = capi.load().bpdq_qmatmul_q8_0_tiles_width
    assert [width(*s) for s in SHAPES] == [64, 64, 0] + [128] * 7
    assert width(129, 9000, 64) == 128 and width(16, 14400, 32) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", SHAPES + [(129, 9000, 64)])
def test_product_is_the_scalar_reference_bit_for_bit(lib, oracle, M, N, K):
    rng = np.random.default_rng(M * 7 + N + K)
    W = synth.q8_0_matrix(N, K, rng).reshape(N, K // 32, 34)
    X = synth.activations(K, rng, rows=M)
    W[0, 0, 2:], X[0, :32] = 0x80, -3.0                      # -128 against -127: the largest sum of a block
    W[1, 0, :2] = np.frombuffer(np.float16(3e-7).tobytes(), np.uint8)      # scales below fp16's normal numbers, on both sides
    X[1, :32] *= 1e-6
    X[2, :32] = 0.0
    assert_bits_equal(tiles_matmul(lib, W.reshape(-1), X, M, N, K), oracle.qmatmul_q8_0(W.reshape(-1), X, M, N, K).reshape(M, N))


def forward_in(lib, cfg, model, n, less):
    """Logits and greedy tokens of a prompt in a workspace that is `less` bytes short of the full one."""
    toks, pos = np.random.default_rng(1).integers(0, cfg.vocab_size, n).astype(np.int32), np.arange(n, dtype=np.int32)
    dev = llama.DeviceLlama(model, lib)
    try:
        dev.retile()
        d_tok, d_pos, logits, out = Dev(lib, toks), Dev(lib, pos), Dev(lib, nbytes=4 * n * cfg.vocab_size, fill=0xFF), Dev(lib, nbytes=8 * n)
        size = lib.bpdq_llama_forward_workspace_bytes(C.byref(dev.cfg), n) - less
        ws = Dev(lib, nbytes=size, fill=0xEE)
        assert lib.bpd_llama_forward_ws_cuda(d_tok.ptr, n, C.byref(dev.weights), C.byref(dev.tiles), C.byref(dev.cfg), d_pos.ptr, 0, dev.d_k,
                                             dev.d_v, logits.ptr, out.ptr, ws.ptr, size, dev.stream) == 0
        assert lib.bpdq_stream_sync(dev.stream) == 0
        assert lib.bpdq_last_status() == 0
        return logits.read(np.uint32), out.read(np.int64)
    finally:
        dev.close()


def wide_only(n, K):
    """What the activations of K columns take in the wide kernel beyond the narrow one."""
    return (K // 32) * (-(-n // 128) * 80 * 128 - -(-n // 64) * 36 * 64)


# heads of 32 or 128, feed-forward, layers, tokens.  In the first the wide kernel takes q/k/v and gate/up as one launch each, where
# the narrow one takes a launch each, on tiles of 128 and of 32 tokens; in the others the down projection too, which then forms silu(gate) * up as it quantizes: whole and partly
# filled tiles of 128 tokens
@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,ff,layers,n", [(8, 2, 32, 704, 2, 300), (8, 2, 32, 704, 2, 30), (16, 4, 128, 2048, 1, 300), (16, 4, 128, 2080, 1, 384)])
def test_forward_in_a_workspace_of_the_narrow_kernel(lib, heads, kv_heads, dim, ff, layers, n):
    """A caller's scratch that holds only the narrow kernel's activations is still enough, and gives the same bits."""
    assert (lib.bpdq_qmatmul_q8_0_tiles_width(n, heads * dim, ff) > 0) == (heads == 16)
    cfg = llama.make_config(layers, heads, kv_heads, dim, ff, 500, n)
    model = llama.SyntheticLlama(cfg, seed=5)
    full, short = (forward_in(lib, cfg, model, n, less) for less in (0, wide_only(n, max(ff, heads * dim))))
    assert np.array_equal(full[0], short[0]) and np.array_equal(full[1], short[1])
