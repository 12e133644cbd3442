"""bf16 products whose tiles fill little of the chip: K in ranges over the CTAs of a cluster, tiles of any multiple of 16 tokens."""
import ctypes as C

import numpy as np
import pytest

from oracle import hybrid_oracle as ho
from tests import hybrid_models as hm
from tests import test_hybrid_gpu as hybrid
from tests import test_vuzelix_gpu as vuzelix
from tests.test_hybrid_gpu import done
from tests.util import Dev, normwise

pytestmark = pytest.mark.gpu


def cut(lib, T, N, K):
    """Tokens of a tile and ranges of K of such a product."""
    tokens, ranges = C.c_int(), C.c_int()
    assert lib.bpdq_linear_bf16_tiles(T, N, K, C.byref(tokens), C.byref(ranges)) == 0
    return tokens.value, ranges.value


# one range, or several joined on tiles of 16 tokens: K blocks that the ranges do not divide, a last block of 16; one row, a last tile that is short
@pytest.mark.parametrize("T,N,K", [(2, 1, 512), (16, 128, 1040), (17, 200, 2000), (50, 128, 8208), (100, 300, 1296), (130, 129, 4096), (250, 256, 656),
                                   (300, 640, 528)])
def test_ranges(lib, T, N, K):
    rng = np.random.default_rng(T + N + K)
    W, x = hm.bf16_round(rng.standard_normal((N, K))), hm.bf16_round(rng.standard_normal((T, K)))
    dW, dx, do = Dev(lib, hm.bf16_bits(W)), Dev(lib, hm.bf16_bits(x)), Dev(lib, nbytes=4 * T * N + 64, fill=0xFF)
    done(lib, lib.bpd_linear_bf16_cuda(dW.ptr, dx.ptr, do.ptr, T, N, K, 1, None))
    raw = do.read(np.uint8)
    assert (raw[4 * T * N:] == 0xFF).all()
    assert normwise(raw[:4 * T * N].view(np.float32).reshape(T, N), x.astype(np.float64) @ W.T.astype(np.float64)) < 2e-5


# several ranges on tiles of several steps of 16 tokens, which the CTAs of a cluster finish in turn: fewer steps than CTAs' halves, as many, and
# more, so that a half takes a second one; ragged rows and tokens
JOINED = [(48, 1990, 4112, 1), (200, 1990, 4112, 1), (48, 2000, 10752, 1), (600, 976, 3088, 2), (590, 1095, 3088, 2), (600, 1096, 4112, 2)]


@pytest.mark.parametrize("T,N,K,turns", JOINED)
def test_joined_tiles(lib, T, N, K, turns):
    tokens, ranges = cut(lib, T, N, K)
    assert tokens > 16 and ranges > 1 and (tokens > 32 * ranges) == (turns > 1)
    test_ranges(lib, T, N, K)


@pytest.mark.parametrize("T,N,K", [(70, 1000, 4112), (600, 1096, 3088)])
def test_joined_epilogues(lib, T, N, K):
    """GELU, cap, log decay and write share on joined sums."""
    tokens, ranges = cut(lib, T, N, K)
    assert tokens > 16 and ranges > 1
    vuzelix.test_mapped_products(lib, 1, T, N, K)


# width, feed-forward, products (rows, columns) that have to be joined on tiles of several steps: the residual step with its rows fetched a turn ahead;
# gates with a tanh norm's input, the mixers' first products with step sizes
@pytest.mark.parametrize("width,ff,products", [(1096, 3088, [(1104, 3088)]), (3088, 548, [(1120, 3088), (1168, 3088), (1088, 3088)])])
def test_joined_products_of_a_model(lib, width, ff, products):
    T = 600
    for N, K in products:
        tokens, ranges = cut(lib, T, N, K)
        assert tokens > 32 * ranges and ranges > 1, (N, tokens, ranges)
    layers = [hm.layer("mamba2", hm.mamba2(6, 64, 20, 3, 4, 4), ff)] if width == 1096 else [
        hm.layer("mamba2", hm.mamba2(16, 32, 16, 4, 1, 4), ff), hm.layer("retention", hm.retention(2, 16, 250, 16, [0.9, 0.99]))]
    cfg = hm.config(97, width, layers)
    w, toks = hm.weights(cfg, 3), hm.tokens(cfg, T, 4)
    _, want = ho.Model(cfg, w).run(toks)
    m = hybrid.device(cfg, w, lib, "bfloat16", capacity=640)
    e = hybrid.Engine(m)
    got = m.residuals(e.slots.acquire(), toks)
    e.close()
    m.close()
    for i in range(len(layers)):
        assert np.max(hm.row_errors(got[i], want[i])) < 4e-2, i
