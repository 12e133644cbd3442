"""bf16 products whose tiles fill little of the chip: K in ranges over the CTAs of a cluster, tiles of any multiple of 16 tokens."""
import numpy as np
import pytest

from tests import hybrid_models as hm
from tests.test_hybrid_gpu import done
from tests.util import Dev, normwise

pytestmark = pytest.mark.gpu


# K blocks that the ranges do not divide, a last block of 16; one row, tiles of one and of several steps of 16 tokens, the last one short
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
