"""bf16 products of tiles that two CTAs share: ragged rows, tokens and K, every epilogue, and a model whose products are such."""
import numpy as np
import pytest

from tests import hybrid_models as hm
from tests import test_hybrid_gpu as hybrid
from tests import test_linear_ranges_gpu as ranges
from tests import test_vuzelix_gpu as vuzelix

pytestmark = pytest.mark.gpu


# rows that end in the first and in the second CTA of a pair, or leave it none; a last tile of few tokens, of fewer than the second CTA's; K blocks of
# 64 and a last one of 16
@pytest.mark.parametrize("T,N,K", [(560, 14336, 1040), (900, 9728 - 1, 1040), (901, 9728 - 129, 1040), (1100, 9728 - 200, 1088)])
def test_products(lib, T, N, K):
    assert lib.bpdq_linear_bf16_ctas(T, N, K) == 2
    ranges.test_ranges(lib, T, N, K)


@pytest.mark.parametrize("T,N,K", [(900, 9600, 1040)])
def test_epilogues(lib, T, N, K):
    """GELU, cap, log decay and write share."""
    assert lib.bpdq_linear_bf16_ctas(T, N, K) == 2
    vuzelix.test_mapped_products(lib, 1, T, N, K)


def test_model(lib):
    """Gates, and the residual step behind a wide model's products: a portion of them against portions of 100 tokens, whose products are not shared."""
    width, ff, T = 9600, 1040, 900
    assert lib.bpdq_linear_bf16_ctas(T, width, ff) == 2 and lib.bpdq_linear_bf16_ctas(100, width, ff) == 1
    cfg = hm.config(97, width, [hm.layer("retention", hm.retention(2, 16, 16, 16, [0.9, 0.99]), ff)])
    w, toks = hm.weights(cfg, 3), hm.tokens(cfg, T, 4)
    m = hybrid.device(cfg, w, lib, "bfloat16", capacity=1024)
    e = hybrid.Engine(m, slots=2)
    a, b = e.slots.acquire(), e.slots.acquire()
    got = m.residuals(a, toks)[0]
    want = np.concatenate([m.residuals(b, toks[t:t + 100])[0] for t in range(0, T, 100)])
    assert lib.bpdq_last_status() == 0
    e.close()
    m.close()
    assert np.max(hm.row_errors(got, want)) < 4e-2
