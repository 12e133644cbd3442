"""fp32 products of several tokens on both tile widths, and one-token products of two rows per warp, plain and with their epilogues."""
import numpy as np
import pytest

from oracle import hybrid_oracle as ho
from tests import hybrid_models as hm
from tests import test_hybrid_gpu as hybrid
from tests import test_vuzelix_gpu as vuzelix

pytestmark = pytest.mark.gpu


# tiles of 64 tokens: more than one tile of 16 per SM, ragged rows and tokens, a last slab of 16 columns; 16 tokens of more rows than two tiles per SM;
# tiles of 16: at that line
@pytest.mark.parametrize("T,N,K", [(100, 2050, 80), (65, 3000, 336), (64, 2369, 48), (16, 2 * 148 * 64 + 1, 32), (12, 2 * 148 * 64, 32)])
def test_fp32(lib, T, N, K):
    hybrid.test_linear(lib, 0, T, N, K)


@pytest.mark.parametrize("T,N,K", [(100, 2050, 80), (130, 1300, 16)])
def test_fp32_epilogues(lib, T, N, K):
    vuzelix.test_mapped_products(lib, 0, T, N, K)


@pytest.mark.parametrize("bf16", hybrid.ACTS)
@pytest.mark.parametrize("N", [2 * 8 * 148 + 1, 2 * 8 * 148 + 2, 2 * 8 * 148])
def test_one_token_rows_in_pairs(lib, bf16, N):
    """Beyond the rows that give every warp one, the last of an odd number alone."""
    vuzelix.test_mapped_products(lib, bf16, 1, N, 48)


def test_fp32_gates(lib):
    """Gate and up rows side by side on tiles of 64 tokens, a last token tile of 36."""
    cfg = hm.config(97, 40, [hm.layer("retention", hm.retention(1, 16, 16, 16, [0.9]), 801)])
    w, toks = hm.weights(cfg, 7), hm.tokens(cfg, 100, 8)
    _, want = ho.Model(cfg, w).run(toks)
    m = hybrid.device(cfg, w, lib, "float32")
    e = hybrid.Engine(m)
    got = m.residuals(e.slots.acquire(), toks)
    e.close()
    m.close()
    assert np.max(hm.row_errors(got[0], want[0])) < 1e-5
