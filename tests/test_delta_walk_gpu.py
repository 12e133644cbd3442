"""Prompts of the gated delta rule where the walk over its chunks changes: one and two blocks of value columns per CTA (up to as many CTAs as the
device has SMs, and beyond), an odd last block, a second half of the keys that is empty, short or whole, fewer and more chunks than stages.  The oracle
and the tolerances are those of the other delta rule tests."""
import pytest

from tests.test_vuzelix_gpu import delta_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,G,D,V", [
    (100, 2, 2, 128, 16), (40, 37, 37, 128, 64), (40, 19, 1, 128, 128), (36, 50, 25, 112, 48), (66, 3, 3, 80, 32),      # 128 keys and fewer
    (70, 2, 1, 256, 32), (50, 40, 40, 256, 64), (50, 52, 4, 144, 48), (33, 3, 1, 250, 40),                              # 256 and fewer
    (90, 2, 2, 64, 48), (34, 50, 2, 64, 48), (80, 1, 1, 32, 16), (49, 2, 1, 48, 64), (130, 3, 3, 16, 144),              # 64 and fewer
])
def test_walk(lib, T, H, G, D, V):
    delta_case(lib, 1, T, H, G, D, V, 7 * T + D + V)
