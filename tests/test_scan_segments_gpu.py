"""A long portion of a decaying state in segments that run side by side: the same bounds as one chain (tests/test_hybrid_gpu.py)."""
import pytest

from tests import test_hybrid_gpu as hybrid

# at the portion from which segments pay (three chunks of 64 stay one chain, four do not), a last segment of one token, segments
# of several chunks with a shorter last one; value columns in two slices, keys that do not fill their tile
SHAPES = [(192, 2, 1, 16, 32), (193, 2, 1, 16, 32), (449, 2, 1, 128, 64), (1000, 74, 2, 48, 64), (520, 9, 3, 240, 80)]


@pytest.mark.gpu
@pytest.mark.parametrize("ssm", [0, 1])
@pytest.mark.parametrize("T,H,G,N,V", SHAPES)
def test_segments(lib, ssm, T, H, G, N, V):
    hybrid.test_decayed_scan(lib, 1, ssm, T, H, G, N, V)
