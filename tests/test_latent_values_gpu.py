"""Latent attention whose CTAs of a head join the splits of keys a slice each (a cluster), and each on its own: both sides of the line."""
import pytest

from tests.test_hybrid_gpu import ACTS, latent_case

pytestmark = pytest.mark.gpu


# tokens, keys before them, heads, value columns, rank: 10 and 11 blocks of 64 keys with 4 tokens, 9 and 10 with 2; a rank that the slices
# do not divide, one slice without columns (2 rows of 16 over 5 CTAs), more value columns than a cluster takes
@pytest.mark.parametrize("bf16", ACTS)
@pytest.mark.parametrize("T,pos,H,V,R", [(4, 636, 2, 48, 208), (4, 637, 2, 48, 208), (2, 574, 3, 72, 500), (2, 575, 3, 72, 500), (3, 800, 2, 160, 24), (3, 800, 2, 272, 96)])
def test_shared_and_alone(lib, bf16, T, pos, H, V, R):
    latent_case(lib, bf16, T, pos, H, 24, 6, V, R, T + pos)
