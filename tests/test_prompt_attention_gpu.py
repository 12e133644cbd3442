"""Attention of prompts on tiles of 128 rows x 128 keys: the cases and bounds of the latent and grouped kernels at the edges of tiles."""
import numpy as np
import pytest

from bpd_substrate_b200.engine import Engine
from bpd_substrate_b200.vuzelix import VuzelixSpec
from tests import hybrid_models as hm
from tests import test_hybrid_gpu as hybrid
from tests import test_vuzelix_gpu as vuzelix
from tests import vuzelix_models as vm

pytestmark = pytest.mark.gpu


# whole tiles and one row more, blocks that end inside the context, padded sizes, value slices of 64 and 128, two kinds of key pieces
@pytest.mark.parametrize("T,pos,H,D,r,V,R", [(128, 0, 2, 64, 64, 64, 64), (129, 0, 1, 128, 64, 128, 96), (200, 65, 3, 128, 64, 128, 128), (131, 500, 2, 64, 64, 192, 64),
                                             (255, 1, 1, 64, 128, 256, 64), (140, 3, 2, 60, 50, 120, 70), (384, 128, 1, 64, 64, 64, 64)])
def test_latent(lib, T, pos, H, D, r, V, R):
    hybrid.latent_case(lib, 1, T, pos, H, D, r, V, R, T + pos)


class Known:
    """The library, the host knowing the position of the portion that is checked."""

    def __init__(self, lib, T, context):
        self.lib, self.T, self.context = lib, T, context

    def __getattr__(self, name):
        return getattr(self.lib, name)

    def bpd_grouped_attention_cuda(self, *a):
        return self.lib.bpd_grouped_attention_context_cuda(*a[:8], self.context if a[7] == self.T else 0, *a[8:])


# one row beyond what the split kernel takes, rows of 1, 2, 4 and 16 heads, chunks inside a block, across blocks and none, value slices
@pytest.mark.parametrize("T,pos,H,G,D,V,chunk", [(65, 0, 1, 1, 64, 64, 0), (17, 100, 8, 2, 128, 128, 0), (128, 0, 2, 2, 64, 64, 0), (40, 90, 4, 1, 64, 192, 64),
                                                 (130, 5, 2, 1, 128, 128, 37), (70, 260, 16, 1, 60, 60, 128), (257, 127, 1, 1, 64, 128, 200), (90, 300, 4, 2, 192, 64, 1)])
@pytest.mark.parametrize("cap,sink", [(2.0, 1), (60.0, 1), (0.0, 0)])
def test_grouped(lib, T, pos, H, G, D, V, chunk, cap, sink):
    vuzelix.attention_case(Known(lib, T, pos + T), 1, T, pos, H, G, D, V, chunk, cap=cap, sink=sink)


# chunks just longer than those that stay on the smaller tiles, and about as long as a block
@pytest.mark.parametrize("T,pos,H,G,D,V,chunk", [(130, 5, 2, 1, 128, 128, 65), (40, 90, 4, 1, 64, 192, 80), (90, 300, 4, 2, 192, 64, 100), (300, 11, 4, 2, 64, 64, 127), (70, 260, 16, 1, 60, 60, 129)])
@pytest.mark.parametrize("cap,sink", [(14.0, 1), (0.0, 0)])
def test_grouped_short_chunks(lib, T, pos, H, G, D, V, chunk, cap, sink):
    test_grouped(lib, T, pos, H, G, D, V, chunk, cap, sink)


# values of several slices, rows of 64 and 128 heads of few tokens, one token (which stays where the position is read from the device)
@pytest.mark.parametrize("T,pos,H,G,D,V", [(33, 150, 2, 1, 128, 320), (33, 100, 2, 1, 64, 512), (2, 150, 2, 1, 128, 320), (1, 150, 2, 1, 128, 320), (2, 130, 128, 1, 64, 64), (1, 130, 128, 1, 64, 64),
                                           (2, 130, 64, 1, 128, 128), (1, 130, 64, 1, 128, 128)])
@pytest.mark.parametrize("cap,sink", [(14.0, 1), (0.0, 0)])
def test_grouped_many_columns_and_heads(lib, T, pos, H, G, D, V, cap, sink):
    test_grouped(lib, T, pos, H, G, D, V, 0, cap, sink)


# a portion that fills the cache's last row, and one that begins again at its first
@pytest.mark.parametrize("T,pos,rows", [(100, 100, 200), (100, 100, 199), (100, 101, 200), (70, 260, 330), (70, 260, 300)])
def test_grouped_at_the_end_of_the_rows(lib, T, pos, rows):
    vuzelix.attention_case(Known(lib, T, pos + T), 1, T, pos, 4, 2, 64, 64, 80, rows)


class ShortPortions(VuzelixSpec):
    portion = 128           # a cache of chunk + 128 rows


# a token's rows beyond the split kernel's: 128 heads on a key head, values of 320; recorded at 100 keys (the larger tiles' contexts begin at 96), and
# replayed beyond a block of keys, a chunk and the cache's rows
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,chunk", [(128, 1, 64, 64, 0), (2, 1, 128, 320, 0), (128, 1, 64, 64, 90), (2, 1, 128, 320, 90)])
def test_recorded_tokens(lib, heads, kv_heads, dim, vdim, chunk):
    """One-token steps that are replayed give the bits of those that are launched."""
    cfg = vm.config(97, 64, 2, [vm.layer("attention", vm.attention(heads, kv_heads, dim, vdim, chunk, 0.3, 15.0))])
    w, toks = vm.weights(cfg, 8), hm.tokens(cfg, 270, 9)
    results = []
    for use_graph in (True, False):
        m = vuzelix.device(cfg, w, lib, "bfloat16", capacity=300, spec_class=ShortPortions, use_graph=use_graph)
        e = Engine(m)
        e.feed("a", toks[:99])
        results.append(np.stack([e.feed("a", toks[t:t + 1], [0])[0][0] for t in range(99, 270)]))
        e.close()
        m.close()
    assert lib.bpdq_last_status() == 0
    assert np.isfinite(results[0]).all() and np.array_equal(*results)
