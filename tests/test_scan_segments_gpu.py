"""A long portion of a decaying state in segments that run side by side: the same bounds as one chain (tests/test_hybrid_gpu.py)."""
import numpy as np
import pytest

from bpd_substrate_b200 import capi
from bpd_substrate_b200.sequences import Sequence
from oracle import hybrid_oracle as ho
from tests import hybrid_models as hm
from tests import test_hybrid_gpu as hybrid

# at the portion from which segments pay (three chunks of 64 stay one chain, four do not), a last segment of one token, segments
# of several chunks with a shorter last one; value columns in two slices, keys that do not fill their tile
SHAPES = [(192, 2, 1, 16, 32), (193, 2, 1, 16, 32), (449, 2, 1, 128, 64), (1000, 74, 2, 48, 64), (520, 9, 3, 240, 80)]


@pytest.mark.gpu
@pytest.mark.parametrize("ssm", [0, 1])
@pytest.mark.parametrize("T,H,G,N,V", SHAPES)
def test_segments(lib, ssm, T, H, G, N, V):
    hybrid.test_decayed_scan(lib, 1, ssm, T, H, G, N, V)


@pytest.mark.parametrize("bytes_off", range(0, 20, 4))
def test_only_aligned_states_are_cut(bytes_off):
    """The fold moves 16 bytes of a state at a time.  (148 SMs are assumed where there is no device.)"""
    cut = capi.load().bpdq_decayed_scan_segments
    assert (cut((1 << 20) + bytes_off, 2048, 8, 256, 256, 1) > 1) == (bytes_off % 16 == 0)
    assert cut(1 << 20, 192, 8, 256, 256, 1) == 1 and cut(1 << 20, 2048, 8, 256, 256, 0) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("bytes_off", [0, 4, 8])
def test_whole_model(lib, bytes_off):
    """A portion that is cut, in a model whose recurrent states lie at any multiple of four bytes."""
    cfg = hm.config(97, 64, [hm.layer("retention", hm.retention(3, 40, 24, 12, [0.5, 0.98, 0.999])),
                             hm.layer("retention", hm.retention(2, 16, 130, 16, [1.0, 0.9], base=1e4), 33)])
    w, toks = hm.weights(cfg, 5), hm.tokens(cfg, 300, 6)
    _, want = ho.Model(cfg, w).run(toks)
    m = hybrid.device(cfg, w, lib, "bfloat16", capacity=512)
    slots = hybrid.Engine(m).slots
    block = lib.bpdq_alloc(slots.layout.slot_bytes + 16)
    try:
        assert lib.bpdq_memset_async(block, 0, slots.layout.slot_bytes + 16, m.stream) == 0
        got = m.residuals(Sequence(0, block + bytes_off, 512), toks)
        assert lib.bpdq_last_status() == 0
    finally:
        lib.bpdq_free(block)
        slots.close()
        m.close()
    for i in range(2):
        assert np.max(hm.row_errors(got[i], want[i])) < 4e-2, i
