"""A step that brings its results to the host gives the bits that its buffers hold on the device, whatever way inputs and results take."""
import numpy as np
import pytest

from bpd_substrate_b200.engine import Engine
from tests import hybrid_models as hm
from tests import test_hybrid_gpu as hybrid

pytestmark = pytest.mark.gpu


def on_device(m, seq, tokens, want):
    """The same step, its results read from the device's buffers."""
    m.launch(seq, tokens, want)
    logits, picked = np.empty((len(want), m.vocab), np.float32), np.empty(len(want), np.int64)
    assert m.lib.bpdq_stream_sync(m.stream) == 0
    m.lib.bpdq_d2h(logits.ctypes.data, m.lib.bpdq_hybrid_logits(m.plan), logits.nbytes)
    m.lib.bpdq_d2h(picked.ctypes.data, m.lib.bpdq_hybrid_picked(m.plan), picked.nbytes)
    return logits, picked


@pytest.mark.parametrize("vocab", [97, 4096 + 4, 2 * 4096 + 1])       # one slice of a row and several, rows that end inside 16 bytes
def test_results(lib, vocab):
    cfg = hm.config(vocab, 64, [hm.layer("retention", hm.retention(2, 16, 16, 16, [0.5, 0.98]), 33)])
    m = hybrid.device(cfg, hm.weights(cfg, 5), lib, "bfloat16", capacity=8300)
    e = Engine(m, slots=2)
    a, b = e.slots.acquire(), e.slots.acquire()
    toks = hm.tokens(cfg, 8300, 6)
    # inputs as one launch's arguments (3 and 4 words, 4096) or copied (4097 words and more); choices alone and logits; rows beyond the
    # pinned memory (40 and 300 of 8193 logits); recorded one-token steps in between
    at = 0
    for n, want in [(2, [1]), (1, [0]), (1, [0]), (1, [0]), (3, range(3)), (4094, [4093]), (1, [0]), (4090, [5, 0, 4089, 5, 77]), (1, [0]), (40, range(40)),
                    (1, [0]), (1, [0]), (1, [0, 0]), (1, [])]:
        part, want = toks[at:at + n], list(want)
        ref = on_device(m, a, part, want)
        choices_alone = n % 2 == 0
        logits, picked = m.step(b, part, want, not choices_alone)
        assert (logits is None) == choices_alone
        if not choices_alone:
            assert np.array_equal(logits.view(np.uint32), ref[0].view(np.uint32)), n
        assert np.array_equal(picked, ref[1]) and np.array_equal(picked, np.argmax(ref[0], 1) if want else picked), n
        at += n
    for seq in (a, b):
        e.slots.release(seq)
    a, b = e.slots.acquire(), e.slots.acquire()
    ref, (logits, picked) = on_device(m, a, toks[:300], list(range(300))), m.step(b, toks[:300], range(300))
    assert np.array_equal(logits.view(np.uint32), ref[0].view(np.uint32)) and np.array_equal(picked, ref[1])
    assert m.lib.bpdq_last_status() == 0
    e.close()
    m.close()


def churn(depth=40):
    """Leaves other numbers where earlier calls had their frames."""
    a = np.full(64, 12345, np.int32)
    return int(a[depth]) + (churn(depth - 1) if depth else 0)


@pytest.mark.parametrize("places", [[2], [0, 1, 2]])
def test_recorded_by_the_caller(lib, places):
    """A step inside the caller's own recording: replays read the caller's tokens and stand at the recorded position, long after the call has returned."""
    cfg = hm.config(97, 64, [hm.layer("latent_attention", hm.latent(2, 16, 8, 16, 24, 20, 0.3), 33)] * 2)
    s = lib.bpdq_stream_create()
    m = hybrid.device(cfg, hm.weights(cfg, 5), lib, "bfloat16", capacity=128, stream=s)
    e = Engine(m, slots=2)
    a, b = e.slots.acquire(), e.slots.acquire()
    toks = hm.tokens(cfg, 46, 7)
    for seq in (a, b):
        m.step(seq, toks[:40])
    mine, want = np.array(toks[43:46], np.int32), np.array(places, np.int32)
    assert lib.bpdq_graph_begin(s) == 0
    rc = lib.bpdq_hybrid_forward(m.plan, mine.ctypes.data, 3, 40, a.base, want.ctypes.data, want.size, None, 0, s)
    graph = lib.bpdq_graph_end(s)
    assert rc == 0 and graph
    mine[:] = toks[40:43]
    churn()
    assert lib.bpdq_graph_launch(graph, s) == 0
    assert lib.bpdq_stream_sync(s) == 0
    logits, picked = np.empty((want.size, 97), np.float32), np.empty(want.size, np.int64)
    lib.bpdq_d2h(logits.ctypes.data, lib.bpdq_hybrid_logits(m.plan), logits.nbytes)
    lib.bpdq_d2h(picked.ctypes.data, lib.bpdq_hybrid_picked(m.plan), picked.nbytes)
    lib.bpdq_graph_destroy(graph)
    ref = m.step(b, toks[40:43], places)
    assert np.array_equal(logits.view(np.uint32), ref[0].view(np.uint32)) and np.array_equal(picked, ref[1])
    # (the cache rows it wrote are those of positions 40 to 42: the next tokens agree too)
    a.length += 3
    assert np.array_equal(m.step(a, toks[43:46], [2])[0], m.step(b, toks[43:46], [2])[0])
    assert lib.bpdq_last_status() == 0
    e.close()
    m.close()
    lib.bpdq_stream_destroy(s)


def test_one_recording_per_slot(lib):
    """Whatever is asked of a slot's one-token steps, one recording gives the bits of launched steps; few outlive the
    engine's slots."""
    cfg = hm.config(5000, 64, [hm.layer("retention", hm.retention(2, 16, 16, 16, [0.5, 0.98]), 33), hm.layer("latent_attention", hm.latent(2, 16, 8, 16, 24, 20, 0.3))])
    w, toks = hm.weights(cfg, 5), hm.tokens(cfg, 40, 6)
    m, plain = (hybrid.device(cfg, w, lib, "bfloat16", capacity=64, use_graph=g) for g in (True, False))
    e, f = Engine(m, slots=2), Engine(plain, slots=2)
    held = [(e.slots.acquire(), f.slots.acquire()) for _ in range(2)]
    for t in range(24):
        a, b = held[t % 5 % 2]
        ref = plain.step(b, toks[t:t + 1], [0])
        if t % 3 == 0:
            got = on_device(m, a, toks[t:t + 1], [0])
        else:
            got = m.step(a, toks[t:t + 1], [0], t % 3 == 1)
        assert np.array_equal(got[1], ref[1]) and (got[0] is None or np.array_equal(got[0].view(np.uint32), ref[0].view(np.uint32))), t
        if t == 10:
            for s in held:
                assert np.array_equal(*(x.step(q, toks[24:40], range(16))[0] for x, q in zip((m, plain), s)))
        assert lib.bpdq_hybrid_recordings(m.plan) <= 2
    assert lib.bpdq_hybrid_recordings(m.plan) == 2 and lib.bpdq_hybrid_recordings(plain.plan) == 0
    e.close()
    # recordings of slots that have gone: a few wait for the next engine, as many engines as there are
    many = [Engine(m, slots=7) for _ in range(3)]
    for i, other in enumerate(many):
        for k in range(7):
            other.feed(k, toks[:1], [0])
    assert lib.bpdq_hybrid_recordings(m.plan) <= 21 + 2
    for other in many:
        other.close()
    assert lib.bpdq_hybrid_recordings(m.plan) == 8
    f.slots.release(held[0][1])
    again = Engine(m, slots=7)          # (at one of their addresses, or not)
    for x, y in zip([again.feed("x", toks[t:t + 1], [0]) for t in range(4)], [f.feed("x", toks[t:t + 1], [0]) for t in range(4)]):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])
    again.close()
    assert lib.bpdq_hybrid_recordings(m.plan) == 8 and lib.bpdq_last_status() == 0
    m.close()
    plain.close()
    f.close()               # (after its model)
