"""Attention of the Q8_0 Llama over more than a few keys, through the C ABI, against 64-bit sums.

Bound: 1e-5 of the largest output.  A score adds up to 16 truncated tensor-core sums, each within 2^-23 of sum |q_d k_d| scale (about 7 for
these inputs): the worst score is off by 1.3e-5, and with it its key's weight.  A row's output is off by that times sum w |v - out|, which is
at most 0.8 for values of unit variance (one key that holds all the weight has none of it), against a largest output of 3 to 4: below 4e-6 of it."""
import numpy as np
import pytest

from tests.util import Dev


def expected(q, k, v, off, scale, n_kv):
    """Scores, softmax and sums in binary64; query t sees keys 0 .. off + t."""
    T, H, D = q.shape
    rep = H // k.shape[1]
    q, k, v = q.astype(np.float64), k.astype(np.float64), v.astype(np.float64)
    out = np.empty((T, H, D))
    for h in range(H):
        s = q[:, h] @ k[:, h // rep].T * scale
        s[np.arange(len(k))[None] >= np.minimum(off + 1 + np.arange(T), n_kv)[:, None]] = -np.inf
        e = np.exp(s - s.max(axis=1, keepdims=True))
        out[:, h] = (e / e.sum(axis=1, keepdims=True)) @ v[:, h // rep]
    return out


def attend(lib, q, k, v, off, scale, n_kv):
    T, H, D = q.shape
    d = [Dev(lib, a) for a in (q, k, v)]
    out = Dev(lib, nbytes=q.nbytes + 64, fill=0xFF)
    assert lib.bpd_gqa_attn_cuda(d[0].ptr, d[1].ptr, d[2].ptr, out.ptr, T, n_kv, H, k.shape[1], D, scale, off, int(k.dtype == np.float16), None) == 0
    lib.bpdq_sync()
    assert lib.bpdq_last_status() == 0
    raw = out.read(np.uint8)
    assert (raw[q.nbytes:] == 0xFF).all()
    return raw[:q.nbytes].view(np.float32).reshape(q.shape)


def inputs(T, S, H, HKV, D, kind, seed):
    rng = np.random.default_rng(seed)
    return (1.5 * rng.standard_normal((T, H, D), dtype=np.float32), rng.standard_normal((S, HKV, D), dtype=np.float32).astype(kind),
            rng.standard_normal((S, HKV, D), dtype=np.float32).astype(kind))


# queries, keys before them, heads, key heads, head size: contexts just beyond the short ones, at and around a block of 64 keys and
# a cluster's stretches; one query and as many as a tile needs; heads per key head from 1 to 8, groups with heads left over
SHAPES = [(1, 64, 8, 2, 64), (1, 127, 4, 4, 128), (1, 128, 6, 2, 128), (1, 1100, 8, 1, 128), (2, 700, 10, 2, 64), (3, 64, 4, 2, 64),
          (65, 0, 32, 8, 128), (128, 0, 32, 32, 64), (129, 63, 24, 8, 128), (200, 1, 16, 2, 64), (700, 3, 8, 4, 64), (130, 500, 10, 2, 128)]


@pytest.mark.gpu
@pytest.mark.parametrize("T,off,H,HKV,D", SHAPES)
@pytest.mark.parametrize("kind", [np.float16, np.float32])
def test_attention_against_64_bits(lib, T, off, H, HKV, D, kind):
    q, k, v = inputs(T, off + T, H, HKV, D, kind, T + off)
    q[0] *= 40.0                       # one row with a peaked softmax, one of zeros (all weights equal)
    q[-1, 0] = 0.0
    scale = np.float32(D ** -0.5)
    got, want = attend(lib, q, k, v, off, scale, off + T), expected(q, k, v, off, float(scale), off + T)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.gpu
def test_attention_never_reads_beyond_the_keys_that_count(lib):
    """n_kv below the last query's position caps what it sees; rows behind are poison."""
    q, k, v = inputs(100, 200, 8, 2, 128, np.float16, 1)
    k[150:], v[150:] = np.nan, np.nan
    got, want = attend(lib, q, k, v, 90, 0.1, 150), expected(q, k[:150], v[:150], 90, 0.1, 150)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.gpu
def test_values_that_are_not_finite_reach_only_the_queries_that_see_them(lib):
    """A prompt whose token 70 has an infinite value and token 90 a NaN key: earlier queries are as before, others carry it."""
    T = 128
    q, k, v = inputs(T, T, 32, 8, 128, np.float16, 2)
    want = expected(q, k, v, 0, 0.1, T)
    v[70, 3, 5], k[90, 1, 7] = np.inf, np.nan
    got = attend(lib, q, k, v, 0, 0.1, T)
    clean = np.ones(got.shape, bool)
    clean[70:, 12:16, 5] = False
    clean[90:, 4:8] = False
    assert np.abs(got - want)[clean].max() <= 1e-5 * np.abs(want).max()
    assert np.isposinf(got[70:, 12:16, 5]).all() and np.isnan(got[90:, 4:8]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("kind,T", [(np.float32, 1), (np.float16, 128)])
def test_softmax_weights(lib, kind, T):
    """Weights one by one, against binary64: scores 0, -1, -2, ... and fractions between them down to where a weight is no normal number any more;
    key i's value is one in column i and zero elsewhere, so that output i is its weight.  A weight is a rounded argument reduction (the score's last
    bits), a polynomial (5e-9), a sum of 127 weights and a division, each a few 2^-24: 5e-7 of it.  The tiles hold a weight times 2^10 as two fp16
    numbers, the low one a multiple of 2^-24: off by up to 2^-35 = 3e-11."""
    D, keys, H, HKV = 128, 128, 32, 8
    rng = np.random.default_rng(3)
    want_s = -np.concatenate([[0.0], np.linspace(0.5, 100.0, 67), rng.uniform(0.0, 12.0, 60)])
    k = np.zeros((keys, HKV, D), kind)
    k[:, :, 0] = want_s[:, None]                                    # (fp16: the nearest number is the score)
    scores = k[:, 0, 0].astype(np.float64)
    v = np.repeat(np.eye(keys, D, dtype=kind)[:, None], HKV, 1)
    q = np.zeros((T, H, D), np.float32)
    q[:, :, 0] = 1.0
    off = keys - T
    assert lib.bpdq_gqa_attn_kernel(T, keys, H, HKV, D, off, int(kind == np.float16)) == (2 if T > 1 else 1)
    got = attend(lib, q, k, v, off, np.float32(1.0), keys)[-1]      # the last query sees every key
    e = np.exp(scores)
    want = e / e.sum()
    assert np.array_equal(got, np.broadcast_to(got[0], got.shape))
    small = 3e-11 if T > 1 else 1e-37
    assert np.all(np.abs(got[0].astype(np.float64) - want) <= 5e-7 * want + small)


# queries, keys before them, heads, key heads, head size, fp16: kernel (0 a CTA per query and head, 1 keys over a cluster, 2 tiles)
@pytest.mark.parametrize("T,off,H,HKV,D,f16,kernel", [
    (1, 63, 32, 8, 128, 1, 0), (1, 64, 32, 8, 128, 1, 1), (300, 0, 32, 8, 128, 1, 2), (300, 0, 32, 8, 128, 0, 1), (300, 0, 32, 8, 96, 1, 0),
    # fp32 heads of 64 that share nothing: short prompts, those a few keys further on, long ones
    (65, 0, 16, 16, 64, 0, 0), (65, 10, 16, 16, 64, 0, 1), (100, 0, 32, 32, 64, 0, 0), (65, 30, 32, 32, 64, 0, 1), (210, 0, 32, 32, 64, 0, 1),
    (128, 0, 32, 16, 64, 0, 1)])
def test_kernel_of_a_call(T, off, H, HKV, D, f16, kernel):
    """On 148 SMs, which are assumed where there is no device."""
    from bpd_substrate_b200 import capi
    assert capi.load().bpdq_gqa_attn_kernel(T, off + T, H, HKV, D, off, f16) == kernel


@pytest.mark.gpu
@pytest.mark.parametrize("T,off", [(65, 0), (65, 10), (100, 0)])
def test_short_prompts_of_unshared_fp32_heads(lib, T, off):
    """Both kernels that such prompts take."""
    q, k, v = inputs(T, off + T, 16, 16, 64, np.float32, T)
    got, want = attend(lib, q, k, v, off, np.float32(0.125), off + T), expected(q, k, v, off, 0.125, off + T)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


# clusters of 8 and 16 CTAs: results joined by all warps (up to 32 per CTA) and by a thread each
@pytest.mark.gpu
@pytest.mark.parametrize("T,off,H,HKV,D", [(1, 300, 4, 4, 64), (1, 511, 8, 4, 128), (1, 400, 8, 2, 64), (2, 300, 6, 2, 64), (1, 300, 8, 2, 128), (1, 513, 4, 4, 64), (1, 1500, 3, 1, 128), (1, 4000, 32, 8, 128),
                                           (3, 600, 4, 2, 64)])
@pytest.mark.parametrize("kind", [np.float16, np.float32])
def test_joined_parts(lib, T, off, H, HKV, D, kind):
    """Parts of a cluster whose maxima lie far apart, in one CTA's stretch, in every CTA's, and nowhere."""
    q, k, v = inputs(T, off + T, H, HKV, D, kind, off)
    scale = np.float32(D ** -0.5)
    q[:, 0] = 0.0                                  # all keys alike
    q[:, 1] *= 30.0                                # one key, somewhere
    k[off // 3] = 4 * k[off // 3]                  # and one that many look at
    got, want = attend(lib, q, k, v, off, scale, off + T), expected(q, k, v, off, float(scale), off + T)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
