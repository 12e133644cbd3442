"""The gated norm and the causal convolution at the edges of their load widths: parts around a warp's and a CTA's channels, few and many parts, channels
that are multiples of eight, four, two and none, tiles of tokens with remainders, pointers that only the narrower loads can take.  References in
fp64; a bf16 result is a rounding (to eight bits: 2^-8 of a value at most) of fp32 arithmetic, whose fast sigmoid and sums stay within 1e-5."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def sigmoid(z):
    return 1.0 / (1.0 + torch.exp(-z))


def acts(rng, rows, ld, dtype, offset):
    """rows x ld values, `offset` elements into an allocation."""
    flat = torch.from_numpy(rng.standard_normal(offset + rows * ld).astype(np.float32)).to(dtype).cuda()
    return flat[offset:].view(rows, ld)


def close(got, want, dtype):
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    got, scale = got.double(), want.abs().max()
    assert torch.isfinite(got).all()
    assert ((got - want).abs() <= want.abs() * (tol + 1e-5) + 1e-6 * scale).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,parts,part,offset", [
    (70, 1, 8, 0), (9, 8, 128, 0), (70, 1, 256, 0), (33, 2, 264, 0), (33, 2, 512, 0), (33, 2, 520, 0), (65, 1, 1024, 0), (65, 1, 1032, 0), (65, 1, 2056, 0),
    (65, 1, 4096, 0), (65, 1, 4104, 0), (65, 1, 8192, 0), (65, 1, 8200, 0), (66, 1, 516, 0), (66, 1, 512, 4), (66, 1, 4096, 4), (66, 3, 65, 0), (1, 8, 512, 0), (2, 1, 4096, 0)])
@pytest.mark.parametrize("form", [0, 1, 2])
def test_gated_norm(lib, dtype, T, parts, part, offset, form):
    n, rng = parts * part, np.random.default_rng(T + part)
    extra = 8 if part % 8 == 0 else 4 if part % 4 == 0 else 1
    o, g = acts(rng, T, n + extra, dtype, offset), acts(rng, T, 2 * n, dtype, offset)
    w = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    y = torch.full((offset + T * n,), float("nan"), dtype=dtype, device="cuda")[offset:].view(T, n)
    torch.cuda.synchronize()
    assert lib.bpd_gated_norm_cuda(o.data_ptr(), n + extra, g.data_ptr(), 2 * n, w.data_ptr() if form else None, y.data_ptr(), n, T, parts, part, part,
                                   parts, form, 1e-5, int(dtype == torch.bfloat16), None) == 0
    torch.cuda.synchronize()
    v, z = o[:, :n].double(), g[:, :n].double()
    gate = sigmoid(z) if form == 2 else z * sigmoid(z)
    if form == 1:
        v = v * gate
    r = v.view(T, parts, part)
    r = (r / torch.sqrt((r * r).mean(-1, keepdim=True) + 1e-5)).view(T, n)
    if form:
        r = r * w.double()
    close(y, r if form == 1 else r * gate, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,channels,taps,offset", [(1, 8, 4, 0), (7, 512, 4, 0), (8, 516, 3, 0), (9, 514, 4, 0), (17, 101, 2, 0), (64, 1028, 4, 0), (40, 520, 6, 0),
                                                    (23, 512, 4, 2), (23, 512, 4, 1), (15, 512, 1, 0)])
def test_causal_conv(lib, dtype, T, channels, taps, offset):
    rng = np.random.default_rng(T + channels)
    ld = channels + (8 if channels % 8 == 0 else 4 if channels % 4 == 0 else 2 if channels % 2 == 0 else 1)
    x = acts(rng, T, ld, dtype, offset)
    w, b, tail = (torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda() for s in ((taps, channels), channels, (max(taps - 1, 1), channels)))
    old, y = tail.clone(), torch.full((offset + T * channels,), float("nan"), dtype=dtype, device="cuda")[offset:].view(T, channels)
    torch.cuda.synchronize()
    assert lib.bpd_causal_conv_silu_cuda(x.data_ptr(), ld, y.data_ptr(), T, channels, taps, w.data_ptr(), b.data_ptr(), tail.data_ptr(),
                                         int(dtype == torch.bfloat16), None) == 0
    torch.cuda.synchronize()
    seen = torch.cat([old[:taps - 1].double(), x[:, :channels].double()])
    a = b.double() + sum(w[j].double() * seen[j:j + T] for j in range(taps))
    close(y, a * sigmoid(a), dtype)
    if taps > 1:
        assert torch.equal(tail.double(), seen[T:])


# tiles of 16 and 24 tokens with whole and ragged last ones, every load width; more tiles than a grid's second dimension takes; windows longer than a tile
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,channels,taps,offset", [(19001, 512, 4, 0), (19007, 130, 3, 0), (19016, 101, 2, 0), (48000, 64, 4, 0), (50011, 34, 4, 0), (50017, 33, 4, 0),
                                                    (524296, 8, 4, 0), (524289, 3, 2, 0), (30, 12, 19, 0), (3, 8, 12, 0)])
def test_causal_conv_tiles(lib, dtype, T, channels, taps, offset):
    test_causal_conv(lib, dtype, T, channels, taps, offset)


# parts at the edges of every number of warps and loads, in channels that only loads of four take and on pointers that only they take
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,parts,part,offset", [(70, 1, 4, 0), (33, 2, 100, 0), (33, 2, 128, 4), (33, 2, 132, 0), (33, 2, 136, 0), (33, 2, 252, 0), (65, 1, 256, 4), (65, 1, 260, 0),
                                                 (65, 1, 508, 0), (65, 1, 1020, 0), (65, 1, 1028, 0), (65, 1, 2044, 0), (65, 1, 2048, 4), (65, 1, 2052, 0), (65, 1, 4092, 0),
                                                 (65, 1, 4100, 0), (65, 1, 8188, 0), (65, 1, 8192, 4), (1, 8, 2048, 0), (2, 1, 2052, 0), (64, 1, 8192, 0)])
def test_gated_norm_narrow_loads(lib, dtype, T, parts, part, offset):
    for form in (0, 1, 2):
        test_gated_norm(lib, dtype, T, parts, part, offset, form)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,part,offset", [(70, 256, 1), (70, 512, 2), (3, 1024, 1), (65, 4096, 3)])
def test_gated_norm_anywhere(lib, dtype, T, part, offset):
    """Rows that begin where no load of several channels may."""
    for form in (0, 1, 2):
        test_gated_norm(lib, dtype, T, 1, part, offset, form)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,channels,taps,offset", [(23, 512, 4, 1), (9, 514, 4, 2), (23, 512, 6, 1), (40, 130, 3, 3)])
def test_causal_conv_floats_anywhere(lib, dtype, T, channels, taps, offset):
    """Weights, biases and window at any float."""
    rng = np.random.default_rng(T + channels)
    x = acts(rng, T, channels, dtype, 0)
    w, b, tail = (acts(rng, 1, n, torch.float32, offset).view(-1, channels) for n in (taps * channels, channels, (taps - 1) * channels))
    old, y = tail.clone(), torch.full((T, channels), float("nan"), dtype=dtype, device="cuda")
    torch.cuda.synchronize()
    assert lib.bpd_causal_conv_silu_cuda(x.data_ptr(), channels, y.data_ptr(), T, channels, taps, w.data_ptr(), b.data_ptr(), tail.data_ptr(),
                                         int(dtype == torch.bfloat16), None) == 0
    torch.cuda.synchronize()
    seen = torch.cat([old.double(), x.double()])
    a = b.double() + sum(w[j].double() * seen[j:j + T] for j in range(taps))
    close(y, a * sigmoid(a), dtype)
    assert torch.equal(tail.double(), seen[T:])
