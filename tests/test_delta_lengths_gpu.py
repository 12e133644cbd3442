"""Keys and queries of a gated delta rule whose square lengths leave fp32: a prompt's chunks, whatever kernel takes them, scale such tokens to zeros, as the walk token
by token does.  Beside them ordinary tokens, and short ones whose squares are far below the lengths' epsilon.  Outputs and state against the walk over the same
tokens in portions that the chunked kernels do not take; both are fp32 sums of at most `T` terms of unit vectors (4e-5, as in the other delta rule tests, of
the state; bf16 outputs a rounding)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(lib, u, lg, beta, H, D, V, portions):
    state = torch.zeros(H, D, V, device="cuda")
    out = torch.full((u.shape[0], H, V), float("nan"), dtype=torch.bfloat16, device="cuda")
    at, ld = 0, u.shape[1]
    torch.cuda.synchronize()
    while at < u.shape[0]:
        n = min(portions, u.shape[0] - at)
        p = u.data_ptr() + 2 * at * ld
        assert lib.bpd_delta_rule_cuda(p, p + 2 * H * D, p + 4 * H * D, ld, lg.data_ptr() + 4 * at * H * D, beta.data_ptr() + 4 * at * H, D ** -0.5, 1e-6, state.data_ptr(),
                                       out.data_ptr() + 2 * at * H * V, None, None, 0.0, n, H, H, D, V, V, 1, None) == 0
        at += n
    torch.cuda.synchronize()
    return out.double().cpu(), state.double().cpu()


@pytest.mark.parametrize("T,H,D,V", [(40, 2, 32, 16), (70, 1, 128, 32), (100, 3, 256, 48)])
@pytest.mark.parametrize("longest", [1e10, 1e19, 1e37])
def test_lengths(lib, T, H, D, V, longest):
    rng = np.random.default_rng(T)
    k, q, v = (rng.standard_normal((T, H * n)) for n in (D, D, V))
    for t in (3, 5, 17, 33):      # (no token has both: their product, which the walk forms of the vectors as they are, stays in fp32's range)
        k[t] *= longest / 8
        q[t + 1] *= longest / 8
    k[7], q[9] = k[7] * 1e-25, q[9] * 1e-25
    k[20, 1::2] = 0.0
    u = torch.from_numpy(np.concatenate([q, k, v], 1).clip(-longest, longest).astype(np.float32)).to(torch.bfloat16).cuda()
    lg = -torch.from_numpy(rng.uniform(0, 0.5, (T, H, D)).astype(np.float32)).cuda()
    beta = torch.from_numpy(rng.uniform(0.1, 1, (T, H)).astype(np.float32)).cuda()
    (out, state), (want, want_state) = run(lib, u, lg, beta, H, D, V, T), run(lib, u, lg, beta, H, D, V, 16)
    assert torch.isfinite(want).all() and torch.isfinite(out).all()
    assert (state - want_state).abs().max() < 4e-5 * want_state.abs().max()
    assert (out - want).abs().max() < 2.0 ** -7 * want.abs().max()
