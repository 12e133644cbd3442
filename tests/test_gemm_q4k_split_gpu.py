"""The tcgen05 Q4_K product with K split over the CTAs of a cluster: ranges of unequal length, fewer tokens than ranges, and the
choice between the two tensor-core kernels, which no result may show."""
import numpy as np
import pytest

from bpd_substrate_b200 import synth
from tests.test_gemm_q4k_gpu import TOL, run
from tests.util import normwise

pytestmark = pytest.mark.gpu


# super-blocks per row that two, three, five and seven ranges do not divide; one token, tokens around each padding
@pytest.mark.parametrize("T,N,K", [(1, 128, 7 * 256), (3, 200, 11 * 256), (5, 128, 56 * 256), (17, 384, 13 * 256), (31, 128, 17 * 256),
                                   (64, 130, 23 * 256), (50, 640, 9 * 256)])
def test_uneven_ranges(lib, oracle, T, N, K):
    rng = np.random.default_rng(T + N + K)
    W, X = synth.q4k_matrix(N, K, rng), synth.activations(K, rng, rows=T)
    _, ref64 = oracle.qmm_q4k_q8k(W, X, T, N, K)
    assert normwise(run(lib, "tc5", W, X, T, N, K), ref64) <= TOL


# tokens, rows, columns, kernel on 148 SMs (0 passes over the weights, 1 mma.sync, 2 tcgen05): few tokens of small, long, many and very many
# rows; more tokens of long rows and of more row tiles than SMs; a remainder behind a pass of 64
@pytest.mark.parametrize("T,N,K,kernel", [(1, 20000, 1024, 0), (2, 14336, 4096, 0), (2, 14336, 1024, 1), (3, 4096, 2048, 0), (3, 14336, 4096, 1), (4, 1024, 4096, 2),
                                          (4, 4096, 2048, 1), (8, 500, 14336, 2), (16, 57344, 1024, 1), (64, 57344, 1024, 2), (16, 4096, 4096, 2), (65, 4096, 1024, 1),
                                          (64, 100, 4096, 1)])
def test_kernel_of_a_call(lib, T, N, K, kernel):
    if lib.bpdq_sm_count() != 148:
        pytest.skip("the lines are those of 148 SMs")
    assert lib.bpdq_qmm_q4k_q8k_kernel(T, N, K) == kernel


# both sides of the dispatcher's lines: 2 to 4 tokens, short and long rows, few and many of them
@pytest.mark.parametrize("T,N,K", [(3, 1024, 4352), (4, 1024, 4096), (4, 1024, 4352), (2, 14336, 512), (9, 512, 8192), (16, 8192, 512), (33, 260, 2048), (70, 300, 1024)])
def test_dispatcher(lib, oracle, T, N, K):
    rng = np.random.default_rng(T * N + K)
    W, X = synth.q4k_matrix(N, K, rng), synth.activations(K, rng, rows=T)
    _, ref64 = oracle.qmm_q4k_q8k(W, X, T, N, K)
    assert normwise(run(lib, "dispatch", W, X, T, N, K), ref64) <= TOL


# more row tiles than clusters of two run at once: one range each, in two waves
@pytest.mark.parametrize("T", [16, 40])
def test_more_tiles_than_sms(lib, oracle, T):
    N, K = 149 * 128 - 5, 1024
    rng = np.random.default_rng(T)
    W, X = synth.q4k_matrix(N, K, rng), synth.activations(K, rng, rows=T)
    _, ref64 = oracle.qmm_q4k_q8k(W, X, T, N, K)
    assert normwise(run(lib, "tc5", W, X, T, N, K), ref64) <= TOL
