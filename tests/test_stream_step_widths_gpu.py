"""Residual streams at the widths where a thread has two groups of columns (1025 to 2048), for every number of streams the kernel is made for.  The
reference and the tolerances are those of the other stream tests."""
import pytest

from tests.test_vuzelix_gpu import test_stream_step as step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("T,S,W", [(3, 4, 1024), (3, 4, 1040), (2, 8, 2048), (40, 2, 1500), (2, 5, 2040), (2, 1, 2049)])
def test_widths(lib, bf16, T, S, W):
    step(lib, bf16, T, S, W)
