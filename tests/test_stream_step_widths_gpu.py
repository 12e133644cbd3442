"""Residual streams around the sizes where a thread has two groups of columns (three and four streams of 1537 to 2048 columns, 500 to 2000 tokens).  The
reference and the tolerances are those of the other stream tests."""
import pytest

from tests.test_vuzelix_gpu import test_stream_step as step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("T,S,W", [(3, 4, 1024), (3, 4, 1040), (2, 8, 2048), (40, 2, 1500), (2, 5, 2040), (2, 1, 2049)])
def test_widths(lib, bf16, T, S, W):
    step(lib, bf16, T, S, W)


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("T,S,W", [(500, 4, 2048), (501, 3, 1540), (499, 4, 1552), (500, 3, 1536), (500, 4, 2052), (500, 2, 1600), (500, 5, 1600), (2000, 3, 1552), (2001, 4, 1552)])
def test_two_groups(lib, bf16, T, S, W):
    step(lib, bf16, T, S, W)
