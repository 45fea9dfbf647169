"""The FP32 transforms where a CTA's lines fill an SM (sizes above 7140 or so: two
columns and 512 threads a CTA), each first radix and odd stages among them, and the
last sizes below (the bound of tests/test_gpu_fft_sizes.py)."""
import pytest

from tests.test_gpu_fft_sizes import test_transforms_match_fp64 as _match

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7056, 7168, 7290, 7500, 7776, 8000, 8064])
def test_large_sizes(n):
    _match(n, n % 7 == 0)
