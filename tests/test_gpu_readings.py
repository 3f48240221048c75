"""GPU test of the roundoff reading at generous lengths, where the words are
small and so are their roundoff errors."""
import pytest

import cudalucas_b200 as cl

pytestmark = pytest.mark.gpu


# cluster, 16 elements per thread, short rows (longer lengths need more bits per
# word for their carries, and words of 2^20 and more have no places below 2^-32)
@pytest.mark.parametrize("n,bits,kernels", [(8192, 6.8, 0), (12288, 7.0, 0), (12288, 7.0, cl.native.LL_KERNELS_NO_CLUSTER),
                                            (16384, 7.0, cl.native.LL_KERNELS_NO_CLUSTER)])
def test_small_roundoff_errors_are_read_to_their_last_places(n, bits, kernels):
    """The reading is the maximum of remainders that are multiples of the last
    place of small words, and is not rounded to multiples of 2^-32.  (The generic
    kernels are no measure here: their carries do not settle with 7 bits.)"""
    q = int(n * bits) | 1
    with cl.LLContext(q, n, tuning={"kernels": kernels}) as c:
        c.start(q // 3)
        c.step(60, errchk=True)
        e = [c.step(1, errchk=True) for _ in range(30)]
    assert 0 < max(e) < 1e-6
    assert any(x * 2**32 % 1 for x in e), e
