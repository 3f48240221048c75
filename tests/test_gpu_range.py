"""GPU test of words beyond the exact FP64 range in every kind of row kernel: the
step reports the largest possible error, at once and after infinities and NaN
have gone through the carries, and never a wait that ran out."""
import numpy as np
import pytest

import cudalucas_b200 as cl
from cudalucas_b200.fftbench import exponent_for

pytestmark = pytest.mark.gpu

NO_PIPE = cl.native.LL_KERNELS_NO_PIPE


# cluster; rows of 4, 8 and 16 elements per thread; persistent rows and columns
# in three shapes; the last without them
@pytest.mark.parametrize("W,H,kernels", [(256, 24, 0), (256, 320, 0), (512, 320, 0), (512, 1024, 0), (1024, 1024, 0),
                                         (1024, 1568, 0), (1280, 1280, 0), (3072, 1536, 0), (4096, 4096, 0),
                                         (1280, 1280, NO_PIPE)])
def test_words_beyond_the_exact_range_report_the_largest_error(W, H, kernels):
    n = 2 * W * H
    q = exponent_for(n)
    rng = np.random.default_rng(n)
    with cl.LLContext(q, n, tuning={"width": W, "kernels": kernels}) as c:
        for digits in (np.full(n, 1 << 29, dtype=np.int32),
                       rng.integers(-(1 << 31), 1 << 31, n, dtype=np.int64).astype(np.int32)):
            for k in (1, 2, 12, 70):
                c.load_digits(digits, 5)
                assert c.step(k, errchk=True) == 1.0, k
                c.load_digits(digits, 5)
                assert c.step(k, report=True) == 1.0, k
        c.start(7)
        assert c.step(20, report=True) < 0.4
        got = c.res64()
    with cl.LLContext(q, n, tuning={"width": W, "kernels": kernels}) as c:
        c.start(7)
        c.step(20, report=True)
        assert got == c.res64()
