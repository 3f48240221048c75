"""CPU test of the choice of row kernels, through ll_context_bytes (a row kernel
with few elements per thread has other tables and carry rows than one with
16): a flag that is not about rows leaves them as they are."""
import ctypes

import pytest

from cudalucas_b200 import native
from cudalucas_b200.fftbench import exponent_for

K = 1024


def _bytes(n, **tuning):
    t = native.Tuning()
    for k, v in tuning.items():
        setattr(t, k, v)
    return native.lib().ll_context_bytes(exponent_for(n), n, ctypes.byref(t))


@pytest.mark.parametrize("nk,width", [(10, 256), (50, 256), (60, 256), (160, 256), (392, 256), (128, 512), (320, 512),
                                      (800, 512)])
@pytest.mark.parametrize("flag", [native.LL_KERNELS_NO_PREFETCH, native.LL_KERNELS_CLUSTER8, native.LL_KERNELS_NO_CLUSTER,
                                  native.LL_KERNELS_FUSED, native.LL_KERNELS_NO_PIPE])
def test_flags_that_are_not_about_rows_keep_the_short_rows(nk, width, flag):
    n = nk * K
    assert _bytes(n, width=width, kernels=flag) == _bytes(n, width=width)
    assert _bytes(n, width=width, kernels=flag | native.LL_KERNELS_LONG_ROWS) != _bytes(n, width=width)


@pytest.mark.parametrize("nk", [12, 14, 56])
def test_two_launches_in_place_of_the_fused_kernel_have_its_rows(nk):
    n = nk * K
    long_rows = _bytes(n, kernels=native.LL_KERNELS_LONG_ROWS)
    assert long_rows != _bytes(n)
    assert _bytes(n, kernels=native.LL_KERNELS_NO_CLUSTER) == _bytes(n, kernels=native.LL_KERNELS_FUSED) == long_rows


@pytest.mark.parametrize("nk,width", [(512, 256), (1024, 512), (1024, 1024)])
def test_many_rows_or_longer_ones_have_16_elements(nk, width):
    n = nk * K
    assert _bytes(n, width=width, kernels=native.LL_KERNELS_LONG_ROWS) == _bytes(n, width=width)
