"""GPU tests of bounded waits that run out.  The limit of the waits inside a
pass is set so low that a wait not satisfied at its first look has expired; the
kernels then finish early, the call returns LL_ERR_TIMEOUT and the GPU stays
usable."""
import numpy as np
import pytest

import cudalucas_b200 as cl
from cudalucas_b200 import native
from cudalucas_b200.fftbench import exponent_for

pytestmark = pytest.mark.gpu

# persistent row pass alone (4 and 1 groups of threads), both passes (3 groups;
# one group with two slots; one group with one slot)
PIPE = [(1024, 1568), (4096, 392), (1280, 1280), (3072, 1536), (4096, 4096)]


def _expire(c):
    """Steps until a wait has run out (at the latest within a few iterations:
    some CTA looks for its predecessor's carries before they are there)."""
    c.wait_limit(-1)
    with pytest.raises(cl.LLError) as e:
        for _ in range(50):
            c.step(3, errchk=True)
    assert e.value.status == native.LL_ERR_TIMEOUT
    c.wait_limit(0)


def _res64(W, H, k):
    n = 2 * W * H
    q = exponent_for(n)
    with cl.LLContext(q, n, tuning={"width": W}) as c:
        c.start(q // 3)
        c.step(k, report=True)
        return c.res64()


@pytest.mark.parametrize("W,H", PIPE)
def test_expired_wait_is_reported_and_leaves_the_gpu_usable(W, H):
    n = 2 * W * H
    q = exponent_for(n)
    want = _res64(W, H, 70)
    with cl.LLContext(q, n, tuning={"width": W}) as c:
        c.start(q // 3)
        _expire(c)
        # the fault stays until the state is loaded again
        with pytest.raises(cl.LLError):
            c.step(1, errchk=True)
    assert _res64(W, H, 70) == want


# rows of 4, 8 and 16 elements per thread beside the persistent passes, the
# generic kernels' neighbours in one context's life
@pytest.mark.parametrize("W,H", PIPE + [(256, 320), (512, 720), (512, 1024), (1024, 1024), (2048, 1024)])
def test_digits_loaded_after_an_expired_wait_give_the_right_residue(W, H):
    """Carries and flags that came after the wait had run out are gone when
    digits are loaded (from the host, or from the device checkpoint)."""
    n = 2 * W * H
    q = exponent_for(n)
    want = _res64(W, H, 70)
    with cl.LLContext(q, n, tuning={"width": W}) as c:
        for _ in range(3):
            c.start(q // 3)
            _expire(c)
            c.start(q // 3)
            assert c.step(70, report=True) < 0.4
            assert c.res64() == want
        c.start(q // 3)
        c.device_checkpoint()
        _expire(c)
        c.device_restore()
        assert c.step(70, report=True) < 0.4
        assert c.res64() == want
