"""GPU test of the steps of few iterations that 32K to 56K run as one cluster
launch, between steps of more that run as two launches per iteration."""
import numpy as np
import pytest

import cudalucas_b200 as cl
from cudalucas_b200.fftbench import exponent_for
from oracle.binding import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk", [32, 36, 42, 48, 56])
def test_few_iterations_in_one_launch_equal_two_launches(nk):
    """Steps of 1 to 7 iterations run in the cluster: the hand-off's parity, the
    place of the -2 and the carry rows are used again by the second iteration.
    From 8 on a step is two launches per iteration.  After every step the digits
    are those of a context without the cluster; the residue at the end is the
    oracle's."""
    n = nk * 1024
    q = exponent_for(n)
    off = q // 3
    steps = [2, 8, 3, 7, 9, 1, 5, 64, 7, 7, 6, 130, 4]
    with cl.LLContext(q, n) as c, cl.LLContext(q, n, tuning={"kernels": cl.native.LL_KERNELS_NO_CLUSTER}) as d:
        assert c.shape["cluster"] and not d.shape["cluster"]
        c.start(off)
        d.start(off)
        for k in steps:
            e, f = c.step(k, report=True), d.step(k, report=True)
            assert e < 0.4 and e <= 2 * f + 1e-3 and f <= 2 * e + 1e-3, (k, e, f)
            x, xo = c.read_digits()
            y, yo = d.read_digits()
            assert xo == yo and np.array_equal(x, y), k
        # steps without a report in between: the state alone is handed on
        for k in (3, 8, 7, 2):
            c.step(k)
            d.step(k)
        assert c.step(7, report=True) < 0.4
        d.step(7, report=True)
        x, xo = c.read_digits()
        y, yo = d.read_digits()
        assert xo == yo and np.array_equal(x, y)
        got = c.res64()
    o = Oracle(q, n)
    o.start(off)
    o.step(sum(steps) + 27)
    assert got == o.res64()
