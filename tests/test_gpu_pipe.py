"""GPU tests of the persistent passes and of the rows with few elements per
thread, at the edges of what they accept: every row and column length they are
compiled for, odd numbers of units, the fewest and the most row groups.  The
digits are compared with the generic kernels' and the residue with the
oracle's."""
import numpy as np
import pytest

import cudalucas_b200 as cl
from cudalucas_b200.fftbench import exponent_for

pytestmark = pytest.mark.gpu

GENERIC, NO_CLUSTER = 1, 8


def _run(q, n, digits, offset, k, tuning):
    with cl.LLContext(q, n, tuning=tuning) as c:
        c.load_digits(digits, offset)
        err = c.step(k, report=True)
        d, o = c.read_digits()
        return d, o, err, c.shape


def _random_digits(q, n, seed):
    rng = np.random.default_rng(seed)
    packed = rng.integers(0, 1 << 32, (q + 31) // 32, dtype=np.uint32)
    packed[-1] &= np.uint32((1 << (q % 32)) - 1)
    return cl.balance_digits(cl.unpack_bits(packed, q, n), q, n), int(rng.integers(0, q))


def _compare(W, H, k):
    n = 2 * W * H
    q = exponent_for(n)
    digits, offset = _random_digits(q, n, W + H)
    d, o, err, shape = _run(q, n, digits, offset, k, {"width": W})
    assert shape["W"] == W and shape["wide_specialised"] and shape["tall_specialised"]
    g, go, gerr, _ = _run(q, n, digits, offset, k, {"width": W, "kernels": GENERIC, "rows_per_cta": 2 if W <= 2048 else 1})
    assert o == go == offset * pow(2, k, q) % q
    assert np.array_equal(cl.standardize(d, q, n)[0], cl.standardize(g, q, n)[0])
    # two arithmetics of the same accuracy: their largest roundoff of k
    # iterations agree within a factor of two, as everywhere in these tests
    assert err < 0.4 and err <= 2 * gerr + 1e-3 and gerr <= 2 * err + 1e-3, (err, gerr)


# rows 256*M and columns 256*M of the persistent passes; 130 iterations run two
# replays of the step graph and single launches after them
@pytest.mark.parametrize("W,H", [
    (1024, 1568), (1280, 1280), (1536, 1536), (2048, 800), (2304, 672), (2560, 1280), (3072, 576), (3584, 448),
    (4096, 392), (1024, 1792), (2048, 2048), (2304, 2304), (512, 2560), (512, 3072), (512, 3584), (512, 4096),
    (1536, 1620), (1792, 2688), (1024, 3402), (4096, 4096)])
def test_persistent_passes(W, H):
    _compare(W, H, 130)


# at most 400 groups of two rows: 16 to 800 rows; one group more runs 16
# elements per thread
@pytest.mark.parametrize("W,H", [(256, 100), (256, 128), (256, 784), (256, 800), (256, 1024), (512, 128), (512, 320),
                                 (512, 800), (512, 1024)])
def test_rows_with_few_elements(W, H):
    _compare(W, H, 70)


@pytest.mark.parametrize("W,H", [(768, 224), (768, 576), (1024, 192), (1024, 800), (1280, 576)])
def test_opt_in_rows(W, H):
    n = 2 * W * H
    q = exponent_for(n)
    digits, offset = _random_digits(q, n, W + H)
    a = _run(q, n, digits, offset, 70, {"width": W, "kernels": NO_CLUSTER})
    b = _run(q, n, digits, offset, 70, {"width": W, "kernels": NO_CLUSTER | 32})
    assert a[1] == b[1] and np.array_equal(a[0], b[0])
    assert b[2] < 0.4 and b[2] <= 2 * a[2] + 1e-3 and a[2] <= 2 * b[2] + 1e-3


NO_PIPE = 64
ROWS = {1024, 1280, 1536, 1792, 2048, 2304, 2560, 3072, 3584, 4096}


# both sides of the lines: 3000K and 9000K (rows of 1792) for rows, columns of
# 1280 and 2304K for columns; rows of 768 and columns of other lengths never
@pytest.mark.parametrize("W,H,rows,columns", [
    (1024, 1024, False, False), (1024, 1568, True, False), (2560, 576, False, False), (3072, 576, True, False),
    (1792, 1792, False, True), (1792, 2688, True, False), (768, 3072, False, True), (2048, 1024, True, False),
    (512, 2048, False, False), (512, 2304, False, True), (1280, 1280, True, True), (4096, 4096, True, True)])
def test_persistent_passes_run_where_the_rule_says(W, H, rows, columns):
    n = 2 * W * H
    q = exponent_for(n)
    with cl.LLContext(q, n, tuning={"width": W}) as c:
        assert (c.shape["wide_persistent"], c.shape["tall_persistent"]) == (rows, columns)
    with cl.LLContext(q, n, tuning={"width": W, "kernels": NO_PIPE}) as c:
        assert c.shape["W"] == W and not c.shape["wide_persistent"] and not c.shape["tall_persistent"]


@pytest.mark.parametrize("W,H", [(1024, 1568), (1280, 1280), (1536, 1536), (1792, 2688), (2048, 2048), (2304, 2304),
                                 (2560, 1280), (3072, 1536), (3584, 1792), (4096, 392), (512, 2304), (512, 3584)])
def test_persistent_passes_equal_a_launch_per_unit(W, H):
    """Same shape, same carry arithmetic: the digits are the same bit for bit;
    and the residue after a few iterations is the oracle's."""
    from oracle.binding import Oracle, set_threads
    n = 2 * W * H
    q = exponent_for(n)
    digits, offset = _random_digits(q, n, W + H)
    d, o, err, _ = _run(q, n, digits, offset, 130, {"width": W})
    g, go, gerr, _ = _run(q, n, digits, offset, 130, {"width": W, "kernels": NO_PIPE})
    assert o == go and np.array_equal(d, g)
    assert err <= 2 * gerr + 1e-3 and gerr <= 2 * err + 1e-3, (err, gerr)
    if n > 3 << 20:
        return
    with cl.LLContext(q, n, tuning={"width": W}) as c:
        c.start(q // 5)
        c.step(6)
        c.step(2, report=True)
        got = c.res64()
    set_threads(16)
    try:
        ref = Oracle(q, n)
        ref.start(q // 5)
        ref.step(8)
        assert got == ref.res64()
    finally:
        set_threads(1)


@pytest.mark.parametrize("W,H", [(2304, 2304), (3072, 2304), (3072, 3072), (1792, 2688), (4096, 2304), (1536, 1536),
                                 (3584, 3584)])
def test_persistent_passes_are_as_accurate_as_a_launch_per_unit(W, H):
    """Mean over 200 iterations of the largest roundoff, same digits on both
    sides.  A single maximum scatters by about 8 %, so the means by 0.6 % each:
    3 % is more than three times the scatter of their ratio."""
    n = 2 * W * H
    q = exponent_for(n)
    mean = []
    for kernels in (0, NO_PIPE):
        with cl.LLContext(q, n, tuning={"width": W, "kernels": kernels}) as c:
            assert c.shape["wide_persistent"] == (kernels == 0)
            c.start(q // 3)
            c.step(64, errchk=True)
            mean.append(sum(c.step(1, errchk=True) for _ in range(200)) / 200)
    assert mean[0] <= 1.03 * mean[1], mean
