"""GPU tests of the launches that a batch chooses for its members: as alone
while the batch is small, 16 elements per thread when it fills the GPU, launch
preferences at long lengths, members with persistent passes in turn."""
import ctypes

import pytest

import cudalucas_b200 as cl
from cudalucas_b200 import native
from cudalucas_b200.workloads import next_prime

pytestmark = pytest.mark.gpu
K = 1024


def _qs(n, count):
    out = [next_prime(int(17.4 * n))]
    while len(out) < count:
        out.append(next_prime(out[-1] + 1))
    return out


def _shape(handle):
    c = cl.LLContext.__new__(cl.LLContext)
    c._h = ctypes.c_void_p(handle)
    s = c.shape
    c._h = ctypes.c_void_p()  # the batch owns it
    return s


def _members(b):
    return [_shape(native.lib().ll_batch_member(b._h, i)) for i in range(len(b))]


def _solo(q, n, off, k):
    with cl.LLContext(q, n) as c:
        c.start(off)
        c.step(k, report=True)
        return c.res64(), c.shape


# on both sides of 1700K words in all; a preference with 16-element rows (640K),
# with short (160K) and with alternative ones (1152K); none (50K)
@pytest.mark.parametrize("nk,count,as_alone", [(640, 1, True), (640, 3, True), (160, 10, True), (160, 11, False),
                                               (50, 34, True), (50, 35, False), (1152, 1, True), (1152, 2, False),
                                               (896, 2, True), (1600, 1, True), (14336, 1, True)])
def test_launch_of_a_member(nk, count, as_alone):
    n = nk * K
    qs = _qs(n, count)
    want, alone = _solo(qs[0], n, qs[0] // 3, 23)
    with cl.LLBatch(qs, [n] * count, graph_iters=10) as b:
        shapes = _members(b)
        b.start([q // 3 for q in qs])
        b.step(23, report=True)  # two replays and three iterations after them
        got = b.res64()
    assert all((s["W"], s["threads_wide"]) == (shapes[0]["W"], shapes[0]["threads_wide"]) for s in shapes)
    assert ((shapes[0]["W"], shapes[0]["threads_wide"]) == (alone["W"], alone["threads_wide"])) == as_alone
    assert got[0] == want
    assert got[-1] == _solo(qs[-1], n, qs[-1] // 3, 23)[0]


@pytest.mark.parametrize("by_length", [True, False])
def test_members_with_persistent_passes_among_others(by_length):
    """Two members that run in turn, one longer one, a class of two and one of
    one length: graph replays, then the iterations after them."""
    ns = [3200 * K, 160 * K, 3200 * K, 3136 * K, 160 * K, 640 * K]
    qs = [next_prime(int(17.2 * n) + 1000 * i) for i, n in enumerate(ns)]
    offs = [(q * 5) // 9 for q in qs]
    with cl.LLBatch(qs, ns, graph_iters=8, by_length=by_length) as b:
        m = _members(b)
        assert [s["wide_persistent"] or s["tall_persistent"] for s in m] == [True, False, True, True, False, False]
        b.start(offs)
        b.step(16)
        b.step(29, report=True)
        got = b.res64()
        b.step(3)
        b.step(8, report=True)
        again = b.res64()
    for q, n, o, r, r2 in zip(qs, ns, offs, got, again):
        assert r == _solo(q, n, o, 45)[0], q
        assert r2 == _solo(q, n, o, 56)[0], q
