"""GPU test of contexts made and released in numbers and from several threads:
they share pages of pinned memory for the read-back of their state."""
import threading

import pytest

import cudalucas_b200 as cl
from oracle import exact

pytestmark = pytest.mark.gpu


def test_many_contexts_read_back_their_own_state():
    """More contexts than a page holds; every second one released and made
    again, so that slots and pages are reused."""
    q, n = 86243, 4096
    made = [cl.LLContext(q, n) for _ in range(130)]
    for i, c in enumerate(made):
        c.start(i)
    for c in made[::2]:
        c.close()
    made = made[1::2] + [cl.LLContext(q, n) for _ in range(65)]
    for i, c in enumerate(made):
        c.start(i)
    errs = [c.step(20 + i % 7, report=True) for i, c in enumerate(made)]
    assert all(0 < e < 0.4 for e in errs)
    want = {k: exact.res64(q, k) for k in range(20, 27)}
    for i, c in enumerate(made):
        assert c.res64() == want[20 + i % 7]
        c.close()


def test_contexts_of_several_threads():
    q, n = 216091, 12288
    want = exact.res64(q, 150)
    got, failed = [], []

    def work(k):
        try:
            for r in range(6):
                with cl.LLContext(q, n) as c:
                    c.start(1000 * k + r)
                    assert c.step(150, report=True) < 0.4
                    got.append(c.res64())
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and got == [want] * 36
