"""The order in which the persistent row pass works on its units (tickets in
kernels_pipe.cuh): every unit once, a unit's predecessor at an earlier ticket
(else CTAs could wait for one that has not been drawn), the extra tickets
before the units that take their carries and before the units they read."""
import pytest


def unit(k, chains, length, units):
    i, j = divmod(k, chains)
    first = j * length
    if first >= units:
        return -1
    if i == 0:
        return (units if j == 0 else first) - 1
    return first + i - 1 if first + i - 1 < units else -1


@pytest.mark.parametrize("slots", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("units", [196, 224, 256, 392, 400, 640, 784, 896, 1152, 1536, 1701, 2048, 2187])
def test_ticket_order(slots, units):
    chains = slots * max(1, min(32 // slots, units // (4 * slots)))
    length = -(-units // chains)
    assert chains % slots == 0 and chains <= 64  # a flag per run
    ticket = {}
    extra = {}
    for k in range(chains * (length + 1)):
        u = unit(k, chains, length, units)
        if u < 0:
            continue
        if k < chains:
            extra[k] = (k, u)
        else:
            assert u not in ticket
            ticket[u] = k
    assert sorted(ticket) == list(range(units))
    for u, k in ticket.items():
        pred = units - 1 if u == 0 else u - 1
        if u % length == 0:  # the first of a run takes its carries from the run's extra ticket
            ek, eu = extra[u // length]
            assert eu == pred and ek < k
        else:
            assert ticket[pred] == k - chains
    for run, (k, u) in extra.items():  # the unit an extra ticket reads is drawn later
        assert k < ticket[u]
        assert u % length == length - 1 or u == units - 1
