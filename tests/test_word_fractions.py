"""The specialised row kernels compare weight exponents as 32-bit fractions of
a turn (WordSize in kernels_static.cuh).  Every comparison has to agree with
the integer rule: word size big iff (E - D) mod n < b, wrapped iff E < D."""
import numpy as np
import pytest

from cudalucas_b200 import engine

LENGTHS = [n for n in engine.fft_table() if n <= 1 << 25]


@pytest.mark.parametrize("n", [64, 1000 * 4, *LENGTHS[::9], 1 << 25])
@pytest.mark.parametrize("bits", [1.01, 17.6, 18.37])
def test_fractions_agree_with_integers(n, bits):
    q = int(n * bits) | 1
    b = q % n
    rng = np.random.default_rng(n)
    E = np.concatenate([rng.integers(0, n, 4000), [0, 1, n - 1, b, (b - 1) % n, (b + 1) % n] * 60])
    D = np.concatenate([rng.integers(0, n, 4000), np.repeat([0, 1, n - 1, b, (b - 1) % n, n // 2], 60)])
    D[:1000] = (E[:1000] - b) % n        # on the limit
    D[1000:2000] = (E[1000:2000] - b + 1) % n  # one step below it
    D[2000:3000] = E[2000:3000]          # equal exponents: no wrap
    turn = 2.0 ** 32 / n
    lim = np.uint32(b * turn)
    F = (E * turn + 0.5 * turn).astype(np.uint64).astype(np.uint32)
    Df = (D * turn).astype(np.uint64).astype(np.uint32)
    f = F - Df  # wraps in 32 bits
    np.testing.assert_array_equal(f < lim, (E - D) % n < b)
    np.testing.assert_array_equal(F < Df, E < D)
