"""The work that a user of the engine has it do, as measurable cases.

A solo case is one Lucas-Lehmer test taken up from a checkpoint: the digits go
host -> device (LLContext.load_digits), the iterations run in calls of `chunk`
iterations with the roundoff error read back after each (LLContext.step, as
the command-line tester does every ErrorIterations), and the digits and the
shift come back (LLContext.read_digits).  A batch case starts `count` tests of
different exponents and lengths and advances them together (LLBatch).

The lengths are those that the length policy picks for the exponent, or those
of the benchmark (12K, 3200K, 18432K)."""
import math

import numpy as np

from cudalucas_b200 import LLBatch, LLContext, engine, workloads

K = 1024
ERROR_LIMIT = 0.40  # the command-line tester's ErrorLimit
# drawn cases: words times iterations at most (the largest listed case has
# 3.9e9), and less where every iteration is a call of its own
MOST_WORDS, MOST_WORDS_SINGLE = 3.6e9, 6e8


def _solo(name, q, n, iters, chunk):
    return {"name": name, "kind": "solo", "q": q, "n": n, "iters": iters, "chunk": chunk}


def listed():
    return [
        # the smallest call: one iteration of a short test, e.g. a spot check
        _solo("12K_single", 216091, 12 * K, 1, 1),
        # the benchmark's short test, in the tester's error-check intervals
        _solo("12K", 216091, 12 * K, 5000, 100),
        # self-test exponents at the lengths the policy picks: short, ...
        _solo("42K", 859433, 42 * K, 3000, 100),
        _solo("160K", 2976221, 160 * K, 4000, 100),
        # ... middle (exponents of batched and served work), ...
        _solo("720K", 13466917, 720 * K, 2000, 100),
        _solo("1600K", 30402457, 1600 * K, 1200, 100),
        # the benchmark's headline length, long calls
        _solo("3200K", 57885161, 3200 * K, 1000, 1000),
        # the careful round-off test at the length the policy picks for that
        # exponent: the error is read back after every iteration
        _solo("3136K_careful", 57885161, 3136 * K, 300, 1),
        # a double check near the current wavefront
        _solo("8064K", 147162241, 8064 * K, 400, 100),
        # the benchmark's 100-million-digit exponent: state larger than L2
        _solo("18432K", 332192831, 18432 * K, 200, 100),
        # the longest supported length
        _solo("32768K", 580000027, 32768 * K, 110, 100),
        # batched mode over the benchmark's range of exponents
        {"name": "batch_32", "kind": "batch", "count": 32, "lo": 1e6, "hi": 2e7, "pick": 7, "iters": 400},
    ]


def draw(rng):
    if rng.random() < 0.15:
        lo = 10 ** rng.uniform(5.3, 6.7)
        count = rng.randint(3, 32)
        return {"kind": "batch", "count": count, "lo": lo, "hi": min(2e7, 10 * lo), "pick": rng.randrange(1000),
                "iters": rng.randint(50, 400)}
    q = workloads.next_prime(10 ** rng.uniform(math.log10(86243), math.log10(5.8e8)))
    n = engine.choose_fft_length(q)
    chunk = rng.choice([1, 37, 100, 100, 1000])
    most = min(5000.0, (MOST_WORDS_SINGLE if chunk == 1 else MOST_WORDS) / n)
    iters = max(1, int(10 ** rng.uniform(math.log10(max(1.0, most / 8)), math.log10(most))))
    return {"kind": "solo", "q": q, "n": n, "iters": iters, "chunk": chunk}


def _members(case, seed):
    """The batch's exponents and lengths: those of the benchmark's generator,
    each moved down to another prime by the seed (the length still fits)."""
    rng = np.random.default_rng([case["pick"], seed])
    base = workloads.batch_exponents(case["count"], case["lo"], case["hi"], seed=case["pick"])
    return [(workloads.next_prime(q - int(rng.integers(1000, 3000))), n) for q, n in base]


class _Solo:
    def __init__(self, case, seed):
        q, n = case["q"], case["n"]
        rng = np.random.default_rng(seed)
        # a residue in the middle of a test: every bit random
        packed = rng.integers(0, 1 << 32, (q + 31) // 32, dtype=np.uint32)
        packed[-1] &= np.uint32((1 << (q % 32)) - 1)
        self.digits = engine.balance_digits(engine.unpack_bits(packed, q, n), q, n)
        self.offset = int(rng.integers(0, q))
        self.iters, self.chunk = case["iters"], case["chunk"]
        self.ctx = LLContext(q, n)


class _Batch:
    def __init__(self, case, seed):
        members = _members(case, seed)
        rng = np.random.default_rng(seed)
        self.offsets = [int(rng.integers(0, q)) for q, _ in members]
        self.iters = case["iters"]
        self.batch = LLBatch([q for q, _ in members], [n for _, n in members])


def prepare(case, seed):
    return _Batch(case, seed) if case["kind"] == "batch" else _Solo(case, seed)


def run(state):
    if isinstance(state, _Batch):
        state.batch.start(state.offsets)
        err = state.batch.step(state.iters, report=True)
        return {"res64": np.array(state.batch.res64(), dtype=np.uint64).view(np.int64),
                "within_limit": bool(err.max() < ERROR_LIMIT)}
    c = state.ctx
    c.load_digits(state.digits, state.offset)
    left, worst = state.iters, 0.0
    while left:
        k = min(left, state.chunk)
        left -= k
        worst = max(worst, c.step(k, report=left == 0, errchk=True))
    digits, offset = c.read_digits()
    # what a tester does with the roundoff error is to compare it with its
    # limit: the value itself is a reading of the arithmetic's order
    return {"digits": digits, "offset": offset, "within_limit": worst < ERROR_LIMIT}


def _iteration_flops(n):
    m = n // 2  # complex points: two transforms and the pointwise squares
    return 10.0 * m * math.log2(m) + 20.0 * m


def _iteration_bytes(n):
    # a state beyond the chip's shared memory and registers (about 70 MB) is
    # read and written once by every iteration
    return 16.0 * n if 8 * n > 70e6 else 0.0


def work(case):
    if case["kind"] == "batch":
        members = _members(case, 0)
        return {"bytes": sum(4.0 * n + case["iters"] * _iteration_bytes(n) for _, n in members),
                "flops": sum(case["iters"] * _iteration_flops(n) for _, n in members)}
    n, k = case["n"], case["iters"]
    return {"bytes": 8.0 * n + k * _iteration_bytes(n), "flops": k * _iteration_flops(n)}


def exact(case, seed):
    """The outputs are whole numbers, which have to stay equal; of them the
    shift has a value in closed form."""
    if case["kind"] == "batch":
        return None
    offset = int(prepare_offset(case, seed))
    return {"digits": None, "offset": offset * pow(2, case["iters"], case["q"]) % case["q"], "within_limit": None}


def prepare_offset(case, seed):
    rng = np.random.default_rng(seed)
    rng.integers(0, 1 << 32, (case["q"] + 31) // 32, dtype=np.uint32)
    return rng.integers(0, case["q"])
