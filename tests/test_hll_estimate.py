"""The estimate from HyperLogLog registers (cqlops_hll_estimate): the sum of 2^-r in any order, and as fast for registers
that are alike as for others (CPU)."""
import math
import time

import numpy as np
import pytest


@pytest.fixture(scope="module")
def estimate():
    from computeql_gb300 import build, native
    build.build()
    lib = native.load_ops()
    return lambda r: lib.cqlops_hll_estimate(r.ctypes.data, len(r))


def plain(r):
    m = float(len(r))
    alpha = {16: 0.673, 32: 0.697, 64: 0.709}.get(len(r), 0.7213 / (1.0 + 1.079 / m))
    total = 0.0
    for x in r.tolist():
        total += 1.0 / float(1 << x)
    e, zeros = alpha * m * m / total, int((r == 0).sum())
    return m * math.log(m / zeros) if e <= 2.5 * m and zeros else e


@pytest.mark.parametrize("m", [1, 16, 32, 64, 1024, 4096, 8192])
@pytest.mark.parametrize("kind", ["zeros", "alike", "drawn", "to 40", "to 41", "to 63"])
def test_equals_the_sum_in_order(estimate, m, kind):
    rng = np.random.default_rng(m)
    r = {"zeros": np.zeros(m), "alike": np.full(m, 9), "drawn": rng.geometric(0.5, m), "to 40": rng.integers(0, 41, m), "to 41": rng.integers(0, 42, m),
         "to 63": rng.integers(0, 64, m)}[kind].astype(np.uint32)
    assert estimate(r) == plain(r)


def test_registers_that_are_alike_take_no_longer(estimate):
    rng = np.random.default_rng(2)

    def best(r):
        times = []
        for _ in range(200):
            t = time.perf_counter()
            for _ in range(10):
                estimate(r)
            times.append(time.perf_counter() - t)
        return min(times)

    assert best(np.zeros(4096, dtype=np.uint32)) < 1.5 * best(rng.geometric(0.5, 4096).astype(np.uint32))
