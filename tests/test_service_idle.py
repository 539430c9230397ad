"""While a long batch runs, the service's worker sleeps: the process takes a small
part of a core."""
import time

import numpy as np
import pytest

from rodv_b200 import Service, workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _long_pair():
    """One pair of 30,000 x 60,000 bases: a few hundred milliseconds on the GPU."""
    rng = np.random.default_rng(6)
    hap = workloads._random_seq(rng, 60000)
    n = 30000
    return Batch.from_regions([([hap], [hap[:n].copy()], [np.full(n, 30, np.uint8)],
                                *[[np.full(n, v, np.uint8)] for v in (45, 45, 10)])])


def test_a_long_batch_keeps_no_core_busy():
    b = _long_pair()
    rng = np.random.default_rng(7)
    small = Batch.from_regions([workloads.random_region(rng, 10, 3)])
    sv = Service(0)
    try:
        want = sv.wait(sv.submit(b))
        want_small = sv.wait(sv.submit(small))
        t = sv.submit(b)
        time.sleep(0.02)  # packed and launched
        wall, cpu = time.perf_counter(), time.process_time()
        got = sv.wait(t)
        wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
        assert np.array_equal(got, want)
        assert wall > 0.05
        assert cpu < 0.4 * wall, (cpu, wall)
        # a request that arrives meanwhile
        t = sv.submit(b)
        time.sleep(0.02)
        assert np.array_equal(sv.wait(sv.submit(small)), want_small)
        assert np.array_equal(sv.wait(t), want)
    finally:
        sv.close()
