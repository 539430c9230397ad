"""A launch that fails after others of its call were made: the call reports it, and
what was launched before it has ended when the call (or, in the service, the
failed batch) is over, so that the next batch's upload, into the same arena,
meets no kernel of the failed one.  The failure is made on the host
(rodv_fault_inject_launch: the n-th next launch is not made)."""
import numpy as np
import pytest

from rodv_b200 import Engine, RodvError, Service, _lib, workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu
RODV_ERR_CUDA = 5


def _batch(seed, scale):
    """Regions of every single-pass class and some multi-pass reads."""
    rng = np.random.default_rng(seed)
    regs = [workloads.random_region(rng, int(rng.integers(1, 40)), int(rng.integers(1, 12)))
            for _ in range(int(20 * scale))]
    for n in (300, 900, 1700):
        hap = workloads._random_seq(rng, n + 300)
        regs.append(([hap], [hap[:n].copy()] * 3, [workloads._quals(rng, n, 20, 40)] * 3,
                     *[[np.full(n, v, np.uint8)] * 3 for v in (45, 45, 10)]))
    return Batch.from_regions(regs)


class _Fault:
    def __init__(self, nth):
        self.nth = nth

    def __enter__(self):
        assert _lib.load().rodv_fault_inject_launch(self.nth) == 0

    def __exit__(self, *exc):
        _lib.load().rodv_fault_inject_launch(0)


@pytest.fixture(scope="module")
def batches(engine):
    bs = [_batch(1, 4.0), _batch(2, 1.0)]
    return [(b, engine.batch(b)) for b in bs]


@pytest.mark.parametrize("nth", [1, 2, 3, 5, 8])
def test_batch_call(batches, nth):
    eng = Engine(0)
    try:
        for b, want in batches:
            with _Fault(nth), pytest.raises(RodvError) as ei:
                eng.batch(b)
            assert ei.value.status == RODV_ERR_CUDA
            for other, ref in batches:
                assert np.array_equal(eng.batch(other), ref)
    finally:
        eng.close()


@pytest.mark.parametrize("nth", [1, 2, 3, 5, 8])
def test_service_batch(batches, nth):
    sv = Service(0)
    try:
        for b, want in batches:
            with _Fault(nth):
                t = sv.submit(b)
                with pytest.raises(RodvError) as ei:
                    sv.wait(t)
            assert ei.value.status == RODV_ERR_CUDA
            tickets = [sv.submit(other) for other, _ in batches]
            for t, (_, ref) in zip(tickets, batches):
                assert np.array_equal(sv.wait(t), ref)
    finally:
        sv.close()


@pytest.mark.parametrize("nth", [1, 3, -1])
def test_device_batch(batches, nth):
    """A launch that fails while the step is captured, of the FP32 part or (-1: the
    last) of the FP64 part: the next run captures again."""
    eng = Engine(0)
    try:
        for b, want in batches:
            db = eng.upload(b)
            launches = db.run()["kernel_launches"]
            db.free()
            db = eng.upload(b)
            with _Fault(nth if nth > 0 else launches), pytest.raises(RodvError) as ei:
                db.run()
            assert ei.value.status == RODV_ERR_CUDA
            for _ in range(2):
                assert db.run()["kernel_launches"] == launches
                assert np.array_equal(db.download(), want)
            db.free()
    finally:
        eng.close()
