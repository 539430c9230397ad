"""Statistics of a host call.  Device times of one cut in ranges: the ranges' kernels
overlap, and time is counted once.  Downloaded bytes: each range's counters (a
block of 512 bytes) and results come back in one copy."""
import numpy as np
import pytest

from rodv_b200 import workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu


def test_overlapping_ranges_are_timed_once(engine):
    rng = np.random.default_rng(12)
    regions = []
    for _ in range(80):
        haps, reads, quals = workloads._region(rng, 8, (300, 500), 80, (100, 250), 0.01, 0.001)
        regions.append((haps, reads, *[[q[f] for q in quals] for f in range(4)]))
    b = Batch.from_regions(regions * 8)
    assert 1e10 < b.cells() < 6e10  # several ranges
    engine.batch(b)
    db = engine.upload(b)
    db.run()
    whole = db.run()["device_ms"]
    db.free()
    for _ in range(3):
        st = engine.batch(b, stats=True)[1]
        assert 0 < st["fp32_ms"] <= st["device_ms"] <= st["total_ms"]
        assert st["device_ms"] >= 0.9 * whole


def test_downloaded_bytes(engine):
    rng = np.random.default_rng(13)
    one = Batch.from_regions([workloads.random_region(rng, 20, 5)])
    assert engine.batch(one, stats=True)[1]["d2h_bytes"] == 512 + 8 * one.num_pairs
