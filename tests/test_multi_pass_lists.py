"""The FP64 launch over a multi-pass class's list takes the positions that a rescue
filled and passes over the others; a block that finds a long run of empty ones
keeps no other warp of it waiting.  With the short wait limit
(rodv_fault_inject_wait(2): 4,096 polls, under a millisecond) a million empty
positions, and as many with a few filled ones among them, give the results of
the same regions without the limit."""
import numpy as np
import pytest

from rodv_b200 import _lib
from rodv_b200.batch import REGION_DTYPE, Batch

pytestmark = pytest.mark.gpu
L, READS, HAPS = 256, 100, 10000


def _batch(per_row, rescued):
    """One region of READS x HAPS pairs on one-base haplotypes: reads that are
    one long insertion at a gap continuation quality of 0 (per-row gaps) or 1
    (uniform gaps), accepted in FP32; `rescued` of them with expensive gaps."""
    n = READS * L
    gaps = [np.full(n, 10, np.uint8), np.full(n, 10, np.uint8), np.full(n, 1, np.uint8)]
    if per_row:
        gaps[2][:] = 0
        gaps[2][::L] = 10
    for r in [k * (READS // rescued) for k in range(rescued)]:
        gaps[2][r * L:(r + 1) * L] = 20
    off = np.arange(READS, dtype=np.uint64) * L
    return Batch(np.array([(0, HAPS, 0, READS)], dtype=REGION_DTYPE),
                 np.full(HAPS, ord("A"), np.uint8), np.arange(HAPS, dtype=np.uint64),
                 np.ones(HAPS, np.uint32), np.full(n, ord("A"), np.uint8),
                 np.full(n, 30, np.uint8), *gaps, off, np.full(READS, L, np.uint32))


@pytest.mark.parametrize("rescued", [0, 2])
@pytest.mark.parametrize("per_row", [False, True])
def test_long_runs_of_empty_positions(engine, per_row, rescued):
    b = _batch(per_row, rescued)
    want, st = engine.batch(b, stats=True)
    assert st["fp64_pairs"] == rescued * HAPS
    lib = _lib.load()
    assert lib.rodv_fault_inject_wait(2) == 0
    try:
        got = engine.batch(b)
    finally:
        lib.rodv_fault_inject_wait(0)
    assert np.array_equal(got, want)
