"""Multi-pass sweeps with many items per block: reads of one to nine passes, ending
at the passes' edges, some rejected by FP32 after a pass or two and some not, in a
batch of several items for every block of the grid.  The block's warps take the
items' passes in whatever order they come free; every region's results are the
bits it gives alone, as the only item of its block (those calls are checked
against the oracle elsewhere)."""
import numpy as np
import pytest

from rodv_b200 import workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu

# one pass (255, uniform gaps), the edges of 256-row passes, nine passes
LENGTHS = [255, 256, 257, 510, 511, 512, 767, 768, 1023, 1024, 1025, 1300, 2047, 2048]


@pytest.mark.parametrize("use_double", [False, True])
@pytest.mark.parametrize("per_row", [False, True])
def test_many_items_per_block(engine, per_row, use_double):
    rng = np.random.default_rng(11 + per_row)
    regions = []
    for g in range(1400):
        n = LENGTHS[g % len(LENGTHS)]
        hap = workloads._random_seq(rng, n + int(rng.integers(1, 40)))
        if g % 7 == 0:
            hap = hap[:int(rng.integers(1, 50))]  # fewer columns than a chunk
        reads, quals = [], []
        for k in range(2 if g % 5 == 0 else 1):  # same-haplotype and two-haplotype items
            noisy = (g + k) % 3 == 0
            rd = np.resize(hap, n).copy()
            rd[rng.random(n) < (0.15 if noisy else 0.002)] = ord("A")
            reads.append(rd)
            quals.append([workloads._quals(rng, n, 25, 40)] +
                         ([workloads._quals(rng, n, 30, 45) for _ in range(3)] if per_row else
                          [np.full(n, v, np.uint8) for v in (45, 45, 10)]))
        regions.append(([hap], reads, *[[q[f] for q in quals] for f in range(4)]))
    b = Batch.from_regions(regions)
    got, st = engine.batch(b, use_double=use_double, stats=True)
    if not use_double:
        assert 0 < st["fp64_pairs"] < st["pairs"]
    off = b.out_offsets()
    for g in range(len(regions)):
        alone = engine.batch(Batch.from_regions([regions[g]]), use_double=use_double)
        assert np.array_equal(alone, got[int(off[g]):int(off[g + 1])]), g
