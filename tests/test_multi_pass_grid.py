"""Multi-pass launches on both sides of the grid at which they change kernels (the
one for few blocks, the one for full grids): n copies of one region around one,
two, three, four and six items for every SM give n times the bits that the region
gives alone."""
import numpy as np
import pytest
import torch

from rodv_b200 import workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nreads,nhaps", [(2, 1), (1, 2), (3, 2)])  # same, two-haplotype, both
@pytest.mark.parametrize("per_sm", [1, 2, 3, 4, 6])
def test_around_the_grid_of_few_blocks(engine, per_sm, nreads, nhaps):
    rng = np.random.default_rng(29)
    haps = [workloads._random_seq(rng, 321 + 9 * k) for k in range(nhaps)]
    reads = []
    for k in range(nreads):  # two passes; the last read is noisy
        rd = haps[0][:280 + 13 * k].copy()
        rd[rng.random(rd.size) < (0.2 if k == nreads - 1 else 0.005)] = ord("A")
        reads.append(rd)
    quals = [[workloads._quals(rng, r.size, 20, 40), *(np.full(r.size, v, np.uint8)
              for v in (45, 45, 10))] for r in reads]
    region = (haps, reads, *[[q[f] for q in quals] for f in range(4)])
    alone = engine.batch(Batch.from_regions([region]))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (per_sm * sms - 1, per_sm * sms, per_sm * sms + 1):
        got = engine.batch(Batch.from_regions([region] * n))
        assert np.array_equal(got, np.tile(alone, n)), n
