"""Batches whose uniform-gap reads share one set of gap qualities run the kernels
that take the gap priors as launch constants; one region with other (uniform)
gap qualities in the batch moves every uniform class to the kernels that take
them per read.  Both compute the same operations on the same values, so the
common regions' results are the same bits, and both match the oracle."""
import numpy as np
import pytest

import oracle
from rodv_b200 import workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu

# read lengths at the edges of the classes (32R - 2 and 32R - 1), of the
# two-haplotype kernels (odd counts) and of the multi-pass strips
EDGES = [1, 14, 30, 31, 62, 63, 94, 126, 127, 158, 190, 222, 254, 255, 256, 300, 511, 520]


def _regions(rng, gaps, counts):
    out = []
    for n_reads, n_haps in counts:
        haps, reads, quals = workloads._region(rng, n_haps, (260, 700), n_reads, (20, 260), 0.01,
                                               0.001)
        reads = [workloads._random_seq(rng, EDGES[k % len(EDGES)]) if k % 5 == 4 else
                 np.resize(r, EDGES[(k + n_haps) % len(EDGES)]) for k, r in enumerate(reads)]
        n = [len(r) for r in reads]
        out.append((haps, reads, [workloads._quals(rng, x, 10, 40) for x in n],
                    *[[np.full(x, g, np.uint8) for x in n] for g in gaps]))
    return out


@pytest.mark.parametrize("use_double", [False, True])
@pytest.mark.parametrize("gaps", [(45, 45, 10), (40, 40, 12), (30, 30, 1)])
def test_constant_and_per_read_gap_priors_agree(engine, gaps, use_double):
    rng = np.random.default_rng(sum(gaps) + use_double)
    regions = _regions(rng, gaps, [(19, 3), (1, 2), (36, 5), (7, 1)])
    other = _regions(rng, (38, 38, 15), [(6, 2)])
    alone = Batch.from_regions(regions)
    got, st = engine.batch(alone, use_double=use_double, stats=True)
    mixed = engine.batch(Batch.from_regions(regions + other), use_double=use_double)
    assert np.array_equal(got, mixed[:len(got)])
    if not use_double and gaps[2] >= 10:  # cheap gap extension (1): nothing underflows FP32
        assert 0 < st["fp64_pairs"] < st["pairs"]
    ref = oracle.batch_log10(alone, oracle.FP64 if use_double else oracle.REFERENCE)
    fin = np.isfinite(ref)
    assert np.array_equal(got[~fin], ref[~fin])
    # FP32: the reference tests' tolerance; FP64: the golden file's
    assert np.abs(got[fin] - ref[fin]).max() < (1e-9 if use_double else 1e-5)
