"""Which batches the host-buffer call cuts in ranges: not those whose regions refer to
haplotypes and reads out of order, where every range would pack and upload most of
the batch again, and not those with haplotypes or reads of no region, whose bases
would go unchecked."""
import numpy as np
import pytest

from rodv_b200 import RodvError, workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu
RODV_ERR_INVALID_BASE = 3


@pytest.fixture(scope="module")
def batch():
    """480 regions of 4 x 40 pairs, about 3e9 cells."""
    rng = np.random.default_rng(8)
    regions = []
    for _ in range(60):
        haps, reads, quals = workloads._region(rng, 4, (240, 260), 40, (150, 200), 0.01, 0.001)
        regions.append((haps, reads, *[[q[f] for q in quals] for f in range(4)]))
    return Batch.from_regions(regions * 8)


def test_shuffled_regions_are_uploaded_once(engine, batch):
    assert 2.2e9 < batch.cells() < 8e9
    want, st = engine.batch(batch, stats=True)
    order = np.random.default_rng(9).permutation(len(batch.regions))
    shuffled = Batch(batch.regions[order], *[getattr(batch, f) for f in (
        "hap_bases", "hap_offsets", "hap_lengths", "read_bases", "base_quals", "ins_quals",
        "del_quals", "gcp_quals", "read_offsets", "read_lengths")])
    got, st2 = engine.batch(shuffled, stats=True)
    off = batch.out_offsets()
    parts = [want[int(off[g]):int(off[g + 1])] for g in order]
    assert np.array_equal(got, np.concatenate(parts))
    assert st2["h2d_bytes"] < 1.25 * st["h2d_bytes"]


@pytest.mark.parametrize("what", ["hap", "read"])
@pytest.mark.parametrize("end", [False, True])
def test_bases_of_no_region_are_checked(engine, batch, what, end):
    """A haplotype or read that no region refers to, first or last of its array,
    with a base outside A, C, G, T, N."""
    lo = 0 if end else 1
    regions = batch.regions.copy()
    f = {k: getattr(batch, k) for k in ("hap_bases", "hap_offsets", "hap_lengths", "read_bases",
                                        "base_quals", "ins_quals", "del_quals", "gcp_quals",
                                        "read_offsets", "read_lengths")}

    def with_bad(names, offsets, lengths, start):
        n = len(f[names[0]])
        for k, name in enumerate(names):
            f[name] = np.concatenate([f[name], np.array([ord("X") if k == 0 else 30], np.uint8)])
        at = len(f[offsets]) if end else 0
        f[offsets] = np.insert(f[offsets], at, np.uint64(n))
        f[lengths] = np.insert(f[lengths], at, np.uint32(1))
        regions[start] += lo

    if what == "hap":
        with_bad(["hap_bases"], "hap_offsets", "hap_lengths", "hap_start")
    else:
        with_bad(["read_bases", "base_quals", "ins_quals", "del_quals", "gcp_quals"],
                 "read_offsets", "read_lengths", "read_start")
    with pytest.raises(RodvError) as ei:
        engine.batch(Batch(regions, *f.values()))
    assert ei.value.status == RODV_ERR_INVALID_BASE
