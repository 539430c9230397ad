"""Forced FP64 on per-row-gap reads: the kernels of the classes up to two, four, six
and eight rows per lane, one launch in a small batch and a launch for each in a
large one, give the bits that each read gives alone, at the classes' edges, and
match the oracle."""
import numpy as np
import pytest

import oracle
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu
# the edges of the classes (32R - 1 bases in R rows per lane)
LENS = [1, 30, 31, 32, 63, 64, 95, 96, 127, 128, 159, 160, 191, 192, 223, 224, 255]


@pytest.mark.parametrize("longest", [63, 127, 191, 255])
def test_small_and_large_batches(engine, longest):
    rng = np.random.default_rng(longest)
    base = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 330)]
    haps = [base[:270 + 20 * k].copy() for k in range(3)]
    lens = [n for n in LENS if n <= longest]
    reads, quals = [], []
    for n in lens:
        at = int(rng.integers(0, 270 - n))
        reads.append(base[at:at + n].copy())
        quals.append([rng.integers(6, 44, n).astype(np.uint8)] +
                     [rng.integers(lo, 45, n).astype(np.uint8) for lo in (20, 20, 5)])
        quals[-1][2][0] = quals[-1][1][0] ^ 2  # per-row gaps, one-base reads among them

    def region(ids):
        return (haps, [reads[i] for i in ids], *[[quals[i][f] for i in ids] for f in range(4)])

    every = list(range(len(lens)))
    small, st1 = engine.batch(Batch.from_regions([region(every)]), use_double=True, stats=True)
    n = 12000 // (len(haps) * len(lens)) + 1
    copies, st = engine.batch(Batch.from_regions([region(every)] * n), use_double=True, stats=True)
    assert (copies.reshape(n, -1) == small).all()
    assert st1["kernel_launches"] == 1 and st["kernel_launches"] == (longest + 1) // 64
    ref = oracle.batch_log10(Batch.from_regions([region(every)]), oracle.FP64)
    fin = np.isfinite(ref)
    assert np.array_equal(small[~fin], ref[~fin])
    assert np.abs(small[fin] - ref[fin]).max() < 1e-9  # the golden file's
    for i in every:
        alone = engine.batch(Batch.from_regions([region([i])]), use_double=True)
        assert np.array_equal(alone, small.reshape(len(haps), -1)[:, i]), lens[i]
