"""Per-row-gap read pairs that share a chain item's lanes.

CPU: the plan with stacking of all reads (rodv_debug_chain_plan, stack 2) holds
the chain kernel's rules and computes the same reads with per-row priors, and
leaves the same one over, as the plan without it.  GPU: the stacked pairs give
the bits the same pairs give alone, and match the oracle."""
import numpy as np
import pytest

import oracle
from rodv_b200.batch import Batch
from test_chain_plan import NO, WARP, plan, single_pass


def _rows(items):
    """Reads computed with per-row priors, and the lanes each item uses."""
    return sorted(r for cls, pairs in items if cls % 2 == 0 for p in pairs for r in p)


@pytest.mark.parametrize("ipw", [(2, 2, 2, 2, 1, 1, 1, 1), (1,) * 8])
@pytest.mark.parametrize("seed", range(10))
def test_plan_with_per_row_stacking(seed, ipw):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 200))
    lengths = [int(v) for v in rng.integers(1, 300, n)]
    uniform = [bool(u) for u in rng.random(n) < (0.0, 0.5, 0.1, 0.95)[seed % 4]]
    items, left = plan(lengths, uniform, ipw, 2)
    old, old_left = plan(lengths, uniform, ipw, 1)
    for cls, pairs in items:
        g, rows = ipw[cls // 2], (cls // 2 + 1) * ipw[cls // 2]
        extra = 1 if cls % 2 else 0  # the sum row
        assert all(y != NO for _, y in pairs)
        assert cls % 2 == 0 or all(uniform[r] for p in pairs for r in p)
        used = sum((max(lengths[x], lengths[y]) + extra) // rows + 1 for x, y in pairs)
        assert used <= WARP // g
    placed = sorted(r for _, pairs in items for p in pairs for r in p) + ([left] if left != NO else [])
    assert sorted(placed) == [r for r in range(n) if single_pass(lengths[r], uniform[r])]
    assert left == old_left and _rows(items) == _rows(old)
    assert len(items) <= len(old)


@pytest.mark.gpu
def test_stacked_per_row_pairs_match_the_same_pairs_alone(engine):
    rng = np.random.default_rng(7)
    base = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 300)]
    haps = [base[:200 + 20 * k].copy() for k in range(4)]
    # neighbours in length pair up; class edges (32R - 1) and lane edges
    lens = [1, 2, 7, 8, 15, 16, 30, 31, 32, 33, 55, 56, 63, 64, 79, 95, 96, 111, 126, 127, 128,
            143, 159, 160, 175, 191, 192, 207, 223, 224, 239, 240, 254, 255]
    reads, quals = [], []
    for n in lens:
        at = int(rng.integers(0, 300 - n))
        reads.append(base[at:at + n].copy())
        quals.append([rng.integers(6, 44, n).astype(np.uint8)] +
                     [rng.integers(lo, 45, n).astype(np.uint8) for lo in (20, 20, 5)])
        quals[-1][1][0] ^= 1  # no read has uniform gaps, one-base reads among them
        quals[-1][2][0] = quals[-1][1][0] ^ 2

    def region(ids):
        return (haps, [reads[i] for i in ids], *[[quals[i][f] for i in ids] for f in range(4)])

    # enough copies of the region (20,400 pairs) that its pairs share items
    copies = engine.batch(Batch.from_regions([region(range(len(lens)))] * 150))
    got = copies.reshape(150, len(haps), len(lens))
    assert (got == got[0]).all()
    got = got[0]
    # the reference tests' tolerance
    ref = oracle.batch_log10(Batch.from_regions([region(range(len(lens)))]))
    assert np.abs(got.ravel() - ref).max() < 1e-5
    for i in range(0, len(lens), 2):
        alone = engine.batch(Batch.from_regions([region([i, i + 1])])).reshape(len(haps), 2)
        assert np.array_equal(alone, got[:, i:i + 2]), lens[i]
