"""A batch just above the size from which host-buffer calls are cut in ranges (2e9
cells), with uniform, per-row-gap and multi-pass reads and odd read counts: the
ranges' results are the bits of the batch in one resident piece, in all three
outputs of the host call."""
import numpy as np
import pytest

from rodv_b200 import Engine, workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _batch():
    rng = np.random.default_rng(3)
    regions = []
    for g in range(60):
        haps, reads, quals = workloads._region(rng, int(rng.integers(2, 14)), (200, 600),
                                               int(rng.integers(21, 160)), (50, 250), 0.01, 0.001)
        fields = [[q[f] for q in quals] for f in range(4)]
        if g % 6 == 1:  # per-row gap qualities
            for f in (1, 2, 3):
                fields[f] = [workloads._quals(rng, len(r), 8, 45) for r in reads]
        if g % 9 == 2:  # a multi-pass read
            reads[0] = np.resize(haps[0], 700)
            fields[0][0] = workloads._quals(rng, 700, 10, 40)
            for f, v in ((1, 45), (2, 45), (3, 10)):
                fields[f][0] = np.full(700, v, np.uint8)
        regions.append((haps, reads, *fields))
    return Batch.from_regions(regions)


def test_ranges_match_one_piece(engine):
    b = _batch()
    assert 2.2e9 < b.cells() < 8e9
    db = engine.upload(b)
    db.run()
    whole = db.download()
    db.free()
    got, st = engine.batch(b, stats=True)
    assert st["pairs"] == b.num_pairs and st["cells"] == b.cells()
    assert np.array_equal(got, whole)
    raw, prec = engine.batch_raw(b)
    assert int(prec.sum()) == st["fp64_pairs"]
    # an FP64 result differs from its raw likelihood by the log10 alone
    k = np.flatnonzero((prec == 1) & np.isfinite(whole))
    assert np.allclose(np.log10(raw[k]) - 307.050595577260822, whole[k], rtol=0, atol=1e-12)
    fp64 = Engine(0, force_fp64=True)
    try:
        db = fp64.upload(b)
        db.run()
        assert np.array_equal(engine.batch(b, use_double=True), db.download())
        db.free()
    finally:
        fp64.close()
