"""Device memory of multi-pass calls: boundary rows for the grids that a batch's own
launches have, and a batch below 2e10 cells whose ranges do not fit in three lanes
is computed in one piece."""
import ctypes

import numpy as np
import pytest
import torch

from rodv_b200 import Engine, _lib, workloads
from rodv_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _long(rng, hap_len, read_len, gaps, noise=0.01):
    hap = workloads._random_seq(rng, hap_len)
    read = np.resize(hap, read_len).copy()
    read[rng.random(read_len) < noise] = ord("A")
    quals = [workloads._quals(rng, read_len, 20, 40)] + [np.full(read_len, g, np.uint8) for g in gaps]
    if gaps[0] != gaps[1]:
        quals[1][0] += 1  # per-row gaps
    return ([hap], [read], *[[q] for q in quals])


def _used(make_call):
    """Device bytes that a fresh engine's call takes."""
    eng = Engine(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    out = make_call(eng)
    after = torch.cuda.mem_get_info()[0]
    eng.close()
    return before - after, out


@pytest.mark.parametrize("gaps", [(45, 45, 10), (40, 45, 10)])
@pytest.mark.parametrize("pairs", [1, 40])
def test_boundary_rows_of_a_few_pairs(gaps, pairs):
    # a block's rows take 16 or 24 bytes a column each; 8 rows a block, FP32
    # items of up to two pairs of one or both kinds, or FP64 ones
    rng = np.random.default_rng(3)
    hap_len = 60000
    b = Batch.from_regions([_long(rng, hap_len, 300, gaps) for _ in range(pairs)])
    torch.zeros(1, device="cuda")
    used, out = _used(lambda e: e.batch(b))
    assert np.isfinite(out).all()
    assert used < pairs * 8 * (hap_len + 72) * 24 + (64 << 20)


@pytest.mark.parametrize("kind,nth", [(0, 1), (0, 2), (0, 3), (1, 2), (1, 4)])
def test_ranges_that_do_not_fit_go_in_one_piece(engine, kind, nth):
    rng = np.random.default_rng(4)
    b = Batch.from_regions([_long(rng, 3000, 1500, (45, 45, 10)) for _ in range(3)] * 600)
    assert 4e9 < b.cells() < 2e10
    want, st = engine.batch(b, stats=True)
    lib = _lib.load()
    live = [ctypes.c_uint64(), ctypes.c_uint64()]
    lib.rodv_debug_live_allocations(*map(ctypes.byref, live))
    eng = Engine(0)
    assert lib.rodv_fault_inject_alloc(kind, nth) == 0
    try:
        got, st2 = eng.batch(b, stats=True)
    finally:
        lib.rodv_fault_inject_alloc(kind, 0)
    assert np.array_equal(got, want)
    assert st2["pairs"] == st["pairs"] and st2["fp64_pairs"] == st["fp64_pairs"]
    eng.close()
    now = [ctypes.c_uint64(), ctypes.c_uint64()]
    lib.rodv_debug_live_allocations(*map(ctypes.byref, now))
    assert [x.value for x in now] == [x.value for x in live]
