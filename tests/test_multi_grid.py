"""Grids and kernel choice of multi-pass launches.

CPU: the rules of multi_grid.h, compiled and run.  GPU: every tuned variant (strip
height 8 or 4 rows, 2 or 4 warps), with one set of gap qualities in the batch and
with several: launches of at most 8 warps per SM, those beside them counted, run
the kernels for few blocks, larger ones the kernels of 12 warps per SM (the
profiler's kernel names: <precision, R, gap form, same haplotype, blocks per SM,
warps>), and all give the bits of the default variant."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest
import torch

from rodv_b200 import Engine, workloads
from rodv_b200.batch import Batch

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_rules(tmp_path):
    exe = tmp_path / "multi_grid_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I",
                    os.path.join(os.path.dirname(HERE), "rodv_b200", "csrc"),
                    os.path.join(HERE, "multi_grid_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout + r.stderr


def _batch(n, reads, several_gaps):
    """n regions of one haplotype and `reads` reads of three to five 128-row strips;
    several_gaps: every second region's reads have other (uniform) gap qualities."""
    rng = np.random.default_rng(17)
    kinds = []
    for k in range(6):
        hap = workloads._random_seq(rng, 420 + 7 * k)
        rds = [np.resize(hap, 300 + 60 * (k % 4) + j).copy() for j in range(reads)]
        for j, rd in enumerate(rds):
            rd[rng.random(rd.size) < (0.2 if (j + k) % 3 == 0 else 0.004)] = ord("A")
        gaps = (40, 40, 12) if several_gaps and k % 2 else (45, 45, 10)
        quals = [[workloads._quals(rng, r.size, 20, 40), *(np.full(r.size, v, np.uint8)
                  for v in gaps)] for r in rds]
        kinds.append(([hap], rds, *[[q[f] for q in quals] for f in range(4)]))
    return Batch.from_regions([kinds[k % 6] for k in range(n)])


def _pipe_kernels(engine, b):
    """Results, and {(precision, R, gap form, same haplotype): blocks x warps per SM}."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = engine.batch(b)
    found = {}
    for e in prof.key_averages():
        m = re.search(r"forward_pipe_kernel<rodv::(\w+), (\d), (\d), (\w+), (\d), (\d)>", e.key)
        if m:
            found[m[1], int(m[2]), int(m[3]), m[4] == "true"] = int(m[5]) * int(m[6])
    return out, found


@pytest.mark.gpu
@pytest.mark.parametrize("several_gaps", [False, True])
@pytest.mark.parametrize("variant", range(4))
def test_variants_and_their_kernels(engine, tmp_path, variant, several_gaps):
    p = torch.cuda.get_device_properties(0)
    sms, warps = p.multi_processor_count, 4 if variant & 1 else 2
    cache = tmp_path / "tune"
    cache.write_text("".join(f"{p.name.replace(' ', '_')}_sm{sms} {c} {v} {v}\n" for c, v in
                             ((c, variant if c >= 16 else 0) for c in range(18))))
    eng = Engine(0, tune_cache=str(cache))
    try:
        assert eng.tuned_variants()["fp32"][17] == variant
        few = 8 * sms // warps  # blocks
        form = 1 if several_gaps else 2
        # (regions, reads): same-haplotype items alone, then with half as many
        # two-haplotype items beside them
        for n, reads, full in ((few - 1, 2, False), (few, 2, False), (few + 1, 2, True),
                               (4 * few, 2, True), (2 * few // 3 - 2, 3, False),
                               (2 * few // 3 + 2, 3, True)):
            b = _batch(n, reads, several_gaps)
            got, kernels = _pipe_kernels(eng, b)
            assert np.array_equal(got, engine.batch(b)), (n, reads)
            if not kernels:
                pytest.skip("the profiler sees no kernels here")
            R = 4 if variant & 2 else 8
            assert kernels["F32x2", R, form, True] == (12 if full else 8), (n, reads, kernels)
            if reads == 3:
                assert kernels["F32x2", R, form, False] == (12 if full else 8), (n, kernels)
    finally:
        eng.close()
