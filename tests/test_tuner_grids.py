"""The autotuner times the multi-pass kernels that full grids run (the profiler's
kernel names: <precision, R, gap form, same haplotype, blocks per SM, warps>), on
at least three rounds of items."""
import re

import pytest
import torch

from rodv_b200 import Engine

pytestmark = pytest.mark.gpu


def test_multi_pass_variants_are_timed_on_full_grids(capfd):
    from torch.profiler import ProfilerActivity, profile
    eng = Engine(0, verbose=True)
    try:
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            eng.autotune(force=True)
    finally:
        eng.close()
    names = [e.key for e in prof.key_averages()]
    if not any("forward" in n for n in names):
        pytest.skip("the profiler sees no kernels here")
    shape = re.compile(r"forward_pipe_kernel<rodv::F32x2, (\d), 2, true, (\d), (\d)>")
    seen = {(int(m[1]), int(m[3])): int(m[2]) * int(m[3]) for m in map(shape.search, names) if m}
    assert seen == {(8, 2): 12, (8, 4): 12, (4, 2): 12, (4, 4): 12}, seen
    lines = re.findall(r"tune FP\d\d class 1[67] .*, (\d+) items on (\d+) blocks",
                       capfd.readouterr().err)
    assert len(lines) == 16
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for items, blocks in lines:
        assert int(blocks) % sms == 0 and int(items) >= 3 * int(blocks), (items, blocks)
