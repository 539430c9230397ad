"""The packer's conversion of bases and qualities to row words and base codes
(rodv_b200/csrc/pack_rows.h): a C++ check of the host's form against row_word
and the code table over lengths, alignments, both gap forms and every byte
value, compiled and run on the CPU with and without SSE2."""
import os
import platform
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(NVCC))), "include")


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA),
                    reason="needs g++ and the CUDA headers")
@pytest.mark.parametrize("flags", [[], ["-U__SSE2__"]])
def test_pack_rows(tmp_path, flags):
    if flags and platform.machine() not in ("x86_64", "AMD64"):
        pytest.skip("the host has one form")
    exe = tmp_path / "pack_rows_check"
    subprocess.run(["g++", "-O2", "-std=c++17", *flags, "-I", CUDA, "-I",
                    os.path.join(ROOT, "rodv_b200", "csrc"),
                    os.path.join(HERE, "pack_rows_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout + r.stderr
