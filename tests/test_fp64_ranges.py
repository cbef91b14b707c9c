"""The branch-free FP64 divide and square root over all operands that their callers
admit, and at quotients and roots next to the middle between two FP64 numbers
(tests/fp64_range_check.cu, whose argument is the number of trials)."""
import subprocess

import pytest

from test_index_host import ROOT, _nvcc


@pytest.mark.gpu
@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_fp64_divide_and_root_over_their_ranges(tmp_path):
    exe = str(tmp_path / "fp64_range_check")
    r = subprocess.run([_nvcc(), "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-fmad=false", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-I", f"{ROOT}/verona_b200/csrc", "-I", f"{ROOT}/include",
                        f"{ROOT}/tests/fp64_range_check.cu", "-o", exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([exe, "1000000000"], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
