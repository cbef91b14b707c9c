"""The branch-free FP64 forms against the general ones (tests/fp64_check.cu):
on the host the rule that chooses between them and their algebra, on the GPU
their divide and square root too. Bit for bit, built as the FP64 units are."""
import subprocess

import pytest

from test_index_host import ROOT, _nvcc

pytestmark = pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")


def _check(tmp_path, *args):
    exe = str(tmp_path / "fp64_check")
    r = subprocess.run([_nvcc(), "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-fmad=false", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-I", f"{ROOT}/verona_b200/csrc", "-I", f"{ROOT}/include",
                        f"{ROOT}/tests/fp64_check.cu", "-o", exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


def test_fp64_fast_forms_on_the_host(tmp_path):
    _check(tmp_path)


@pytest.mark.gpu
def test_fp64_fast_forms_on_the_device(tmp_path):
    _check(tmp_path, "device")
