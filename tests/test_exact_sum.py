"""The metrics' per-thread sums (csrc/isti_device.cuh, ExactSum), built for the host with nvcc."""
import os
import subprocess

import pytest

from imagebasedspatiotemporalinterpolation_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sum_is_no_less_exact_than_double(tmp_path):
    nvcc = _build._nvcc()
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "exact_sum_test")
    cmd = [nvcc, "-std=c++20", "-O2", "-fmad=false", "-Xcompiler", "-ffp-contract=off", _build.CUDA_ARCH, "-I", _build.INCLUDE, "-I", _build.CSRC,
           os.path.join(ROOT, "tests", "cpp", "exact_sum_test.cu"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert res.returncode == 0, res.stdout + res.stderr
    assert res.stdout.startswith("ok"), res.stdout
