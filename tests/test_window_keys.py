"""The reprojection's window selection (csrc/isti_kernels.cuh, window_keys), built for the host
with nvcc: minima over tile rows against the reference's scan, with ties and special depths."""
import os
import subprocess

import pytest

from imagebasedspatiotemporalinterpolation_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_window_minima_select_the_scan_s_keys(tmp_path):
    nvcc = _build._nvcc()
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "window_keys_test")
    cmd = [nvcc, "-std=c++20", "-O1", _build.CUDA_ARCH, "-I", _build.INCLUDE, "-I", _build.CSRC,
           os.path.join(ROOT, "tests", "cpp", "window_keys_test.cu"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300, env=env)
    assert res.returncode == 0, res.stdout + res.stderr
    assert res.stdout.startswith("ok "), res.stdout
