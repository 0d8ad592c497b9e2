"""Device helpers built for the host with nvcc: the reprojection's window selection (csrc/isti_kernels.cuh,
window_keys: minima over tile rows against the reference's scan, with ties and special depths) and the
division by a constant (csrc/isti_device.cuh, divided_by)."""
import os
import subprocess

import pytest

from imagebasedspatiotemporalinterpolation_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("source", ["window_keys_test", "divided_by_test"])
def test_device_helper_on_the_host(source, tmp_path):
    nvcc = _build._nvcc()
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / source)
    cmd = [nvcc, "-std=c++20", "-O1", "-Xcompiler", "-ffp-contract=off", _build.CUDA_ARCH, "-I", _build.INCLUDE, "-I", _build.CSRC,
           os.path.join(ROOT, "tests", "cpp", source + ".cu"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300, env=env)
    assert res.returncode == 0, res.stdout + res.stderr
    assert res.stdout.startswith("ok"), res.stdout
