"""The weight gradient's work splits: none without units (on the host), and the gradients of a training
step whose splits do not divide its units against those of its images one by one."""
import os
import subprocess

import pytest

from imagebasedspatiotemporalinterpolation_gb300 import _build
from imagebasedspatiotemporalinterpolation_gb300.flownet import FlowNet

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_split_without_units(tmp_path):
    nvcc = _build._nvcc()
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "wgrad_splits_test")
    cmd = [nvcc, "-std=c++20", "-O1", _build.CUDA_ARCH, "-I", _build.INCLUDE, "-I", _build.CSRC,
           os.path.join(ROOT, "tests", "cpp", "wgrad_splits_test.cu"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr
    assert res.stdout.startswith("ok"), res.stdout


# A batch of 2^k images: the loss's weight of a pixel, and with it every bf16 gradient behind it, is that
# of the single image times an exact 2^-k.  Left is the order of the f32 sums: 1e-4 of the largest gradient.
@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 8])
def test_step_gradients_equal_the_images_mean(cuda, n):
    import torch
    net = FlowNet(seed=6)
    g = torch.Generator(device="cuda").manual_seed(31)
    x = torch.randn(n, 272, 480, 16, generator=g, device="cuda").bfloat16()
    label = torch.randn(n, 272, 480, 4, generator=g, device="cuda") * 0.5
    want = torch.zeros_like(net.grads(), dtype=torch.float64)
    for i in range(n):
        net.backward(x[i:i + 1].contiguous(), label[i:i + 1].contiguous())
        torch.cuda.synchronize()
        want += net.grads().double() / n
    for _ in range(4):  # back to back
        net.backward(x, label)
    got = net.grads().clone()
    torch.cuda.synchronize()
    assert net.device_status() == 0
    for layer in range(11):
        w, b = net.offsets(layer)
        for lo, hi in ((w, b), (b, net.offsets(layer + 1)[0] if layer < 10 else got.numel())):
            assert (got[lo:hi] - want[lo:hi]).abs().max().item() <= 1e-4 * want[lo:hi].abs().max().item(), f"layer {layer}"
    net.close()
