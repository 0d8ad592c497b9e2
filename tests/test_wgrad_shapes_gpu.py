"""The weight gradient's work splits against torch: row lengths around its segments, channel counts that
put all accumulators, one row of taps or one block of output channels into a CTA, 1x1 images."""
import ctypes as C

import pytest

from imagebasedspatiotemporalinterpolation_gb300 import native

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


# tolerance: f32 accumulation of exact bf16 products in another order than torch's, as a share of the largest gradient
@pytest.mark.parametrize("taps,cin,cout", [(9, 16, 16), (9, 32, 32), (9, 64, 64), (9, 240, 112), (9, 256, 128), (9, 96, 128), (1, 256, 128),
                                           (1, 16, 16)], ids=str)
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (2, 3, 64), (1, 2, 65), (2, 5, 128), (1, 4, 129), (3, 2, 200)], ids=str)
def test_wgrad_matches_torch(cuda, taps, cin, cout, n, h, w):
    import torch
    lib = native.load()
    torch.manual_seed(1000 * cin + 10 * cout + w)
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    x = torch.randn(n, h, w, cin, device="cuda").bfloat16()
    dy = torch.randn(n, h, w, cout, device="cuda").bfloat16()
    k = 3 if taps == 9 else 1
    ref = torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2), (cout, cin, k, k), dy.double().permute(0, 3, 1, 2), padding=k // 2)
    ref = ref.permute(0, 2, 3, 1).reshape(cout, taps, cin)
    nbytes = lib.isti_unet_wgrad_scratch_bytes(taps, n, h, w, cin, cout)
    scratch = torch.empty(nbytes // 4 + 1, dtype=torch.float32, device="cuda")
    dw = torch.full((cout, taps, cin), float("nan"), device="cuda")
    assert lib.isti_unet_wgrad(taps, _p(dy), _p(x), n, h, w, cin, cout, _p(dw), 0, _p(scratch), nbytes, _p(status), None) == native.ISTI_OK
    torch.cuda.synchronize()
    assert int(status[0].item()) == native.ISTI_OK
    assert (dw - ref).abs().max().item() <= 1e-4 * ref.abs().max().item()
