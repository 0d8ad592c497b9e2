"""A key tile of the persistent multi-pair launch that never arrives (test hook): the block that waited for it
takes further work before it sees the call's status word.  It must announce nothing more on the barrier
whose phase did not complete; the call reports ISTI_ERR_TIMEOUT and the next one renders bit for bit."""
import pytest

from imagebasedspatiotemporalinterpolation_gb300 import native, scene
from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer

pytestmark = pytest.mark.gpu

WAIT_LIMIT = 1 << 12  # polls of the barrier before giving up (twice): well under a second


@pytest.mark.parametrize("frames", [1, 3])
@pytest.mark.parametrize("widths", [(960, 960), (960, 957)], ids=["tma", "tma-plain"])
def test_block_goes_on_after_a_withheld_tile(cuda, widths, frames):
    import torch
    jobs, wants = [], []
    ref = Renderer()
    for i, w in enumerate(widths):  # pair 0: 30 x 270 blocks, more than fit the GPU at a time
        seq = scene.Sequence(w, 540, 2, seed=4700 + i)
        clients = [seq.client(0, 1 + b) for b in range(frames)]
        frame = DeviceFrame.from_host(seq.frame(0))
        want = [torch.zeros((540, w, 4), dtype=torch.uint8, device="cuda") for _ in clients]
        ref.render_batch(want, clients, frame, chain=False)
        jobs.append(([torch.zeros_like(o) for o in want], clients, frame))
        wants.append(want)
    r = Renderer()
    r.set_pair_units(32, 256)  # the persistent launch
    for withheld in [(5, 5), (900, 100), (-1, -1), (500, 270), (-1, -1)]:
        for outs, _, _ in jobs:
            for o in outs:
                o.zero_()
        r.test_withhold_tile(*withheld, WAIT_LIMIT)
        r.render_pairs(jobs)
        torch.cuda.synchronize()
        assert r.device_status() == (native.ISTI_ERR_TIMEOUT if withheld[0] >= 0 else native.ISTI_OK)
        if withheld[0] < 0:
            for (outs, _, _), want in zip(jobs, wants):
                for a, b in zip(outs, want):
                    assert torch.equal(a, b)
    r.close()
    ref.close()
