"""Reprojection blocks that hold their frames' results in groups: batches of up to 8 frames, for view
counts that are constants of the kernel (2, 4, 6) and not (8), must equal frame-by-frame renders."""
import numpy as np
import pytest

from imagebasedspatiotemporalinterpolation_gb300 import native
from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer
from imagebasedspatiotemporalinterpolation_gb300.scene import Sequence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", [native.ARITH_IEEE, native.ARITH_REFERENCE_GPU])
@pytest.mark.parametrize("mode", [0, 1, 3])
@pytest.mark.parametrize("aux", [(), (-0.3,), (-0.3, 0.3), (-0.3, 0.3, 0.6)], ids=len)
@pytest.mark.parametrize("size", [(162, 70), (97, 61)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_grouped_batches_equal_frames_in_order(cuda, size, aux, mode, arith):
    import torch
    w, h = size
    seq = Sequence(w, h, 2, seed=911, aux_offsets=aux, shadows=True, max_speed=3.0, frames_per_anchor=9, shadow_frames_per_anchor=9)
    frame = DeviceFrame.from_host(seq.frame(0))
    r = Renderer()
    r.set_arithmetic(arith)
    prev = torch.from_numpy(np.random.default_rng(3).integers(0, 256, (h, w, 4), dtype=np.uint8)).cuda()
    for n in (4, 5, 7, 8):
        clients = [seq.client(0, 1 + b, mode=mode) for b in range(n)]
        single = []
        running = prev.clone()
        for c in clients:
            alone = prev.clone()
            r.render(alone, c, frame)
            r.render(running, c, frame)
            single.append((alone, running.clone()))
        for chain in (False, True):
            outs = [prev.clone() for _ in clients]
            r.render_batch(outs, clients, frame, chain=chain)
            for k, o in enumerate(outs):
                assert torch.equal(o, single[k][int(chain)]), f"{n} frames, chain {chain}, frame {k}"
    r.close()
