"""Kernels that start before the kernels in front of them have finished: they must not read through the
read-only path what those write, and calls back to back on one renderer, each with other keyframes, sizes
and poses than the one before, must give what each gives alone."""
import os
import re

import pytest

from imagebasedspatiotemporalinterpolation_gb300 import _build, native
from imagebasedspatiotemporalinterpolation_gb300.flownet import FlowNet
from imagebasedspatiotemporalinterpolation_gb300.metrics import Quality
from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer
from imagebasedspatiotemporalinterpolation_gb300.scene import Sequence


@pytest.mark.parametrize("source", ["isti_kernels.cuh", "isti_learned.cuh", "isti_batch.cuh", "isti_metrics.cu"])
def test_no_read_only_loads(source):
    """Every image, table and intermediate of these kernels may have been written by a kernel that still ran
    when they started (the rule in isti_pdl.cuh)."""
    with open(os.path.join(_build.CSRC, source)) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert not re.findall(r"__ldg|__restrict__|ld\.global\.nc|__ldca", code)


def _scenes(aux):
    """Keyframe pairs of different sizes (the second has an odd width) and poses, with clients."""
    out = []
    for i, (w, h) in enumerate([(320, 180), (243, 161), (320, 180), (402, 150)]):
        seq = Sequence(w, h, 2, seed=940 + i, aux_offsets=aux, shadows=bool(aux), max_speed=3.0)
        out.append((seq, DeviceFrame.from_host(seq.frame(0)), (h, w, 4)))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("aux", [(), (-0.3, 0.3)], ids=["main", "aux"])
@pytest.mark.parametrize("mode", [0, 1, 3, 4])
def test_renders_back_to_back_equal_renders_alone(cuda, mode, aux, captured):
    import torch
    scenes = _scenes(aux)
    calls = [(scenes[i % 4], [scenes[i % 4][0].client(0, 1 + b, mode=mode) for b in range(1 + i % 3)]) for i in range(12)]
    wants = []
    for (_, frame, shape), clients in calls:
        alone = Renderer()
        want = [torch.full(shape, 5, dtype=torch.uint8, device="cuda") for _ in clients]
        torch.cuda.synchronize()
        alone.render_batch(want, clients, frame)
        torch.cuda.synchronize()
        alone.close()
        wants.append(want)
    outs = [[torch.empty_like(o) for o in want] for want in wants]
    r, stream, graph = Renderer(), torch.cuda.Stream(), torch.cuda.CUDAGraph()

    def chain():
        for ((_, frame, _), clients), out in zip(calls, outs):
            r.render_batch(out, clients, frame, stream=stream)

    def clear():
        for o in sum(outs, []):
            o.fill_(5)
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        clear()
        chain()  # sizes the arena
        if captured:
            stream.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                chain()
    for turn in range(3):
        with torch.cuda.stream(stream):
            clear()
            graph.replay() if captured else chain()
        torch.cuda.synchronize()
        for i, (out, want) in enumerate(zip(outs, wants)):
            for a, b in zip(out, want):
                assert torch.equal(a, b), f"turn {turn} call {i}"
    assert r.device_status() == native.ISTI_OK
    r.close()


@pytest.mark.gpu
def test_learned_calls_back_to_back_equal_calls_alone(cuda):
    import torch
    scenes = _scenes(())
    net = FlowNet(seed=8)
    calls = [(scenes[i % 4], [scenes[i % 4][0].client(0, 1 + b) for b in range(1 + i % 3)]) for i in range(12)]

    def one(r, out, call):
        (_, frame, _), clients = call
        r.render_learned(out, clients, frame, net, iterations=1)

    wants, outs = [], []
    for call in calls:
        alone = Renderer()
        want = [torch.full(call[0][2], 5, dtype=torch.uint8, device="cuda") for _ in call[1]]
        outs.append([o.clone() for o in want])
        torch.cuda.synchronize()
        one(alone, want, call)
        torch.cuda.synchronize()
        alone.close()
        wants.append(want)
    r = Renderer()
    torch.cuda.synchronize()
    for call, out in zip(calls, outs):
        one(r, out, call)
    torch.cuda.synchronize()
    for i, (out, want) in enumerate(zip(outs, wants)):
        for a, b in zip(out, want):
            assert torch.equal(a, b), f"call {i}"
    r.close()
    net.close()


@pytest.mark.gpu
def test_metrics_right_behind_the_render_they_measure(cuda):
    """PSNR, SSIM and FLIP enqueued behind the render that writes their image, another frame each time."""
    import torch
    scenes = _scenes(())[::2]  # one size
    truth = torch.full(scenes[0][2], 90, dtype=torch.uint8, device="cuda")
    r, q = Renderer(), Quality(320, 180)
    clients = [(frame, seq.client(0, b)) for seq, frame, _ in scenes for b in (1, 2, 3)]
    wants = []
    for frame, c in clients:
        out = torch.full_like(truth, 5)
        r.render(out, c, frame)
        torch.cuda.synchronize()
        wants.append((q(out, truth), q.flip(out, truth)))
    out, moments, flips = torch.empty_like(truth), [], []
    for frame, c in clients:
        out.fill_(5)
        r.render(out, c, frame)
        moments.append(q.launch(out, truth).clone())
    for frame, c in clients:
        out.fill_(5)
        r.render(out, c, frame)
        flips.append(q.flip(out, truth))
    for m, f, w in zip(moments, flips, wants):
        assert m.tolist() == [w[0]["mse"], w[0]["psnr"], w[0]["ssim"]]
        assert f == w[1]
    r.close()


@pytest.mark.gpu
def test_network_right_behind_its_weights(cuda):
    """Training steps, each followed at once by an inference and a learned render with the new weights (a
    dependent launch in between), against the same steps waited for one by one."""
    import torch
    seq, frame, shape = _scenes(())[0]
    clients = [seq.client(0, b) for b in (1, 2)]
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(2, 48, 136, 16, generator=g, device="cuda").bfloat16()
    label = torch.randn(2, 48, 136, 4, generator=g, device="cuda")

    def steps(waits):
        net, r, got = FlowNet(seed=9), Renderer(), []
        wait = torch.cuda.synchronize if waits else lambda: None
        wait()
        for _ in range(8):
            net.backward(x, label)
            wait()
            net.adam(1e-2)
            wait()
            flow = net.forward(x)
            wait()
            net.adam(1e-2)
            wait()
            outs = [torch.full(shape, 5, dtype=torch.uint8, device="cuda") for _ in clients]
            wait()
            r.render_learned(outs, clients, frame, net, iterations=1)
            wait()
            got += [flow, *outs]
        torch.cuda.synchronize()
        r.close()
        net.close()
        return got

    for i, (a, b) in enumerate(zip(steps(False), steps(True))):
        assert torch.equal(a, b), f"output {i}"
