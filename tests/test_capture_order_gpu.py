"""Calls inside CUDA graph captures and event chains, where the kernel launched first does not follow a
kernel: after nothing, after a copy, after a join with another stream, and before one."""
import numpy as np
import pytest

from imagebasedspatiotemporalinterpolation_gb300 import native
from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer, pack_shadow_entries, rgb8_to_rgba8, unpack_shadows
from imagebasedspatiotemporalinterpolation_gb300.scene import Sequence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 4])
@pytest.mark.parametrize("captured", [False, True])
def test_render_after_copies_and_joins(cuda, captured, mode):
    """The keyframes' colour arrives by copies on another stream that the render's stream joins; the output
    is copied out there after the render.  Every replay (or turn) must show the colour of its turn."""
    import torch
    seq = Sequence(162, 98, 2, seed=921, aux_offsets=(0.3,), shadows=True, max_speed=3.0)
    host = seq.frame(0)
    frame, client = DeviceFrame.from_host(host), seq.client(0, 2, mode=mode)
    colors = [frame.fwd.color.clone(), 255 - frame.fwd.color]
    r = Renderer()
    wants = []
    for c in colors:
        for view in frame.views():
            view.color.copy_(c)
        out = torch.zeros((98, 162, 4), dtype=torch.uint8, device="cuda")
        r.render(out, client, frame)
        torch.cuda.synchronize()
        wants.append(out)
    assert not torch.equal(*wants)
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    src, out, got = torch.empty_like(colors[0]), torch.empty_like(wants[0]), torch.empty_like(wants[0])

    def chain():
        fork, join, done, back = (torch.cuda.Event() for _ in range(4))
        out.zero_()
        fork.record(main)
        with torch.cuda.stream(side):
            side.wait_event(fork)
            for view in frame.views():
                view.color.copy_(src)
            join.record(side)
        main.wait_event(join)
        r.render(out, client, frame, main)
        done.record(main)
        with torch.cuda.stream(side):
            side.wait_event(done)
            got.copy_(out)
            back.record(side)
        main.wait_event(back)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(main):
        if captured:
            with torch.cuda.graph(graph, stream=main):
                chain()
    torch.cuda.synchronize()
    for turn in range(6):
        with torch.cuda.stream(main):
            src.copy_(colors[turn % 2])
            graph.replay() if captured else chain()
        torch.cuda.synchronize()
        assert torch.equal(got, wants[turn % 2]), f"turn {turn}"
    r.close()


@pytest.mark.parametrize("captured", [False, True])
def test_uploads_and_renders_in_one_chain(cuda, captured):
    """Colour expansion, sparse shadows and a render back to back, the colour written by a copy before."""
    import torch
    seq = Sequence(161, 97, 2, seed=922, shadows=True, max_speed=3.0)
    host, client = seq.frame(0), seq.client(0, 1)
    frame = DeviceFrame.from_host(host)
    entries = [torch.from_numpy(pack_shadow_entries(v.shadow_info, v.shadow_a, v.shadow_b)).cuda() for v in (host.fwd, host.bwd)]
    colors = [torch.from_numpy(np.ascontiguousarray(host.fwd.color[..., :3])).cuda(), torch.full((97, 161, 3), 40, dtype=torch.uint8, device="cuda")]
    r = Renderer()
    stream, rgb = torch.cuda.Stream(), torch.empty_like(colors[0])
    out = torch.empty((97, 161, 4), dtype=torch.uint8, device="cuda")
    src = torch.empty_like(rgb)

    def chain():
        out.zero_()
        rgb.copy_(src)
        rgb8_to_rgba8(frame.fwd.color, rgb, stream)
        rgb8_to_rgba8(frame.bwd.color, rgb, stream)
        for v, e in zip((frame.fwd, frame.bwd), entries):
            unpack_shadows(v.shadow_info, v.shadow_a, v.shadow_b, e, clear_entries=e, stream=stream)
        r.render(out, client, frame, stream)

    wants = []
    for c in colors:  # every step waited for
        frame.fwd.color[..., :3] = c
        frame.bwd.color[..., :3] = c
        want = torch.zeros_like(out)
        torch.cuda.synchronize()
        r.render(want, client, frame)
        torch.cuda.synchronize()
        wants.append(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        chain()
        stream.synchronize()
        if captured:
            with torch.cuda.graph(graph, stream=stream):
                chain()
    for turn in range(6):
        with torch.cuda.stream(stream):
            src.copy_(colors[turn % 2])
            graph.replay() if captured else chain()
        stream.synchronize()
        assert not torch.equal(*wants)
        assert torch.equal(out, wants[turn % 2]), f"turn {turn}"
    assert r.device_status() == native.ISTI_OK
    r.close()


@pytest.mark.parametrize("render_on_default", [True, False])
def test_implicit_order_with_the_default_stream(cuda, render_on_default):
    """A stream made by cudaStreamCreate and the default stream wait for each other without events.  The
    keyframes' colour arrives on one of them behind a delay, the render runs on the other, where the
    kernel before it was enqueued earlier than that, and the output is read on the first."""
    import ctypes
    import torch
    handle = ctypes.c_void_p()
    assert torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle)) == torch.cuda.cudart().cudaError.success
    default, blocking = torch.cuda.default_stream(), torch.cuda.ExternalStream(handle.value)
    at, other = (default, blocking) if render_on_default else (blocking, default)
    seq = Sequence(162, 98, 2, seed=921, aux_offsets=(0.3,), shadows=True, max_speed=3.0)
    frame, client = DeviceFrame.from_host(seq.frame(0)), seq.client(0, 2)
    colors = [frame.fwd.color.clone(), 255 - frame.fwd.color]
    r = Renderer()
    out = torch.zeros((98, 162, 4), dtype=torch.uint8, device="cuda")
    wants = []
    for c in colors:
        for view in frame.views():
            view.color.copy_(c)
        r.render(out.zero_(), client, frame)
        torch.cuda.synchronize()
        wants.append(out.clone())
    torch.cuda.synchronize()
    for turn in range(6):
        with torch.cuda.stream(at):
            out.zero_()
        with torch.cuda.stream(other):
            torch.cuda._sleep(4_000_000)  # about 2 ms
            for view in frame.views():
                view.color.copy_(colors[turn % 2])
        r.render(out, client, frame, at)
        with torch.cuda.stream(other):
            got = out.clone()
        torch.cuda.synchronize()
        assert torch.equal(got, wants[turn % 2]), f"turn {turn}"
    r.close()
    torch.cuda.cudart().cudaStreamDestroy(handle.value)
