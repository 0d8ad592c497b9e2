"""isti_render_pairs' persistent launch, asked for by unit sizes: pairs of every size and number would
otherwise be rendered as batches.  Its staging buffers under capture, the call after a timeout, and large
pairs whose reprojection blocks hold their frames in groups."""
import pytest

from imagebasedspatiotemporalinterpolation_gb300 import native, scene
from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer

pytestmark = pytest.mark.gpu


def _persistent():
    r = Renderer()
    r.set_pair_units(32, 256)
    return r


def _pair(seq, k, frames, ref, mode=0):
    """(render_pairs job with zeroed outputs, the outputs of render_batch)"""
    import torch
    clients = [seq.client(k, 1 + b, mode=mode) for b in range(frames)]
    frame = DeviceFrame.from_host(seq.frame(k))
    want = [torch.zeros((seq.height, seq.width, 4), dtype=torch.uint8, device="cuda") for _ in clients]
    ref.render_batch(want, clients, frame, chain=False)
    return ([torch.zeros_like(w) for w in want], clients, frame), want


def _equal(jobs, wants):
    import torch
    for i, ((outs, _, _), want) in enumerate(zip(jobs, wants)):
        for k, (a, b) in enumerate(zip(outs, want)):
            assert torch.equal(a, b), f"pair {i} frame {k}: {int((a != b).any(-1).sum())} pixels differ"


def _clear(jobs):
    import torch
    for outs, _, _ in jobs:
        for o in outs:
            o.zero_()
    torch.cuda.synchronize()


def test_captured_and_uncaptured_calls_keep_their_parameters(cuda):
    import torch
    seq, ref = scene.Sequence(320, 180, 4, seed=4300), Renderer()
    (job_a, want_a), (job_b, want_b) = _pair(seq, 0, 3, ref), _pair(seq, 1, 3, ref)
    r, stream, graph = _persistent(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        r.render_pairs([job_a], stream=stream)  # sizes the arena and both staging buffers
    stream.synchronize()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            r.render_pairs([job_a], stream=stream)
    for _ in range(3):
        _clear([job_a, job_b])
        with torch.cuda.stream(stream):
            r.render_pairs([job_b], stream=stream)  # uncaptured, other parameters
            graph.replay()                          # must still render pair a
        stream.synchronize()
        assert r.device_status() == native.ISTI_OK
        _equal([job_a, job_b], [want_a, want_b])
    r.close()
    ref.close()


def test_call_after_a_stalled_one(cuda):
    import torch
    seq, ref = scene.Sequence(320, 180, 4, seed=4400, aux_offsets=(-0.3, 0.3), shadows=True), Renderer()
    jobs, wants = zip(*[_pair(seq, k, 3, ref) for k in range(3)])
    r = _persistent()
    for stalled in (1, -1, 0, 2, -1):
        _clear(jobs)
        r.test_stall_pair(stalled, 4096)
        r.render_pairs(jobs)
        torch.cuda.synchronize()
        assert r.device_status() == (native.ISTI_ERR_TIMEOUT if stalled >= 0 else native.ISTI_OK)
        if stalled < 0:
            _equal(jobs, wants)
    r.close()
    ref.close()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("frames", [6, 8])
@pytest.mark.parametrize("aux", [(), (-0.3, 0.3)], ids=["main", "aux"])
def test_frames_in_groups(cuda, aux, frames, mode):
    """Six and eight frames are more than a block's results take at a time (rule_group_frames)."""
    import torch
    ref, jobs, wants = Renderer(), [], []
    for i, (w, h) in enumerate([(1280, 720), (643, 361), (1920, 1080)]):
        seq = scene.Sequence(w, h, 2, seed=4800 + i, aux_offsets=aux, shadows=bool(aux), frames_per_anchor=9, shadow_frames_per_anchor=9)
        job, want = _pair(seq, 0, frames, ref, mode)
        jobs.append(job)
        wants.append(want)
    r = _persistent()
    r.render_pairs(jobs)
    torch.cuda.synchronize()
    assert r.device_status() == native.ISTI_OK
    _equal(jobs, wants)
    r.close()
    ref.close()
