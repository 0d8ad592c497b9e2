"""The work that is measured: what a program built on this library has it do, call by call.

Every case goes through the public Python classes (Renderer, Quality, FlowNet and the upload
helpers).  Sizes are those of the tests and the benchmark -- 640x360, 1280x720, 1920x1080 and
2064x2208 per eye, up to two aux cameras, up to eight frames per call, the trained network and
its training batch -- and ragged ones between them.

Scenes: a ground plane, moving spheres, one directional light with soft shadows, ray-cast on
the GPU with plain torch (the distribution of scene.Sequence: at most ~1.2 degrees and 5 cm of
camera movement per 1/30 s keyframe interval, client frames at 120 Hz; for the learned cases
the network's training distribution).
"""
import math

import numpy as np
import torch

from imagebasedspatiotemporalinterpolation_gb300 import native, train_flownet
from imagebasedspatiotemporalinterpolation_gb300.flownet import FlowNet
from imagebasedspatiotemporalinterpolation_gb300.metrics import Quality
from imagebasedspatiotemporalinterpolation_gb300.renderer import (DeviceFrame, DeviceView, Renderer, pack_shadow_entries, render_info,
                                                                  rgb8_to_rgba8, unpack_shadows)
from imagebasedspatiotemporalinterpolation_gb300.scene import Client, Pose, perspective, right_vector, view_matrix

DT = 1.0 / 30.0
FRAMES_PER_KEYFRAME = 4
EYES = (-0.032, 0.032)  # half the interpupillary distance, metres
PPD = native.FLIP_DEFAULT_PPD


def listed():
    return [
        # One small frame per call: the lowest-latency use (a preview, a phone), where launches count.
        {"name": "frame_640x360", "kind": "render", "w": 640, "h": 360, "aux": 0, "aux_div": 1, "shadows": False, "mode": 0, "frames": 1,
         "chain": False, "fast": True, "motion": "f16x3"},
        # The frame loop: one call per client frame, three cameras, soft shadows, the library's default arithmetic.
        {"name": "frame_1080p_3cam", "kind": "render", "w": 1920, "h": 1080, "aux": 2, "aux_div": 1, "shadows": True, "mode": 0, "frames": 1,
         "chain": False, "fast": False, "motion": "f16x3"},
        # The benchmark's step: the three client frames of one keyframe interval in one call, the reference's GPU arithmetic.
        {"name": "interval_1080p_3cam", "kind": "render", "w": 1920, "h": 1080, "aux": 2, "aux_div": 1, "shadows": True, "mode": 0,
         "frames": 3, "chain": True, "fast": True, "motion": "f16x3"},
        # A headset server: three times x two eyes of one keyframe pair per call, main camera only.
        {"name": "stereo_2064x2208", "kind": "render", "w": 2064, "h": 2208, "aux": 0, "aux_div": 1, "shadows": False, "mode": 0, "frames": 6,
         "chain": False, "fast": False, "motion": "f16x3"},
        # The linear bidirectional mode (7x7 window, 5 steps) with a half-resolution aux camera, three chained frames.
        {"name": "bidirectional_1366x768", "kind": "render", "w": 1366, "h": 768, "aux": 1, "aux_div": 2, "shadows": True, "mode": 1,
         "frames": 3, "chain": True, "fast": True, "motion": "f16x3"},
        # The splatting mode (no search) at an odd size with the reference's float4 motion images.
        {"name": "splatting_853x481", "kind": "render", "w": 853, "h": 481, "aux": 0, "aux_div": 1, "shadows": False, "mode": 3, "frames": 2,
         "chain": True, "fast": False, "motion": "f32x4"},
        # The timewarp fallback (mode 4), one frame per call, one aux camera behind it.
        {"name": "timewarp_1080p", "kind": "render", "w": 1920, "h": 1080, "aux": 1, "aux_div": 1, "shadows": False, "mode": 4, "frames": 1,
         "chain": False, "fast": False, "motion": "f16x3"},
        # The learned initialiser's call: a U-Net and one search step instead of splatting and three.
        {"name": "learned_1080p", "kind": "learned", "w": 1920, "h": 1080, "frames": 3},
        # Many keyframe pairs of different sizes in one call (several headsets served together).
        {"name": "pairs_mixed", "kind": "pairs", "w": 1280, "h": 720, "w2": 1920, "h2": 1080, "w3": 2064, "h3": 2208, "pairs": 6, "frames": 3},
        # The evaluation loop: PSNR, SSIM and LDR-FLIP (with its map) of a rendered frame against the truth.
        {"name": "metrics_1080p", "kind": "metrics", "w": 1920, "h": 1080},
        # A training step of the flow initialiser (the start of a run): loss and all gradients of a batch at quarter resolution.
        {"name": "train_480x272x8", "kind": "train", "w": 1920, "h": 1080, "batch": 8},
        # A new keyframe of three cameras arriving in the compact upload forms: RGB colour and sparse shadows.
        {"name": "ingest_1080p_3cam", "kind": "ingest", "w": 1920, "h": 1080, "cams": 3},
    ]


def _size(rng, lo, hi):
    """A frame size with the pixel count spread over its logarithm, any parity, common aspects."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.choice((16 / 9, 16 / 9, 4 / 3, 1.0, 2064 / 2208))
    w = max(96, int(math.sqrt(n * aspect)))
    return w, max(64, int(n / w))


def draw(rng):
    kind = rng.choice(("render",) * 6 + ("learned", "pairs", "metrics", "train", "ingest"))
    big = 2064 * 2208
    if kind == "render":
        mode = rng.choice((0, 0, 0, 1, 2, 3, 4))
        aux = rng.choice((0, 0, 1, 2))
        frames = rng.randint(1, 6)
        w, h = _size(rng, 200_000, min(big, 12_000_000 / frames / (1 + aux) / (2 if mode == 1 else 1)))
        aux_div = rng.choice((1, 1, 2))
        if aux_div == 2:
            w, h = w // 2 * 2, h // 2 * 2
        return {"kind": kind, "w": w, "h": h, "aux": aux, "aux_div": aux_div, "shadows": rng.random() < 0.5, "mode": mode, "frames": frames,
                "chain": rng.random() < 0.5, "fast": rng.random() < 0.5, "motion": rng.choice(("f16x3", "f16x3", "f32x4"))}
    if kind == "learned":
        frames = rng.randint(1, 4)
        w, h = _size(rng, 200_000, min(big, 8_000_000 / frames))
        return {"kind": kind, "w": w, "h": h, "frames": frames}
    if kind == "pairs":
        frames, pairs = rng.randint(1, 4), rng.randint(2, 8)
        sizes = [_size(rng, 200_000, min(big, 30_000_000 / pairs / frames)) for _ in range(3)]
        sizes = [(w // 2 * 2, h) for w, h in sizes]  # panels of headsets: even widths
        return {"kind": kind, "w": sizes[0][0], "h": sizes[0][1], "w2": sizes[1][0], "h2": sizes[1][1], "w3": sizes[2][0], "h3": sizes[2][1],
                "pairs": pairs, "frames": frames}
    if kind == "train":
        w, h = _size(rng, 500_000, 1920 * 1080)
        return {"kind": kind, "w": w, "h": h, "batch": rng.randint(1, 8)}
    w, h = _size(rng, 200_000, big)
    if kind == "metrics":
        return {"kind": kind, "w": w, "h": h}
    return {"kind": kind, "w": w, "h": h, "cams": rng.randint(1, 3)}


# ------------------------------------------------------------------ scenes (ray-cast with torch)

class _Scene:
    """Seeded spheres over a chequered ground, two keyframe poses."""

    def __init__(self, seed, n_spheres=64, max_speed=0.5, max_rot_deg=1.2, max_step_m=0.05):
        g = np.random.default_rng([int(seed), n_spheres])
        n = int(n_spheres)
        self.c = g.uniform(-10.0, 10.0, (n, 2))
        self.r = g.uniform(0.2, 1.5, n)
        speed, angle = g.uniform(0.0, max_speed, n), g.uniform(0.0, 2.0 * math.pi, n)
        self.v = np.stack([speed * np.cos(angle), speed * np.sin(angle)], 1)
        self.albedo = torch.from_numpy(np.concatenate([g.uniform(0.0, 1.0, (n, 3)), np.zeros((2, 3))]).astype(np.float32)).cuda()
        light = np.array([0.45, 0.8, 0.35])
        self.light = light / np.linalg.norm(light)
        a = Pose(np.array([0.0, 2.5, -15.0]), 0.0, math.radians(-8.0))
        d = g.standard_normal(3)
        d *= g.uniform(0.0, max_step_m) / max(1e-9, np.linalg.norm(d))
        yaw, pitch = np.radians(g.uniform(-max_rot_deg, max_rot_deg, 2)) * np.array([1.0, 0.5])
        self.poses = (a, Pose(a.eye + d, a.yaw + yaw, a.pitch + pitch))

    def camera(self, w, h, t, offset=0.0):
        """(viewproj, eye) of the camera at time t (in keyframe intervals), `offset` metres to its right."""
        p = self.poses[0].lerp(self.poses[1], t)
        eye = p.eye + right_vector(p.yaw, p.pitch) * offset
        return perspective(90.0, w / h, 0.1, 100.0) @ view_matrix(eye, p.yaw, p.pitch), eye

    def centres(self, time):
        c = self.c + self.v * time
        return np.stack([c[:, 0], self.r, c[:, 1]], 1)

    def visibility(self, p, obj, time, shift):
        """Fraction of the light's disc (2 degrees) seen from the points p (three f32 images) moved by `shift` with their spheres."""
        theta = math.radians(2.0)
        if shift:
            v = torch.from_numpy(np.concatenate([self.v, np.zeros((2, 2))]).astype(np.float32)).cuda()[obj] * shift
            p = (p[0] + v[..., 0], p[1], p[2] + v[..., 1])
        vis = torch.ones_like(p[0])
        lx, ly, lz = (float(x) for x in self.light)
        for i, (cx, cy, cz) in enumerate(self.centres(time)):
            dx, dy, dz = float(cx) - p[0], float(cy) - p[1], float(cz) - p[2]
            along = dx * lx + dy * ly + dz * lz
            dist = torch.sqrt(dx * dx + dy * dy + dz * dz)
            r = float(self.r[i])
            beta = torch.asin(torch.clamp(r / dist, max=1.0))
            alpha = torch.acos(torch.clamp(along / dist, -1.0, 1.0))
            cover = torch.clamp((beta + theta - alpha) / (2.0 * theta), 0.0, 1.0)
            vis = torch.where((along > 0) & (dist > r) & (obj != i), vis * (1.0 - cover), vis)
        return vis

    def cast(self, w, h, vp, eye, k, shadow_frames=0):
        """Images of one camera at keyframe k (0 or 1; a fraction: the client's time): colour, z, the
        motion to the other keyframe (f32, three components) and, with shadow_frames, shadow A / B / info."""
        dev = torch.device("cuda")
        time, sign = k * DT, (1.0 if k < 1 else -1.0)
        x = 2.0 * (torch.arange(w, device=dev, dtype=torch.float64) + 0.5) / w - 1.0
        y = 2.0 * (torch.arange(h, device=dev, dtype=torch.float64) + 0.5) / h - 1.0
        inv = np.linalg.inv(vp)
        far = [(inv[i, 0] * x[None, :] + inv[i, 1] * y[:, None] + (inv[i, 2] + inv[i, 3])) for i in range(4)]
        d = [far[i] / far[3] - float(eye[i]) for i in range(3)]
        length = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        d = [a / length for a in d]
        n = len(self.r)
        obj = torch.full((h, w), n + 1, device=dev, dtype=torch.int64)  # n: the ground, n + 1: the sky
        ground = -float(eye[1]) / torch.where(d[1] < -1e-12, d[1], torch.full_like(d[1], -1e-12))
        hit = (d[1] < -1e-12) & (ground < length)
        best = torch.where(hit, ground, length)
        obj[hit] = n
        centres = self.centres(time)
        for i in range(n):
            oc = eye - centres[i]
            b = d[0] * float(oc[0]) + d[1] * float(oc[1]) + d[2] * float(oc[2])
            disc = b * b - float(oc @ oc - self.r[i] ** 2)
            t = -b - torch.sqrt(torch.clamp(disc, min=0.0))
            closer = (disc > 0) & (t > 1e-6) & (t < best)
            best = torch.where(closer, t, best)
            obj[closer] = i
        p = [float(eye[i]) + d[i] * best for i in range(3)]
        sky = obj == n + 1

        def ndc(q):
            r = [vp[i, 0] * q[0] + vp[i, 1] * q[1] + vp[i, 2] * q[2] + vp[i, 3] for i in range(4)]
            return [r[i] / r[3] for i in range(3)]

        z = torch.where(sky, torch.ones_like(best), ndc(p)[2]).float()
        v = torch.from_numpy(np.concatenate([self.v, np.zeros((2, 2))])).cuda()[obj] * (sign * DT)
        q = ndc([p[0] + v[..., 0], p[1], p[2] + v[..., 1]])
        here = ndc(p)
        moving = obj < n
        motion = torch.stack([torch.where(moving, a - b, torch.zeros_like(a)) for a, b in zip(q, here)], -1).float()

        cf = torch.from_numpy(np.concatenate([centres, np.zeros((2, 3))]).astype(np.float32)).cuda()[obj]
        pf = [a.float() for a in p]
        normal = torch.stack(pf, -1) - cf
        normal /= torch.linalg.norm(normal, dim=-1, keepdim=True)
        lambert = (normal * torch.from_numpy(self.light.astype(np.float32)).cuda()).sum(-1).clamp(min=0.0)
        lambert = torch.where(obj == n, torch.full_like(lambert, float(self.light[1])), lambert)
        chequer = 0.3 + 0.3 * ((torch.floor(p[0]) + torch.floor(p[2])).long() & 1).float()
        albedo = torch.where((obj == n)[..., None], chequer[..., None], self.albedo[obj])
        up = d[1].float().clamp(min=0.0)
        sky_rgb = torch.stack([0.35 + 0.2 * up, 0.5 + 0.25 * up, 0.75 + 0.2 * up], -1)

        def shade(vis):
            lin = albedo * (0.2 + 0.8 * lambert * vis)[..., None]
            lin = torch.where(sky[..., None], sky_rgb, lin).clamp(0.0, 1.0)
            s = torch.where(lin <= 0.0031308, 12.92 * lin, 1.055 * lin ** (1.0 / 2.4) - 0.055)
            out = torch.full((h, w, 4), 255, dtype=torch.uint8, device=dev)
            out[..., :3] = torch.round(s * 255.0).to(torch.uint8)
            return out

        color = shade(self.visibility(pf, obj, time, 0.0))
        images = {"color": color, "z": z.contiguous(), "motion": motion.contiguous(), "viewproj": vp.astype(np.float32),
                  "inv_viewproj": inv.astype(np.float32)}
        if shadow_frames:
            levels = []
            for j in range(shadow_frames):
                dt = sign * j * DT / shadow_frames
                vis = self.visibility(pf, obj, time + dt, dt)
                levels.append(torch.where(sky, torch.zeros_like(vis), torch.floor((1.0 - vis) * 4.0).clamp(0, 3)).to(torch.int32))
            stack = torch.stack(levels)
            lo, hi = stack.amin(0), stack.amax(0)
            field = sum(lv << (2 * j) for j, lv in enumerate(levels))
            field = torch.where(lo != hi, field, torch.zeros_like(field))
            info = torch.full((h, w, 4), 255, dtype=torch.uint8, device=dev)
            for c in range(3):
                info[..., c] = ((field >> (16 - 8 * c)) & 255).to(torch.uint8)
            images.update(shadow_a=shade(1.0 - lo.float() / 3.0), shadow_b=shade(1.0 - hi.float() / 3.0), shadow_info=info)
        return images


def _view(im, motion_format):
    m = im["motion"].half() if motion_format == "f16x3" else torch.nn.functional.pad(im["motion"], (0, 1))
    return DeviceView(im["color"], im["z"], m.contiguous(), im.get("shadow_a"), im.get("shadow_b"), im.get("shadow_info"), im["viewproj"],
                      im["inv_viewproj"])


def _pair(scene, w, h, aux, aux_div, shadows, motion_format):
    """The two keyframes of every camera as the renderer takes them."""
    n = FRAMES_PER_KEYFRAME if shadows else 0
    views = []
    for cam in range(1 + aux):
        vw, vh = (w, h) if cam == 0 else (w // aux_div, h // aux_div)
        offset = (0.0, -0.3, 0.3)[cam]
        views.append([_view(scene.cast(vw, vh, *scene.camera(vw, vh, float(k), offset), k, n), motion_format) for k in (0, 1)])
    frame = DeviceFrame(*views[0])
    for curr, nxt in views[1:]:
        frame.aux_curr.append(curr)
        frame.aux_next.append(nxt)
        frame.aux_priority.append(3 if shadows else 2)
    return frame


def _client(scene, w, h, t, mode, offset=0.0):
    vp, _ = scene.camera(w, h, t, offset)
    return Client(w, h, float(np.float32(t)), vp.astype(np.float32), np.linalg.inv(vp).astype(np.float32), FRAMES_PER_KEYFRAME,
                  FRAMES_PER_KEYFRAME, False, mode)


def _clients(scene, w, h, frames, mode, stereo):
    """The next `frames` client frames: t = 1/4, 2/4, 3/4, ... of the interval, for each eye in turn when `stereo`."""
    eyes = EYES if stereo else (0.0,)
    steps = -(-frames // len(eyes))
    return [render_info(_client(scene, w, h, (i // len(eyes) + 1) / (steps + 1), mode, eyes[i % len(eyes)])) for i in range(frames)]


# ------------------------------------------------------------------ the cases

def prepare(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "render":
        scene = _Scene(seed)
        frame = _pair(scene, w, h, case["aux"], case["aux_div"], case["shadows"], case["motion"])
        r = Renderer()
        r.set_arithmetic(native.ARITH_REFERENCE_GPU if case["fast"] else native.ARITH_IEEE)
        return {"kind": kind, "renderer": r, "frame": frame, "chain": case["chain"],
                "infos": _clients(scene, w, h, case["frames"], case["mode"], case["frames"] == 6 and case["aux"] == 0),
                "outs": [frame.fwd.color.clone() for _ in range(case["frames"])]}
    if kind == "learned":
        n = int(np.random.default_rng(int(seed)).integers(16, 257))
        scene = _Scene(seed, n, 1.0, 5.0, 0.1)
        frame = _pair(scene, w, h, 0, 1, False, "f16x3")
        return {"kind": kind, "renderer": Renderer(), "frame": frame, "net": train_flownet.load(),
                "infos": _clients(scene, w, h, case["frames"], 0, False), "outs": [frame.fwd.color.clone() for _ in range(case["frames"])]}
    if kind == "pairs":
        sizes = ((w, h), (case["w2"], case["h2"]), (case["w3"], case["h3"]))
        jobs = []
        for i in range(case["pairs"]):
            pw, ph = sizes[i % 3]
            scene = _Scene(1000 * int(seed) + i)
            frame = _pair(scene, pw, ph, 0, 1, False, "f16x3")
            jobs.append(([frame.fwd.color.clone() for _ in range(case["frames"])], _clients(scene, pw, ph, case["frames"], 0, False), frame))
        return {"kind": kind, "renderer": Renderer(), "jobs": jobs}
    if kind == "metrics":
        truth, test = _metric_images(case, seed)
        return {"kind": kind, "quality": Quality(w, h), "truth": truth, "test": test}
    if kind == "train":
        b = train_flownet.Batcher(w, h, case["batch"])
        b.fill([int(seed) * 1000 + i for i in range(case["batch"])])
        return {"kind": kind, "net": FlowNet(seed=int(seed)), "x": b.x, "label": b.label}
    cams = []
    for c in range(case["cams"]):
        scene = _Scene(1000 * int(seed) + c)
        vp, eye = scene.camera(w, h, 1.0, (0.0, -0.3, 0.3)[c])
        now, before = scene.cast(w, h, vp, eye, 1, FRAMES_PER_KEYFRAME), scene.cast(w, h, vp, eye, 0, FRAMES_PER_KEYFRAME)
        entries = [torch.from_numpy(pack_shadow_entries(*[im[n].cpu().numpy() for n in ("shadow_info", "shadow_a", "shadow_b")])).cuda()
                   for im in (now, before)]
        cams.append({"rgb": now["color"][..., :3].contiguous(), "rgba": torch.empty_like(now["color"]), "entries": entries[0],
                     "before": entries[1], "images": [torch.zeros_like(now["color"]) for _ in range(3)]})
    return {"kind": kind, "cams": cams}


def _metric_images(case, seed):
    """(truth, test): the client's frame at t = 1/2 and the same frame as interpolation leaves it -- the truth
    blended with the earlier keyframe near moving edges, a pixel of drift in places, a little noise."""
    w, h = case["w"], case["h"]
    scene = _Scene(seed)
    truth = scene.cast(w, h, *scene.camera(w, h, 0.5), 0.5)["color"]
    early = scene.cast(w, h, *scene.camera(w, h, 0.0), 0)["color"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    coarse = torch.rand((1, 1, h // 32 + 2, w // 32 + 2), generator=g, device="cuda")
    mask = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear")[0, 0]
    test = torch.where((mask > 0.8)[..., None], early, truth)
    test = torch.where(((mask > 0.3) & (mask < 0.4))[..., None], torch.roll(truth, 1, 1), test)
    noise = torch.randint(-2, 3, (h, w, 3), generator=g, device="cuda")
    test = test.clone()
    test[..., :3] = torch.where((mask < 0.2)[..., None], (test[..., :3].int() + noise).clamp(0, 255).to(torch.uint8), test[..., :3])
    return truth.contiguous(), test.contiguous()


def run(state):
    kind = state["kind"]
    if kind == "render":
        outs, infos = state["outs"], state["infos"]
        if len(outs) == 1:
            state["renderer"].render(outs[0], infos[0], state["frame"])
        else:
            state["renderer"].render_batch(outs, infos, state["frame"], chain=state["chain"])
        return outs
    if kind == "learned":
        state["renderer"].render_learned(state["outs"], state["infos"], state["frame"], state["net"], 1)
        return state["outs"]
    if kind == "pairs":
        state["renderer"].render_pairs(state["jobs"])
        return [o for outs, _, _ in state["jobs"] for o in outs]
    if kind == "metrics":
        q = state["quality"]
        values = q.launch(state["test"], state["truth"])
        mean, fmap = q.flip(state["test"], state["truth"], with_map=True)
        return {"quality": values, "flip": mean, "map": fmap}
    if kind == "train":
        net = state["net"]
        net.backward(state["x"], state["label"])
        return net.grads()
    out = []
    for cam in state["cams"]:
        rgb8_to_rgba8(cam["rgba"], cam["rgb"])
        unpack_shadows(*cam["images"], cam["entries"], clear_entries=cam["before"])
        out += [cam["rgba"], *cam["images"]]
    return out


# ------------------------------------------------------------------ what a pass cannot do without

_LAYERS = ((9, 16, 32, 1), (9, 32, 64, 2), (9, 64, 96, 4), (9, 96, 128, 8), (1, 128, 96, 8), (9, 96, 96, 4), (1, 96, 64, 4), (9, 64, 64, 2),
           (1, 64, 32, 2), (9, 32, 32, 1), (1, 32, 4, 1))  # taps, channels in, channels out, scale


def _net_size(w, h):
    q = [(-(-s // 4) + 7) // 8 * 8 for s in (w, h)]
    return q[0], q[1], sum(2.0 * taps * ci * co * (q[0] // s) * (q[1] // s) for taps, ci, co, s in _LAYERS)


def work(case):
    kind, px = case["kind"], case["w"] * case["h"]
    if kind == "render":
        per = 4 + 4 + (6 if case["motion"] == "f16x3" else 16) + (12 if case["shadows"] else 0)
        views = 2 * px + 2 * case["aux"] * (case["w"] // case["aux_div"]) * (case["h"] // case["aux_div"])
        if case["mode"] == 4:  # the forward keyframe's z, and a colour per output pixel
            return {"bytes": 4 * px + 8 * px * case["frames"], "flops": 0}
        return {"bytes": per * views + 4 * px * case["frames"], "flops": 0}
    if kind == "learned":
        return {"bytes": 14 * 2 * px + 4 * px * case["frames"], "flops": case["frames"] * _net_size(case["w"], case["h"])[2]}
    if kind == "pairs":
        sizes = (px, case["w2"] * case["h2"], case["w3"] * case["h3"])
        return {"bytes": sum((28 + 4 * case["frames"]) * sizes[i % 3] for i in range(case["pairs"])), "flops": 0}
    if kind == "metrics":  # both images; the map (11 + 11 taps of five moments, 21 + 21 of seven and nine filters, per channel or image)
        return {"bytes": 2 * 2 * 4 * px + 4 * px, "flops": px * (3 * 2 * 22 * 5 + 2 * 2 * 21 * 16)}
    if kind == "train":
        qw, qh, flops = _net_size(case["w"], case["h"])
        return {"bytes": case["batch"] * qw * qh * (32 + 16) + 8 * 339268, "flops": 3 * flops * case["batch"]}
    return {"bytes": case["cams"] * 7 * px, "flops": 0}


# ------------------------------------------------------------------ in 64 bits

def exact(case, seed):
    if case["kind"] == "metrics":
        truth, test = _metric_images(case, seed)
        mse, psnr, ssim = _exact_quality(test, truth)
        mean, fmap = _exact_flip(test, truth)
        return {"quality": torch.tensor([mse, psnr, ssim], dtype=torch.float64), "flip": mean, "map": fmap}
    if case["kind"] == "train":
        s = prepare(case, seed)
        return _exact_gradients(s["net"], s["x"], s["label"])
    return None  # rendered frames and images are bytes


def _rgb(image):
    return image[..., :3].permute(2, 0, 1)[:, None].double() / 255.0


def _separable(x, fx, fy):
    """x (n, 1, h, w) filtered with fx along its rows and fy along its columns, no padding."""
    x = torch.nn.functional.conv2d(x, fx.reshape(1, 1, 1, -1))
    return torch.nn.functional.conv2d(x, fy.reshape(1, 1, -1, 1))


def _exact_quality(a, b):
    x, y = _rgb(a), _rgb(b)
    mse = float(((x - y) ** 2).mean())
    g = torch.exp(-(torch.arange(11, dtype=torch.float64, device=x.device) - 5.0) ** 2 / (2.0 * 1.5 ** 2))
    g = g / g.sum()
    f = lambda v: _separable(torch.nn.functional.pad(v, (5, 5, 5, 5)), g, g)  # noqa: E731
    mx, my = f(x), f(y)
    vx, vy, cov = f(x * x) - mx * mx, f(y * y) - my * my, f(x * y) - mx * my
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    ssim = ((2 * mx * my + c1) * (2 * cov + c2)) / ((mx * mx + my * my + c1) * (vx + vy + c2))
    return mse, -10.0 * math.log10(mse), float(ssim.mean())


_TO_XYZ = ((10135552 / 24577794, 8788810 / 24577794, 4435075 / 24577794), (2613072 / 12288897, 8788810 / 12288897, 887015 / 12288897),
           (1425312 / 73733382, 8788810 / 73733382, 70074185 / 73733382))
_TO_RGB = ((3.241003275, -1.537398934, -0.498615861), (-0.969224334, 1.875930071, 0.041554224), (0.055639423, -0.204011202, 1.057148933))
_WHITE = (0.950428545, 1.0, 1.088900371)
_INV_WHITE = (1.052156925, 1.0, 0.918357670)


def _mix(m, v):
    return [m[i][0] * v[0] + m[i][1] * v[1] + m[i][2] * v[2] for i in range(3)]


def _hunt_lab(rgb):
    xyz = [v * s for v, s in zip(_mix(_TO_XYZ, rgb), _INV_WHITE)]
    d = 6.0 / 29.0
    f = [torch.where(v > d ** 3, v.clamp(min=d ** 3) ** (1.0 / 3.0), v / (3 * d * d) + 4.0 / 29.0) for v in xyz]
    lum = 116.0 * f[1] - 16.0
    return lum, 0.01 * lum * 500.0 * (f[0] - f[1]), 0.01 * lum * 200.0 * (f[1] - f[2])


def _hyab(p, q):
    return torch.sqrt(((p[0] - q[0]) ** 2).clamp(min=1e-15)) + torch.sqrt((p[1] - q[1]) ** 2 + (p[2] - q[2]) ** 2)


def _exact_flip(test, truth):
    """LDR-FLIP (Andersson et al. 2020) with the reference's filters, as sums of separable ones."""
    dev = test.device
    rc = math.ceil(3.0 * math.sqrt(0.04 / (2.0 * math.pi ** 2)) * PPD)
    x = torch.arange(-rc, rc + 1, dtype=torch.float64, device=dev) / PPD
    csf = {b: torch.exp(-math.pi ** 2 * x * x / b) for b in (0.0047, 0.0053, 0.04, 0.025)}
    w1, w2 = 34.1 * math.sqrt(math.pi / 0.04), 13.5 * math.sqrt(math.pi / 0.025)
    norm = w1 * csf[0.04].sum() ** 2 + w2 * csf[0.025].sum() ** 2
    sd = 0.5 * 0.082 * PPD
    rf = math.ceil(3.0 * sd)
    y = torch.arange(-rf, rf + 1, dtype=torch.float64, device=dev)
    gauss = torch.exp(-y * y / (2.0 * sd * sd))
    signed = lambda v: v / torch.where(v < 0, -v[v < 0].sum(), v[v > 0].sum())  # noqa: E731
    edge, point, gauss = signed(-y * gauss), signed((y * y / (sd * sd) - 1.0) * gauss), gauss / gauss.sum()

    def pad(v, r):
        return torch.nn.functional.pad(v[None, None], (r, r, r, r), mode="replicate")

    def features(image):
        v = [c[0] for c in _rgb(image)]
        lin = [torch.where(c > 0.04045, ((c.clamp(min=0.04045) + 0.055) / 1.055) ** 2.4, c / 12.92) for c in v]
        xyz = [c * s for c, s in zip(_mix(_TO_XYZ, lin), _INV_WHITE)]
        lum, cx, cz = 116.0 * xyz[1] - 16.0, 500.0 * (xyz[0] - xyz[1]), 200.0 * (xyz[1] - xyz[2])
        ga, gr = csf[0.0047] / csf[0.0047].sum(), csf[0.0053] / csf[0.0053].sum()
        fl, fx = _separable(pad(lum, rc), ga, ga)[0, 0], _separable(pad(cx, rc), gr, gr)[0, 0]
        fz = ((w1 * _separable(pad(cz, rc), csf[0.04], csf[0.04]) + w2 * _separable(pad(cz, rc), csf[0.025], csf[0.025])) / norm)[0, 0]
        yy = (fl + 16.0) / 116.0
        back = [(yy + fx / 500.0) * _WHITE[0], yy, (yy - fz / 200.0) * _WHITE[2]]
        lab = _hunt_lab([c.clamp(0.0, 1.0) for c in _mix(_TO_RGB, back)])
        ny = pad((lum + 16.0) / 116.0, rf)
        size = lambda f: torch.sqrt(_separable(ny, f, gauss) ** 2 + _separable(ny, gauss, f) ** 2)[0, 0]  # noqa: E731
        return lab, size(edge), size(point)

    (lab_r, edge_r, point_r), (lab_t, edge_t, point_t) = features(truth), features(test)
    one = lambda *v: [torch.tensor(c, dtype=torch.float64, device=dev) for c in v]  # noqa: E731
    cmax = float(_hyab(_hunt_lab(one(0, 1, 0)), _hunt_lab(one(0, 0, 1))) ** 0.7)
    power, knee = _hyab(lab_r, lab_t) ** 0.7, 0.4 * cmax
    dec = torch.where(power < knee, 0.95 / knee * power, 0.95 + (power - knee) / (cmax - knee) * 0.05)
    feat = torch.maximum((edge_r - edge_t).abs(), (point_t - point_r).abs()).clamp(min=1e-15)
    fmap = dec ** (1.0 - torch.sqrt(feat / math.sqrt(2.0)))
    return float(fmap.mean()), fmap


def _exact_gradients(net: FlowNet, x, label):
    """All parameter gradients (flat, in the library's order) of the Huber loss of the U-Net, in 64 bits."""
    flat = net.params().double().requires_grad_(True)
    conv, weights = torch.nn.functional.conv2d, []
    for i, (taps, ci, co, _) in enumerate(_LAYERS):
        wo, bo = net.offsets(i)
        k = 3 if taps == 9 else 1
        weights.append((flat[wo:wo + taps * ci * co].reshape(co, k, k, ci).permute(0, 3, 1, 2), flat[bo:bo + co], k // 2))
    layer = lambda i, v: conv(v, weights[i][0], weights[i][1], padding=weights[i][2])  # noqa: E731
    relu, pool = torch.relu, lambda v: torch.nn.functional.avg_pool2d(v, 2)  # noqa: E731
    up = lambda v: v.repeat_interleave(2, 2).repeat_interleave(2, 3)  # noqa: E731
    total = label.shape[0] * label.shape[1] * label.shape[2]
    for i in range(x.shape[0]):  # one sample at a time: the loss is a sum over them
        v = x[i:i + 1].double().permute(0, 3, 1, 2)
        e1 = relu(layer(0, v))
        e2 = relu(layer(1, pool(e1)))
        e3 = relu(layer(2, pool(e2)))
        e4 = relu(layer(3, pool(e3)))
        d3 = relu(layer(5, up(layer(4, e4)) + e3))
        d2 = relu(layer(7, up(layer(6, d3)) + e2))
        d1 = relu(layer(9, up(layer(8, d2)) + e1))
        want = label[i:i + 1].double().permute(0, 3, 1, 2)
        valid = ~torch.isnan(want)
        err = torch.where(valid, layer(10, d1) - torch.nan_to_num(want), torch.zeros_like(want))
        size = err.abs()
        (torch.where(size < 1, 0.5 * err * err, size - 0.5).sum() / total).backward(retain_graph=True)
    return flat.grad
