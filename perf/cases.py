"""The work a host has this backend do, as cases that can be timed and compared.

A case is a dict of plain values; :func:`prepare` makes what a host holds
before the call (a resident world, a context, the inputs), :func:`run` is one
pass through the public entry points, :func:`work` what that pass cannot do
without and :func:`exact` the answer in 64 bits where there is a closed form
of it (the denoiser and the guide; a march that stops within a tolerance has
none).

The sizes are the repository's own configurations: the small plain scene at
256 x 256 and 16 spp; the full-size one at 1920 x 1080; the serving mix over
scenes of 256 to 16384 primitives with its 1280 x 720 interactive sessions;
the enclosed room for the learned guide; the city at 3840 x 2160 and 32
surfaces; and the transport's ray pools for a host that keeps its own
transport.
"""
from __future__ import annotations

import ctypes
import math
import os

import numpy as np
import torch

import kodanuki_gb300 as K
from kodanuki_gb300.scene import Scene

SCENES = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden", "scenes")

# how each scene's octree is built: the benchmark's for the full-size scene
# and the city, the serving run's for its scenes, the tests' for the others
BUILDS = {"c2": (7, 11, 32), "c5": (7, 11, 32), "c1": (6, 10, 64), "serve_256": (6, 10, 64), "serve_1024": (6, 10, 64), "serve_4096": (6, 10, 64)}
TESTED = (5, 10, 64)

# march-form program steps a sample of a frame runs (kdn_frame_stats), for
# the operation counts: two floating-point operations a step
STEPS_A_SAMPLE = {"c2": 1040, "c5": 600}
STEPS_ELSE = 500

_worlds: dict[str, K.Backend] = {}


def world(name: str) -> K.Backend:
    """A scene's resident world, built once as a render host keeps it; each
    state draws it through a context of its own (kdn_open_sharing)."""
    if name not in _worlds:
        b = K.Backend(0)
        b.load(Scene.load(os.path.join(SCENES, name + ".npz")))
        b.build(*BUILDS.get(name, TESTED))
        _worlds[name] = b
    return _worlds[name]


def listed() -> list[dict]:
    return [
        # a host that keeps the transport passes its worker's pool of 512
        # slots through kdn_extend each step: the smallest call there is
        {"name": "extend_pool", "kind": "extend", "scene": "c1", "rays": 512, "on_device": False},
        # a host with its rays on the device: a large odd-sized batch in the
        # full-size scene, half of it camera rays, half scattered ones
        {"name": "extend_million", "kind": "extend", "scene": "c2", "rays": 1_000_003, "on_device": True},
        # the smallest request of the serving mix: a preview frame
        {"name": "frame_preview", "kind": "frame", "scene": "serve_256", "width": 320, "height": 240, "samples": 1, "surfaces": 8},
        # the small plain configuration whole
        {"name": "frame_small", "kind": "frame", "scene": "c1", "width": 256, "height": 256, "samples": 16, "surfaces": 8},
        # an interactive session's frame: 1 spp with the reconstruction chain
        {"name": "frame_session", "kind": "frame", "scene": "serve_4096", "width": 1280, "height": 720, "samples": 1, "surfaces": 8, "denoise": True},
        # the full-size configuration's frame, at a quarter of its samples
        {"name": "frame_full", "kind": "frame", "scene": "c2", "width": 1920, "height": 1080, "samples": 16, "surfaces": 16, "denoise": True},
        # the city's progressive 4K frame
        {"name": "frame_city", "kind": "frame", "scene": "c5", "width": 3840, "height": 2160, "samples": 1, "surfaces": 32, "denoise": True},
        # an odd-sized frame of the rarer parts: scattering bodies, the Sobol
        # sampler, a sample count that divides nothing
        {"name": "frame_ragged", "kind": "frame", "scene": "scatter_small", "width": 641, "height": 359, "samples": 3, "surfaces": 8, "sobol": True},
        # a burst of the serving mix: previews, stills and interactive
        # frames of three resident scenes at once
        {"name": "serve_burst", "kind": "serve", "requests": 6, "slots": 8},
        # a frame of the enclosed room drawn from the learned guide
        {"name": "frame_guided", "kind": "guided", "scene": "room", "width": 960, "height": 540, "samples": 4, "surfaces": 8, "table_log2": 19},
        # a training batch of the guide, forward and backward
        {"name": "guide_gradients", "kind": "gradients", "rows": 65_536, "table_log2": 14},
        # the denoiser over a host's own feature buffers on the device
        {"name": "denoise_1080p", "kind": "denoise", "width": 1920, "height": 1080, "demodulated": True},
    ]


def _between(rng, low: float, high: float) -> int:
    """A whole number spread over the logarithm of the range."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(["extend", "frame", "frame", "frame", "frame", "serve", "guided", "gradients", "query", "denoise"])
    if kind == "extend":
        n = _between(rng, 100, 1_000_000)
        return {"kind": kind, "scene": rng.choice(["c1", "c2", "serve_1024"]), "rays": n, "on_device": n > 50_000 or rng.random() < 0.3}
    if kind == "frame":
        scene = rng.choice(["c1", "c2", "serve_256", "serve_1024", "serve_4096", "scatter_small", "glass_small", "rough_small", "films_small", "patterns_small", "lamps_small"])
        width = _between(rng, 96, 1920)
        height = max(8, int(width * rng.uniform(0.5, 1.0)))
        samples = min(rng.choice([1, 1, 2, 3, 4, 5, 16]), max(1, 16_000_000 // (width * height)))
        case = {"kind": kind, "scene": scene, "width": width, "height": height, "samples": samples, "surfaces": rng.choice([4, 8, 8, 12, 16]),
                "denoise": rng.random() < 0.5, "sobol": rng.random() < 0.2}
        if case["denoise"] and rng.random() < 0.4:
            # a film factor above 1: drawn at a fraction of the shown size, then the upscale member
            factor = rng.choice([2, 3, 4])
            case.update(factor=factor, phase=rng.randrange(factor * factor), width=max(width // factor, 8) * factor, height=max(height // factor, 8) * factor)
        return case
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(3, 7), "slots": rng.choice([4, 8])}
    if kind == "guided":
        width = _between(rng, 96, 1280)
        return {"kind": kind, "scene": "room", "width": width, "height": max(8, int(width * rng.uniform(0.5, 0.8))), "samples": rng.choice([1, 2, 3, 4]), "surfaces": 8,
                "table_log2": rng.choice([14, 17, 19])}
    if kind == "gradients":
        return {"kind": kind, "rows": _between(rng, 500, 200_000), "table_log2": rng.choice([12, 13, 14, 15])}
    if kind == "query":
        return {"kind": kind, "rows": _between(rng, 500, 500_000), "table_log2": rng.choice([14, 17, 19])}
    width = _between(rng, 65, 2560)
    return {"kind": kind, "width": width, "height": max(33, int(width * rng.uniform(0.4, 0.8))), "demodulated": rng.random() < 0.5}


# ---- inputs ----

def _camera(scene: Scene, rng: np.random.Generator) -> np.ndarray:
    """The scene's camera turned a little about its target, as a viewer's is."""
    cam = K.scene_blocks(scene)["shot.camera"].copy()
    eye, target = cam["eye"][0].copy(), cam["target"][0]
    a = rng.uniform(-0.05, 0.05)
    d = eye - target
    eye[0] = target[0] + d[0] * math.cos(a) - d[1] * math.sin(a)
    eye[1] = target[1] + d[0] * math.sin(a) + d[1] * math.cos(a)
    cam["eye"][0] = eye
    return cam


def _rays(scene: Scene, n: int, rng: np.random.Generator) -> np.ndarray:
    """Half camera rays, half from points about the target in even directions."""
    cam = _camera(scene, rng)
    eye, target, up = cam["eye"][0], cam["target"][0], cam["up"][0]
    forward = (target - eye) / np.linalg.norm(target - eye)
    right = np.cross(forward, up)
    right /= np.linalg.norm(right)
    above = np.cross(right, forward)
    reach = math.tan(float(cam["fov"][0]) / 2)
    rays = np.zeros(n, K.RAY_DTYPE)
    m = n // 2
    u, v = rng.uniform(-1, 1, m) * reach * 16 / 9, rng.uniform(-1, 1, m) * reach
    d = forward + u[:, None] * right + v[:, None] * above
    rays["origin"][:m] = eye
    rays["origin"][m:] = target + np.linalg.norm(target - eye) * rng.uniform(-0.5, 0.5, (n - m, 3))
    e = rng.normal(size=(n - m, 3))
    rays["direction"][:m] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["direction"][m:] = e / np.linalg.norm(e, axis=1, keepdims=True)
    rays["far"] = np.inf
    rays["within"] = 0xFFFFFFFF
    return rays


def _guide_params(table_log2: int, weights: int, rng: np.random.Generator):
    """A guide past its start: weights and a table that carry signal."""
    shapes = [(64, 48), (64, 64), (64, 64), (48, 64)]
    w = np.concatenate([rng.uniform(-1, 1, (n, k)).ravel() * 2 * math.sqrt(6.0 / (n + k)) for n, k in shapes]).astype(np.float32)
    w[weights - 8 * 64:] = 0.0  # the output layer's unused rows
    t = rng.random((16 << table_log2) * 2, dtype=np.float32)
    return w, t - np.float32(0.5)


def _guide_rows(lo, hi, n: int, rng: np.random.Generator, columns: int) -> np.ndarray:
    def unit():
        d = rng.normal(size=(n, 3))
        return d / np.linalg.norm(d, axis=1, keepdims=True)
    parts = [rng.uniform(lo, hi, size=(n, 3)), unit()]
    if columns == 10:
        parts += [unit(), rng.exponential(1.0, (n, 1))]
    return np.ascontiguousarray(np.concatenate(parts, axis=1), np.float32)


def _guide(table_log2: int, rng: np.random.Generator, lo, hi, trained: bool) -> K.Guide:
    g = K.Guide(0, table_log2=table_log2, seed=2, region=(lo, hi), learning_rate=1e-2, batch=16384, max_steps=256, sample_capacity=1 << 18)
    if trained:
        g.train(_guide_rows(lo, hi, 128, np.random.default_rng(1), 10), batch=128, steps=1)  # frames draw from a trained guide alone
    g.set_params(*_guide_params(table_log2, g.weight_count, rng))
    return g


UNIT = (np.full(3, -1.0), np.full(3, 1.0))


def _features(width: int, height: int, seed: int) -> dict:
    """Feature buffers of a frame on the device: a floor and balls in front of
    a sky, 1-spp light with its history's length and second moment."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dev = dict(device="cuda")
    y, x = torch.meshgrid(torch.arange(height, **dev, dtype=torch.float32), torch.arange(width, **dev, dtype=torch.float32), indexing="ij")
    u, v = (x + 0.5) / width * 2 - 1, 1 - (y + 0.5) / height * 2
    leaf = torch.where(v < 0.3, 0, -1).to(torch.int32)
    distance = torch.where(v < 0.3, 4.0 / (0.35 - v).clamp(min=0.05), torch.full_like(v, float("inf")))
    normal = torch.zeros(height, width, 3, **dev)
    normal[..., 2] = (v < 0.3).float()
    balls = torch.rand(24, 4, generator=g, **dev)
    for k in range(24):
        cx, cy, r = balls[k, 0] * 2 - 1, balls[k, 1] * 1.2 - 0.8, 0.05 + 0.15 * balls[k, 2]
        dx, dy = (u - cx) / r, (v - cy) / r * height / width
        inside = dx * dx + dy * dy < 1
        dz = (1 - dx * dx - dy * dy).clamp(min=0).sqrt()
        ball = torch.stack([dx, -dz, dy], dim=-1)
        normal = torch.where(inside[..., None], ball, normal)
        distance = torch.where(inside, 3.0 + 4.0 * balls[k, 3] - r * dz, distance)
        leaf = torch.where(inside, torch.full_like(leaf, k + 1), leaf)
    tint = torch.rand(25, 3, generator=g, **dev) * 0.6 + 0.2
    hit = (leaf >= 0)[..., None]
    albedo = torch.where(hit, tint[leaf.clamp(min=0).long()], torch.zeros(3, **dev))
    base = torch.where(hit, (0.3 + 0.7 * normal[..., 2:3].abs()), 0.8 + 0.2 * v[..., None])
    noise = -torch.log(torch.rand(height, width, 3, generator=g, **dev).clamp(min=1e-6))
    colour = base * noise
    luma = colour @ torch.tensor([0.2126, 0.7152, 0.0722], **dev)
    # most pixels have a history, a disoccluded band has none yet
    length = torch.randint(4, 30, (height, width), generator=g, **dev).float()
    length = torch.where((x / width * 7 + y / height * 3) % 2 < 0.5, torch.ones_like(length), length)
    moment = luma * luma * (1 + torch.rand(height, width, generator=g, **dev))
    return {"colour": colour.contiguous(), "moment": moment.contiguous(), "length": length.contiguous(), "distance": distance.half().contiguous(),
            "normal": normal.half().contiguous(), "albedo": albedo.half().contiguous(), "leaf": leaf.contiguous()}


REACH = math.tan(0.35)


def _lens(width: int, height: int):
    """eye, forward, right, up, reach, aspect"""
    return [0.0, 0.0, 1.0, 0.0, 1.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0, 1.0, REACH, width / height]


class Holder:
    """A server with its tickets' scenes, closed with the state."""

    def __init__(self, slots: int, scenes: list[str]):
        self.server = K.Server(0, slots=slots)
        self.ids = [self.server.add_scene(world(s)) for s in scenes]

    def __del__(self):
        try:
            self.server.close()
        except Exception:
            pass


SERVED = ["serve_256", "serve_1024", "serve_4096"]


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "extend":
        base = world(case["scene"])
        rays = _rays(base.scene, case["rays"], rng)
        state = {"case": case, "backend": base.share(), "rays": rays}
        if case["on_device"]:
            state["rays"] = torch.from_numpy(rays.view(np.uint8).reshape(case["rays"], -1)).cuda()
            state["hits"] = torch.zeros(case["rays"], K.HIT_DTYPE.itemsize // 4, dtype=torch.float32, device="cuda")
            state["stream"] = torch.cuda.Stream()
        return state
    if kind in ("frame", "guided"):
        base = world(case["scene"])
        b = base.share()
        b.upload("shot.camera", _camera(base.scene, rng))
        state = {"case": case, "backend": b, "seed": int(rng.integers(1, 1 << 30))}
        if kind == "guided":
            lo = np.asarray(base.scene.region_lower, np.float64)
            state["guide"] = _guide(case["table_log2"], rng, lo, lo + np.asarray(base.scene.region_size, np.float64), True)
            b.set_guide(state["guide"], 0.5, K.GUIDE_SAMPLE)
        return state
    if kind == "serve":
        requests = []
        for k in range(case["requests"]):
            # the serving mix: 30% interactive session frames, stills of the mix's smaller sizes
            if k % 3 == 2:
                requests.append(dict(scene=k % 3, width=1280, height=720, samples=1, denoise=True, interactive=True, session=k + 1))
            else:
                w, h = [(320, 240), (640, 480)][k % 2]
                requests.append(dict(scene=(k + 1) % 3, width=w, height=h, samples=[1, 4, 16, 4, 1][k % 5]))
            requests[-1]["seed"] = int(rng.integers(1, 1 << 30))
        return {"case": case, "holder": Holder(case["slots"], SERVED), "requests": requests}
    if kind == "gradients":
        return {"case": case, "guide": _guide(case["table_log2"], rng, *UNIT, False), "rows": _guide_rows(*UNIT, case["rows"], rng, 10)}
    if kind == "query":
        return {"case": case, "guide": _guide(case["table_log2"], rng, *UNIT, False), "rows": _guide_rows(*UNIT, case["rows"], rng, 6)}
    w, h = case["width"], case["height"]
    lens = _lens(w, h)
    f = K.DenoiseFrame(w, h, 1 if case["demodulated"] else 0, 0)
    for k in range(3):
        f.eye[k], f.forward[k], f.right[k], f.up[k] = lens[k], lens[3 + k], lens[6 + k], lens[9 + k]
    f.reach, f.aspect = lens[12], lens[13]
    return {"case": case, "backend": world("c1").share(), "frame": f, "features": _features(w, h, seed), "out": torch.zeros(h, w, 3, device="cuda"),
            "stream": torch.cuda.Stream()}


# ---- one pass ----

HIT_FIELDS = ("kind", "distance", "point", "normal", "leaf", "other", "share")


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "extend":
        b = state["backend"]
        if case["on_device"]:
            hits = state["hits"]
            b._check(b.lib.kdn_extend_device(b.handle, ctypes.c_void_p(state["rays"].data_ptr()), case["rays"], ctypes.c_void_p(hits.data_ptr()),
                                             ctypes.c_void_p(state["stream"].cuda_stream)))
            whole = hits.view(torch.int32)
            return {"kind": whole[:, 0], "distance": hits[:, 1], "point": hits[:, 2:5], "normal": hits[:, 5:8], "leaf": whole[:, 8], "other": whole[:, 9], "share": hits[:, 10]}
        hits = b.extend(state["rays"])
        return {name: hits[name] for name in HIT_FIELDS}
    if kind in ("frame", "guided"):
        return state["backend"].render(case["width"], case["height"], case["samples"], surfaces=case["surfaces"], seed=state["seed"], denoise=case.get("denoise", False),
                                       sobol=case.get("sobol", False), factor=case.get("factor", 1), phase=case.get("phase", 0))
    if kind == "serve":
        server, ids = state["holder"].server, state["holder"].ids
        tickets = []
        for r in state["requests"]:
            r = dict(r, scene=ids[r["scene"]])
            tickets.append(server.submit(surfaces=8, **r))
        images = []
        for t in tickets:
            status, _, image = server.wait(t)
            if status != K.KDN_OK:
                raise RuntimeError(f"a request ended with status {status}")
            images.append(image)
        return images
    if kind == "gradients":
        loss, dw, dt = state["guide"].gradients(state["rows"])
        return {"loss": loss, "weights": dw, "table": dt}
    if kind == "query":
        return state["guide"].query(state["rows"])
    b, t = state["backend"], state["features"]
    b._check(b.lib.kdn_denoise_device(b.handle, ctypes.byref(state["frame"]), *[ctypes.c_void_p(t[k].data_ptr()) for k in
                                      ("colour", "moment", "length", "distance", "normal", "albedo", "leaf")], ctypes.c_void_p(state["out"].data_ptr()),
                                      ctypes.c_void_p(state["stream"].cuda_stream)))
    return state["out"]


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "extend":
        n = case["rays"]
        return {"bytes": n * (36 + 56), "flops": n * 2 * 230}
    if kind in ("frame", "guided"):
        px = case["width"] * case["height"]
        drawn = px // case.get("factor", 1) ** 2 * case["samples"]
        return {"bytes": 12 * px, "flops": 2.0 * drawn * STEPS_A_SAMPLE.get(case["scene"], STEPS_ELSE) + (drawn * 3.0 * 28672 * 0.5 if kind == "guided" else 0)}
    if kind == "serve":
        shown = [1280 * 720 if k % 3 == 2 else [320 * 240, 640 * 480][k % 2] for k in range(case["requests"])]
        samples = sum(n * (1 if k % 3 == 2 else [1, 4, 16, 4, 1][k % 5]) for k, n in enumerate(shown))
        return {"bytes": 12 * sum(shown), "flops": 2.0 * samples * STEPS_ELSE}
    if kind == "gradients":
        return {"bytes": case["rows"] * 40 + 4 * (14336 * 2 + (32 << case["table_log2"])) + (64 << case["table_log2"]), "flops": 3.0 * 28672 * case["rows"]}
    if kind == "query":
        return {"bytes": case["rows"] * (24 + 160) + 28672, "flops": 28672.0 * case["rows"]}
    px = case["width"] * case["height"]
    return {"bytes": px * (12 + 4 + 4 + 2 + 6 + 6 + 4 + 12), "flops": px * 4 * 25 * 40.0}


# ---- in 64 bits ----

RESOLUTIONS = [16, 22, 30, 42, 58, 80, 111, 153, 212, 294, 406, 561, 776, 1072, 1482, 2048]


def _guide_outputs(rows: torch.Tensor, w: torch.Tensor, table: torch.Tensor, log2: int, lo, hi) -> torch.Tensor:
    """The 48 outputs of the guide's network: a hash grid of the position
    (Mueller et al. 2022) into 48-64-64-64-48 with ReLUs."""
    dev = rows.device
    u = ((rows[:, 0:3] - torch.as_tensor(lo, device=dev)) / torch.as_tensor(hi - lo, device=dev)).clamp(0, 1)
    table = table.reshape(16, 1 << log2, 2)
    feats = []
    for level, n in enumerate(RESOLUTIONS):
        x = u * n
        c0 = x.floor().clamp(max=n - 1)
        f = x - c0
        c0 = c0.long()
        dense = (n + 1) ** 3 <= 1 << log2
        total = 0
        for c in range(8):
            o = [(c >> a) & 1 for a in range(3)]
            g = [c0[:, a] + o[a] for a in range(3)]
            i = g[0] + (n + 1) * (g[1] + (n + 1) * g[2]) if dense else (g[0] ^ (g[1] * 2654435761) ^ (g[2] * 805459861)) & ((1 << log2) - 1)
            weight = 1.0
            for a in range(3):
                weight = weight * (f[:, a] if o[a] else 1 - f[:, a])
            total = total + weight[:, None] * table[level][i]
        feats.append(total)
    ones = torch.ones(len(rows), 1, dtype=torch.float64, device=dev)
    x = torch.cat(feats + [rows[:, 3:6], ones, torch.zeros(len(rows), 12, dtype=torch.float64, device=dev)], dim=1)
    at = 0
    for layer, (n, k) in enumerate([(64, 48), (64, 64), (64, 64), (48, 64)]):
        x = x @ w[at:at + n * k].reshape(n, k).T
        at += n * k
        if layer < 3:
            x = x.relu()
    return x


def _mixture(out: torch.Tensor):
    o = out[:, :40].reshape(-1, 8, 5)
    mean = o[:, :, 2:5]
    return torch.softmax(o[:, :, 0], dim=1), o[:, :, 1].clamp(-2, 8).exp(), mean / mean.norm(dim=2, keepdim=True)


def _exact_guide(case: dict, seed: int):
    rng = np.random.default_rng(seed)
    w, t = _guide_params(case["table_log2"], 14336, rng)
    gradients = case["kind"] == "gradients"
    rows = torch.from_numpy(_guide_rows(*UNIT, case["rows"], rng, 10 if gradients else 6)).double().cuda()
    w, t = torch.from_numpy(w).double().cuda(), torch.from_numpy(t).double().cuda()
    if not gradients:
        with torch.no_grad():
            share, kappa, mean = _mixture(_guide_outputs(rows, w, t, case["table_log2"], *UNIT))
        return torch.cat([share[..., None], kappa[..., None], mean], dim=2).reshape(-1, 40)
    w.requires_grad_(True)
    t.requires_grad_(True)
    loss = 0.0
    for part in rows.split(1 << 15):
        share, kappa, mean = _mixture(_guide_outputs(part, w, t, case["table_log2"], *UNIT))
        cosine = (mean * part[:, None, 6:9]).sum(2)
        density = kappa.log() - math.log(2 * math.pi) - torch.log1p(-torch.exp(-2 * kappa)) + kappa * (cosine - 1)
        each = -(part[:, 9] * torch.logsumexp(share.log() + density, dim=1)).sum() / len(rows)
        each.backward()
        loss += float(each.detach())
    return {"loss": np.float64(loss), "weights": w.grad, "table": t.grad}


def _shifted(a: torch.Tensor, i: int, j: int) -> torch.Tensor:
    """a at (x + i, y + j), zero outside."""
    h, w = a.shape[:2]
    out = torch.zeros_like(a)
    if abs(i) < w and abs(j) < h:
        out[max(0, -j):h - max(0, j), max(0, -i):w - max(0, i)] = a[max(0, j):h - max(0, -j), max(0, i):w - max(0, -i)]
    return out


def _exact_denoise(case: dict, seed: int):
    """The SVGF-like filter as the reference's denoisedFrame states it."""
    w, h = case["width"], case["height"]
    f = {k: (v if k == "leaf" else v.double()) for k, v in _features(w, h, seed).items()}
    lens = torch.tensor(_lens(w, h), dtype=torch.float64, device="cuda")
    luma = lambda c: 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]  # noqa: E731
    sky = (f["leaf"] < 0) | ~torch.isfinite(f["distance"])
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64) + 0.5, torch.arange(w, device="cuda", dtype=torch.float64) + 0.5, indexing="ij")
    side = lens[12] * lens[13]
    heading = lens[3:6] + lens[6:9] * (side * (2 * x / w - 1))[..., None] + lens[9:12] * (lens[12] * (1 - 2 * y / h))[..., None]
    heading = heading / heading.norm(dim=2, keepdim=True)
    distance = torch.where(sky, 0.0, f["distance"])
    point = heading * distance[..., None]
    normal = torch.where(sky[..., None], 0.0, f["normal"])
    offset = (point * normal).sum(2)
    near = torch.where(sky, 0.0, 1 / (0.02 * distance.clamp(min=1e-9)))
    divisor = torch.where(f["albedo"] < 1e-3, 1.0, f["albedo"])
    by = torch.ones_like(divisor) if case["demodulated"] else divisor
    light = f["colour"] / by
    spread = (f["moment"] - luma(f["colour"]) ** 2).clamp(min=0)
    variance = torch.where(f["length"] >= 4, spread / (f["length"] * luma(by) ** 2), -1.0)
    inside = torch.ones(h, w, dtype=torch.float64, device="cuda")
    skyf = sky.double()

    def quick(v):  # 2^(v log2 e), the mantissa from the fitted quadratic
        e = v.clamp(min=-30) * 1.44269504
        part = e - e.floor()
        return torch.where(v > -30, (1 + part * (0.66023 + part * 0.33977)) * torch.exp2(e.floor()), 0.0)

    def weight(i, j, lum, plane, dev):
        facing = (normal * _shifted(normal, i, j)).sum(2) + skyf * _shifted(skyf, i, j)
        power = torch.where(facing > 0.5, facing, 0.0) ** 128
        away = ((_shifted(point, i, j) * normal).sum(2) - offset).abs() * plane
        return _shifted(inside, i, j) * power * quick(-away - (_shifted(lum, i, j) - lum).abs() * dev)

    lum = luma(light)
    s, q, n = 0, 0, 0
    for j in range(-3, 4):
        for i in range(-3, 4):
            k = weight(i, j, lum, near, 0.0)
            s, q, n = s + k * _shifted(lum, i, j), q + k * _shifted(lum, i, j) ** 2, n + k
    some = n > 0
    n = torch.where(some, n, 1.0)
    variance = torch.where(variance < 0, torch.where(some, (q / n - (s / n) ** 2).clamp(min=0), 0.0), variance)
    spline, gauss = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16], [0.25, 0.5, 0.25]
    for step in (1, 2, 4, 8):
        lum = luma(light)
        vs, vw = 0, 0
        for j in range(3):
            for i in range(3):
                k = gauss[i] * gauss[j]
                vs, vw = vs + k * _shifted(variance, i - 1, j - 1), vw + k * _shifted(inside, i - 1, j - 1)
        dev = 1 / (4 * (vs / vw).sqrt() + 1e-4 + 1e-3 * lum)
        c, v, n = 0, 0, 0
        for j in range(-2, 3):
            for i in range(-2, 3):
                k = weight(i * step, j * step, lum, near / step, dev) * (spline[i + 2] * spline[j + 2])
                c, v, n = c + k[..., None] * _shifted(light, i * step, j * step), v + k * k * _shifted(variance, i * step, j * step), n + k
        some = n > 0
        n = torch.where(some, n, 1.0)
        light = torch.where(some[..., None], c / n[..., None], light)
        variance = torch.where(some, v / n ** 2, variance)
    share = (1 / (1 + f["length"] / 8))[..., None]
    held = f["colour"] * divisor if case["demodulated"] else f["colour"]
    return light * divisor * share + held * (1 - share)


def exact(case: dict, seed: int):
    if case["kind"] in ("gradients", "query"):
        return _exact_guide(case, seed)
    if case["kind"] == "denoise":
        return _exact_denoise(case, seed)
    return None
