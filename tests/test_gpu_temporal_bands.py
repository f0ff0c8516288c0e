"""The temporal member's plane tests near their thresholds, against the oracle,
which works in double: whichever of FP32 and double answers a test, it is
double's answer.  Of unit normals, and of normals a thousand long (the buffers
are a caller's), whose dots cancel and whose offsets FP32 knows a thousand times
less well.  A test answered otherwise takes a pixel's history from other pixels,
whose lengths are other whole numbers: the length tells (a bilinear blend, FP32
against double: 1e-5)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 256, 192
REACH, DEPTH_SHARE, COSINE, BAND = 0.42, 0.03, 0.9, 1e-5


def lens(eye):
    return np.array([*eye, 0, 0, -1, 1, 0, 0, 0, 1, 0, REACH, W / H], np.float64)


def half(a):
    return np.asarray(a, np.float32).astype(np.float16).astype(np.float32)


def headings():
    y, x = np.mgrid[0:H, 0:W]
    return np.stack([(2 * (x + 0.5) / W - 1) * REACH * W / H, (1 - 2 * (y + 0.5) / H) * REACH, -np.ones((H, W))], axis=-1).reshape(-1, 3)


def near_unit(rng, n):
    """Unit normals, some 0.9 alike, and points up to 1 apart."""
    a = rng.normal(size=(n, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(a, rng.normal(size=(n, 3)))
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    cosine = np.where(rng.random(n) < 0.5, rng.uniform(0.88, 0.92, n), rng.uniform(0.95, 1.0, n))[:, None]
    return half(a), half(cosine * a + np.sqrt(1 - cosine ** 2) * b), half(rng.uniform(5, 6, n)), half(rng.uniform(5, 6, n)), rng.normal(size=3) * 0.02


def near_long(rng, n):
    """Normals 1000 long: alike, with the eye moved by some 6e-5 of a distance;
    and such whose dots are the few tenths that two millions leave."""
    a = rng.normal(size=(n, 3))
    a *= 1000.0 / np.linalg.norm(a, axis=1, keepdims=True)
    b = a.copy()
    odd = rng.random(n) < 0.3
    a[odd] = [1.0, 1000.0, 1000.0]
    b[odd] = np.stack([half(rng.uniform(0.85, 0.95, odd.sum())), np.full(odd.sum(), 1000.0), np.full(odd.sum(), -1000.0)], axis=1)
    d = half(rng.uniform(5, 6, n))
    return half(a), half(b), d, d, rng.normal(size=3) * 2e-4


@pytest.mark.parametrize("make", [near_unit, near_long])
@pytest.mark.parametrize("seed", [1, 2])
def test_plane_tests_near_their_thresholds_are_doubles(make, seed):
    import torch
    import kodanuki_gb300 as K
    import oracle.port as op
    rng = np.random.default_rng(seed)
    n = W * H
    normal, last_normal, distance, last_distance, shift = make(rng, n)
    eye = np.array([0.3, -0.2, 10.0])
    now, before = lens(eye), lens(eye + shift)
    light = half(rng.uniform(0.1, 2.0, (n, 3)))
    ones, leaf = np.ones((n, 3), np.float32), np.full(n, 3, np.uint32)
    surface = {"distance": distance, "normal": normal, "leaf": leaf, "albedo": ones}
    state = np.zeros(n, op.TPIXEL_DTYPE)
    state["colour"], state["moment"] = half(rng.uniform(0.1, 2.0, (n, 3))), 1.0
    state["length"], state["distance"], state["normal"], state["leaf"], state["albedo"] = rng.integers(1, 200, n), last_distance, last_normal, leaf, 1.0
    want, _ = op.temporal(W, H, True, False, True, now, before, light, surface, surface, state)

    # the inputs do come near: of a pixel's own place in the frame before
    h = headings()
    unit = h / np.linalg.norm(h, axis=1, keepdims=True)
    n64, l64 = normal.astype(np.float64), last_normal.astype(np.float64)
    alike = (n64 * l64).sum(axis=1)
    off = np.abs(((shift + unit * last_distance[:, None] - unit * distance[:, None]) * n64).sum(axis=1))
    scale = 1.0 if make is near_unit else 1e3
    assert (np.abs(alike - COSINE) < BAND * scale ** 2).any()
    assert ((alike > COSINE) & (np.abs(off - DEPTH_SHARE * distance) < BAND * scale * 2 * distance)).any()

    dev = torch.device("cuda:0")
    keep, bufs = [], K.TemporalBuffers()

    def bind(name, a, bits=None):
        t = torch.from_numpy(np.ascontiguousarray(a) if bits is None else np.ascontiguousarray(np.asarray(a, np.float32).astype(np.float16)).view(np.int16)).to(dev)
        keep.append(t)
        setattr(bufs, name, t.data_ptr())
        return t

    bind("light", light)
    for prefix in ("first", "centre"):
        bind(f"{prefix}_distance", distance, 16)
        bind(f"{prefix}_normal", normal, 16)
        bind(f"{prefix}_albedo", ones, 16)
        bind(f"{prefix}_leaf", leaf.view(np.int32))
    bind("before_colour", state["colour"].astype(np.float32))
    bind("before_moment", state["moment"].astype(np.float32))
    bind("before_length", state["length"])
    bind("before_distance", last_distance, 16)
    bind("before_normal", last_normal, 16)
    bind("before_leaf", leaf.view(np.int32))
    length = bind("length", np.zeros(n, np.float32))
    for name, size in (("colour", 3 * n), ("moment", n), ("image", 3 * n)):
        bind(name, np.zeros(size, np.float32))
    fr = K.TemporalFrame(W, H, 1, 0, 1, 1, 0, 1, 0)
    for k in range(14):
        fr.now[k], fr.before[k] = float(now[k]), float(before[k])
    with K.Backend(0) as b:
        b._check(b.lib.kdn_temporal_device(b.handle, ctypes.byref(fr), ctypes.byref(bufs), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
    got = length.cpu().numpy().astype(np.float64)
    apart = np.abs(got - want["length"]) > 1e-5 * np.maximum(want["length"], 1.0)
    assert not apart.any(), f"{apart.sum()} of {n} pixels"
