"""Marches of many small steps on the device against the same march in numpy's
FP32: rays that skim a plane for up to the 65536-step cap, and rays far from
their start whose steps over it become too small to move them, which end as
capped misses.  One cell (no octree), so a step is the plane's height alone;
every operation is rounded once, the multiply-add through double."""
import numpy as np
import pytest

from helpers import host_backend  # noqa: F401  (the tests' path)
from test_fused_march import Program

pytestmark = pytest.mark.gpu

CAP = 1 << 16
f32 = np.float32


def marched(o, d, size):
    """(kind, distance) of a ray over the plane z = 0 in one cell [-size/2, size/2)."""
    t = f32(0)
    up = np.inf
    for a in range(3):
        inv = f32(1) / (d[a] if abs(d[a]) >= f32(1e-12) else np.copysign(f32(1e-12), d[a]))
        up = min(up, max((f32(-size / 2) - o[a]) * inv, (f32(size / 2) - o[a]) * inv))
    step = 0
    while step < CAP and t <= up:
        p = [f32(np.float64(d[a]) * np.float64(t) + np.float64(o[a])) for a in range(3)]
        step += 1
        tol = f32(2e-6) * max(f32(1), max(abs(x) for x in p) * f32(0.25))
        if p[2] < tol:
            return 1, t
        on = min(t + p[2], max(f32(up), t) + max(f32(1e-5), abs(t) * f32(2e-6)))
        if on == t:
            return 0, t
        t = on
    return 0, t


def test_skimming_and_standing_rays_match_fp32():
    import kodanuki_gb300 as K
    from kodanuki_gb300.scene import STEP_DTYPE
    size = 512.0
    rng = np.random.default_rng(5)
    p = Program()
    p.op(2 + 2)  # the point's z
    p.op(9, 0, p.const(0.0))
    steps = np.zeros(len(p.steps), STEP_DTYPE)
    for k, s in enumerate(p.steps):
        steps[k] = s
    refs = np.zeros(1, K.PROGRAM_REF_DTYPE)
    refs[0] = (0, len(steps), len(steps) - 1)
    region = np.zeros(1, K.REGION_DTYPE)
    region["lower"], region["size"] = -size / 2, size
    n = 160
    rays = np.zeros(n, K.RAY_DTYPE)
    for i in range(n):
        if i % 4 == 0:  # skims: a small height, hardly any slope (capped, leaving, or landing)
            rays["origin"][i] = (-200, 0, 10 ** rng.uniform(-3.5, -1))
            d = np.array([1, 0.2, rng.choice([-1, 1]) * 10 ** rng.uniform(-8, -4)])
        else:  # from afar to about the origin, where a step may be too small to move it
            d = np.array([0.6, rng.uniform(-0.2, 0.2), -0.8])
            d /= np.linalg.norm(d)
            rays["origin"][i] = rng.uniform(-1, 1, 3) * (1, 1, 0) - d * rng.uniform(110, 250)
        rays["direction"][i] = d / np.linalg.norm(d)
    rays["far"] = np.inf
    rays["within"] = 0xFFFFFFFF
    with K.Backend(0) as b:
        for name, block in (("scene.steps", steps), ("scene.programs", refs), ("scene.leaves", np.zeros(1, np.uint32)), ("geometry.region", region)):
            b.upload(name, block)
        b.build(0, 0, 1 << 30)
        hits = b.extend(rays)
    with np.errstate(all="ignore"):
        want = [marched(r["origin"], r["direction"], size) for r in rays]
    kinds = np.array([k for k, _ in want])
    assert np.array_equal(hits["kind"], kinds)
    landed = kinds == 1
    assert landed.any() and (~landed[np.arange(n) % 4 != 0]).any(), "some land and some stand"
    assert np.array_equal(hits["distance"][landed], np.array([t for _, t in want], np.float32)[landed])
