"""Programs whose minimum, maximum or smooth minimum joins a slab, a sphere or a
box with a coordinate itself (a half-space through the origin): the coordinate
is the point's at whichever way a ray is marched.

On the host a turn's steps against a plain double evaluation, within 3.1e-5
(test_fused_march.py has the bound).  On the device many rays a warp, marched a
step a turn, against few, marched by all lanes: equal to the bit; and every hit
lies on the surface.  A march lands below a tolerance of 2e-6 (coordinates are
below 4), and o + d * t is rounded to 2^-24 of values below 8, so a hit's value
in double is within 3e-6 of zero and FP32's bound above: 4e-5."""
import numpy as np
import pytest

from helpers import host_backend
from test_fused_march import Program
from test_march_form import MAX, MIN, NEG, PX, SMIN, SUB, evaluate

import kodanuki_gb300 as K
from kodanuki_gb300.scene import STEP_DTYPE


def half_ball(p):
    p.op(MAX, p.sphere((0.1, -0.2, 0.05), 0.6), p.op(PX + 2))


def wedge(p):
    p.op(MAX, p.op(MAX, p.op(PX), p.op(PX + 2)), p.sphere((0.0, 0.0, 0.0), 0.8))


def cut_slab(p):
    p.op(MAX, p.op(MAX, p.slab(0, 0.1, 0.2), p.op(PX + 1)), p.sphere((0.0, 0.0, 0.0), 0.9))


def ground(p):
    p.op(MIN, p.op(PX + 2), p.box((0.1, 0.2, 0.3), (0.3, 0.2, 0.4), 0.05))


def blended(p):
    p.op(SMIN, p.slab(0, 0.1, 0.2), p.op(PX + 1), p.const(0.3))


def joined_after(p):  # a primitive, its maximum with a coordinate, then another primitive
    a = p.op(MAX, p.box((-0.3, 0.0, 0.1), (0.2, 0.3, 0.4), 0.02), p.op(NEG, p.op(PX + 1)))
    p.op(MIN, p.op(MAX, p.sphere((0.5, 0.1, 0.0), 0.4), p.op(PX)), a)


SHAPES = [half_ball, wedge, cut_slab, ground, blended, joined_after]


def world(b, shape):
    p = Program()
    shape(p)
    steps = np.array(p.steps, STEP_DTYPE)
    refs = np.zeros(1, K.PROGRAM_REF_DTYPE)
    refs[0] = (0, len(steps), len(steps) - 1)
    region = np.zeros(1, K.REGION_DTYPE)
    region["lower"], region["size"] = -2.0, 4.0
    for block, value in (("scene.steps", steps), ("scene.programs", refs), ("scene.leaves", np.zeros(1, np.uint32)), ("geometry.region", region)):
        b.upload(block, value)
    return steps


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("build", [(0, 0, 1 << 30), (3, 3, 1 << 30)], ids=["whole", "level3"])
def test_a_turns_steps_match_programs(shape, build):
    rng = np.random.default_rng(4)
    b = host_backend()
    checked = 0
    try:
        world(b, shape)
        b.build(*build)
        for i in range(b.world_stats()["cells"]):
            level, place, _, kept = b.world_cell(i)
            if not kept:
                continue
            side = 4.0 / (1 << level)
            pts = (-2.0 + side * (np.array(place) + rng.random((24, 3)))).astype(np.float32)
            got = b.world_march(i, pts)
            if got.shape[0] == 0:
                continue
            _, result, cut = kept[0]
            want = evaluate(cut, int(result), pts.astype(np.float64))
            assert np.abs(got[0] - want).max() <= 3.1e-5
            checked += len(pts)
    finally:
        b.close()
    assert checked >= 24


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_many_rays_hit_where_few_do(shape):
    rng = np.random.default_rng(5)
    n = 200_000  # tens of rays a warp
    rays = np.zeros(n, K.RAY_DTYPE)
    o = rng.normal(size=(n, 3))
    o *= 1.7 / np.linalg.norm(o, axis=1, keepdims=True)
    d = rng.uniform(-0.6, 0.6, (n, 3)) - o
    rays["origin"], rays["direction"] = o, d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["far"], rays["within"] = np.inf, 0xFFFFFFFF
    with K.Backend(0) as b:
        steps = world(b, shape)
        rays["inside"] = evaluate(steps, len(steps) - 1, rays["origin"].astype(np.float64)) < 0
        b.build(0, 0, 1 << 30)
        many = b.extend(rays)
        few = np.concatenate([b.extend(rays[k:k + 500]) for k in range(0, 5000, 500)])
    assert many[:5000].tobytes() == few.tobytes()
    at = many["point"][many["kind"] == 1].astype(np.float64)
    assert len(at) > n // 10
    assert np.abs(evaluate(steps, len(steps) - 1, at)).max() <= 4e-5
