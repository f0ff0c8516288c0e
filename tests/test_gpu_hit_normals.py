"""Normals of hits on programs of each operation the hit kernel's common stretch
holds, and of some it does not, against central differences of the program in
double.

At a point where the gradient is smooth (the same to 4e-3 at 1e-3 around it) a
hit point off by the tolerance, some 1e-5, and FP32's roundings of a few dozen
steps move it by less than 1e-3."""
import numpy as np
import pytest

from test_fused_march import Program
from test_march_form import ABS, ADD, MAX, MIN, MUL, NEG, POSSQ, PX, SMIN, SQRT, SUB, evaluate

pytestmark = pytest.mark.gpu


def made(name):
    p = Program()
    if name == "slab":
        p.op(MAX, p.slab(0, 0.1, 0.4), p.op(MAX, p.slab(1, -0.1, 0.5), p.slab(2, 0.0, 0.6)))
    elif name == "negative":
        p.op(MAX, p.slab(2, 0.3, 0.2, negative=True), p.sphere((0.0, 0.0, 0.0), 0.8))
    elif name == "sphere":
        p.sphere((0.1, -0.2, 0.05), 0.7)
    elif name == "box":
        p.box((0.05, 0.0, -0.1), (0.5, 0.4, 0.3), 0.1)
    elif name == "product":
        p.op(MUL, p.op(NEG, p.op(NEG, p.sphere((0.0, 0.1, 0.0), 0.6))), p.op(ADD, p.const(0.5), p.op(MUL, p.op(PX), p.const(0.05))))
    elif name == "least":
        p.op(MIN, p.sphere((0.4, 0.0, 0.0), 0.5), p.op(MIN, p.sphere((-0.4, 0.0, 0.0), 0.5), p.box((0.0, 0.0, 0.0), (0.2, 0.2, 0.8), 0.05)))
    elif name == "smooth":
        p.op(SMIN, p.sphere((0.35, 0.0, 0.0), 0.4), p.box((-0.3, 0.0, 0.0), (0.3, 0.3, 0.3), 0.05), p.const(0.3))
    elif name == "repeated":
        p.op(MAX, p.op(SUB, p.op(ABS, p.repeated(0, 0.1, 0.5)), p.const(0.1)), p.sphere((0.0, 0.0, 0.0), 0.9))
    else:  # a cone of positive parts, part by part
        q = [p.op(POSSQ, p.op(SUB, p.op(ABS, p.op(PX + k)), p.const(0.3))) for k in range(3)]
        p.op(SUB, p.op(SQRT, p.op(ADD, p.op(ADD, q[0], q[1]), q[2])), p.const(0.2))
    return p


@pytest.mark.parametrize("name", ["slab", "negative", "sphere", "box", "product", "least", "smooth", "repeated", "parts"])
def test_normals_match_central_differences(name):
    import kodanuki_gb300 as K
    from kodanuki_gb300.scene import STEP_DTYPE
    p = made(name)
    steps = np.zeros(len(p.steps), STEP_DTYPE)
    for k, s in enumerate(p.steps):
        steps[k] = s
    refs = np.zeros(1, K.PROGRAM_REF_DTYPE)
    refs[0] = (0, len(steps), len(steps) - 1)
    region = np.zeros(1, K.REGION_DTYPE)
    region["lower"], region["size"] = -4.0, 8.0
    rng = np.random.default_rng(3)
    n = 1000
    rays = np.zeros(n, K.RAY_DTYPE)
    o = rng.normal(size=(n, 3))
    o *= 3.0 / np.linalg.norm(o, axis=1, keepdims=True)
    d = rng.uniform(-0.6, 0.6, (n, 3)) - o
    rays["origin"], rays["direction"] = o, d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["far"], rays["within"] = np.inf, 0xFFFFFFFF
    with K.Backend(0) as b:
        for block, value in (("scene.steps", steps), ("scene.programs", refs), ("scene.leaves", np.zeros(1, np.uint32)), ("geometry.region", region)):
            b.upload(block, value)
        b.build(0, 0, 1 << 30)
        hits = b.extend(rays)
    d, hits = rays["direction"][hits["kind"] == 1], hits[hits["kind"] == 1]

    def gradient(at):
        g = np.stack([evaluate(steps, len(steps) - 1, at + e) - evaluate(steps, len(steps) - 1, at - e) for e in 1e-6 * np.eye(3)], axis=1)
        return g / np.linalg.norm(g, axis=1, keepdims=True)

    at = hits["point"].astype(np.float64)
    with np.errstate(all="ignore"):
        want = gradient(at)
        smooth = (want * d).sum(axis=1) < -0.01  # a grazing hit's normal is turned to the ray
        for e in 1e-3 * np.concatenate([np.eye(3), -np.eye(3)]):
            smooth &= np.abs(gradient(at + e) - want).max(axis=1) < 4e-3
    assert smooth.sum() > 50
    assert np.abs(hits["normal"][smooth] - want[smooth]).max() < 1e-3
