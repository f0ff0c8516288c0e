"""Which steps of a program the march form makes primitives of (world.h
MarchForm).  A primitive works out three slabs and a root whatever it holds, so
a single step that other forms read (the offset of a turned body, one operation)
stays that step, and a run of steps, or a slab that primitives are joined with,
is one; the values are the programs' either way."""
import os
import subprocess

import numpy as np
import pytest

from helpers import host_backend
from test_fused_march import Program
from test_march_form import ABS, ADD, MAX, MIN, MUL, NEG, POSSQ, PX, SQRT, SUB, evaluate

import kodanuki_gb300 as K
from kodanuki_gb300.scene import STEP_DTYPE

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRIMITIVE, FMA = 16, 0


@pytest.fixture(scope="module")
def forms(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("forms") / "march_forms")
    csrc = os.path.join(ROOT, "kodanuki_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), "-I", csrc, os.path.join(ROOT, "tests", "march_forms.cpp"),
                    os.path.join(csrc, "octree.cpp"), "-lpthread", "-o", out], check=True, capture_output=True, text=True)

    def of(p):
        text = "\n".join(f"{o} {a} {b} {c} {v!r}" for o, a, b, c, v, _ in p.steps)
        r = subprocess.run([out], input=text, capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.split("\n") if line]
    return of


def turned(p, q, rows):
    return [p.op(ADD, p.op(ADD, p.op(MUL, p.const(r[0]), q[0]), p.op(MUL, p.const(r[1]), q[1])), p.op(MUL, p.const(r[2]), q[2])) for r in rows]


ROWS = [(0.8, -0.36, 0.48), (0.6, 0.48, -0.64), (0.0, 0.8, 0.6)]


def half_space(p):
    q = [p.op(SUB, p.op(PX + k), p.const(c)) for k, c in enumerate((0.3, -0.2, 0.1))]
    p.op(SUB, turned(p, q, ROWS[:1])[0], p.const(0.25))


def turned_box(p):
    q = turned(p, [p.op(SUB, p.op(PX + k), p.const(c)) for k, c in enumerate((0.1, 0.2, -0.3))], ROWS)
    q = [p.op(ADD, p.op(SUB, p.op(ABS, q[k]), p.const(0.3)), p.const(0.02)) for k in range(3)]
    total = p.op(ADD, p.op(ADD, p.op(POSSQ, q[0]), p.op(POSSQ, q[1])), p.op(POSSQ, q[2]))
    p.op(SUB, p.op(ADD, p.op(SQRT, total), p.op(MIN, p.op(MAX, q[0], p.op(MAX, q[1], q[2])), p.const(0.0))), p.const(0.02))


def mirrored(p):  # |x - c|, c - y and |z| in products
    a = p.op(ABS, p.op(SUB, p.op(PX), p.const(0.2)))
    b = p.op(SUB, p.const(0.3), p.op(PX + 1))
    c = p.op(ABS, p.op(PX + 2))
    p.op(SUB, p.op(ADD, p.op(MUL, a, a), p.op(ADD, p.op(MUL, b, c), p.op(MUL, a, c))), p.const(0.4))


def joined_in_product(p):  # a maximum of a coordinate and a number, read by a product
    a = p.op(MAX, p.op(PX), p.const(0.3))
    b = p.op(MAX, p.op(SUB, p.op(PX + 1), p.const(0.1)), p.op(PX + 2))
    p.op(SUB, p.op(MUL, a, b), p.const(0.1))


@pytest.mark.parametrize("shape", [half_space, turned_box, mirrored])
def test_single_steps_of_other_forms_are_no_primitives(forms, shape):
    p = Program()
    shape(p)
    kinds = [f for f, _, rare in forms(p)]
    assert PRIMITIVE not in kinds and FMA in kinds


def test_slabs_that_primitives_are_joined_with_are_primitives(forms):
    p = Program()
    p.op(MAX, p.op(SUB, p.op(PX), p.const(0.4)), p.op(MAX, p.op(NEG, p.op(SUB, p.op(PX + 1), p.const(0.2))), p.sphere((0.0, 0.1, 0.2), 0.6)))
    assert {f for f, _, _ in forms(p)} == {PRIMITIVE}


@pytest.mark.parametrize("shape", [half_space, turned_box, mirrored, joined_in_product])
def test_values_are_the_programs(shape):
    """FP32 against double: 64 roundings of values below 8 (test_fused_march.py)."""
    p = Program()
    shape(p)
    steps = np.array(p.steps, STEP_DTYPE)
    refs = np.zeros(1, K.PROGRAM_REF_DTYPE)
    refs[0] = (0, len(steps), len(steps) - 1)
    region = np.zeros(1, K.REGION_DTYPE)
    region["lower"], region["size"] = -1.0, 2.0
    b = host_backend()
    try:
        for name, block in (("scene.steps", steps), ("scene.programs", refs), ("scene.leaves", np.zeros(1, np.uint32)), ("geometry.region", region)):
            b.upload(name, block)
        b.build(0, 0, 1 << 30)
        pts = np.random.default_rng(6).uniform(-1, 1, (4000, 3)).astype(np.float32)
        assert np.abs(b.world_march(0, pts)[0] - evaluate(steps, len(steps) - 1, pts.astype(np.float64))).max() <= 3.1e-5
    finally:
        b.close()
