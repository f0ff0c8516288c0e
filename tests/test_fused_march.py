"""The fused steps of the march form (world.h MarchForm) against a plain
double evaluation of the programs they stand for: slabs, spheres, rounded
boxes and a repetition, alone and joined, kept whole (no cut) and cut by the
cells of a small octree, where a box loses axes, its corners and edges square
an axis whole, and an inside term stays or goes.

The tolerance is FP32's: a program of n steps over values below V rounds each
step by at most V * 2^-24 and the root of a sum of squares loses at most the
square root's 2^-22 more (the host's root is correctly rounded), so 64 steps
over |values| < 8 stay within 64 * 8 * 2^-24 = 3.1e-5 away from roots near
zero, where an error e of the sum becomes sqrt(e): the points are kept where
the distance to every centre and edge is above 1e-2, which bounds the root's
amplification by 1 / (2 * 1e-2) of the sum's relative error times its size."""
import numpy as np
import pytest

from helpers import host_backend
from test_march_form import ABS, ADD, CONSTANT, DIV, FLOOR, MAX, MIN, MUL, NEG, POSSQ, PX, SMIN, SQRT, SUB, evaluate

import kodanuki_gb300 as K
from kodanuki_gb300.scene import STEP_DTYPE


class Program:
    def __init__(self):
        self.steps = []

    def op(self, opcode, a=0, b=0, c=0, value=0.0):
        self.steps.append((opcode, a, b, c, value, 0))
        return len(self.steps) - 1

    def const(self, v):
        return self.op(CONSTANT, value=v)

    def sphere(self, centre, radius):
        d = [self.op(SUB, self.op(PX + k), self.const(centre[k])) for k in range(3)]
        y2 = self.op(MUL, d[1], d[1])
        xy = self.op(ADD, self.op(MUL, d[0], d[0]), y2)
        root = self.op(SQRT, self.op(ADD, self.op(MUL, d[2], d[2]), xy))
        return self.op(SUB, root, self.const(radius))

    def box(self, centre, half, round_, axes=3):
        q = []
        for k in range(axes):
            u = self.op(ABS, self.op(SUB, self.op(PX + k), self.const(centre[k])))
            q.append(self.op(ADD, self.op(SUB, u, self.const(half[k])), self.const(round_)))
        total = self.op(POSSQ, q[0])
        for k in range(1, axes):
            total = self.op(ADD, total, self.op(POSSQ, q[k]))
        most = q[-1]
        for k in range(axes - 2, -1, -1):
            most = self.op(MAX, q[k], most)
        inside = self.op(MIN, most, self.const(0.0))
        return self.op(SUB, self.op(ADD, self.op(SQRT, total), inside), self.const(round_))

    def repeated(self, axis, centre, period):
        u = self.op(SUB, self.op(PX + axis), self.const(centre))
        k = self.op(FLOOR, self.op(ADD, self.op(DIV, u, self.const(period)), self.const(0.5)))
        return self.op(SUB, u, self.op(MUL, self.const(period), k))

    def slab(self, axis, centre, half, negative=False):
        u = self.op(SUB, self.op(PX + axis), self.const(centre))
        u = self.op(NEG, u) if negative else self.op(ABS, u)
        return self.op(SUB, u, self.const(half))


def programs():
    out = []
    for axis in range(3):
        p = Program()
        p.slab(axis, 0.3, 0.2)
        out.append(p)
        p = Program()
        p.slab(axis, -0.4, 0.1, negative=True)
        out.append(p)
    p = Program()
    p.sphere((0.1, -0.2, 0.3), 0.5)
    out.append(p)
    for axes in (1, 2, 3):
        p = Program()
        p.box((0.05, -0.1, 0.15), (0.4, 0.3, 0.5), 0.02, axes)
        out.append(p)
    p = Program()  # a union, a smooth union and a cut of the three
    a, b, c = p.sphere((-0.5, 0.1, 0.0), 0.3), p.box((0.3, 0.2, -0.1), (0.2, 0.3, 0.25), 0.05), p.sphere((0.2, -0.5, 0.2), 0.35)
    p.op(SMIN, p.op(MIN, a, b), c, p.const(0.08))
    out.append(p)
    p = Program()
    a, b = p.box((0.0, 0.0, 0.0), (0.5, 0.4, 0.45), 0.03), p.sphere((0.4, 0.3, 0.2), 0.3)
    p.op(MAX, a, p.op(NEG, b))
    out.append(p)
    p = Program()  # balls in a row: a repeated coordinate beside two plain ones
    d = [p.repeated(0, 0.05, 0.4)] + [p.op(SUB, p.op(PX + k), p.const(0.1 * k)) for k in (1, 2)]
    total = p.op(ADD, p.op(MUL, d[2], d[2]), p.op(ADD, p.op(MUL, d[0], d[0]), p.op(MUL, d[1], d[1])))
    p.op(SUB, p.op(SQRT, total), p.const(0.15))
    out.append(p)
    return out


@pytest.mark.parametrize("build", [(0, 0, 1 << 30), (2, 2, 1 << 30), (4, 4, 1 << 30)], ids=["whole", "level2", "level4"])
def test_fused_steps_match_programs(build):
    rng = np.random.default_rng(3)
    checked = 0
    for p in programs():
        steps = np.zeros(len(p.steps), STEP_DTYPE)
        for k, s in enumerate(p.steps):
            steps[k] = s
        refs = np.zeros(1, K.PROGRAM_REF_DTYPE)
        refs[0] = (0, len(steps), len(steps) - 1)
        region = np.zeros(1, K.REGION_DTYPE)
        region["lower"], region["size"] = -1.0, 2.0
        b = host_backend()
        try:
            for name, block in (("scene.steps", steps), ("scene.programs", refs), ("scene.leaves", np.zeros(1, np.uint32)), ("geometry.region", region)):
                b.upload(name, block)
            b.build(*build)
            for i in range(b.world_stats()["cells"]):
                level, place, _, kept = b.world_cell(i)
                if not kept:
                    continue
                side = 2.0 / (1 << level)
                pts = (-1.0 + side * (np.array(place) + rng.random((24, 3)))).astype(np.float32)
                got = b.world_march(i, pts)
                if got.shape[0] == 0:
                    continue
                _, result, cut = kept[0]
                want = evaluate(cut, int(result), pts.astype(np.float64))
                # away from a root of a sum near zero (see above)
                roots = [evaluate(cut[:k + 1], k, pts.astype(np.float64)) for k in range(len(cut)) if cut[k]["opcode"] == SQRT]
                clear = np.all([(r > 1e-2) | (r == 0) for r in roots], axis=0) if roots else np.ones(len(pts), bool)
                # and from a floor's step, where FP32 and double may take either side
                for k in range(len(cut)):
                    if cut[k]["opcode"] == FLOOR:
                        a = evaluate(cut[:k], int(cut[k]["a"]), pts.astype(np.float64))
                        clear &= np.abs(a - np.round(a)) > 1e-5
                assert np.abs(got[0] - want)[clear].max(initial=0.0) <= 3.1e-5
                checked += int(clear.sum())
        finally:
            b.close()
    assert checked >= 200
