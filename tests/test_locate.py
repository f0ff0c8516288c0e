"""Locating a point by the tabled walls, the grid and the bricks below it
(world.h kEntryLeaf) names the leaf the descent from the root names: trees
shallower than the grid, of odd and even depths below it, and deeper than the
tabled walls; and regions so far from the origin that FP32 has room for few
walls, or for none."""
import numpy as np
import pytest

from helpers import host_backend
from test_fused_march import Program

import kodanuki_gb300 as K
from kodanuki_gb300.scene import STEP_DTYPE


@pytest.mark.parametrize("depth", [1, 6, 7, 8, 9, 10, 13])
@pytest.mark.parametrize("lower,size", [(-1.0, 2.0), (1000.0, 2.0), (-61.2, 122.4), (1e6, 1.0)])
def test_locate_names_the_descents_leaf(depth, lower, size):
    p = Program()
    # a ball small enough that its cells at the depth are few
    radius = size * min(0.3, 12.0 / (1 << depth))
    p.sphere([lower + 0.37 * size] * 3, radius)
    steps = np.zeros(len(p.steps), STEP_DTYPE)
    for k, s in enumerate(p.steps):
        steps[k] = s
    refs = np.zeros(1, K.PROGRAM_REF_DTYPE)
    refs[0] = (0, len(steps), len(steps) - 1)
    region = np.zeros(1, K.REGION_DTYPE)
    region["lower"], region["size"] = lower, size
    b = host_backend()
    try:
        for name, block in (("scene.steps", steps), ("scene.programs", refs), ("scene.leaves", np.zeros(1, np.uint32)), ("geometry.region", region)):
            b.upload(name, block)
        b.build(depth, depth, 1 << 30)
        rng = np.random.default_rng(depth)
        lo, sz = np.float64(np.float32(lower)), np.float64(np.float32(size))
        near = lower + 0.37 * size + rng.normal(size=(4000, 3)) * radius
        walls = lo + sz * rng.integers(0, (1 << min(depth, 12)) + 1, (4000, 3)) / (1 << min(depth, 12))
        outside = lo + sz * (rng.random((1000, 3)) * 1.4 - 0.2)
        odd = np.array([[np.nan, lo, lo], [np.inf, -np.inf, lo], [-np.inf] * 3, [3e38] * 3])
        pts = np.concatenate([near, walls, lo + sz * rng.random((4000, 3)), outside, odd]).astype(np.float32)
        located, descended = b.world_locate(pts)
        assert np.array_equal(located, descended)
    finally:
        b.close()
