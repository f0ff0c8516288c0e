"""Frames of more chunks than there are lanes: groups of chunks one after the
other, a last group that is partly empty, and lanes whose chunks end at
different rounds (bodies that scatter hold some chunks' paths far longer than
others'), are the frame drawn in one group, to the bit.

A chunk is at least 65536 / 4 paths, which the smaller budget asks for: 2048
pixels of 8 samples.  Each chunk launches its camera, a trace, hits, a shading
and its fold at least."""
import numpy as np
import pytest

from helpers import scene

pytestmark = pytest.mark.gpu

WIDTH, HEIGHT, SAMPLES, LANES = 320, 208, 8, 4
PATH_BYTES = 420


@pytest.mark.parametrize("name", ["c1_small", "scatter_small", "glass_small"])
@pytest.mark.parametrize("march_budget", [0, 16])
def test_frames_in_groups_of_chunks_equal_frames_in_one(name, march_budget):
    import kodanuki_gb300 as K
    sc = scene(name)
    with K.Backend(0) as b:
        b.load(sc)
        b.build(5, 10, 64)
        b.set_march_budget(march_budget)
        whole = b.render(WIDTH, HEIGHT, SAMPLES, surfaces=8, seed=3)
        launches = b.frame_stats().launches
        for paths in (65536, 100_000):
            b.set_frame_budget(paths * PATH_BYTES)
            assert np.array_equal(b.render(WIDTH, HEIGHT, SAMPLES, surfaces=8, seed=3), whole)
            chunks = -(-WIDTH * HEIGHT // -(-(paths // LANES) // SAMPLES))
            assert chunks > LANES and chunks % LANES != 0
            assert b.frame_stats().launches > launches
            assert b.frame_stats().launches >= 5 * chunks
