"""A frame cut into many chunks of paths (kdn_set_frame_budget), whose rounds
end at different times (bodies that scatter hold some chunks' paths far longer
than others'), is the frame drawn in few, to the bit: a path reads nothing of
another's."""
import numpy as np
import pytest

from helpers import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["c1_small", "scatter_small", "glass_small"])
@pytest.mark.parametrize("march_budget", [0, 16])
def test_frames_in_many_chunks_equal_frames_in_few(name, march_budget):
    import kodanuki_gb300 as K
    sc = scene(name)
    w, h, surfaces = int(sc.render["width"]), int(sc.render["height"]), int(sc.render["surfaces"])
    with K.Backend(0) as b:
        b.load(sc)
        b.build(5, 10, 64)
        b.set_march_budget(march_budget)
        whole = b.render(w, h, 8, surfaces=surfaces, seed=3)
        launches = b.frame_stats().launches
        for budget in (1 << 19, 1 << 21):
            b.set_frame_budget(budget)
            assert np.array_equal(b.render(w, h, 8, surfaces=surfaces, seed=3), whole)
        assert b.frame_stats().launches >= launches
