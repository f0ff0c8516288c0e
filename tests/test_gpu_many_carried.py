"""Carried marches are counted one by one however many of them one warp has: a
frame on one SM, whose 16 warps carry some 80 000 rays each in a launch, counts
what the frame on all SMs counts."""
import numpy as np
import pytest

from helpers import scene

pytestmark = pytest.mark.gpu


def test_counts_of_carried_rays_do_not_depend_on_the_warps():
    import kodanuki_gb300 as K
    sc = scene("c1_small")
    with K.Backend(0) as b:
        b.load(sc)
        b.build(5, 10, 64)
        b.set_march_budget(1)
        whole = b.render(1024, 1024, 5, surfaces=1, seed=3)
        want = b.frame_stats()
        b._check(b.lib.kdn_set_sm_limit(b.handle, 1))
        one = b.render(1024, 1024, 5, surfaces=1, seed=3)
        got = b.frame_stats()
    assert np.array_equal(one, whole)
    assert want.carried_rays > 1024 * 1024 * 5
    assert (got.carried_rays, got.capped_rays) == (want.carried_rays, want.capped_rays)
