"""A launch's rays, few or many a warp: each ray's hit is the one it has in a
launch of few, whatever shares its warp (a ray's march reads nothing of
another's, so the hits are equal to the bit)."""
import numpy as np
import pytest

from helpers import golden_rays, scene

pytestmark = pytest.mark.gpu

POOL, WARPS = 64, 16  # rays a warp holds, warps an SM


@pytest.fixture(scope="module")
def few():
    import kodanuki_gb300 as K
    b = K.Backend(0)
    b.load(scene("c2"))
    b.build(7, 10, 96)
    rays = golden_rays("c2")[0][:499]
    yield b, rays, b.extend(rays)
    b.close()


@pytest.mark.parametrize("a_warp, more", [(0, 1), (0, 33), (1, 0), (1, 1), (33, -1), (POOL, -1), (POOL, 0), (POOL, 1), (3 * POOL, 7)])
def test_hits_do_not_depend_on_the_launch(few, a_warp, more):
    import torch
    backend, rays, want = few
    n = a_warp * WARPS * torch.cuda.get_device_properties(0).multi_processor_count + more
    at = np.arange(n) * 7 % len(rays)
    assert backend.extend(rays[at]).tobytes() == want[at].tobytes()
