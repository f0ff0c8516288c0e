"""A launch's rays, few or many a warp: each ray's hit is the one it has in a
launch of few, which are marched by all of a warp's lanes from registers (a
ray's march reads nothing of another's and every way to march it rounds alike,
so the hits are equal to the bit)."""
import numpy as np
import pytest

from helpers import golden_rays, scene

pytestmark = pytest.mark.gpu

POOL, WARPS = 64, 16  # rays a warp holds, warps an SM


def rays_of(name, sc):
    if name in ("c1", "c2"):
        return golden_rays(name)[0][:499]
    import kodanuki_gb300 as K
    rng = np.random.default_rng(7)
    lo, size = np.asarray(sc.region_lower, np.float32), np.asarray(sc.region_size, np.float32)
    rays = np.zeros(499, K.RAY_DTYPE)
    rays["origin"] = lo + size * rng.uniform(0.3, 0.7, (499, 3)).astype(np.float32)
    d = rng.normal(size=(499, 3))
    rays["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["far"], rays["within"] = np.inf, 0xFFFFFFFF
    return rays


@pytest.fixture(scope="module", params=["c1", "c2", "c5", "patterns_small", "rough_small"])
def few(request):
    import kodanuki_gb300 as K
    sc = scene(request.param)
    b = K.Backend(0)
    b.load(sc)
    b.build(6, 10, 64)
    rays = rays_of(request.param, sc)
    yield b, rays, b.extend(rays)
    b.close()


@pytest.mark.parametrize("a_warp, more", [(0, 1), (1, 1), (5, 0), (33, -1), (POOL, -1), (POOL, 1), (3 * POOL, 7)])
def test_hits_do_not_depend_on_the_launch(few, a_warp, more):
    import torch
    backend, rays, want = few
    n = a_warp * WARPS * torch.cuda.get_device_properties(0).multi_processor_count + more
    at = np.arange(n) * 7 % len(rays)
    assert backend.extend(rays[at]).tobytes() == want[at].tobytes()
