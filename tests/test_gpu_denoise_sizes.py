"""The denoiser at sizes where its blocks and rows do not come out even."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width, height", [(1, 1), (5, 3), (31, 9), (33, 17), (64, 48), (97, 65), (160, 33)])
@pytest.mark.parametrize("demodulated", [False, True])
def test_odd_sizes_match_the_oracle(width, height, demodulated):
    """Frames smaller than a block, of sizes that are no multiple of a block or
    of a pass's rows, with sky, young and old pixels, against the oracle's
    denoiser (float for float the reference's).  A pixel's filtered light is a
    mean of at most 25 taps over four passes, each weight of some twenty
    roundings and a power of 128 (128 roundings of the facing): a relative
    1e-4 covers 4 * (128 + 20) * 2^-24 = 3.5e-5 twice over."""
    import kodanuki_gb300 as K
    import oracle.port as op
    rng = np.random.default_rng(width * 1000 + height)
    n = width * height
    colour = rng.exponential(1.0, (n, 3)).astype(np.float32)
    lum = colour @ np.array([0.2126, 0.7152, 0.0722], np.float32)
    moment = (lum * lum * (1 + rng.random(n))).astype(np.float32)
    length = np.where(rng.random(n) < 0.4, 1, rng.integers(4, 40, n)).astype(np.float32)
    normal = rng.normal(size=(n, 3)) * 0.1 + (0, 0, 1)
    normal = (normal / np.linalg.norm(normal, axis=1, keepdims=True)).astype(np.float16)
    distance = (5 + rng.random(n)).astype(np.float16)
    leaf = rng.integers(0, 3, n).astype(np.uint32)
    sky = rng.random(n) < 0.1
    leaf[sky], distance[sky], normal[sky] = 0xFFFFFFFF, np.inf, 0
    albedo = rng.random((n, 3)).astype(np.float16)
    albedo[rng.random(n) < 0.1] = 0
    lens = np.array([0, 0, 1, 0, 1, 0, 1, 0, 0, 0, 0, 1, 0.4, width / height])
    with K.Backend(0) as b:
        out = b.denoise(width, height, demodulated, lens, colour, moment, length, distance, normal, albedo, leaf)
    want = op.denoise(width, height, demodulated, lens, colour.astype(np.float64), moment.astype(np.float64), length, distance.astype(np.float32),
                      normal.astype(np.float64), leaf, albedo.astype(np.float64))
    assert np.abs(out - want.reshape(out.shape)).max() <= 1e-4 * max(1.0, np.abs(want).max())
