"""The denoiser over light whose square FP32 does not hold: the history's second
moment is infinite, as the temporal member leaves it, and a pixel's variance is
the oracle's, which works in double.  The bound is the odd sizes' (a relative
1e-4 of the frame's brightest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("demodulated", [False, True])
@pytest.mark.parametrize("scale", [1e18, 1e20, 1e30])
def test_bright_frames_match_the_oracle(demodulated, scale):
    import kodanuki_gb300 as K
    import oracle.port as op
    width, height = 40, 24
    rng = np.random.default_rng(int(np.log10(scale)))
    n = width * height
    colour = (scale * rng.uniform(0.5, 1.5, (n, 3))).astype(np.float32)
    with np.errstate(over="ignore"):
        lum = colour @ np.array([0.2126, 0.7152, 0.0722], np.float32)
        moment = (lum * lum * np.float32(1.5)).astype(np.float32)
    assert np.isinf(moment).all() == (scale > 1e19)
    length = rng.integers(4, 40, n).astype(np.float32)
    normal = np.tile(np.array([0, 0, 1], np.float16), (n, 1))
    distance = np.full(n, 5, np.float16)
    leaf = np.zeros(n, np.uint32)
    albedo = rng.uniform(0.2, 0.9, (n, 3)).astype(np.float16)
    lens = np.array([0, 0, 1, 0, 1, 0, 1, 0, 0, 0, 0, 1, 0.01, width / height])
    with K.Backend(0) as b:
        out = b.denoise(width, height, demodulated, lens, colour, moment, length, distance, normal, albedo, leaf)
    with np.errstate(all="ignore"):
        want = op.denoise(width, height, demodulated, lens, colour.astype(np.float64), moment.astype(np.float64), length, distance.astype(np.float32),
                          normal.astype(np.float64), leaf, albedo.astype(np.float64)).reshape(out.shape)
    assert np.isfinite(want).all()
    assert np.abs(out - want).max() <= 1e-4 * np.abs(want).max()
