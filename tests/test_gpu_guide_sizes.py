"""The guide's training kernel at the edges of its tiles (128 samples) and of
a launch (a block takes several tiles where there are more than SMs) against
the CPU oracle.

The bars are those of 16-bit operands: 2e-2 of a gradient's norm, and where
the sample is one, one unit of 64 more whose ReLU falls the other way
(1 / sqrt(64) of the norm)."""
import numpy as np
import pytest

from oracle.port import guide as G
from test_gpu_guide import HI, LO, LOG2, _guide, _livelier, _rows, _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 2 * 152 * 128 + 5])
def test_gradients_at_the_edges_of_tiles(n):
    rng = np.random.default_rng(29)
    with _guide() as g:
        ws, table = _livelier(g, rng)
        p, nv = _rows(rng, n)
        d = rng.normal(size=(n, 3))
        d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        w = rng.uniform(0.5, 3.0, n).astype(np.float32)
        loss, dw, dt = g.gradients(np.concatenate([p, nv, d, w[:, None]], axis=1))
        want_loss, want_dws, want_dt, _ = G.gradients(p, nv, d, w, ws, table, LO, HI, LOG2)
    bar = 2e-2 + (0.125 if n == 1 else 0.0)
    assert abs(loss - want_loss) <= bar * max(1.0, abs(want_loss))
    for a, b in zip([*_weights(dw), dt], [*want_dws, want_dt]):
        assert np.linalg.norm(a.ravel() - b.ravel()) <= bar * np.linalg.norm(b)
