"""The list build's rows against a brute-force search: sizes about the sub-leaf (8), leaf (32) and batch
edges, and search radii so uneven that a leaf's sub-leaves reach very different candidates.  Lists
are exact sets: d^2 in doubles, without fused operations, as the build's exact test rounds it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 32, 33, 64, 65, 129, 1000, 3001])
@pytest.mark.parametrize("spread", [1.0, 30.0])
def test_rows_match_brute_force(n, spread):
    from blackhole_nebula_simulator_b200 import ops

    rng = np.random.default_rng(n)
    centres = rng.uniform(-5.0, 5.0, (5, 3))
    pos = centres[rng.integers(0, 5, n)] + rng.normal(0.0, 0.7, (n, 3))
    h = 0.1 * np.exp(rng.uniform(0.0, np.log(spread), n) * (rng.random(n) < 0.05))
    nb = ops.find_neighbours(pos, h)
    off, idx = nb.offset.cpu().numpy(), nb.index.cpu().numpy()
    d = pos[:, None, :] - pos[None, :, :]
    d2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]
    r = 2.0 * np.maximum(h[:, None], h[None, :])
    row, col = np.nonzero(d2 < r * r)
    assert np.array_equal(np.diff(off), np.bincount(row, minlength=n))
    assert np.array_equal(idx, col)
