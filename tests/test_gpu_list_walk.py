"""The list build's candidate walk at its limits: leaves whose frontiers outgrow a warp's and a block's
buffers, lists shared out over many work items, and bounding boxes so large that the walk's grid
resolves nothing.  The lists are exact sets, known without a reference."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 3000, 40_000, 420_000])
def test_one_particle_reaches_all(n):
    """Every particle alone but for one whose search radius covers the box: its row is everything,
    the others hold it and themselves."""
    from blackhole_nebula_simulator_b200 import ops

    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    cells = rng.permutation(side**3)[:n]
    pos = np.stack([cells // side**2, cells // side % side, cells % side], 1) + 0.2 * rng.random((n, 3))
    h = np.full(n, 0.3)
    big = n // 2
    h[big] = side  # 2 h covers the diagonal
    nb = ops.find_neighbours(pos, h)
    off, idx = nb.offset.cpu().numpy(), nb.index.cpu().numpy()
    count = np.full(n, 2)
    count[big] = n
    assert np.array_equal(np.diff(off), count)
    assert np.array_equal(idx[off[big] : off[big + 1]], np.arange(n))
    rest = np.delete(np.arange(n), big)
    assert np.array_equal(idx[off[rest]], np.minimum(rest, big))
    assert np.array_equal(idx[off[rest] + 1], np.maximum(rest, big))


@pytest.mark.parametrize("far", [1e5, 1e9, 1e13, 1e200])
def test_a_particle_far_away_changes_no_list(far):
    from blackhole_nebula_simulator_b200 import ops

    rng = np.random.default_rng(3)
    pos = rng.uniform(0.0, 1.0, (2000, 3)) + 40.0
    h = rng.uniform(0.04, 0.06, 2000)
    a = ops.find_neighbours(pos, h)
    b = ops.find_neighbours(np.concatenate([pos, [[far, -far, far]]]), np.append(h, 0.05))
    off, idx = b.offset.cpu().numpy(), b.index.cpu().numpy()
    assert np.array_equal(off[:-1], a.offset.cpu().numpy())
    assert np.array_equal(idx[:-1], a.index.cpu().numpy()) and idx[-1] == 2000
