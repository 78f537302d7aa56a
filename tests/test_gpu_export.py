"""Lists exported in the caller's order, at the row lengths where the export's sorting networks
change over (128, 256, 512 and 1024 entries) and one entry beyond."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 128, 129, 256, 257, 512, 513, 1024, 1025, 1500])
def test_every_row_holds_the_whole_clump(n):
    """n particles inside one another's search radius, and a second clump of 40 far away: each row is
    its whole clump, ascending."""
    from blackhole_nebula_simulator_b200 import ops

    rng = np.random.default_rng(n)
    pos = np.concatenate([rng.uniform(0.0, 1.0, (n, 3)), rng.uniform(50.0, 51.0, (40, 3))])
    order = rng.permutation(n + 40)
    first = np.flatnonzero(order < n)  # the first clump's places after the shuffle
    second = np.flatnonzero(order >= n)
    nb = ops.find_neighbours(pos[order], np.full(n + 40, 2.0))
    off, idx = nb.offset.cpu().numpy(), nb.index.cpu().numpy()
    for i in range(n + 40):
        expected = first if order[i] < n else second
        assert np.array_equal(idx[off[i] : off[i + 1]], expected), f"row {i} of {n}"
