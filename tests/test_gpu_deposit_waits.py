"""Host waits of a box deposition: one where no support holds eight centres or reaches the box (the
mass outside and the trilinear count come back with the lists' length), one more for the gather."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,shift,waits", [(0.2, 0.0, 1), (4.0, 100.0, 1), (4.0, 0.0, 2)])
def test_host_waits(cells, shift, waits):
    from blackhole_nebula_simulator_b200 import _lib
    from blackhole_nebula_simulator_b200 import gasgrid as gg

    rng = np.random.default_rng(3)
    n, box = 200, gg.CartesianBox(centre=(0.0, 0.0, 0.0), size=16.0, n=16)
    x = rng.uniform(-7.0, 7.0, (n, 3)) + shift
    before = _lib.lib().nb_sync_count()
    g = gg.deposit_box(x, np.full(n, cells), np.ones(n), np.ones(n), np.zeros((n, 3)), box)
    assert _lib.lib().nb_sync_count() - before == waits
    assert g.n_trilinear == (n if cells < 1.0 else 0)
    assert abs(float(g.mass.sum()) + g.outside - n) < 1e-9 * n
    assert (g.outside == n) == (shift > 0.0)
