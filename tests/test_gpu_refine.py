"""refine_sums by itself, on coarse grids down to a single cell, against the CPU oracle.

Positive coarse sums: every fine sum is eight positive terms times a ratio of volumes and of masses.
The volumes differ from NumPy's by a few ulp of their factors (r2^3 - r1^3 and cos th1 - cos th2 lose
at most a factor of ten on these grids), so 1e-13 holds fifty such roundings.
"""

import numpy as np
import pytest
import torch

from tests.conftest import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radii", [(2.0, 200.0), (200.0, 2.0)])
@pytest.mark.parametrize("shape,coarsen", [((8, 4, 8), (2, 4, 4)), ((8, 4, 8), (8, 4, 8)),
                                           ((3, 2, 5), (1, 2, 5)), ((3, 1, 4), (3, 1, 2)),
                                           ((8, 8, 8), (2, 4, 4))])  # fmt: skip
def test_refine_sums_matches_the_oracle(shape, coarsen, radii):
    from blackhole_nebula_simulator_b200 import gasgrid as gg
    from oracle import deposit as odep

    g = gg.LogSphericalGrid(r_min=radii[0], r_max=radii[1], nr=shape[0], nth=shape[1], nph=shape[2])
    gc = gg.coarse_log_grid(g, coarsen)
    acc = np.random.default_rng(7).uniform(0.5, 2.0, (*gc.shape, gg.N_FIELDS))
    ref = odep.refine_sums(acc, gc, g, coarsen)
    out = gg.refine_sums(torch.as_tensor(acc, device="cuda"), gc, g, coarsen)
    check("fine sums", ref, out.cpu().numpy(), rtol=1e-13)
