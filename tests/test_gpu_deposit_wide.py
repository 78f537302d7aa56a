"""Box deposition of supports that all reach every brick: more list entries than are held at once
(2^28), so the lists are made in parts.

The sums are additive over the particles: the whole against two halves that each fit.  Every cell
adds positive masses in another order, 40,000 of them: a few ulp of the sum, so 1e-12.  The lists'
room is bounded by 2^28 entries of 4 bytes and a quarter to spare, 1.34 GB, and the records take 96
bytes a particle: 1.45 GB hold both (all the entries at once would take 1.6 GB).
"""

import numpy as np
import pytest
import torch

from tests.conftest import check

pytestmark = pytest.mark.gpu


def test_lists_of_wide_supports_are_made_in_parts():
    from blackhole_nebula_simulator_b200 import gasgrid as gg

    rng = np.random.default_rng(9)
    n, box = 40_000, gg.CartesianBox(centre=(1.0, -2.0, 0.5), size=8.0, n=160)
    # 2 h = 7.1 from 0.05 about the centre: past the corners, 4 sqrt 3 away
    p = [torch.as_tensor(a, device="cuda") for a in (
        np.asarray(box.centre) + rng.uniform(-0.05, 0.05, (n, 3)), rng.uniform(3.55, 3.6, n),
        rng.uniform(0.5, 2.0, n), rng.uniform(1e4, 1e6, n), rng.normal(size=(n, 3)))]  # fmt: skip

    def scratch():  # device memory in use but for the caching allocator's
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free - torch.cuda.memory_reserved()

    gg.deposit_box(*[a[:100] for a in p], box, "cubic")
    before = scratch()
    whole = gg.deposit_box(*p, box, "cubic")
    kept = scratch() - before
    parts = [gg.deposit_box(*[a[k : k + n // 2] for a in p], box, "cubic") for k in (0, n // 2)]
    check("mass", sum(a.mass for a in parts).cpu().numpy(), whole.mass.cpu().numpy(), rtol=1e-12)
    check("outside", sum(a.outside for a in parts), whole.outside, rtol=1e-12)
    assert whole.n_trilinear == 0
    assert kept < 1.45e9
