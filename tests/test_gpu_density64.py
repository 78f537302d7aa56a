"""The FP64 density operator where its row kernel changes over: 8 lanes per row (cubic, from 65,536
rows) against 32, rows with more entries inside 2.1 h than the cache holds, and starts from which
the cache is filled again; against the CPU oracle at the tolerances of the golden density test
(h, rho, Omega 1e-12; iterations and flags exact).

The cloud is a jittered lattice with masses within 20 %: from these starts the reference's sums,
taken forward and backward, give the same h to 2e-15 in every row, so 1e-12 is far above what the
order of the sums can do (random positions have rows where a Newton step through df/dh near zero
magnifies it ten thousandfold)."""

import numpy as np
import pytest

from tests.conftest import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel, eta", [("cubic", 1.2), ("wendland_c4", 1.6)])
@pytest.mark.parametrize("start", [0.8, 1.0, 1.35])
@pytest.mark.parametrize("nrows", [1, 7, 65535, 65536])
def test_rows_and_starts_match_the_oracle(kernel, eta, start, nrows):
    from blackhole_nebula_simulator_b200 import ics, ops
    from blackhole_nebula_simulator_b200.config import C_NORM, KERNEL_IDS
    from oracle import native

    n = 3000 if nrows < 100 else 66_000
    ic = ics.cloud(n, kernel=kernel, seed=5)
    rng = np.random.default_rng(nrows)
    mass = ic.mass * np.where(rng.random(n) < 0.5, 1.0, rng.uniform(0.9, 1.1, n))
    h_search = 1.4 * ic.h
    nb = native.find_neighbours(ic.x, h_search)
    rows = np.sort(rng.permutation(n)[:nrows])
    kid = KERNEL_IDS[kernel]
    h, rho, omega, iters, flags = native.density(ic.x, mass, ic.h * start, nb, h_search, kid,
                                                 C_NORM[kid], eta, rows=rows)  # fmt: skip
    got = ops.density_numba(ic.x, mass, ic.h * start, nb, h_search, kernel, eta, rows=rows)
    check("flags", flags, got.flags.cpu().numpy())
    check("iterations", iters, got.iterations.cpu().numpy())
    check("h", h, got.h.cpu().numpy(), rtol=1e-12)
    check("rho", rho, got.rho.cpu().numpy(), rtol=1e-12)
    check("omega", omega, got.omega.cpu().numpy(), rtol=1e-12)
