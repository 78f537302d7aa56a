"""Shared steps, which evaluate every particle without marking or selecting any, against the density
operator on lists of its own: the same guess of h at the same positions gives the same h and rho.
The sums differ by their order alone; on a jittered lattice that is 2e-15 of h, so 1e-12 as in the
golden density test."""

import numpy as np
import pytest

from tests.conftest import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 1500])
@pytest.mark.parametrize("kernel, eta", [("cubic", 1.2), ("wendland_c4", 1.6)])
def test_every_particle_is_evaluated(n, kernel, eta):
    from blackhole_nebula_simulator_b200 import coupled, ics, ops
    from blackhole_nebula_simulator_b200.config import CoupledConfig, HydroConfig

    ic = ics.cloud(n, kernel=kernel, seed=3)
    cc = CoupledConfig(hydro=HydroConfig(kernel=kernel, eta=eta))
    st = coupled.initialise(ic.x, ic.v, ic.u, ic.mass, ic.h, cc)
    for scale in (1e-6, 1.0, 1.0):  # the first on the cached lists
        h = st.h.clone()
        st = coupled.step(st, cc, scale * coupled.stable_dt(st, cc))
        ref = ops.compute_density(st.x, st.mass, h, kernel, eta, h_max=cc.hydro.h_max)
        check("h", ref.h.cpu().numpy(), st.h.cpu().numpy(), rtol=1e-12)
        check("rho", ref.rho.cpu().numpy(), st.rho.cpu().numpy(), rtol=1e-12)
    assert st.reuses >= 1 and st.builds >= 1
    assert np.isfinite(st.a_hydro.cpu().numpy()).all()
