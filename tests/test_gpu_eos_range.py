"""Gas + radiation temperatures over the whole bracket [1, 1e13] K and forty decades of density: u is made
from a known T, which the solve has to give back.

Tolerance: u and rho are rounded on the way (about six roundings of 1.1e-16 each) and T moves by at
most the relative change of u; the solve's own last step leaves some ulps more: 4e-15 in all."""

import numpy as np
import pytest

from tests.conftest import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decade", [-24, -16, -8, 0, 8, 16])
def test_known_temperatures_come_back(decade):
    from blackhole_nebula_simulator_b200 import ops
    from blackhole_nebula_simulator_b200.config import HydroConfig, eos_fields

    hc = HydroConfig(eos="gasrad")
    f = eos_fields(hc)
    rng = np.random.default_rng(decade + 100)
    t = np.exp(rng.uniform(np.log(1.0 + 1e-9), np.log(1e13 * (1 - 1e-9)), 5000))
    t[:2] = 1.0 + 1e-9, 1e13 * (1 - 1e-9)
    rho_si = 10.0**decade * np.exp(rng.uniform(0.0, np.log(1e8), t.size))
    rho = rho_si / f["eos_rho_si"]
    u = (f["eos_a1"] * t + f["eos_a_rad"] * t**4 / (rho * f["eos_rho_si"])) / f["eos_u_si"]
    got = ops.gasrad_state(rho, u, hc.gas_units)[2].cpu().numpy()
    check("T", t, got, rtol=4e-15)
