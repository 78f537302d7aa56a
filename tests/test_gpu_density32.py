"""The FP32 density solve from good and bad guesses of h (rows that fit its cache, rows that walk their
list in every sum, supports that outgrow the cached range), against the FP64 form at the FP32
form's tolerance for h and rho (1e-5)."""

import pytest

from tests.conftest import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel, eta", [("cubic", 1.2), ("wendland_c4", 1.6)])
@pytest.mark.parametrize("guess", [0.55, 1.0, 1.8])
@pytest.mark.parametrize("n", [33, 5001])
def test_fp32_density_follows_fp64(kernel, eta, guess, n):
    from dataclasses import replace

    from blackhole_nebula_simulator_b200 import coupled, ics
    from blackhole_nebula_simulator_b200.config import CoupledConfig, HydroConfig

    ic = ics.cloud(n, kernel=kernel, seed=8)
    hc = HydroConfig(kernel=kernel, eta=eta, switch=False, reconstruction=False, h_max=200.0)
    st = [coupled.initialise(ic.x, ic.v, ic.u, ic.mass, guess * ic.h,
                             CoupledConfig(hydro=replace(hc, precision=p)))
          for p in ("fp64", "fp32")]  # fmt: skip
    for f in ("h", "rho"):
        a, b = (getattr(s, f).cpu().numpy() for s in st)
        check(f, a, b, rtol=1e-5)
