"""The FP32 form with the switch on and the reconstruction off against the FP64 form, at the tolerances
of tests/test_gpu_fp32_errors.py: its records are packed after the switch's update of alpha, for the
touched particles alone where fewer than an eighth of the particles close.

The switch fixture's cloud with its 100 particles nearest to the first one four levels deeper: steps
that close 100, about 500 and all 2,048 particles.  The switch's alpha is a ratio of sums that cancel,
so 1e-3 of its range, as with the reconstruction.
"""

import dataclasses

import numpy as np
import pytest

from tests.conftest import check, golden

pytestmark = pytest.mark.gpu


def _np(t):
    return t.detach().cpu().numpy()


def test_switch_without_reconstruction():
    from blackhole_nebula_simulator_b200 import blocks
    from blackhole_nebula_simulator_b200.config import BlockConfig, CoupledConfig
    from tests.test_gpu_fp32_errors import TOL
    from tests.test_gpu_shock import _switch_hc

    g = golden("switch_blocks.npz")
    n = len(g["h0"])
    offset = np.zeros(n, np.int64)
    offset[np.argsort(np.linalg.norm(g["x0"] - g["x0"][0], axis=1))[:100]] = 4
    out = []
    for prec in ("fp64", "fp32"):
        hc = dataclasses.replace(_switch_hc(prec), reconstruction=False)
        bc = BlockConfig(coupled=CoupledConfig(hydro=hc, cooling_beta=230.0), dt_max=64.0)
        st = blocks.initialise(g["x0"], g["v0"], g["u0"], g["mass"], g["h0"], bc, t_stop=1e6,
                               level_offset=offset)  # fmt: skip
        act = [len(blocks.advance(st, bc)) for _ in range(20)]
        out.append((st, act))
    (a, act_a), (b, act_b) = out
    assert min(act_a) * 8 < n and max(act_a) == n
    check("active counts", np.array(act_a), np.array(act_b))
    check("levels", _np(a.level), _np(b.level))
    for f in ("h", "rho", "u"):
        check(f, _np(getattr(a, f)), _np(getattr(b, f)), rtol=TOL[f])
    for f in ("x", "p"):
        check(f, _np(getattr(a, f)), _np(getattr(b, f)), rtol=TOL[f], per_vector=True)
    amax = np.linalg.norm(_np(a.a_hydro), axis=1).max()
    check("a_hydro", _np(a.a_hydro) / amax, _np(b.a_hydro) / amax, atol=TOL["a_hydro"])
    dmax = np.abs(_np(a.dudt)).max()
    check("dudt", _np(a.dudt) / dmax, _np(b.dudt) / dmax, atol=TOL["dudt"])
    check("alpha", _np(a.alpha), _np(b.alpha), atol=1e-3)
    assert np.ptp(_np(a.alpha)) > 0.5
