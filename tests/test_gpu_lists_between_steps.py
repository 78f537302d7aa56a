"""Operators called between a run's steps on the same context.

An operator's list build takes the place of the lists that the run would reuse, so the run builds its
own again; the cell grid's bounding box is not the run's.  FP64 runs then differ from an undisturbed
one by the order of their sums (1e-15 of h and rho on a jittered lattice, times a few steps: 1e-11
holds it; lists of another search radius miss it by tens of per cent).  Where the lists are reused the
FP32 form gives the same bits.
"""

import pytest
import torch

from tests.conftest import check

pytestmark = pytest.mark.gpu


def _shared(precision, between):
    from blackhole_nebula_simulator_b200 import coupled, ics
    from blackhole_nebula_simulator_b200.config import CoupledConfig, HydroConfig

    ic = ics.cloud(1500, kernel="cubic", seed=3)
    cc = CoupledConfig(hydro=HydroConfig(kernel="cubic", eta=1.2, precision=precision))
    st = coupled.initialise(ic.x, ic.v, ic.u, ic.mass, ic.h, cc)
    for _ in range(3):
        between(st)
        st = coupled.step(st, cc, 1e-6 * coupled.stable_dt(st, cc))
    return st


def _blocks(precision, between):
    from blackhole_nebula_simulator_b200 import blocks, ics
    from blackhole_nebula_simulator_b200.config import BlockConfig, CoupledConfig, HydroConfig

    ic = ics.cloud(1500, kernel="cubic", seed=3)
    bc = BlockConfig(coupled=CoupledConfig(hydro=HydroConfig(kernel="cubic", eta=1.2, precision=precision)),
                     dt_max=16.0)  # fmt: skip
    st = blocks.initialise(ic.x, ic.v, ic.u, ic.mass, ic.h, bc, t_stop=1600.0)
    for _ in range(3):
        between(st)
        blocks.advance(st, bc)
    return st


@pytest.mark.parametrize("run", [_shared, _blocks])
def test_a_list_build_between_steps(run):
    from blackhole_nebula_simulator_b200 import ops

    alone = run("fp64", lambda st: None)
    assert alone.reuses >= 1
    other = run("fp64", lambda st: ops.find_neighbours(st.x + 5.0, 0.6 * st.h))
    for f in ("h", "rho", "a_hydro", "dudt", "u", "x"):
        a, b = (getattr(s, f).cpu().numpy() for s in (alone, other))
        check(f, a, b, atol=1e-11 * abs(a).max())


@pytest.mark.parametrize("run", [_shared, _blocks])
def test_a_cell_grid_between_steps(run):
    from blackhole_nebula_simulator_b200 import ops

    alone = run("fp32", lambda st: None)
    other = run("fp32", lambda st: ops.cell_geometry(1e-3 * st.x + 1e4, st.h))
    assert other.reuses == alone.reuses >= 1
    for f in ("h", "rho", "a_hydro", "dudt", "u", "x"):
        assert torch.equal(getattr(alone, f), getattr(other, f)), f
