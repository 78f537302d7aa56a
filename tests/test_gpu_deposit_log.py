"""The log-spherical deposition's walks of the candidate centres against the CPU oracle.

A particle with up to LOG_WIDE (128) candidates is one thread's, the others a warp's; supports here
run from less than a cell (trilinear) to past the origin, on both sides of that line, on the poles,
across phi = 0 and beyond both ends of the radii.  Split grids put the wide particles on a second
grid in the same launches.

Tolerances: the cell sums differ from the oracle's by the order of their additions and an ulp or two
of a weight (q = sqrt(d^2) (1 / h)); weights of a particle sum to 1 and are smooth in q but for the
support's edge, where they vanish as (2 - q)^3 at least, so 1e-12 of the largest cell mass holds both
(the other depositions' bound); masses outside to 1e-12; counts exactly.
"""

import numpy as np
import pytest

from tests.conftest import check

pytestmark = pytest.mark.gpu


def _np(t):
    return t.detach().cpu().numpy()


def _particles(lg, n, widest):
    rng = np.random.default_rng(n)
    r = np.exp(rng.uniform(np.log(0.6 * lg.r_min), np.log(1.3 * lg.r_max), n))
    th = np.arccos(rng.uniform(-1.0, 1.0, n))
    ph = rng.uniform(0.0, 2.0 * np.pi, n)
    th[: n // 8] = rng.uniform(0.0, 1e-3, n // 8)  # about the poles
    th[n // 8 : n // 4] = np.pi - rng.uniform(0.0, 1e-3, n // 4 - n // 8)
    ph[n // 4 : n // 3] = rng.normal(0.0, 1e-3, n // 3 - n // 4)  # about phi = 0
    x = r[:, None] * np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1)
    x[-1] = 0.0
    h = r * lg.dlnr * np.exp(rng.uniform(np.log(0.2), np.log(widest), n))
    return (x, h, rng.uniform(0.5, 2.0, n), np.exp(rng.uniform(np.log(1e4), np.log(1e7), n)),
            rng.normal(0.0, 0.05, (n, 3)))  # fmt: skip


def _same(ref, res):
    scale = np.abs(ref["mass"]).max()
    check("mass", ref["mass"] / scale, _np(res.mass) / scale, atol=1e-12)
    check("outside", ref["outside"], res.outside, rtol=1e-12)
    check("trilinear count", ref["n_trilinear"], res.n_trilinear)
    for f in ("rho", "t_mass", "t_em", "vel"):
        a = np.asarray(ref[f], dtype=np.float64)
        check(f, a, _np(getattr(res, f)).astype(np.float64), atol=1e-6 * float(np.abs(a).max()))


@pytest.mark.parametrize("n,widest,shape", [(1, 3.0, (24, 12, 24)), (33, 6.0, (24, 12, 24)),
                                            (2000, 6.0, (24, 12, 24)), (700, 3.0, (17, 9, 31)),
                                            (300, 8.0, (5, 2, 1))])  # fmt: skip
@pytest.mark.parametrize("kernel", ["wendland_c4", "cubic"])
def test_candidate_walks_match_the_oracle(n, widest, shape, kernel):
    from blackhole_nebula_simulator_b200 import gasgrid as gg
    from oracle import deposit as odep

    lg = gg.LogSphericalGrid(r_min=2.0, r_max=200.0, nr=shape[0], nth=shape[1], nph=shape[2])
    p = _particles(lg, n, widest)
    _same(odep.deposit_log(*p, lg, kernel), gg.deposit_log(*p, lg, kernel))


@pytest.mark.parametrize("shape,wide_cells", [((24, 12, 24), 3.0), ((24, 12, 24), 1e9),
                                              ((24, 12, 24), 1e-9), ((32, 16, 28), 6.0)])  # fmt: skip
def test_split_grids_match_the_oracle(shape, wide_cells):
    from blackhole_nebula_simulator_b200 import gasgrid as gg
    from oracle import deposit as odep

    lg = gg.LogSphericalGrid(r_min=2.0, r_max=200.0, nr=shape[0], nth=shape[1], nph=shape[2])
    p = _particles(lg, 1500, 6.0)
    gc = gg.coarse_log_grid(lg)
    _same(odep.deposit_log_split(*p, lg, gc, "wendland_c4", wide_cells),
          gg.deposit_log_split(*p, lg, "wendland_c4", wide_cells))  # fmt: skip


def test_split_without_a_coarse_grid_and_no_wide_particle():
    """A grid that the coarse one does not divide is refused only when a particle is wide."""
    from blackhole_nebula_simulator_b200 import gasgrid as gg

    lg = gg.LogSphericalGrid(r_min=2.0, r_max=200.0, nr=23, nth=12, nph=24)
    p = _particles(lg, 300, 3.0)
    a, b = gg.deposit_log_split(*p, lg, wide_cells=1e9), gg.deposit_log(*p, lg)
    check("mass", _np(b.mass), _np(a.mass), rtol=0.0, atol=1e-12 * float(b.mass.max()))
    with pytest.raises(ValueError, match="divisible"):
        gg.deposit_log_split(*p, lg, wide_cells=1e-9)
