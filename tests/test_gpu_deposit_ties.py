"""Which centres the log-spherical deposition counts when a centre lies on the support's edge.

Kernel weights or trilinear ones: the choice is the number of centres with r / h < 2, r from the
reference's own arithmetic (render/gasgrid.py:380-395: centre (rc sin th) cos ph, every operation
rounded).  Each particle's h puts its eighth nearest centre exactly on the edge, r / h = 2 (outside:
seven centres, trilinear), or one rounding of h inside it (eight, the kernel).  Particles
whose seventh, eighth and ninth centres are not clearly apart are left out.  The centres' radii are the device's own
exponentials, so the counts are exact.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _centres(lg):
    """Centres as the reference forms them, from the tables the deposition reads."""
    from blackhole_nebula_simulator_b200 import gasgrid as gg

    tab = gg._device_tables(lg, torch.device("cuda")).cpu().numpy()
    sth, cth = tab[: lg.nth], tab[lg.nth : 2 * lg.nth]
    cph, sph = tab[3 * lg.nth : 3 * lg.nth + lg.nph], tab[3 * lg.nth + lg.nph : 3 * lg.nth + 2 * lg.nph]
    i = torch.arange(lg.nr, dtype=torch.float64, device="cuda")
    rc = lg.r_min * torch.exp((i + 0.5) * lg.dlnr).cpu().numpy()
    rst = (rc[:, None] * sth)[:, :, None]
    z = np.broadcast_to((rc[:, None] * cth)[:, :, None], (lg.nr, lg.nth, lg.nph))
    return np.stack([rst * cph, rst * sph, z], -1).reshape(-1, 3)


def _case(fine):
    """A grid and particles whose eight nearest centres lie inside it: anywhere, or (with shells a
    hundred-thousandth of the radius apart) along a column of centres."""
    from blackhole_nebula_simulator_b200 import gasgrid as gg

    rng = np.random.default_rng(5)
    if not fine:
        lg = gg.LogSphericalGrid(r_min=2.0, r_max=200.0, nr=24, nth=12, nph=24)
        r = np.exp(rng.uniform(np.log(6.0), np.log(80.0), 4000))
        d = rng.normal(size=(4000, 3))
        return lg, r[:, None] * d / np.linalg.norm(d, axis=1, keepdims=True)
    lg = gg.LogSphericalGrid(r_min=40.0, r_max=40.1, nr=250, nth=5, nph=7)
    c = _centres(lg).reshape(*lg.shape, 3)
    at = rng.integers(0, [150, lg.nth, lg.nph], (500, 3)) + [50, 0, 0]
    return lg, c[tuple(at.T)] + rng.uniform(-2e-4, 2e-4, (500, 3))


@pytest.mark.parametrize("kernel", ["cubic", "wendland_c4"])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("fine", [False, True])
def test_centres_on_the_edge_are_counted_as_the_reference_does(kernel, split, fine):
    from blackhole_nebula_simulator_b200 import gasgrid as gg

    lg, x = _case(fine)
    c = _centres(lg)
    edge, clear = np.empty(len(x)), np.empty(len(x), bool)
    for p in range(len(x)):
        e = c - x[p]
        dist = np.sort(np.sqrt(e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1] + e[:, 2] * e[:, 2]))
        edge[p] = dist[7]
        clear[p] = dist[8] > dist[7] * (1.0 + 1e-7) and dist[6] < dist[7] * (1.0 - 1e-7)
    n = int(clear.sum())
    assert n > 0.9 * len(x)
    x, h = x[clear], edge[clear] / 2.0
    one, t, v = np.ones(n), np.full(n, 1e5), np.zeros((n, 3))
    kw = dict(coarsen=(1, 1, 1), wide_cells=1e9) if split else {}
    call = gg.deposit_log_split if split else gg.deposit_log
    assert call(x, h, one, t, v, lg, kernel, **kw).n_trilinear == n
    assert call(x, np.nextafter(h, np.inf), one, t, v, lg, kernel, **kw).n_trilinear == 0
