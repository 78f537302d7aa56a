"""Mass of single particles on a box whose centres all lie close to the support's edge.

There the weights are small differences (2 - q) and their relative error is large, but each particle's
weights are divided by their own sum, so its mass on the grid and outside is its mass to the rounding
of eight or more additions and products: 1e-14.  Supports end between a rounding and a hundredth beyond
the eighth centre; particles on cell corners (eight centres alike), on edges, faces and anywhere, inside
the box and across its faces.  The choice of weights is the oracle's.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["cubic", "wendland_c4"])
@pytest.mark.parametrize("beyond", [0.0, 1e-15, 1e-14, 1e-12, 1e-9, 1e-6, 1e-2])
def test_each_particles_mass_is_on_the_grid_or_outside(kernel, beyond):
    from blackhole_nebula_simulator_b200 import gasgrid as gg
    from oracle import deposit as odep

    rng = np.random.default_rng(11)
    box = gg.CartesianBox(centre=(0.3, -0.7, 0.1), size=1.6, n=12)
    at = rng.integers(0, 13, (24, 3)).astype(float)  # corners, some on the box' faces
    at[6:12, 0] += 0.5
    at[12:18, :2] += 0.5
    at[18:] += rng.uniform(0.0, 1.0, (6, 3))
    x = box.lo + at * box.dx
    axes = [box.lo[d] + (np.arange(-6, 18) + 0.5) * box.dx for d in range(3)]
    c = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    for p in x:
        e = c - p
        r8 = np.sort(np.sqrt(e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1] + e[:, 2] * e[:, 2]))[7]
        h = np.nextafter(r8 / 2.0, np.inf) * (1.0 + beyond)
        one = (p[None], np.array([h]), np.array([1.7]), np.array([1e5]), np.zeros((1, 3)), box, kernel)
        g = gg.deposit_box(*one)
        assert g.n_trilinear == odep.deposit_box(*one)["n_trilinear"]
        assert abs(float(g.mass.sum()) + g.outside - 1.7) <= 1e-14 * 1.7, (p, h)


@pytest.mark.parametrize("kernel", ["cubic", "wendland_c4"])
@pytest.mark.parametrize("beyond", [0.0, 1e-15, 1e-14, 1e-12, 1e-9, 1e-6, 1e-2])
def test_each_particles_mass_on_the_log_grid(kernel, beyond):
    """The same on a log-spherical grid: particles on the polar axis, whose nearest centres are a ring of
    sixteen alike, and anywhere."""
    from blackhole_nebula_simulator_b200 import gasgrid as gg

    rng = np.random.default_rng(12)
    lg = gg.LogSphericalGrid(r_min=2.0, r_max=60.0, nr=30, nth=12, nph=16)
    r = np.exp(rng.uniform(np.log(5.0), np.log(30.0), 40))
    d = rng.normal(size=(40, 3))
    x = r[:, None] * d / np.linalg.norm(d, axis=1, keepdims=True)
    x[:30, :2] = 0.0
    t, rc = lg.tables(), lg.r_centres()
    rst = (rc[:, None] * t["sth"])[:, :, None]
    c = np.stack([rst * t["cph"], rst * t["sph"],
                  np.broadcast_to((rc[:, None] * t["cth"])[:, :, None], lg.shape)], -1).reshape(-1, 3)  # fmt: skip
    for p in x:
        e = c - p
        r8 = np.sort(np.sqrt(e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1] + e[:, 2] * e[:, 2]))[7]
        h = np.nextafter(r8 / 2.0, np.inf) * (1.0 + beyond)
        g = gg.deposit_log(p[None], np.array([h]), np.array([1.7]), np.array([1e5]), np.zeros((1, 3)), lg, kernel)
        assert abs(float(g.mass.sum()) + g.outside - 1.7) <= 1e-14 * 1.7, (p, h)
