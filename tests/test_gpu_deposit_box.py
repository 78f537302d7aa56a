"""The box deposition's bricks, work lists and groups at their edges, against the CPU oracle at the
tolerances of the golden deposition test (cell masses 1e-12 of the largest, counts exact)."""

import numpy as np
import pytest

from tests.conftest import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "nb, n, lo, hi",
    [
        (1, 50, 0.2, 2.0),  # one cell
        (7, 400, 0.1, 1.2),  # below a brick; trilinear and kernel weights mixed
        (8, 5000, 0.85, 0.88),  # one brick, several stretches; supports around sqrt(3) cells
        (9, 700, 0.5, 3.0),  # a ragged second brick
        (33, 300, 2.0, 14.0),  # a warp's and a block's particles (16384 candidate cells)
        (40, 1, 30.0, 30.0),  # one particle wider than the box
    ],
)
def test_box_edges_match_the_oracle(nb, n, lo, hi):
    from blackhole_nebula_simulator_b200 import gasgrid as gg
    from oracle import deposit as odep

    rng = np.random.default_rng(nb * 1000 + n)
    bx = gg.CartesianBox(centre=(3.0, -2.0, 1.0), size=10.0, n=nb)
    x = np.array(bx.centre) + rng.uniform(-8.0, 8.0, (n, 3))  # a part of them beyond the box
    h = bx.dx * np.exp(rng.uniform(np.log(lo), np.log(hi), n)) if hi > lo else np.full(n, lo * bx.dx)
    m = rng.uniform(0.5, 2.0, n)
    t = np.exp(rng.uniform(np.log(1e4), np.log(1e7), n))
    v = rng.normal(0.0, 0.05, (n, 3))
    for kernel in ("cubic", "wendland_c4"):
        ref = odep.deposit_box(x, h, m, t, v, bx, kernel)
        res = gg.deposit_box(x, h, m, t, v, bx, kernel)
        scale = max(np.abs(ref["mass"]).max(), 1e-300)
        check(f"{kernel} mass", ref["mass"] / scale, res.mass.cpu().numpy() / scale, atol=1e-12)
        check(f"{kernel} outside", ref["outside"], res.outside, rtol=1e-12, atol=1e-14 * m.sum())
        check(f"{kernel} trilinear count", ref["n_trilinear"], res.n_trilinear)
        for f in ("rho", "t_mass", "t_em", "vel"):
            a = np.asarray(ref[f], np.float64)
            check(f"{kernel} {f}", a, getattr(res, f).cpu().numpy().astype(np.float64),
                  atol=1e-6 * float(np.abs(a).max()))  # fmt: skip
