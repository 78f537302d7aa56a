"""The FP64 pair passes on row counts around the eight-lane groups and their warps, on rows of every
length from the particle alone upward, against the CPU oracle: every output within 1e-12 of its
largest value (the golden shock tests' tolerance)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _near(name, expected, got):
    got = got.detach().cpu().numpy()
    scale = np.abs(expected).max()
    assert np.all(np.abs(got - expected) <= 1e-12 * scale), (
        f"{name}: {np.abs(got - expected).max() / max(scale, 1e-300):.3g} of the largest value")


@pytest.mark.parametrize("kernel", ["cubic", "wendland_c4"])
@pytest.mark.parametrize("nrows", [1, 3, 4, 5, 31, 33, None])
def test_pair_passes_match_the_oracle(kernel, nrows):
    from blackhole_nebula_simulator_b200 import ics, ops
    from blackhole_nebula_simulator_b200.config import C_NORM, KERNEL_IDS, ShockCapturing
    from oracle import native

    ic = ics.cloud(1200, kernel=kernel, seed=3)
    rng = np.random.default_rng(7)
    # chains of 1 to 12 particles far away: lists of those lengths
    chains = [np.array([5000.0 + 500.0 * k, 0.0, 0.0]) + rng.uniform(0.0, 0.5, (k, 3)) * ic.h[0]
              for k in range(1, 13)]  # fmt: skip
    x = np.concatenate([ic.x, *chains])
    n = len(x)
    order = rng.permutation(n)
    x = np.ascontiguousarray(x[order])
    h = ic.h[0] * rng.uniform(0.8, 1.25, n)
    v, acc = rng.normal(0.0, 1.0, (n, 3)), rng.normal(0.0, 1.0, (n, 3))
    m, rho, om = rng.uniform(0.5, 2.0, n), rng.uniform(0.5, 2.0, n), rng.uniform(0.8, 1.2, n)
    P, u, cs, al = (rng.uniform(0.2, 2.0, n) for _ in range(4))
    kid = KERNEL_IDS[kernel]
    cn = C_NORM[kid]
    nb = native.find_neighbours(x, h)
    assert set(range(1, 13)) <= set(np.diff(nb.offset).tolist())
    rows = None if nrows is None else np.sort(rng.permutation(n)[:nrows])
    k = dict(rows=rows)
    for signal in (0, 1):
        ref = native.forces(x, v, m, h, rho, om, P, nb, kid, cn, u, cs, al, alpha_u=0.7,
                            cond_signal=signal, **k)  # fmt: skip
        got = ops.forces_numba(x, v, m, h, rho, om, P, nb, kernel, u, cs, al,
                               ShockCapturing(alpha_u=0.7, conductivity_signal=signal), **k)
        for f, a in zip(("acc", "dudt", "vsig_max", "dudt_visc", "dudt_cond"), ref):
            _near(f"signal {signal} {f}", a, getattr(got, f))
    plain = ops.forces_numba(x, v, m, h, rho, om, P, nb, kernel, **k)
    ref = native.forces(x, v, m, h, rho, om, P, nb, kid, cn, **k)
    _near("plain acc", ref[0], plain.acc)
    _near("plain dudt", ref[1], plain.dudt)
    a, d = native.disc_forces(x, v, m, h, rho, om, cs, 1.3, nb, kid, cn, **k)
    ga, gd = ops.disc_forces_numba(x, v, m, h, rho, om, cs, 1.3, nb, kernel, **k)
    _near("disc acc", a, ga)
    _near("disc dudt", d, gd)
    gv = native.velocity_gradients(x, v, m, h, nb, kid, cn)
    _near("velocity gradients", gv, ops.velocity_gradients_numba(x, v, m, h, nb, kernel))
    ref = native.gradients(x, v, acc, m, h, nb, kid, cn, **k)
    g = ops.gradients_numba(x, v, acc, m, h, nb, kernel, **k)
    for f, a in zip(("div_v", "curl_v", "ddivv_dt"), ref):
        _near(f, a, getattr(g, f))
    for gate in (0, 1, 2):
        for close in (True, False):
            ref = native.forces(x, v, m, h, rho, om, P, nb, kid, cn, u, cs, al, grad_v=gv,
                                closeness=close, eta_crit=0.9, gate=gate, **k)  # fmt: skip
            sh = ShockCapturing(reconstruction=True, closeness=close, eta_crit=0.9, recon_gate=gate)
            got = ops.forces_numba(x, v, m, h, rho, om, P, nb, kernel, u, cs, al, sh, grad_v=gv, **k)
            for f, a in zip(("acc", "dudt", "vsig_max", "dudt_visc", "dudt_cond"), ref):
                _near(f"gate {gate} close {close} {f}", a, getattr(got, f))
