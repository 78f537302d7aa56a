"""The calls that a user of this framework makes, as timed cases: the operators of the SPH step one
by one, the render-grid deposition, and whole runs of both step schemes, over the sizes that the
package's workloads, tests and benchmark use.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same ranges, ``prepare`` makes a
case's inputs from a seed, ``run`` is one pass through the public API and returns everything it
computed, ``work`` is what that pass cannot do without, and ``exact`` evaluates the same operators in
plain 64-bit torch on pairs found by brute force.
"""

from __future__ import annotations

import math
import os

import numpy as np
import torch

from blackhole_nebula_simulator_b200 import blocks, cooling, coupled, gasgrid, ics, ops, units
from blackhole_nebula_simulator_b200.config import (
    ALPHA_U_MAGMA2,
    COND_VELOCITY,
    C_NORM,
    H_MAX_HOLE,
    HFACT,
    KERNEL_IDS,
    BlockConfig,
    CoupledConfig,
    HydroConfig,
    ShockCapturing,
)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WEIGHTS = os.path.join(ROOT, "blackhole_nebula_simulator_b200", "data", "cooling_mlp.npy")
SKIN = 1.4  # search radius over smoothing length (HydroConfig.skin)
GAMMA = 5.0 / 3.0
DETAIL_BOX = dict(centre=(100.0, 0.0, 0.0), size=64.0, n=160)  # the benchmark's detail box


def listed():
    return [
        # a script or test on the small cloud: one list build, where launches and waits count
        dict(name="lists_cloud_small", kind="lists", gas="cloud", n=4096, kernel="wendland_c4"),
        # the list build of a production-size disc snapshot, lists handed to the caller
        dict(name="lists_torus", kind="lists", gas="torus", n=1_000_003, kernel="cubic"),
        # the h-rho solve of every particle from the last step's h (FP64 operator)
        dict(name="density_cloud", kind="density", gas="cloud", n=262_144, kernel="cubic", rows=1.0),
        # the forces of a block step's active rows: lists tightened, pressure + viscosity +
        # conductivity, and the disc viscosity
        dict(name="forces_torus_rows", kind="forces", gas="torus", n=400_009, kernel="cubic",
             rows=0.37, disc=True),
        # the shock-capturing operators of the reference's default configuration: velocity
        # gradients, switch gradients, forces with the reconstructed jump
        dict(name="shock_streams", kind="shock", gas="streams", n=100_002, kernel="wendland_c4",
             rows=1.0),
        # the gravity flow on its own: test particles and orbit ensembles
        dict(name="orbits", kind="orbits", n=1_000_003),
        # temperatures, pressures and sound speeds of a snapshot with gas + radiation
        dict(name="eos_gasrad", kind="eos", n=300_007),
        # a render frame's two grids: the whole torus on the log-spherical grid, the detail box
        dict(name="deposit_log", kind="deposit_log", gas="torus", n=1_000_003, kernel="cubic"),
        dict(name="deposit_box", kind="deposit_box", gas="torus", n=1_048_576, kernel="cubic"),
        # a short shared-step run of the reference's default physics on the small cloud
        dict(name="shared_cloud_small", kind="shared", gas="cloud", n=4096, kernel="wendland_c4",
             steps=4, precision="fp64", shock=True),
        # the flagship: the first system steps of the 4M torus, FP32 pair form, learned cooling
        dict(name="blocks_torus_4m", kind="blocks", gas="torus", n=4_194_304, kernel="cubic",
             steps=10, precision="fp32", shock=False, network=True),
        # a block run with few active rows per system step, FP64 form, exact cooling
        dict(name="blocks_streams", kind="blocks", gas="streams", n=300_000, kernel="cubic",
             steps=20, precision="fp64", shock=False, network=False),
    ]  # fmt: skip


def draw(rng):
    def size(lo, hi):
        n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
        return n

    kind = rng.choice(["lists", "density", "forces", "shock", "orbits", "eos", "deposit_log",
                       "deposit_box", "shared", "blocks"])  # fmt: skip
    gas = rng.choice(["cloud", "torus", "streams"])
    kernel = rng.choice(["cubic", "wendland_c4"])
    rows = 1.0 if rng.random() < 0.4 else round(math.exp(rng.uniform(math.log(0.01), 0.0)), 4)
    if kind == "lists":
        return dict(kind=kind, gas=gas, n=_even(gas, size(3000, 1_000_000)), kernel=kernel)
    if kind == "density":
        return dict(kind=kind, gas=gas, n=_even(gas, size(4000, 400_000)), kernel=kernel, rows=rows)
    if kind == "forces":
        return dict(kind=kind, gas=gas, n=_even(gas, size(4000, 400_000)), kernel=kernel, rows=rows,
                    disc=rng.random() < 0.5)  # fmt: skip
    if kind == "shock":
        return dict(kind=kind, gas=gas, n=_even(gas, size(4000, 200_000)), kernel=kernel, rows=rows)
    if kind == "orbits":
        return dict(kind=kind, n=size(1000, 2_000_000))
    if kind == "eos":
        return dict(kind=kind, n=size(1000, 2_000_000))
    if kind == "deposit_log":
        return dict(kind=kind, gas="torus", n=size(20_000, 2_000_000), kernel=kernel)
    if kind == "deposit_box":  # fewer particles would not resolve the box' 0.4 cells
        return dict(kind=kind, gas="torus", n=size(300_000, 2_000_000), kernel="cubic")
    if kind == "shared":
        return dict(kind=kind, gas=gas, n=_even(gas, size(2000, 300_000)), kernel=kernel,
                    steps=rng.randint(1, 5), precision=rng.choice(["fp64", "fp32"]),
                    shock=rng.random() < 0.5)  # fmt: skip
    return dict(kind=kind, gas=gas, n=_even(gas, size(8000, 1_000_000)), kernel="cubic",
                steps=rng.randint(4, 16), precision=rng.choice(["fp64", "fp32"]),
                shock=rng.random() < 0.3, network=rng.random() < 0.5)  # fmt: skip


def _even(gas, n):
    return n - n % 2 if gas == "streams" else n  # two equal streams


# ------------------------------------------------------------------------------- inputs
def _rng(seed, tag):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + tag) % (2**62))
    return g


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _torus(n, seed, kernel):
    """The torus of ics.torus (major radius 100, Gaussian minor profile of width 15 cut at 40,
    circular speeds with 1 % noise), drawn on the device."""
    g = _rng(seed, 1)
    big, a, sigma, total = 100.0, 40.0, 15.0, 0.01
    parts, have = [], 0
    while have < n:
        k = int((n - have) * 4) + 4096
        s = sigma * _normal(g, k).abs()
        th, phi = _uniform(g, k, 0.0, 2 * math.pi), _uniform(g, k, 0.0, 2 * math.pi)
        cyl = big + s * torch.cos(th)
        keep = (s <= a) & (_uniform(g, k, 0.0, 1.0) < (s / a) * cyl / (big + a))
        s, th, phi, cyl = s[keep], th[keep], phi[keep], cyl[keep]
        parts.append(torch.stack([cyl * torch.cos(phi), cyl * torch.sin(phi), s * torch.sin(th)], 1))
        have += len(s)
    x = torch.cat(parts)[:n].contiguous()
    r = x.norm(dim=1)
    vc = (r - 2.0) / r * torch.rsqrt(r - 3.0)
    cyl = torch.hypot(x[:, 0], x[:, 1])
    v = torch.stack([-x[:, 1] / cyl, x[:, 0] / cyl, torch.zeros_like(r)], 1) * vc[:, None]
    v = v + 0.01 * vc[:, None] * _normal(g, n, 3)
    vol = 2.0 * math.pi**2 * big * a**2
    f = lambda c: torch.full((n,), c, device="cuda", dtype=torch.float64)  # noqa: E731
    return (x, v, f(units.gas_u_from_temperature(1.0e9)), f(total / n),
            f(HFACT[kernel] * (vol / n) ** (1.0 / 3.0)))  # fmt: skip


def _start(case, seed):
    """x, v, u, mass and the first guess of h of the case's gas."""
    n, kernel = case["n"], case["kernel"]
    if case["kind"] == "lists":
        return _turned(case, seed)
    if case["gas"] == "torus":
        return _torus(n, seed, kernel)
    make = {"cloud": ics.cloud, "streams": ics.streams}[case["gas"]]
    ic = make(n, kernel=kernel, seed=int(seed) % (2**31))
    return tuple(torch.as_tensor(a, device="cuda", dtype=torch.float64).contiguous()
                 for a in (ic.x, ic.v, ic.u, ic.mass, ic.h))  # fmt: skip


def _turned(case, seed):
    """One fixed gas, mirrored and renumbered by the seed: other positions and other lists with the
    same number of entries, so that the results of different seeds have the same shapes."""
    g = _rng(seed, 7)
    at = int(torch.randint(1, case["n"], (1,), generator=g, device="cuda"))
    flip = (2 * torch.randint(0, 2, (3,), generator=g, device="cuda") - 1).to(torch.float64)
    x, v, *rest = (torch.roll(a, at, 0) for a in _start(dict(case, kind="gas"), 12))
    return (x * flip).contiguous(), (v * flip).contiguous(), *rest


def _moving(case, seed):
    """The case's gas in motion: velocities with half a sound speed of noise, 20 % scatter in u,
    viscosity parameters between 0 and 1, accelerations of the order of u / h."""
    x, v, u, mass, h0 = _start(case, seed)
    g, n = _rng(seed, 2), case["n"]
    u = u * _uniform(g, n, 0.8, 1.2)
    cs = torch.sqrt(GAMMA * (GAMMA - 1.0) * u)
    v = (v + 0.5 * cs[:, None] * _normal(g, n, 3)).contiguous()
    alpha = _uniform(g, n, 0.0, 1.0)
    acc = (u / h0)[:, None] * _normal(g, n, 3)
    return x, v, u, mass, h0, cs, alpha, acc.contiguous()


def _rows(case, seed):
    """The active rows of a block step, ascending; None for every particle."""
    if case["rows"] >= 1.0:
        return None
    n = case["n"]
    m = max(1, int(n * case["rows"]))
    return torch.randperm(n, generator=_rng(seed, 3), device="cuda")[:m].sort().values


def _config(case):
    hc = HydroConfig(kernel=case["kernel"], eta=HFACT[case["kernel"]], switch=case["shock"],
                     reconstruction=case["shock"], conductivity_signal=COND_VELOCITY,
                     alpha_u=ALPHA_U_MAGMA2, h_max=H_MAX_HOLE, precision=case["precision"],
                     disc_alpha_av=1.0 if case["gas"] == "torus" else 0.0)  # fmt: skip
    if case["kind"] == "shared":
        return CoupledConfig(hydro=hc)
    net = None
    if case["network"]:
        net = cooling.load_network(WEIGHTS, cooling.mlp_params())
    return BlockConfig(coupled=CoupledConfig(hydro=hc, cooling="brems", cooling_mlp=net),
                       dt_max=256.0 if case["gas"] == "torus" else 4096.0)  # fmt: skip


def _orbit_inputs(case, seed):
    n, g = case["n"], _rng(seed, 4)
    r = torch.exp(_uniform(g, n, math.log(20.0), math.log(3000.0)))
    d = _normal(g, n, 3)
    d = d / d.norm(dim=1, keepdim=True)
    t = torch.linalg.cross(d, _normal(g, n, 3))
    t = t / t.norm(dim=1, keepdim=True)
    x = (r[:, None] * d).contiguous()
    v = torch.rsqrt(r)[:, None] * (_uniform(g, n, 0.5, 1.2)[:, None] * t
                                   + _uniform(g, n, -0.5, 0.5)[:, None] * d)  # fmt: skip
    # the steps of the reference's orbit criterion, eta_orb r^(3/2) and up to four levels below
    dt = 0.00125 * r**1.5 * torch.exp2(-_uniform(g, n, 0.0, 4.0))
    return x, (r / (r - 2.0))[:, None] * v, dt


def _eos_inputs(case, seed):
    """rho over the streams' and the torus' densities, T log-uniform from 1e4 to 1e9 K."""
    n, g = case["n"], _rng(seed, 5)
    hc = HydroConfig(eos="gasrad")
    rho_si = torch.exp(_uniform(g, n, math.log(1e-10), math.log(1e-3)))
    t = torch.exp(_uniform(g, n, math.log(1e4), math.log(1e9)))
    a1 = 1.5 * units.K_B / (units.MU * units.M_P)
    u = (a1 * t + units.A_RAD * t**4 / rho_si) / units.C**2
    return hc, rho_si / hc.gas_units.density_kg_m3, u


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=dict(case))
    if kind == "orbits":
        s["x"], s["p"], s["dt"] = _orbit_inputs(case, seed)
        return s
    if kind == "eos":
        s["hc"], s["rho"], s["u"] = _eos_inputs(case, seed)
        return s
    if kind in ("shared", "blocks"):
        s["ic"] = _start(case, seed)
        s["cfg"] = _config(case)
        return s
    kernel, eta = case["kernel"], HFACT[case["kernel"]]
    x, v, u, mass, h0, cs, alpha, acc = _moving(case, seed)
    # the state that the last step left: converged h, rho, Omega and the lists it used
    d = ops.compute_density(x, mass, h0, kernel, eta, tol=1e-12, skin=SKIN)
    s.update(x=x, mass=mass, kernel=kernel, eta=eta)
    if kind == "lists":
        s.update(h_search=d.h * SKIN)
        return s
    if kind.startswith("deposit"):
        s.update(h=d.h, t=u / units.gas_u_from_temperature(1.0), v=v)
        s["grid"] = (gasgrid.LogSphericalGrid() if kind == "deposit_log"
                     else gasgrid.CartesianBox(**DETAIL_BOX))  # fmt: skip
        return s
    s["rows"] = _rows(case, seed)
    s["lists"] = ops.find_neighbours(x, d.h * SKIN)
    if kind == "density":
        # the guess is the last step's h, one per cent off
        s.update(h_start=d.h * _uniform(_rng(seed, 6), case["n"], 0.99, 1.01), h_search=d.h * SKIN)
        return s
    s.update(v=v, u=u, cs=cs, alpha=alpha, acc=acc, h=d.h, rho=d.rho, omega=d.omega,
             P=(GAMMA - 1.0) * d.rho * u)  # fmt: skip
    if kind == "shock":
        s["shock"] = ShockCapturing(alpha_u=ALPHA_U_MAGMA2, conductivity_signal=COND_VELOCITY,
                                    reconstruction=True, eta_crit=1.0 / eta)  # fmt: skip
        s["lists"] = ops.tighten(s["lists"], x, d.h)
    return s


# ------------------------------------------------------------------------------- one pass
_STATE = ("x", "p", "u", "h", "rho", "a_hydro", "dudt", "vsig_max", "alpha")


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "lists":
        nb = ops.find_neighbours(s["x"], s["h_search"])
        return dict(offset=nb.offset, index=nb.index)
    if kind == "density":
        r = ops.density_numba(s["x"], s["mass"], s["h_start"], s["lists"], s["h_search"],
                              s["kernel"], s["eta"], rows=s["rows"])  # fmt: skip
        return dict(h=r.h, rho=r.rho, omega=r.omega, iterations=r.iterations, flags=r.flags)
    if kind == "forces":
        nb = ops.tighten(s["lists"], s["x"], s["h"], s["rows"])
        f = ops.forces_numba(s["x"], s["v"], s["mass"], s["h"], s["rho"], s["omega"], s["P"], nb,
                             s["kernel"], s["u"], s["cs"], s["alpha"], rows=s["rows"])  # fmt: skip
        out = _force_fields(f)
        if case["disc"]:
            out["disc_acc"], out["disc_dudt"] = ops.disc_forces_numba(
                s["x"], s["v"], s["mass"], s["h"], s["rho"], s["omega"], s["cs"], 1.0, nb,
                s["kernel"], rows=s["rows"])  # fmt: skip
        return out
    if kind == "shock":
        gv = ops.velocity_gradients_numba(s["x"], s["v"], s["mass"], s["h"], s["lists"], s["kernel"])
        g = ops.gradients_numba(s["x"], s["v"], s["acc"], s["mass"], s["h"], s["lists"],
                                s["kernel"], rows=s["rows"])  # fmt: skip
        f = ops.forces_numba(s["x"], s["v"], s["mass"], s["h"], s["rho"], s["omega"], s["P"],
                             s["lists"], s["kernel"], s["u"], s["cs"], s["alpha"], s["shock"],
                             rows=s["rows"], grad_v=gv)  # fmt: skip
        return dict(grad_v=gv, div=g.div_v, curl=g.curl_v, ddiv=g.ddivv_dt, **_force_fields(f))
    if kind == "orbits":
        x1, p1, it = ops.glf_step_many(s["x"], s["p"], s["dt"])
        return dict(x=x1, p=p1, iterations=it)
    if kind == "eos":
        P, cs = ops.eos_state(s["hc"], s["rho"], s["u"])
        return dict(P=P, cs=cs)
    if kind in ("deposit_log", "deposit_box"):
        call = gasgrid.deposit_log_split if kind == "deposit_log" else gasgrid.deposit_box
        g = call(s["x"], s["h"], s["mass"], s["t"], s["v"], s["grid"], s["kernel"])
        return dict(mass=g.mass, rho=g.rho, t_mass=g.t_mass, t_em=g.t_em, vel=g.vel,
                    outside=g.outside, n_trilinear=g.n_trilinear)  # fmt: skip
    if kind == "shared":
        st = coupled.initialise(*s["ic"], s["cfg"])
        for _ in range(case["steps"]):
            coupled.step(st, s["cfg"], coupled.stable_dt(st, s["cfg"]))
        return {k: getattr(st, k) for k in _STATE}
    st = blocks.initialise(*s["ic"], s["cfg"], t_stop=s["cfg"].dt_max * 2.0**20)
    for _ in range(case["steps"]):
        blocks.advance(st, s["cfg"])
    return {k: getattr(st, k) for k in (*_STATE, "omega", "level", "n_end", "luminosity")}


def _force_fields(f):
    return dict(acc=f.acc, dudt=f.dudt, vsig=f.vsig_max, visc=f.dudt_visc, cond=f.dudt_cond)


# ------------------------------------------------------------------------------- necessary work
def work(case):
    """Inputs read once and outputs written once; pair terms counted as in DESIGN.md's kernel table
    (25 per density term and three sums, 75 per force pair, 20 with the disc viscosity)."""
    n, kind = case["n"], case["kind"]
    if kind == "orbits":
        return dict(bytes=n * (7 + 7) * 8, flops=n * 700)
    if kind == "eos":
        return dict(bytes=n * 4 * 8, flops=n * 8 * 60)
    pairs = 4.0 / 3.0 * math.pi * (2.0 * HFACT[case["kernel"]]) ** 3  # inside 2 h
    entries = pairs * SKIN**3  # inside the search radius
    if kind == "lists":
        return dict(bytes=n * (32 + 8) + 8 * n * entries, flops=n * entries * 8)
    if kind == "deposit_log":
        return dict(bytes=n * 72 + 192 * 96 * 192 * 32, flops=n * 8 * 20)
    if kind == "deposit_box":
        h = HFACT[case["kernel"]] * (math.pi**2 * 3.2e5 / n) ** (1.0 / 3.0)
        cells = max(8.0, 4.0 / 3.0 * math.pi * (2.0 * h / 0.4) ** 3) * 0.1  # a tenth is in the box
        return dict(bytes=n * 72 + 160**3 * 32, flops=n * cells * 30)
    if kind in ("shared", "blocks"):
        # per step: the state in and out, one list walk, density and force pairs of the active
        # rows (about half of the particles); the first evaluation builds the lists
        per = 300.0 + 4.0 * entries
        return dict(bytes=n * (per + case["steps"] * (300.0 + 4.0 * entries * 0.5)),
                    flops=n * pairs * (75 + 75) * (1 + 0.5 * case["steps"]))  # fmt: skip
    m = n * case["rows"]
    if kind == "density":
        return dict(bytes=n * 48 + m * (8 * entries + 8 + 40), flops=m * pairs * 75)
    if kind == "forces":
        flops = m * (entries * 8 + pairs * (75 + 20 * case["disc"]))
        return dict(bytes=n * 104 + m * (8 * entries + 8 * pairs + 8 + 56 + 32 * case["disc"]),
                    flops=flops)  # fmt: skip
    return dict(bytes=n * (128 + 72 + 8 * pairs) + m * (24 + 56),
                flops=n * pairs * 60 + m * pairs * (80 + 150))  # fmt: skip


# ------------------------------------------------------------------------------- in 64 bits
_MOST_EXACT = 420_000  # particles whose pairs are found by brute force within seconds


def _f(q, kernel):
    if kernel == "cubic":
        near = 1.0 - 1.5 * q * q + 0.75 * q**3
        far = 0.25 * (2.0 - q) ** 3
        return torch.where(q < 1.0, near, torch.where(q < 2.0, far, torch.zeros_like(q)))
    w = torch.clamp(1.0 - 0.5 * q, min=0.0)
    return w**6 * (35.0 / 12.0 * q * q + 3.0 * q + 1.0)


def _df(q, kernel):
    if kernel == "cubic":
        near = -3.0 * q + 2.25 * q * q
        far = -0.75 * (2.0 - q) ** 2
        return torch.where(q < 1.0, near, torch.where(q < 2.0, far, torch.zeros_like(q)))
    w = torch.clamp(1.0 - 0.5 * q, min=0.0)
    return -7.0 / 3.0 * q * w**5 * (5.0 * q + 2.0)


def _pairs(x, reach, rows, both=False):
    """(position in rows, other particle) of every pair closer than 2 reach of the row (``both``: of
    either particle), the row itself included."""
    order = torch.argsort(x[:, 0])
    xs, rs = x[order], reach[order]
    left = xs[:, 0].contiguous()
    by_x = torch.argsort(x[rows, 0])
    top = float(rs.max())
    outs = []
    for part in by_x.split(1024):
        i = rows[part]
        far = 2.0 * (top if both else float(reach[i].max())) * (1.0 + 1e-9)
        lo = int(torch.searchsorted(left, x[i, 0].min() - far))
        hi = int(torch.searchsorted(left, x[i, 0].max() + far, right=True))
        d2 = sum((xs[None, lo:hi, c] - x[i, c][:, None]) ** 2 for c in range(3))
        r = reach[i][:, None].expand_as(d2)
        if both:
            r = torch.maximum(r, rs[None, lo:hi])
        a, b = torch.nonzero(d2 < (2.0 * r) ** 2, as_tuple=True)
        outs.append((part[a], order[lo + b]))
    return tuple(torch.cat(o) for o in zip(*outs))


def _solve_h(x, mass, start, search, rows, kernel, eta, tol):
    """The Newton-bisection h-rho solve of the rows from ``start`` within (0, search], particle by
    particle in parallel: h, rho, Omega and whether the root lies beyond the search radius."""
    cn = C_NORM[KERNEL_IDS[kernel]]
    q, j = _pairs(x, search, rows)
    r = (x[j] - x[rows[q]]).norm(dim=1)
    m, mi, cap = mass[j], mass[rows], search[rows]
    zero = torch.zeros(len(rows), dtype=torch.float64, device=x.device)

    def sums(h):
        hq = h[q]
        u = r / hq
        f = _f(u, kernel)
        rho = zero.index_add(0, q, m * cn / hq**3 * f)
        drho = zero.index_add(0, q, -m * cn / hq**4 * (3.0 * f + u * _df(u, kernel)))
        return rho, drho

    h = torch.minimum(start[rows], cap)
    h0, lo, hi = h.clone(), zero.clone(), cap.clone()
    done = torch.zeros(len(rows), dtype=torch.bool, device=x.device)
    for _ in range(50):
        rho, drho = sums(h)
        f = rho - mi * (eta / h) ** 3
        df = drho + 3.0 * mi * eta**3 / h**4
        hi = torch.where(~done & (f > 0), h, hi)
        lo = torch.where(~done & ~(f > 0), h, lo)
        new = torch.where(df > 0, h - f / df, 0.5 * (lo + hi))
        new = torch.where((lo <= new) & (new <= hi), new, 0.5 * (lo + hi))
        stop = (new - h).abs() < tol * h0
        h = torch.where(done, h, new)
        done = done | stop
        if bool(done.all()):
            break
    beyond = (h >= cap * (1.0 - 1e-3)) & (sums(cap)[0] - mi * (eta / cap) ** 3 < 0)
    h = torch.where(beyond, cap, h)
    rho, drho = sums(h)
    return h, rho, 1.0 + h / (3.0 * rho) * drho, beyond


def _converged(case, x, mass, h0):
    """h, rho, Omega at the root for every particle."""
    kernel, n = case["kernel"], case["n"]
    h, rho, om = h0.clone(), torch.empty_like(h0), torch.empty_like(h0)
    rows, search = torch.arange(n, device=x.device), h0 * SKIN
    start = h0.clone()
    for _ in range(12):
        a, b, c, beyond = _solve_h(x, mass, start, search, rows, kernel, HFACT[kernel], 1e-13)
        h[rows], rho[rows], om[rows] = a, b, c
        rows = rows[beyond]
        if len(rows) == 0:
            break
        start[rows] = h[rows]
        search[rows] *= 2.0
    return h, rho, om


def _gradient(q, rows, dx, mf, cnt, vecs):
    """Corrected gradients G R^-1 of each vector field (its differences per pair in ``vecs``)."""
    def total(a):
        return torch.zeros(rows, 3, 3, dtype=torch.float64, device=dx.device).index_add(
            0, q, mf[:, None, None] * a[:, :, None] * dx[:, None, :])

    R = -total(dx)
    scale = (R[:, 0, 0] + R[:, 1, 1] + R[:, 2, 2]) / 3.0
    single = (cnt < 4) | ~(scale > 0) | ~(torch.linalg.det(R).abs() >= 1e-6 * scale**3)
    eye = torch.eye(3, dtype=torch.float64, device=dx.device)
    inv = torch.linalg.inv(torch.where(single[:, None, None], eye, R))
    weak = torch.where(scale > 0, 1.0 / scale, torch.zeros_like(scale))
    out = []
    for a in vecs:
        G = total(a)
        out.append(torch.where(single[:, None, None], G * weak[:, None, None], G @ inv))
    return out


def _forces(x, v, mass, h, rho, om, P, u, cs, al, rows, kernel, shock=None, gv=None, disc=None):
    cn = C_NORM[KERNEL_IDS[kernel]]
    q, b = _pairs(x, h, rows, both=True)
    a = rows[q]
    keep = a != b
    q, a, b = q[keep], a[keep], b[keep]
    dx = x[a] - x[b]
    r = dx.norm(dim=1)
    e = dx / r[:, None]
    fa = cn / h[a] ** 4 * _df(r / h[a], kernel)
    fb = cn / h[b] ** 4 * _df(r / h[b], kernel)
    dv = v[a] - v[b]
    vr = (dv * e).sum(1)
    m = mass[b]

    def total(t):
        return torch.zeros(len(rows), *t.shape[1:], dtype=torch.float64, device=x.device).index_add(0, q, t)

    if disc is not None:
        qa = -rho[a] * h[a] / (2.0 * r) * disc * cs[a] * vr / (om[a] * rho[a] ** 2)
        qb = -rho[b] * h[b] / (2.0 * r) * disc * cs[b] * vr / (om[b] * rho[b] ** 2)
        return total(-(m * (qa * fa + qb * fb))[:, None] * e), total(m * qa * vr * fa)
    sh = shock or ShockCapturing()
    zero = torch.zeros_like(vr)
    if gv is None:
        jump, on = vr, vr < 0
        sig = vr.abs()
    else:
        ga = (gv[a] * dx[:, None, :]).sum(2)
        gb = (gv[b] * dx[:, None, :]).sum(2)
        pa, pb = (dx * ga).sum(1), (dx * gb).sum(1)
        ratio = torch.where(pb != 0, pa / torch.where(pb != 0, pb, torch.ones_like(pb)), zero)
        phi = torch.where(ratio > 0, torch.clamp(4.0 * ratio / (1.0 + ratio) ** 2, max=1.0), zero)
        near = torch.minimum(r / h[a], r / h[b])
        fold = torch.exp(-(((near - sh.eta_crit) / sh.eta_fold) ** 2))
        phi = torch.where(near < sh.eta_crit, phi * fold, phi)
        jump = ((v[a] - 0.5 * phi[:, None] * ga - v[b] - 0.5 * phi[:, None] * gb) * e).sum(1)
        on = (jump < 0) & (vr < 0)
        jump = torch.maximum(jump, vr)  # the min-mod gate
        sig = jump.abs()
    va, vb = al[a] * cs[a] + sh.beta * sig, al[b] * cs[b] + sh.beta * sig
    na = P[a] + torch.where(on, -0.5 * rho[a] * va * jump, zero)
    nb = P[b] + torch.where(on, -0.5 * rho[b] * vb * jump, zero)
    ia = 1.0 / (om[a] * rho[a])
    visc = total(torch.where(on, -m * va * 0.5 * jump * vr * fa * ia, zero))
    if sh.conductivity_signal == COND_VELOCITY:
        vu = vr.abs()
    else:
        vu = torch.sqrt((P[a] - P[b]).abs() / (0.5 * (rho[a] + rho[b])))
    cond = total(m * sh.alpha_u * vu * (u[a] - u[b]) * 0.5 * (fa * ia + fb / (om[b] * rho[b])))
    f = m * (na * fa / (om[a] * rho[a] ** 2) + nb * fb / (om[b] * rho[b] ** 2))
    dudt = P[rows] / (om[rows] * rho[rows] ** 2) * total(m * vr * fa) + visc + cond
    cfl = al[a] * cs[a] + sh.beta * vr.abs()
    vsig = cs[rows].scatter_reduce(0, q, cfl, "amax")
    return dict(acc=total(-f[:, None] * e), dudt=dudt, vsig=vsig, visc=visc, cond=cond)


def _gn_dh_dx(x, p):
    r = x.norm(dim=1, keepdim=True)
    px, pp = (p * x).sum(1, keepdim=True), (p * p).sum(1, keepdim=True)
    c = -2.0 * (r - 2.0) / r**4
    radial = (pp / r**2 + 0.5 * (6.0 * r - 16.0) / r**5 * px * px) / r + 1.0 / r**3
    return radial * x + c * px * p


def _gn_dh_dp(x, p):
    r = x.norm(dim=1, keepdim=True)
    return (r - 2.0) / r * p - 2.0 * (r - 2.0) / r**4 * (p * x).sum(1, keepdim=True) * x


def _box_fields(x, h, m, t, v, box, kernel):
    """The box' fields from every (particle, cell centre inside its support) pair, a batch of
    particles at a time; None where a particle covers fewer than eight centres (trilinear)."""
    n, dx = box.n, box.dx
    lo = torch.as_tensor(box.lo, device=x.device)
    first = torch.floor((x - 2.0 * h[:, None] - lo) / dx).long()
    last = torch.floor((x + 2.0 * h[:, None] - lo) / dx).long()
    inside = ((last >= 0) & (first < n)).all(1)
    outside = float(m[~inside].sum())
    vals = torch.stack([m, m * t, m * t**4, m * v[:, 0], m * v[:, 1], m * v[:, 2]], 1)
    x, h, vals, first = x[inside], h[inside], vals[inside], first[inside]
    size = last[inside] - first + 1
    count = size.prod(1)
    acc = torch.zeros(n**3, 6, dtype=torch.float64, device=x.device)
    ends = torch.cumsum(count, 0).cpu().numpy()
    a = 0
    while a < len(x):
        base = int(ends[a - 1]) if a else 0
        b = max(a + 1, int(np.searchsorted(ends, base + 40_000_000)))
        c = count[a:b]
        p = torch.repeat_interleave(torch.arange(a, b, device=x.device), c)
        e = torch.arange(len(p), device=x.device) - (torch.cumsum(c, 0) - c).repeat_interleave(c)
        cell = torch.stack([e // (size[p, 1] * size[p, 2]), e // size[p, 2] % size[p, 1],
                            e % size[p, 2]], 1) + first[p]  # fmt: skip
        q = (lo + (cell.double() + 0.5) * dx - x[p]).norm(dim=1) / h[p]
        near = q < 2.0
        p, cell, w = p[near], cell[near], _f(q[near], kernel)
        if int(torch.bincount(p - a, minlength=b - a).min()) < 8:
            return None
        total = torch.zeros(b - a, dtype=torch.float64, device=x.device).index_add(0, p - a, w)
        share = (w / total[p - a])[:, None] * vals[p]
        ok = ((cell >= 0) & (cell < n)).all(1)
        outside += float(share[~ok, 0].sum())
        cell = cell[ok]
        acc.index_add_(0, (cell[:, 0] * n + cell[:, 1]) * n + cell[:, 2], share[ok])
        a = b
    mass = acc[:, 0]
    mean = torch.where(mass[:, None] > 0, acc / torch.where(mass > 0, mass, torch.ones_like(mass))[:, None],
                       torch.zeros_like(acc))  # fmt: skip
    shape = (n, n, n)
    return dict(mass=mass.view(shape), rho=(mass / dx**3).view(shape), t_mass=mean[:, 1].view(shape),
                t_em=(mean[:, 2] ** 0.25).view(shape), vel=mean[:, 3:].reshape(*shape, 3),
                outside=outside, n_trilinear=None)  # fmt: skip


def exact(case, seed):
    """What ``run`` returns for these inputs, in plain 64-bit torch.  None where only whole numbers
    come back, for whole runs, for the log-spherical grid, and for sizes whose pairs take too long
    to find."""
    kind = case["kind"]
    if kind == "orbits":
        x, p, dt = _orbit_inputs(case, seed)
        dt = dt[:, None]
        ph = p
        for _ in range(10):
            ph = p - 0.5 * dt * _gn_dh_dx(x, ph)
        v = _gn_dh_dp(x, ph)
        y = x + dt * v
        for _ in range(10):
            y = x + 0.5 * dt * (v + _gn_dh_dp(y, ph))
        return dict(x=y, p=ph - 0.5 * dt * _gn_dh_dx(y, ph), iterations=None)
    if kind == "eos":
        hc, rho, u = _eos_inputs(case, seed)
        rs, us = rho * hc.gas_units.density_kg_m3, u * units.C**2
        a1, kb = 1.5 * units.K_B / (units.MU * units.M_P), units.K_B / (units.MU * units.M_P)
        t = torch.minimum(us / a1, (us * rs / units.A_RAD) ** 0.25)  # above the root
        for _ in range(60):  # the energy is convex in T: Newton falls onto the root
            t = t - (a1 * t + units.A_RAD * t**4 / rs - us) / (a1 + 4.0 * units.A_RAD * t**3 / rs)
        gas, rad = rs * kb * t, units.A_RAD * t**4 / 3.0
        beta, g = gas / (gas + rad), 2.0 / 3.0
        P = (gas + rad) / (hc.gas_units.density_kg_m3 * units.C**2)
        g1 = beta + (4.0 - 3.0 * beta) ** 2 * g / (beta + 12.0 * g * (1.0 - beta))
        return dict(P=P, cs=torch.sqrt(g1 * P / rho))
    if kind == "deposit_box":
        x, v, u, mass, h0, *_ = _moving(case, seed)
        h = ops.compute_density(x, mass, h0, case["kernel"], HFACT[case["kernel"]], tol=1e-12).h
        return _box_fields(x, h, mass, u / units.gas_u_from_temperature(1.0), v,
                           gasgrid.CartesianBox(**DETAIL_BOX), case["kernel"])  # fmt: skip
    if kind not in ("density", "forces", "shock") or case["n"] > _MOST_EXACT:
        return None
    kernel, n = case["kernel"], case["n"]
    x, v, u, mass, h0, cs, alpha, acc = _moving(case, seed)
    h, rho, om = _converged(case, x, mass, h0)
    rows = _rows(case, seed)
    rows = torch.arange(n, device=x.device) if rows is None else rows
    if kind == "density":
        start = h * _uniform(_rng(seed, 6), n, 0.99, 1.01)
        a, b, c, _ = _solve_h(x, mass, start, h * SKIN, rows, kernel, HFACT[kernel], 1e-4)
        return dict(h=a, rho=b, omega=c, iterations=None, flags=None)
    P = (GAMMA - 1.0) * rho * u
    if kind == "forces":
        out = _forces(x, v, mass, h, rho, om, P, u, cs, alpha, rows, kernel)
        if case["disc"]:
            out["disc_acc"], out["disc_dudt"] = _forces(x, v, mass, h, rho, om, P, u, cs, alpha,
                                                        rows, kernel, disc=1.0)  # fmt: skip
        return out
    q, b = _pairs(x, h, torch.arange(n, device=x.device), both=True)
    q, b = q[q != b], b[q != b]
    dx = x[q] - x[b]
    r = dx.norm(dim=1)
    mf = mass[b] * C_NORM[KERNEL_IDS[kernel]] / h[q] ** 4 * _df(r / h[q], kernel) / r
    gv, ga = _gradient(q, n, dx, mf, torch.bincount(q, minlength=n), (v[b] - v[q], acc[b] - acc[q]))
    trace = lambda t: t[:, 0, 0] + t[:, 1, 1] + t[:, 2, 2]  # noqa: E731
    curl = torch.stack([gv[:, 2, 1] - gv[:, 1, 2], gv[:, 0, 2] - gv[:, 2, 0],
                        gv[:, 1, 0] - gv[:, 0, 1]], 1).norm(dim=1)  # fmt: skip
    ddiv = trace(ga) - trace(gv @ gv)
    shock = ShockCapturing(alpha_u=ALPHA_U_MAGMA2, conductivity_signal=COND_VELOCITY,
                           reconstruction=True, eta_crit=1.0 / HFACT[kernel])  # fmt: skip
    f = _forces(x, v, mass, h, rho, om, P, u, cs, alpha, rows, kernel, shock, gv)
    return dict(grad_v=gv, div=trace(gv)[rows], curl=curl[rows], ddiv=ddiv[rows], **f)
