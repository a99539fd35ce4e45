"""Timed cases of the radiation hot path: what a user's program calls, over the range it is used in.

Every case goes through a public entry point: the ``sr`` object (spectra, flux maps, power-density
maps, point lists and multi-particle beams, in the default FP64 and in mixed precision), the job
queue, or the differentiable spectrum.  Sizes are those of the repository's configurations (3 GeV,
0.5 A electrons from z = -1 m through 31 periods of 49 mm, screen at 30 m) and of its tests, or odd
numbers between them.  Each pass integrates its trajectory again (``set_trajectory_cache`` drops the
kept one), as a program does that changes the beam or the field between calculations.

Seeds move the beam (position, angle, energy) and the field strength a little; sizes belong to the case.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

QE, ME, HBAR, PLANCK = 1.602176462e-19, 9.10938356e-31, 1.054571596e-34, 6.62606876e-34
LIGHT, EPS0, MU0 = 2.99792458e8, 8.854187817e-12, 1.2566370614e-6
PERIOD, NPERIODS, SCREEN, CURRENT = 0.049, 31, 30.0, 0.5
E1 = 152.25225225225225  # first harmonic on axis, eV

# Flops of one integrand evaluation (trajectory point x output) that the sums cannot do without, a fused
# multiply-add as two: direction and distance ~20, phase ~5, sine and cosine ~20 and three complex
# multiply-adds with the amplitude ~35 (flux); without the geometry for a spectrum; the triple product,
# its square and the fifth power for the power density.
FLOPS = {"flux": 80.0, "spectrum": 50.0, "power_density": 70.0}
STEP_FLOPS = 250.0  # one RK4 step of a particle


def listed():
    return [
        # a first look at a device: few energies, a coarse trajectory; latency is all there is
        dict(name="spectrum_quick", kind="spectrum", precision="fp64", npoints=2001, ne=101, field="undulator"),
        # the on-axis spectrum of configuration 0, as the drop-in gives it by default
        dict(name="spectrum", kind="spectrum", precision="fp64", npoints=20001, ne=1000, field="undulator"),
        # a measured field map (1-D grid), the beam given at its centre (both chains of the trajectory),
        # spectrum around the third harmonic and the total radiated power
        dict(name="field_map", kind="spectrum", precision="fp64", npoints=12001, ne=200, field="grid"),
        # configuration 1 in the default precision: maps at the first and the third harmonic
        dict(name="flux_maps", kind="flux", precision="fp64", npoints=20001, n1=101, n2=101, maps=2, field="undulator"),
        # flux on a curved screen given as a list of points, odd in number
        dict(name="flux_points", kind="points", precision="fp64", npoints=10001, n=2347, field="undulator"),
        # heat load of an elliptically polarising undulator on a mask, default precision
        dict(name="power_density", kind="power_density", precision="fp64", npoints=40001, n1=51, n2=51, field="epu"),
        # a small beam: the random electrons of one call, each with its own trajectory
        dict(name="beam_small", kind="beam", precision="fp64", npoints=10001, ne=300, particles=24, field="undulator"),
        # configuration 1 in mixed precision
        dict(name="flux_maps_mixed", kind="flux", precision="mixed", npoints=20001, n1=101, n2=101, maps=2,
             field="undulator"),
        # configuration 2 in mixed precision: the largest map
        dict(name="power_density_mixed", kind="power_density", precision="mixed", npoints=40001, n1=201, n2=201,
             field="epu"),
        # configuration 3a at a quarter of its particles: emittance and energy spread, 2000 energies
        dict(name="beam_mixed", kind="beam", precision="mixed", npoints=20001, ne=2000, particles=1024,
             field="undulator"),
        # configuration 3b: unequal maps and spectra with their trajectories in one queue
        dict(name="queue", kind="queue", jobs=40, set=3),
        # configuration 4: the spectrum of a perturbed field map and all of its derivatives
        dict(name="adjoint", kind="adjoint", npoints=20001, ne=200, nz=2001),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spectrum", "spectrum", "spectrum", "flux", "flux", "points", "power_density", "power_density",
                       "beam", "beam", "queue", "adjoint"])
    if kind == "queue":
        return dict(kind=kind, jobs=_log(rng, 6, 40), set=rng.randrange(1 << 20))
    if kind == "adjoint":
        return dict(kind=kind, npoints=_log(rng, 4001, 20001), ne=_log(rng, 50, 200), nz=_log(rng, 500, 2001))
    c = dict(kind=kind, precision=rng.choice(["fp64", "fp64", "mixed"]), npoints=_log(rng, 2001, 40001),
             field=rng.choice(["undulator", "undulator", "epu", "grid"]))
    if kind == "spectrum":
        c["ne"] = _log(rng, 50, 2000)
    elif kind == "flux":
        c.update(n1=_log(rng, 8, 128), n2=_log(rng, 8, 128), maps=rng.choice([1, 2]))
    elif kind == "points":
        c["n"] = _log(rng, 100, 8000)
    elif kind == "power_density":
        c.update(n1=_log(rng, 8, 128), n2=_log(rng, 8, 128))
    else:
        c.update(ne=_log(rng, 100, 1000), particles=_log(rng, 4, 256), field="undulator")
    return c


# ------------------------------------------------------------------ the inputs

def _inputs(case, seed):
    """What the seed decides: the beam's position, angle and energy and the field's strength."""
    r = random.Random(seed)
    two_chains = case.get("field") == "grid"
    z0 = 0.0 if two_chains else -1.0
    return dict(x0=[r.uniform(-5e-5, 5e-5), r.uniform(-2e-5, 2e-5), z0],
                d0=[r.uniform(-1e-5, 1e-5), r.uniform(-1e-5, 1e-5), 1.0],
                energy=3.0 * (1.0 + r.uniform(-1e-3, 1e-3)), bpeak=1.0 + r.uniform(-0.01, 0.01),
                start=-1.0 if two_chains else 0.0, stop=1.0 if two_chains else 2.0, photon=1.0 + r.uniform(-0.01, 0.01),
                sample=r.randrange(1 << 30))


def _undulator_by(z, bpeak):
    length = PERIOD * (NPERIODS + 2)
    s = np.sin(2 * math.pi * z / PERIOD)
    f = np.where(np.abs(z) > length / 2 - PERIOD, 0.75, 1.0)
    f = np.where(np.abs(z) > length / 2 - PERIOD / 2, 0.25, f)
    return np.where(np.abs(z) > length / 2, 0.0, f * bpeak * s)


def _field_map(seed, bpeak, nz=2001):
    """A "measured" map on z in [-1.05, 1.05]: the undulator with half a percent of error per pole."""
    z = np.linspace(-1.05, 1.05, nz)
    poles = 2 * (NPERIODS + 2)
    err = np.random.default_rng(seed).normal(0.0, 0.005, poles)
    k = np.clip(np.floor((z + PERIOD * (NPERIODS + 2) / 2) / (PERIOD / 2)).astype(int), 0, poles - 1)
    data = np.zeros((nz, 3))
    data[:, 1] = _undulator_by(z, bpeak) * (1.0 + err[k])
    return float(z[0]), float((z[-1] - z[0]) / (nz - 1)), data


def _fields(case, x):
    """The field list: ("undulator", amplitude, phase) or ("grid", z0, dz, data)."""
    if case["field"] == "grid":
        return [("grid", *_field_map(x["sample"], x["bpeak"]))]
    f = [("undulator", [0.0, x["bpeak"], 0.0], 0.0)]
    if case["field"] == "epu":
        f.append(("undulator", [0.6 * x["bpeak"], 0.0, 0.0], math.pi / 2))
    return f


def _curved_screen(n):
    """n points on a sphere of 30 m around the source, on a golden-angle spiral of 5 mm, facing it."""
    i = np.arange(n) + 0.5
    r, a = 0.005 * np.sqrt(i / n), 2.399963229728653 * i
    x, y = r * np.cos(a), r * np.sin(a)
    p = np.column_stack([x, y, np.sqrt(SCREEN ** 2 - x * x - y * y)])
    return [[q.tolist(), (q / SCREEN).tolist()] for q in p]


def _energy_range(case):
    return (0.98 * 3 * E1, 1.02 * 3 * E1) if case["field"] == "grid" else (100.0, 1000.0)


def _sr(case, x):
    from srsoriginal_b200.sr import sr
    o = sr()
    for f in _fields(case, x):
        if f[0] == "undulator":
            o.add_bfield_undulator(bfield=f[1], period=[0, 0, PERIOD], nperiods=NPERIODS, phase=f[2])
        else:
            o.add_bfield_grid([0, 0, f[1]], [0, 0, f[2]], [1, 1, len(f[3])], f[3])
    extra = {}
    if case["kind"] == "beam":
        extra = dict(sigma_energy_GeV=0.003, beta=[1.5, 0.8], emittance=[1e-9, 8e-12], horizontal_direction=[1, 0, 0],
                     lattice_reference=[0, 0, -1])
        x = dict(x, d0=[0.0, 0.0, 1.0])
    o.set_particle_beam(type="electron", name="beam_0", energy_GeV=x["energy"], x0=x["x0"], d0=x["d0"], current=CURRENT,
                        **extra)
    o.set_ctstartstop(x["start"], x["stop"])
    o.set_npoints_trajectory(case["npoints"])
    return o


def _job_sizes(case):
    from srsoriginal_b200.workloads import config3b_jobs
    return config3b_jobs(case["jobs"], case["set"])


def prepare(case, seed):
    x = _inputs(case, seed)
    if case["kind"] == "queue":
        return _prepare_queue(case, x)
    if case["kind"] == "adjoint":
        return _prepare_adjoint(case, x)
    state = dict(case=case, x=x, sr=_sr(case, x))
    if case["kind"] == "points":
        state["points"] = _curved_screen(case["n"])
    return state


def _prepare_queue(case, x):
    from srsoriginal_b200 import device as D, queue as Q
    from srsoriginal_b200.sr import energy_grid, rectangle_points
    specs = _job_sizes(case)
    part, _ = D.ideal_particle(x["energy"], x["x0"], x["d0"])
    und = D.undulator([0, x["bpeak"], 0], [0, 0, PERIOD], NPERIODS)
    nts = [s["nt"] for s in specs]
    k = len(specs)
    trajs = Q.trajectory_buffers([0.0] * k, [2.0] * k, [0.0] * k, nts)
    jobs = []
    for s, t in zip(specs, trajs):
        nout = s["n"] ** 2 if s["kind"] == "flux" else s["ne"]
        out = torch.empty(nout, dtype=torch.float64, device="cuda")
        if s["kind"] == "flux":
            g = rectangle_points([s["n"], s["n"]], plane="XY", width=[0.01, 0.01], translation=[0, 0, SCREEN])[3]
            jobs.append(Q.flux_job(t, -QE, CURRENT, g, E1 * x["photon"], out))
        else:
            e = torch.tensor(energy_grid(s["ne"], 100.0, 1000.0), dtype=torch.float64, device="cuda")
            jobs.append(Q.spectrum_job(t, -QE, CURRENT, [0, 0, SCREEN], e, out))
    q = Q.JobQueue(jobs, integrate=dict(fields=[und], particles=[part] * k, ctstart=0.0, ctstop=2.0, t0=0.0, npoints=nts))
    return dict(case=case, queue=q, outs=[j[1][-1] for j in jobs])


def _prepare_adjoint(case, x):
    from srsoriginal_b200 import device as D
    from srsoriginal_b200.adjoint import SpectrumProblem
    from srsoriginal_b200.sr import energy_grid
    z0, dz, data = _field_map(x["sample"], x["bpeak"], case["nz"])
    e = torch.tensor(energy_grid(case["ne"], 0.98 * 3 * E1, 1.02 * 3 * E1), dtype=torch.float64, device="cuda")
    problem = SpectrumProblem(fields=[D.grid_z(z0, dz, data[:, 1], None)], obs=(0.0, 0.0, SCREEN), energies=e,
                              npoints=case["npoints"], current=CURRENT)
    grid = torch.tensor(data, dtype=torch.float64, device="cuda", requires_grad=True)
    ic = torch.tensor([*x["x0"][:2], *x["d0"][:2], -1.0, x["energy"]], dtype=torch.float64, requires_grad=True)
    return dict(case=case, problem=problem, grid=grid, ic=ic)


# ------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "queue":
        state["queue"].run()
        return state["outs"]
    if kind == "adjoint":
        from srsoriginal_b200.adjoint import SpectrumFlux, integrated_flux_loss
        state["grid"].grad = state["ic"].grad = None
        flux = SpectrumFlux.apply(state["grid"], None, state["ic"], state["problem"])
        integrated_flux_loss(flux, 1.0).backward()
        return [flux.detach(), state["grid"].grad, state["ic"].grad]
    o, x, p = state["sr"], state["x"], case["precision"]
    o.set_trajectory_cache(True)  # drops the trajectory of the last pass: the beam may have changed
    if kind == "spectrum":
        e, f = o.spectrum_arrays(obs=[0, 0, SCREEN], npoints=case["ne"], energy_range_eV=list(_energy_range(case)),
                                 precision=p)
        return [e, f, o.calculate_total_power()] if case["field"] == "grid" else [e, f]
    if kind == "flux":
        return [o.flux_arrays(energy_eV=E1 * x["photon"] * (2 * m + 1), npoints=[case["n1"], case["n2"]], plane="XY",
                              width=[0.01, 0.01], translation=[0, 0, SCREEN], precision=p) for m in range(case["maps"])]
    if kind == "points":  # the list the reference returns, without the zero entries its dispatch appends
        return np.array([v for _, v in o.calculate_flux(E1 * x["photon"], state["points"], precision=p)[:case["n"]]])
    if kind == "power_density":
        return o.power_density_arrays(npoints=[case["n1"], case["n2"]], plane="XY", width=[0.04, 0.04],
                                      translation=[0, 0, SCREEN], precision=p)
    from srsoriginal_b200.sr import reset_random
    reset_random(x["sample"])  # the same electrons in every pass on this state
    return o.spectrum_arrays(obs=[0, 0, SCREEN], npoints=case["ne"], energy_range_eV=[100, 1000],
                             nparticles=case["particles"], precision=p)


def work(case):
    """Bytes: the outputs, and the trajectory (x, beta, a/c) written once and read once by each sum."""
    kind = case["kind"]
    if kind == "queue":
        b = f = 0.0
        for s in _job_sizes(case):
            nout = s["n"] ** 2 if s["kind"] == "flux" else s["ne"]
            b += 120.0 * s["nt"] + 8.0 * nout
            f += s["nt"] * (FLOPS[s["kind"]] * nout + STEP_FLOPS)
        return dict(bytes=b, flops=f)
    n, parts = case["npoints"], case.get("particles", 1)
    if kind == "adjoint":
        return dict(bytes=72.0 * 3 * n + 48.0 * case["nz"], flops=n * (3 * FLOPS["spectrum"] * case["ne"] + 6 * STEP_FLOPS))
    nout = dict(spectrum=lambda: case["ne"], beam=lambda: case["ne"], points=lambda: case["n"],
                flux=lambda: case["n1"] * case["n2"], power_density=lambda: case["n1"] * case["n2"])[kind]()
    maps = case.get("maps", 1)
    per = FLOPS[dict(points="flux", beam="spectrum").get(kind, kind)]
    read = 72.0 if kind == "power_density" else 48.0
    return dict(bytes=parts * n * (72.0 + maps * read) + 8.0 * nout * maps, flops=parts * n * (per * nout * maps + STEP_FLOPS))


# ------------------------------------------------------------------ the same in plain 64-bit arithmetic

def _trajectory(fields, x, npoints):
    """The fixed-step RK4 trajectory in Python floats: x, beta, a/c as (3, n), dt, gamma.  Forward from ct
    = 0 and backward to the start; a/c of a point is the derivative at the previous step's state."""
    g = x["energy"] / (1e-9 * ME * LIGHT * LIGHT / QE)
    b = math.sqrt(1.0 - 1.0 / (g * g))
    dn = math.sqrt(sum(v * v for v in x["d0"]))
    beta0 = [v / dn * b for v in x["d0"]]
    gamma = 1.0 / math.sqrt(1.0 - sum(v * v for v in beta0))
    q = -QE / ME / gamma
    dt = (x["stop"] - x["start"]) / LIGHT / (npoints - 1)
    nf, nb = int(1 + x["stop"] / LIGHT / dt), int(-x["start"] / LIGHT / dt)
    length, sin, tau = PERIOD * (NPERIODS + 2), math.sin, 2.0 * math.pi

    def field(z):
        bx = by = 0.0
        for f in fields:
            if f[0] == "grid":
                z0, dz, data = f[1:]
                k = int((z - z0) / dz)
                if z <= z0 or z >= z0 + (len(data) - 1) * dz:
                    continue
                k = min(k, len(data) - 2)
                by += data[k] + (data[k + 1] - data[k]) * ((z - z0) - k * dz) / dz
            else:
                ps = f[2] * PERIOD / tau
                if z > length / 2 + ps or z < -length / 2 + ps:
                    continue
                s = sin(tau * (z - ps) / PERIOD)
                if z < -length / 2 + ps + PERIOD or z > length / 2 + ps - PERIOD:
                    s *= 0.25 if z < -length / 2 + ps + PERIOD / 2 or z > length / 2 + ps - PERIOD / 2 else 0.75
                bx += f[1][0] * s
                by += f[1][1] * s
        return bx, by

    fields = [(f[0], f[1], f[2], f[3][:, 1].tolist()) if f[0] == "grid" else f for f in fields]
    n = nf + nb
    X, B, A = np.zeros((3, n)), np.zeros((3, n)), np.zeros((3, n))

    def force(vx, vy, vz, f):
        return q * (-vz * f[1]), q * (vz * f[0]), q * (vx * f[1] - vy * f[0])

    for h, count, first, step in ((dt, nf, nb, 1), (-dt, nb, nb - 1, -1)):
        px, py, pz = x["x0"]
        vx, vy, vz = (v * LIGHT for v in beta0)
        a1 = (0.0, 0.0, 0.0)
        hh, h6 = h * 0.5, h / 6.0
        for i in range(count + (step < 0)):
            k = first + step * (i - (step < 0))
            if step > 0 or i > 0:
                X[:, k] = px, py, pz
                B[:, k] = vx, vy, vz
                A[:, k] = a1
            if i == count - 1 + (step < 0):
                break
            a1 = force(vx, vy, vz, field(pz))
            ux, uy, uz = vx + hh * a1[0], vy + hh * a1[1], vz + hh * a1[2]
            a2 = force(ux, uy, uz, field(pz + hh * vz))
            wx, wy, wz = vx + hh * a2[0], vy + hh * a2[1], vz + hh * a2[2]
            a3 = force(wx, wy, wz, field(pz + hh * uz))
            rx, ry, rz = vx + h * a3[0], vy + h * a3[1], vz + h * a3[2]
            a4 = force(rx, ry, rz, field(pz + h * wz))
            px = px + h6 * (vx + rx + 2.0 * (wx + ux))
            py = py + h6 * (vy + ry + 2.0 * (wy + uy))
            pz = pz + h6 * (vz + rz + 2.0 * (wz + uz))
            vx = vx + h6 * (a1[0] + a4[0] + 2.0 * (a3[0] + a2[0]))
            vy = vy + h6 * (a1[1] + a4[1] + 2.0 * (a3[1] + a2[1]))
            vz = vz + h6 * (a1[2] + a4[2] + 2.0 * (a3[2] + a2[2]))
    return X, B / LIGHT, A / LIGHT, dt, gamma


def _tensors(*arrays):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return [torch.tensor(a, dtype=torch.float64, device=dev) for a in arrays]


def _flux_sum(X, B, dt, points, omegas):
    """|E|^2 with the reference's constants for pairs (points[j], omegas[j]), or one of either."""
    n = X.shape[1]
    nout = max(len(points), len(omegas))
    E = torch.zeros(3, nout, dtype=torch.complex128, device=X.device)
    block = max(1, 20_000_000 // nout)
    i = torch.arange(n, dtype=torch.float64, device=X.device)
    c = torch.full((1, 1), LIGHT, dtype=torch.float64, device=X.device)  # a tensor: torch multiplies by 1/scalar
    for s in range(0, n, block):
        R = [points[:, a][None] - X[a, s:s + block][:, None] for a in range(3)]
        D = torch.sqrt(R[0] * R[0] + R[1] * R[1] + R[2] * R[2])
        ph = omegas[None] * (dt * i[s:s + block][:, None] + D / c)
        k = torch.round(ph / (2 * math.pi))
        ph = (ph - k * 6.28125) - k * (2 * math.pi - 6.28125) - k * 2.4492935982947064e-16
        e = torch.polar(torch.ones_like(ph), ph)
        for a in range(3):
            N = R[a] / D
            E[a] += (torch.complex((B[a, s:s + block][:, None] - N) / D, -(N * (c / omegas[None] / D)) / D) * e).sum(0)
    c0 = -QE / (4 * math.pi * LIGHT * EPS0 * 2.5066282746310002416)
    c2 = 4 * math.pi * CURRENT / (PLANCK * QE * MU0 * LIGHT) * 1e-6 * 0.001
    return c2 * ((c0 * omegas * dt) ** 2 * (E.real ** 2 + E.imag ** 2).sum(0))


def _power(X, B, A, dt, points):
    n, nout = X.shape[1], len(points)
    total = torch.zeros(nout, dtype=torch.float64, device=X.device)
    block = max(1, 10_000_000 // nout)
    for s in range(0, n, block):
        R = torch.stack([points[:, c][None] - X[c, s:s + block][:, None] for c in range(3)])
        D2 = (R * R).sum(0)
        N = R / torch.sqrt(D2)
        b, a = B[:, s:s + block, None], A[:, s:s + block, None]
        V = torch.linalg.cross(N, torch.linalg.cross(N - b, a.expand_as(N), dim=0), dim=0)
        total += ((V * V).sum(0) / (1 - (N * b).sum(0)) ** 5 / D2 * N[2]).sum(0)
    return (total * (QE * CURRENT / (16 * math.pi ** 2 * EPS0 * LIGHT) * dt / 1e6)).abs()


def _rectangle(case, width):
    s1, s2 = width / (case["n1"] - 1), width / (case["n2"] - 1)
    i1, i2 = np.meshgrid(np.arange(case["n1"]), np.arange(case["n2"]), indexing="ij")
    x, y = -width / 2 + s1 * i1.reshape(-1), -width / 2 + s2 * i2.reshape(-1)
    return np.column_stack([x, y, np.full(x.size, SCREEN)])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("queue", "adjoint", "beam"):  # many trajectories, or many more evaluations than 20 s allow
        return None
    x = _inputs(case, seed)
    X, B, A, dt, gamma = _trajectory(_fields(case, x), x, case["npoints"])
    total = (QE * CURRENT) * gamma ** 6 / (6 * math.pi * EPS0 * LIGHT) * dt * float(
        (A ** 2).sum() - (np.cross(B, A, axis=0) ** 2).sum())
    X, B, A = _tensors(X, B, A)
    if kind == "spectrum":
        lo, hi = _energy_range(case)
        e = lo + (hi - lo) / (case["ne"] - 1) * np.arange(1, case["ne"] + 1)
        f = _flux_sum(X, B, dt, *_tensors([[0.0, 0.0, SCREEN]], e * QE / HBAR))
        return [e, f, total] if case["field"] == "grid" else [e, f]
    if kind == "flux":
        xyz = _rectangle(case, 0.01)
        return [(xyz, _flux_sum(X, B, dt, *_tensors(xyz, [E1 * x["photon"] * (2 * m + 1) * QE / HBAR])))
                for m in range(case["maps"])]
    if kind == "points":
        xyz = np.array([p for p, _ in _curved_screen(case["n"])])
        return _flux_sum(X, B, dt, *_tensors(xyz, [E1 * x["photon"] * QE / HBAR]))
    xyz = _rectangle(case, 0.04)
    return xyz, _power(X, B, A, dt, _tensors(xyz)[0])
