"""How the trajectories of few particles are integrated (srs_trajectory_route), and that a particle for which the
parallel iteration does not contract ends in the serial kernel with its bits.  Field maps are what gets there: their
strength is not known before the first pass.  The serial kernel is reached as in test_gpu_exact.py."""
import numpy as np
import pytest

from test_gpu_exact import MANY, _fields

pytestmark = pytest.mark.gpu


def _map(axis, values):
    import torch

    from srsoriginal_b200 import _lib, device as D

    s = np.linspace(-1.05, 1.05, 701)
    by = values(s)
    data = torch.tensor(np.column_stack([0 * by, by, 0 * by]), device="cuda")
    f = _lib.Field()
    f.kind = _lib.GRID
    for a in range(3):
        f.n[a] = len(s) if a == axis else 1
        f.start[a] = s[0] if a == axis else 0.0
        f.step[a] = s[1] - s[0] if a == axis else 0.0
    f.data = D._dptr(data)
    return f, data


MAPS = {
    "wiggler": (2, lambda z: np.sin(2 * np.pi * z / 0.049) * (np.abs(z) < 0.8)),
    "dipole": (2, lambda z: 0.5 + 0 * z),
    # weak where straight flight goes, strong where the particle is turned to
    "wall": (0, lambda x: np.where(x > 0.02, 5.0, 0.1)),
}


def _route(fields, parts, start, npoints):
    import torch

    from srsoriginal_b200 import _lib, device as D

    dt, nf, nb = D.counts(start, start + 2.0, 0.0, npoints)
    out = D.Trajectory(*(torch.empty((len(parts), 3, nf + nb), dtype=torch.float64, device="cuda") for _ in range(3)),
                       dt)
    route = torch.full((len(parts),), -1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib.srs_trajectory_route((_lib.Field * len(fields))(*fields), len(fields),
                                             (_lib.Particle * len(parts))(*parts), len(parts), start, start + 2.0, 0.0,
                                             npoints, D._ptr(out.x), D._ptr(out.beta), D._ptr(out.aoc), D._ptr(route),
                                             D._stream()))
    return out, route


# 0.05 GeV is turned by 8 and 6 rad and given up after the first pass; 0.23 GeV by 1.28 through the wiggler, below
# the limit of 1.3, goes through all sweeps without reproducing every step; 300 and 2001 points by the chain
# kernel, 6001 by runs; one particle of several that is given up gives all up.
@pytest.mark.parametrize("name,energies,npoints,start,route", [
    ("wiggler", [3.0], 2001, -1.0, "PARALLEL"), ("dipole", [0.6], 6001, 0.0, "PARALLEL"),
    ("wiggler", [0.05], 300, 0.0, "GIVEN_UP"), ("dipole", [0.05], 2001, -1.0, "GIVEN_UP"),
    ("dipole", [0.05], 6001, 0.0, "GIVEN_UP"), ("wall", [0.05], 2001, 0.0, "GIVEN_UP"),
    ("wiggler", [0.23], 300, 0.0, "GIVEN_UP"), ("wiggler", [0.23], 6001, 0.0, "GIVEN_UP"),
    ("wiggler", [3.0, 2.5, 3.1, 0.05, 2.9], 1025, -1.0, "GIVEN_UP"),
    ("wiggler", [3.0, 2.5, 3.1, 0.23, 2.9], 1025, 0.0, "GIVEN_UP"),
    ("wiggler", [3.0], 256, 0.0, "SERIAL"), ("wiggler", [3.0] * MANY, 300, 0.0, "SERIAL"),
])
def test_route_and_the_serial_bits(name, energies, npoints, start, route):
    import torch

    from srsoriginal_b200 import _lib, device as D

    f, keep = _map(*MAPS[name])
    z0 = -1.0 if start == 0.0 else 0.0
    parts = [D.ideal_particle(e, [1e-6 * k, 0, z0], [1e-5, 0, 1] if name != "wall" else [0, 0, 1])[0]
             for k, e in enumerate(energies)]
    if name == "wall":
        parts[0].qomg = -abs(parts[0].qomg)  # turned to positive x
    got, taken = _route([f], parts, start, npoints)
    many = D.trajectory([f] + _fields("nothing")[0], (parts * MANY)[:max(MANY, len(parts))], start, start + 2.0, 0.0,
                        npoints)
    torch.cuda.synchronize()
    if name == "wall":
        assert got.x[0, 0].max() > 0.02
    assert taken.tolist() == [getattr(_lib, "ROUTE_" + route)] * len(parts)
    for a in ("x", "beta", "aoc"):
        assert torch.equal(getattr(got, a), getattr(many, a)[:len(parts)]), a


def test_route_of_undulators():
    import torch

    from srsoriginal_b200 import _lib, device as D

    und = _fields("undulator")[0]
    part, _ = D.ideal_particle(3.0, [0, 0, -1.0], [0, 0, 1])
    slow, _ = D.ideal_particle(0.05, [0, 0, -1.0], [0, 0, 1])
    routes = [_route(und, p, 0.0, 1025)[1] for p in ([part], [part] * MANY, [slow])]
    torch.cuda.synchronize()
    want = (_lib.ROUTE_PARALLEL, _lib.ROUTE_LANES, _lib.ROUTE_SERIAL)
    assert [r.tolist() for r in routes] == [[w] * len(r) for w, r in zip(want, routes)]
