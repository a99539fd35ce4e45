"""Trajectories that leave the finite numbers: where the serial kernel gives NaN the parallel-in-time ones give
NaN, and the points before keep its bits.  The serial kernel is reached as in test_gpu_exact.py."""
import numpy as np
import pytest

from test_gpu_exact import MANY, _fields

pytestmark = pytest.mark.gpu


def _same(a, b):
    """Equal bits, or NaN in both."""
    import torch

    return bool(((a.view(torch.int64) == b.view(torch.int64)) | (a.isnan() & b.isnan())).all())


# A map with one sample that is no number, along each axis (the particle flies along z): the positions become
# NaN at that sample (for a map across the flight at once) and are looked up in the map again.
@pytest.mark.parametrize("axis,value,npoints,start", [
    (2, "nan", 2049, -1.0), (2, "inf", 5003, 0.0), (2, "nan", 12001, -1.0), (0, "nan", 1025, 0.0),
    (1, "-inf", 1025, -1.0),
])
def test_maps_with_a_sample_that_is_no_number(axis, value, npoints, start):
    import torch

    from srsoriginal_b200 import _lib, device as D

    s = np.linspace(-1.05, 1.05, 701)
    by = np.sin(2 * np.pi * s / 0.049) * (np.abs(s) < 0.8)
    data = np.column_stack([0 * by, by, 0 * by])
    data[400 if axis == 2 else 350, 1] = float(value)
    data = torch.tensor(data, device="cuda")
    f = _lib.Field()
    f.kind = _lib.GRID
    for a in range(3):
        f.n[a] = len(s) if a == axis else 1
        f.start[a] = s[0] if a == axis else 0.0
        f.step[a] = s[1] - s[0] if a == axis else 0.0
    f.data = D._dptr(data)
    part, _ = D.ideal_particle(3.0, [1e-5, -2e-5, -1.0 if start == 0.0 else 0.0], [3e-6, -5e-6, 1])
    many = D.trajectory([f] + _fields("nothing")[0], [part] * MANY, start, start + 2.0, 0.0, npoints)
    exact = D.trajectory([f], [part], start, start + 2.0, 0.0, npoints)
    shoot = D.trajectory_shoot([f], part, start, start + 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    assert many.x.isnan().any() and not many.x.isnan().all()
    for a in ("x", "beta", "aoc"):
        assert _same(getattr(exact, a)[0], getattr(many, a)[MANY - 1]), a
    for a in ("x", "beta"):  # (a segment's first a/c is formed from the segment before it, NaN or not)
        assert torch.equal(getattr(shoot, a)[0].isnan(), getattr(many, a)[MANY - 1].isnan()), a


# A start height or a charge that is no number, alone and in a batch: the undulator kernels' sines take both for
# finite, so such calls take the serial kernel.
@pytest.mark.parametrize("field", ["undulator", "epu"])
@pytest.mark.parametrize("particles", [1, MANY])
@pytest.mark.parametrize("what", ["z nan", "z inf", "charge nan"])
def test_starts_that_are_no_numbers(field, particles, what):
    import torch

    from srsoriginal_b200 import _lib, device as D

    fields = _fields(field)[0]
    part, _ = D.ideal_particle(3.0, [1e-5, -2e-5, -1.0], [3e-6, -5e-6, 1])
    odd = _lib.Particle(part.x0, part.beta0, float("nan") if what == "charge nan" else part.qomg)
    if what != "charge nan":
        odd.x0[2] = float(what.split()[1])
    parts = [part] * (particles - 1) + [odd]
    got = D.trajectory(fields, parts, 0.0, 2.0, 0.0, 601)
    ref = D.trajectory(fields + _fields("nothing")[0], [part] * (MANY - particles) + parts, 0.0, 2.0, 0.0, 601)
    torch.cuda.synchronize()
    assert not ref.x[-1].isfinite().all()
    for a in ("x", "beta", "aoc"):
        assert _same(getattr(got, a), getattr(ref, a)[-particles:]), a
