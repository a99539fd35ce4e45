"""The trajectories of few and of many particles against the serial kernel with the sign of zero, which particles
that start at -0 keep until a step adds +0: a field component of zero has the serial kernel's sign.  That kernel is
reached as in test_gpu_exact.py."""
import pytest

from test_gpu_exact import MANY, _fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["undulator", "epu", "grid"])
@pytest.mark.parametrize("particles,npoints", [(1, 1025), (1, 6001), (MANY, 1025)])
@pytest.mark.parametrize("start", [0.0, -1.0])
@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("charge", [-1, 1])
def test_zeros_have_the_serial_sign(field, particles, npoints, start, zero, charge):
    import torch

    from srsoriginal_b200 import device as D

    fields, keep = _fields(field)
    part, _ = D.ideal_particle(3.0, [zero, zero, -1.0 if start == 0.0 else zero], [zero, zero, 1],
                               charge=charge * D.QE)
    got = D.trajectory(fields, [part] * particles, start, start + 2.0, 0.0, npoints)
    ref = D.trajectory(fields + _fields("nothing")[0], [part] * MANY, start, start + 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    for a in ("x", "beta", "aoc"):
        g, r = getattr(got, a), getattr(ref, a)[:particles]
        assert torch.equal(g.view(torch.int64), r.view(torch.int64)), a
