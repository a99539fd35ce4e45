"""What is not a number beside the axis that an undulator along z or a map along one axis depends on: the serial
kernel multiplies it by the direction's zeros, which gives NaN, so the faster kernels must not leave it out.  The
serial kernel is reached as in test_gpu_exact.py."""
import pytest

from test_gpu_exact import MANY, _fields
from test_gpu_nonfinite import _same

pytestmark = pytest.mark.gpu


def _compare(fields, parts, npoints):
    import torch

    from srsoriginal_b200 import device as D

    got = D.trajectory(fields, parts, 0.0, 2.0, 0.0, npoints)
    ref = D.trajectory(fields + _fields("nothing")[0], [parts[0]] * (MANY - len(parts)) + parts, 0.0, 2.0, 0.0,
                       npoints)
    torch.cuda.synchronize()
    assert not ref.x[-1].isfinite().all()
    for a in ("x", "beta", "aoc"):
        assert _same(getattr(got, a), getattr(ref, a)[-len(parts):]), a
    return ref


@pytest.mark.parametrize("field,particles", [("undulator", 1), ("epu", 3), ("undulator", MANY), ("grid", 1), ("grid", 3)])
@pytest.mark.parametrize("axis,value", [(0, "nan"), (1, "inf")])
def test_starts_across_the_axis(field, particles, axis, value):
    import torch

    from srsoriginal_b200 import _lib, device as D

    fields, _keep = _fields(field)
    part, _ = D.ideal_particle(3.0, [1e-5, -2e-5, -1.0], [3e-6, -5e-6, 1])
    odd = _lib.Particle(part.x0, part.beta0, part.qomg)
    odd.x0[axis] = float(value)
    ref = _compare(fields, [part] * (particles - 1) + [odd], 2001)
    if particles == 1:
        shoot = D.trajectory_shoot(fields, odd, 0.0, 2.0, 0.0, 2001)
        torch.cuda.synchronize()
        for a in ("x", "beta"):
            assert torch.equal(getattr(shoot, a)[0].isnan(), getattr(ref, a)[-1].isnan()), a


@pytest.mark.parametrize("particles", [1, MANY])
@pytest.mark.parametrize("value", ["nan", "inf"])
def test_centres_across_the_axis(particles, value):
    from srsoriginal_b200 import device as D

    part, _ = D.ideal_particle(3.0, [1e-5, -2e-5, -1.0], [3e-6, -5e-6, 1])
    und = D.undulator([0, 1.0, 0], [0, 0, 0.049], 31)
    und.center[1] = float(value)
    _compare([und], [part] * particles, 601)
