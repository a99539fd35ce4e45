"""Many trajectories of unequal lengths through undulators along z (srs_trajectory_batch, one chain per lane): chains of
a few long steps beside chains of many short ones, whose lanes go on after the short ones' ends.  Bit for bit the
serial kernel's, which is reached as in test_gpu_exact.py."""
import pytest

from test_gpu_exact import MANY, _fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["undulator", "epu"])
def test_short_chains_beside_long_ones(field):
    import torch

    from srsoriginal_b200 import device as D, queue as Q

    fields = _fields(field)[0]
    lengths = [2001, 2, 257, 3, 1024, 2, 255]
    n = MANY + 50
    parts, stop, npts = [], [], []
    for k in range(n):
        parts.append(D.ideal_particle(3.0 - 1e-3 * k, [1e-6 * k, 0, -1.0], [1e-6 * (k % 5), 0, 1])[0])
        npts.append(lengths[k % len(lengths)])
        stop.append(2.0 if npts[-1] > 3 else 100.0)  # steps of up to 100 m, against 1 mm
    start, t0 = [0.0 if k % 3 else -0.5 for k in range(n)], [0.0] * n
    got = Q.trajectory_batch(fields, parts, start, stop, t0, npts)
    ref = Q.trajectory_batch(fields + _fields("nothing")[0], parts, start, stop, t0, npts)
    torch.cuda.synchronize()
    for k in range(n):
        for a in ("x", "beta", "aoc"):
            assert torch.equal(getattr(got[k], a), getattr(ref[k], a)), (k, a)


# The counts of steps and chains between which a batch takes the lanes: 128 steps; not up to a twentieth above 16
# lanes of a warp on each of 592 schedulers (one undulator, one chain), nor above 32.
@pytest.mark.parametrize("field,particles,npoints,start,route", [
    ("undulator", MANY, 128, 0.0, "SERIAL"), ("undulator", MANY, 129, 0.0, "LANES"), ("epu", MANY, 260, -1.0, "LANES"),
    ("undulator", 9472, 129, 0.0, "LANES"), ("undulator", 9473, 129, 0.0, "SERIAL"),
    ("undulator", 9944, 129, 0.0, "SERIAL"), ("undulator", 9945, 129, 0.0, "LANES"), ("epu", 9473, 129, 0.0, "LANES"),
    ("undulator", 4800, 260, -1.0, "LANES"), ("epu", 18944, 129, 0.0, "LANES"), ("epu", 18945, 129, 0.0, "SERIAL"),
    ("undulator", 9473, 260, -1.0, "SERIAL"), ("undulator", 19891, 129, 0.0, "LANES"),
])
def test_route_and_bits_at_the_edges_of_the_rule(field, particles, npoints, start, route):
    import torch

    from srsoriginal_b200 import _lib, device as D
    from test_gpu_exact_route import _route

    fields = _fields(field)[0]
    z0 = -1.0 if start == 0.0 else 0.0
    parts = [D.ideal_particle(3.0 - 1e-2 * k, [1e-6 * k, 0, z0], [1e-6 * k, 0, 1])[0] for k in range(7)]
    parts = (parts * (particles // 7 + 1))[:particles]
    got, taken = _route(fields, parts, start, npoints)
    ref = D.trajectory(fields + _fields("nothing")[0], parts, start, start + 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    assert (taken == getattr(_lib, "ROUTE_" + route)).all()
    for a in ("x", "beta", "aoc"):
        assert torch.equal(getattr(got, a), getattr(ref, a)), a


# A step whose stages lie in different fields lengthens the velocity, by up to 1.06 c^2 here: steps of 1 m through periods
# of 1 / 20.5 m find the field 0, 1, 1, 0 at their stages.  Beside a long trajectory such a short one is integrated
# parallel in time, 0.72 rad per step.
@pytest.mark.parametrize("npoints", [3, 4])
def test_a_step_that_lengthens_the_velocity(npoints):
    import torch

    from srsoriginal_b200 import device as D, queue as Q

    und = [D.undulator([0, 1.0, 0], [0, 0, 1 / 20.5], 121)]
    parts = [D.ideal_particle(0.4183 * npoints / 3, [0, 0, 0], [0, 0, 1])[0] for _ in range(2)]
    args = [0.0, 0.0], [npoints - 1.0, 2.0], [0.0, 0.0], [npoints, 300]
    got = Q.trajectory_batch(und, parts, *args)
    many = Q.trajectory_batch(und + _fields("nothing")[0], parts * MANY, *[a * MANY for a in args])
    torch.cuda.synchronize()
    if npoints == 3:
        assert (got[0].beta ** 2).sum(1).max() > 1.05
    for k in range(2):
        for a in ("x", "beta", "aoc"):
            assert torch.equal(getattr(got[k], a), getattr(many[k], a)), (k, a)
