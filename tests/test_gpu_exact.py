"""The trajectory kernels of few and of many particles against the serial one, bit for bit: few are
integrated parallel in time, many through undulators along z take one lane each.  The serial kernel is
reached by integrating more than 256 particles at once with a field of no amplitude added to the list
(x + 0 is exact)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MANY = 257


def _fields(name):
    import torch

    from srsoriginal_b200 import _lib, device as D

    def shape(kind, b, c, s, rot=(0, 0, 0)):
        f = _lib.Field()
        f.kind = kind
        f.field, f.center, f.sigma_or_width, f.rotations = _lib.v3(b), _lib.v3(c), _lib.v3(s), _lib.v3(rot)
        return f

    if name == "nothing":
        return [shape(_lib.GAUSSIAN, (0, 0, 0), (0, 0, 0), (0, 0, 1.0))], None
    und = D.undulator([0, 1.0, 0], [0, 0, 0.049], 31)
    if name == "undulator":
        return [und], None
    if name in ("epu", "taper"):
        return [und, D.undulator([0.6, 0, 0], [0, 0, 0.049], 31, phase=math.pi / 2,
                                 taper=0.01 if name == "taper" else 0.0)], None
    if name == "none":
        return [], None
    if name == "grid":
        z = np.linspace(-1.05, 1.05, 701)
        by = np.sin(2 * np.pi * z / 0.049) * (np.abs(z) < 0.8)
        data = torch.tensor(np.column_stack([0 * by, by, 0 * by]), device="cuda")
        return [D.grid_z(z[0], z[1] - z[0], by, data)], data
    return [shape(_lib.GAUSSIAN, (0, 1, 0), (0, 0, 0), (0, 0, 0.05)),
            shape(_lib.GAUSSIAN, (0.3, 0.4, 0.2), (0, 0, 0.3), (0.01, 0.02, 0.05), (0.1, 0.2, 0.3)),
            shape(_lib.UNIFORM_BOX, (0, 0.2, 0.1), (0, 0, -0.5), (0, 0, 0.3))], None


# The sizes sit at the edges of the blocks (128 steps), of the chain's tiles (256 states) and of the rule
# (more than 256 steps); "two chains" starts in the middle; 0.05 GeV does not contract and ends in the
# serial kernel.
@pytest.mark.parametrize("field,npoints,energy,start", [
    ("undulator", 257, 3.0, 0.0), ("undulator", 258, 3.0, 0.0), ("undulator", 385, 3.0, 0.0),
    ("undulator", 512, 3.0, 0.0), ("undulator", 513, 3.0, 0.0), ("undulator", 20001, 2.997, 0.0),
    ("undulator", 4097, 3.0, -1.0), ("undulator", 3001, 0.05, 0.0), ("undulator", 16641, 0.5, 0.0),
    ("taper", 9999, 3.0, 0.0), ("epu", 40001, 3.0, 0.0), ("grid", 2049, 3.0, -1.0), ("none", 1025, 3.0, 0.0),
    ("mixed", 5003, 3.0, -0.7),
])
def test_single_trajectory_equals_the_serial_kernel_bitwise(field, npoints, energy, start):
    import torch

    from srsoriginal_b200 import device as D

    fields, keep = _fields(field)
    x0 = [1e-5, -2e-5, -1.0 if start == 0.0 else 0.0]
    part, _ = D.ideal_particle(energy, x0, [3e-6, -5e-6, 1])
    one = D.trajectory(fields, [part], start, start + 2.0, 0.0, npoints)
    many = D.trajectory(fields + _fields("nothing")[0], [part] * MANY, start, start + 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    for a in ("x", "beta", "aoc"):
        assert torch.equal(getattr(one, a)[0], getattr(many, a)[MANY - 1]), a


def test_few_particles_together_equal_the_serial_kernel_bitwise():
    import torch

    from srsoriginal_b200 import device as D

    fields, _ = _fields("undulator")
    rng = np.random.default_rng(5)
    parts = [D.ideal_particle(3.0 * (1 + 1e-3 * rng.normal()), [3e-5 * rng.normal(), 1e-5 * rng.normal(), 0.0],
                              [2e-5 * rng.normal(), 1e-5 * rng.normal(), 1])[0] for _ in range(7)]
    few = D.trajectory(fields, parts, -1.0, 1.0, 0.0, 3001)
    many = D.trajectory(fields + _fields("nothing")[0], parts * 37, -1.0, 1.0, 0.0, 3001)
    torch.cuda.synchronize()
    for a in ("x", "beta", "aoc"):
        assert torch.equal(getattr(few, a), getattr(many, a)[:7]), a


# Chains added by runs (from 4500 steps and 3 per block of 128): the first length that is, a full last block and
# one step in it, full groups of 12 blocks and one block more, two particles whose positions cross many
# binades (x0 = 0), several particles in two chains.
@pytest.mark.parametrize("field,particles,npoints,start", [
    ("undulator", 1, 4608, 0.0), ("undulator", 1, 4609, 0.0), ("undulator", 1, 4612, 0.0), ("epu", 1, 4738, 0.0),
    ("undulator", 2, 6145, 0.0), ("undulator", 4, 12001, -1.0), ("mixed", 2, 12289, -0.5), ("none", 1, 6001, 0.0),
    ("grid", 1, 18434, -1.0),
])
def test_chains_by_runs_equal_the_serial_kernel_bitwise(field, particles, npoints, start):
    import torch

    from srsoriginal_b200 import device as D

    fields, keep = _fields(field)
    rng = np.random.default_rng(npoints)
    parts = [D.ideal_particle(3.0 - 0.3 * i, [1e-6 * i * rng.normal(), 0.0, -1.0 if start == 0.0 else 0.0],
                              [3e-6 * i * rng.normal(), 1e-6 * i, 1])[0] for i in range(particles)]
    few = D.trajectory(fields, parts, start, start + 2.0, 0.0, npoints)
    many = D.trajectory(fields + _fields("nothing")[0], parts * MANY, start, start + 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    for a in ("x", "beta", "aoc"):
        assert torch.equal(getattr(few, a), getattr(many, a)[:particles]), a


def test_batches_beyond_the_scratch_bound_go_half_by_half():
    import torch

    from srsoriginal_b200 import device as D

    fields, _ = _fields("undulator")
    parts = [D.ideal_particle(3.0 - 0.01 * i, [1e-6 * i, 0, -1.0], [1e-7 * i, 0, 1])[0] for i in range(5)]
    n = 6000001  # 5 x 6e6 steps of 144 bytes: 4.3 GB, one particle's 0.9
    all_ = D.trajectory(fields, parts, 0.0, 2.0, 0.0, n)
    for i in (0, 2, 4):
        one = D.trajectory(fields, [parts[i]], 0.0, 2.0, 0.0, n)
        torch.cuda.synchronize()
        for a in ("x", "beta", "aoc"):
            assert torch.equal(getattr(one, a)[0], getattr(all_, a)[i]), (i, a)


# Sizes at the edges of the lane kernel: one, two and four particles per warp, the two chains, a last
# block that is not full.
@pytest.mark.parametrize("field,particles,npoints,start", [
    ("undulator", 257, 2, 0.0), ("undulator", 257, 5001, 0.0), ("undulator", 601, 1025, -1.0),
    ("epu", 1303, 2050, 0.0), ("undulator", 300, 401, 0.0), ("epu", 2500, 333, -1.0),
])
def test_many_particles_equal_the_serial_kernel_bitwise(field, particles, npoints, start):
    import torch

    from srsoriginal_b200 import device as D

    fields, _ = _fields(field)
    rng = np.random.default_rng(particles)
    z0 = -1.0 if start == 0.0 else 0.0
    parts = [D.ideal_particle(3.0 * (1 + 1e-3 * rng.normal()), [3e-5 * rng.normal(), 1e-5 * rng.normal(), z0],
                              [2e-5 * rng.normal(), 1e-5 * rng.normal(), 1])[0] for _ in range(particles)]
    got = D.trajectory(fields, parts, start, start + 2.0, 0.0, npoints)
    ref = D.trajectory(fields + _fields("nothing")[0], parts, start, start + 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    for a in ("x", "beta", "aoc"):
        assert torch.equal(getattr(got, a), getattr(ref, a)), a


# What the lane kernel's phase bound does not cover takes the serial kernel: steps that turn the velocity by more
# than a radian (RK4 grows without bound beyond 2.8), a particle faster than light
@pytest.mark.parametrize("energy,npoints,faster", [(0.02, 60, 1.0), (0.005, 30, 1.0), (3.0, 500, 5.0)])
def test_batches_beyond_the_phase_bound_equal_the_serial_kernel_bitwise(energy, npoints, faster):
    import torch

    from srsoriginal_b200 import _lib, device as D

    und = D.undulator([0, 3.0, 0], [0, 0, 0.049], 31)
    part, _ = D.ideal_particle(energy, [0, 0, -1.0], [1e-4, 0, 1])
    part.beta0 = _lib.v3([faster * b for b in part.beta0])
    a = D.trajectory([und], [part] * MANY, 0.0, 2.0, 0.0, npoints)
    b = D.trajectory([und] + _fields("nothing")[0], [part] * MANY, 0.0, 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    for k in ("x", "beta", "aoc"):
        assert torch.equal(torch.nan_to_num(getattr(a, k), nan=7.0), torch.nan_to_num(getattr(b, k), nan=7.0)), k
