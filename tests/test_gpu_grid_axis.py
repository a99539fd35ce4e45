"""Field maps along one axis: the parallel-in-time kernels evaluate them without the other axes and the rotation.
The same map with its samples repeated along a second axis takes the general interpolation, whose extra
step (a + 0 between equal samples) is exact: the trajectories are equal bit for bit, and the shooting
trajectory stays within its bars (positions and beta 2e-14, a/c 1e-12 of its largest) of them."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(axis, n, shift, second=None):
    import torch

    from srsoriginal_b200 import _lib, device as D

    shape, start, step, tr = [1, 1, 1], [0.0] * 3, [0.0] * 3, [0.0] * 3
    shape[axis], start[axis], step[axis], tr[axis] = n, -0.9, 1.8 / (n - 1), shift
    tr[(axis + 1) % 3] = 0.25 * shift  # (of no consequence: the map does not depend on it)
    z = -0.9 + step[axis] * np.arange(n)
    b = np.stack([np.sin(2 * np.pi * z / 0.049 + 0.3 * c) * 0.8 ** c + 0.01 * c for c in range(3)], axis=-1)
    b[:, axis] *= 0.1
    full = b.reshape(shape + [3])
    if second is not None:
        shape[second], start[second], step[second] = 2, -1.0, 2.0
        full = np.repeat(full, 2, axis=second)
    data = torch.tensor(np.ascontiguousarray(full).reshape(-1, 3), device="cuda")
    f = _lib.Field()
    f.kind = _lib.GRID
    for a in range(3):
        f.n[a] = shape[a]
    f.start, f.step, f.translation = _lib.v3(start), _lib.v3(step), _lib.v3(tr)
    f.data = D._dptr(data)
    return f, data


# The smallest map (one cell), one cell more, an ordinary one, one too large for shared memory (24576 doubles);
# trajectories that enter and leave it; two chains.
@pytest.mark.parametrize("axis,n,shift,start", [(2, 2, 0.0, 0.0), (2, 3, 0.01, 0.0), (2, 1801, 0.0, 0.0),
                                                (2, 1801, -0.0123, -1.0), (2, 9001, 0.003, 0.0), (0, 1801, 0.01, 0.0),
                                                (1, 1200, -0.02, -1.0), (1, 2, 0.0, -1.0)])
def test_map_along_one_axis_equals_the_general_interpolation(axis, n, shift, start):
    import torch

    from srsoriginal_b200 import device as D

    x0, d0 = [1e-5, -2e-5, 3e-5], [2e-6, -1e-6, 3e-6]
    x0[axis], d0[axis] = (-1.0 if start == 0.0 else 0.0), 1.0
    part, _ = D.ideal_particle(3.0, x0, d0)
    one, keep1 = _grid(axis, n, shift)
    two, keep2 = _grid(axis, n, shift, (axis + 2) % 3)
    a = D.trajectory([one], [part], start, start + 2.0, 0.0, 4001)
    b = D.trajectory([two], [part], start, start + 2.0, 0.0, 4001)
    s = D.trajectory_shoot([one], part, start, start + 2.0, 0.0, 4001)
    torch.cuda.synchronize()
    assert a.aoc.abs().max() > 0
    for k, bar in (("x", 2e-14), ("beta", 2e-14), ("aoc", 1e-12)):
        assert torch.equal(getattr(a, k), getattr(b, k)), k
        size = b.aoc.abs().max() if k == "aoc" else 1.0  # (the bar of a/c is relative to its largest)
        assert (getattr(s, k)[0] - getattr(b, k)[0]).abs().max() <= bar * size, k


# The adjoint through such maps against the general corners of the doubled map, whose samples' gradients add up to
# the single map's.  The weights carry one more rounding each; a step's terms are bounded by the adjoint of the
# directions (every gradient with its lever arm) times q h, a gradient passes through at most all steps, and a
# step is ~60 rounded operations.
@pytest.mark.parametrize("axis,n,shift,start", [(2, 2, 0.0, 0.0), (2, 901, 0.01, 0.0), (0, 901, -0.02, 0.0), (1, 300, 0.0, -1.0)])
def test_adjoint_through_a_map_along_one_axis(axis, n, shift, start):
    import torch

    from srsoriginal_b200 import _lib, device as D

    npoints = 385
    x0, d0 = [1e-5, -2e-5, 3e-5], [2e-6, -1e-6, 3e-6]
    x0[axis], d0[axis] = (-1.0 if start == 0.0 else 0.0), 1.0
    part, _ = D.ideal_particle(3.0, x0, d0)
    one, keep = _grid(axis, n, shift)
    tr = D.trajectory([one], [part], start, start + 2.0, 0.0, npoints)
    m = tr.x.shape[-1]
    rng = np.random.default_rng(n)
    gx, gb = (torch.tensor(rng.normal(size=3 * m), device="cuda") for _ in range(2))
    ptr = lambda t: C.c_void_p(t.data_ptr())
    got = []
    for second in (None, (axis + 2) % 3):
        f, data = _grid(axis, n, shift, second)
        grad, ic = torch.zeros_like(data), (C.c_double * 7)()
        _lib.check(_lib.lib.srs_trajectory_adjoint((_lib.Field * 1)(f), 1, (_lib.Particle * 1)(part), start, start + 2.0, 0.0,
                                                   npoints, ptr(tr.x), ptr(tr.beta), ptr(gx), ptr(gb),
                                                   (C.c_void_p * 1)(grad.data_ptr()), None, ic, D._stream()))
        shape = [1, 1, 1]
        shape[axis] = n
        if second is not None:
            shape[second] = 2
            grad = grad.reshape(shape + [3]).sum(dim=second)
        got.append((grad.reshape(n, 3).cpu().numpy(), np.array(ic[:])))
    span = 4.0
    q, h = abs(part.qomg), tr.dt
    sbeta = (gb.abs().sum() + span * gx.abs().sum()).item()
    step = sbeta * q * h
    eps = 60 * m * 2.0 ** -53
    assert np.abs(got[0][0]).max() > 0
    assert np.abs(got[0][0] - got[1][0]).max() <= eps * m * step
    slope = 1.3 * 2 * np.pi / 0.049  # of the field
    assert np.abs(got[0][1][:3] - got[1][1][:3]).max() <= eps * (gx.abs().sum().item() + m * step * slope)
    assert np.abs(got[0][1][3:6] - got[1][1][3:6]).max() <= eps * sbeta
    assert abs(got[0][1][6] - got[1][1][6]) <= eps * m * step * 1.3 / q
