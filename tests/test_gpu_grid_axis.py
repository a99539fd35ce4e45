"""Field maps along one axis: the parallel-in-time kernels evaluate them without the other axes and the rotation.
The same map with its samples repeated along a second axis takes the general interpolation, whose extra
step (a + 0 between equal samples) is exact: the trajectories are equal bit for bit, and the shooting
trajectory stays within its bars (positions and beta 2e-14, a/c 1e-12 of its largest) of them."""
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
