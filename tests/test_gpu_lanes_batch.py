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
