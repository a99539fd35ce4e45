"""The plain FP64 sums at the edges of their tiles and splits (128 outputs per CTA, 128-point tiles,
chunks in multiples of 32 points), against the oracle on the same trajectory: 1e-10 normwise, the bar of
the drop-in (the terms' phases and distances are the oracle's to the last bit, every other operation
carries ~1e-16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _trajectory(npoints):
    import torch

    from srsoriginal_b200 import device as D

    und = D.undulator([0.3, 1.0, 0], [0, 0, 0.049], 31)
    part, _ = D.ideal_particle(3.0, [1e-5, -2e-5, -1], [2e-6, -3e-6, 1])
    t = D.trajectory([und], [part], 0.0, 2.0, 0.0, npoints)
    torch.cuda.synchronize()
    return t, [a[0].cpu().numpy().copy() for a in (t.x, t.beta, t.aoc)]


def _normwise(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("npoints", [2, 31, 33, 128, 129, 1000, 4225])
@pytest.mark.parametrize("nout", [1, 127, 129])
def test_fp64_sums_against_the_oracle(npoints, nout):
    import oracle as O
    import torch

    from srsoriginal_b200 import _lib, device as D

    t, (X, B, A) = _trajectory(npoints)
    rng = np.random.default_rng(1000 * nout + npoints)
    pts = np.column_stack([rng.uniform(-0.01, 0.01, (nout, 2)), rng.uniform(25, 35, nout)])
    nrm = rng.normal(size=(nout, 3))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    e = np.sort(rng.uniform(50, 1500, nout))
    dp, dn, de = (torch.tensor(v.reshape(-1), device="cuda") for v in (pts, nrm, e))
    out = torch.empty(nout, dtype=torch.float64, device="cuda")
    D.flux(t, -D.QE, 0.5, 152.25, out, points=dp, precision=_lib.FP64)
    assert _normwise(out.cpu().numpy(), O.flux(X, B, t.dt, pts, 152.25, -O.QE, 0.5)) < TOL
    D.spectrum(t, -D.QE, 0.5, [1e-3, 2e-3, 30.0], de, out, precision=_lib.FP64)
    assert _normwise(out.cpu().numpy(), O.spectrum(X, B, t.dt, [1e-3, 2e-3, 30.0], e, -O.QE, 0.5)) < TOL
    if npoints > 2:  # the first point's a/c is 0: two points radiate nothing
        for directional in (0, 1):
            D.power_density(t, -D.QE, 0.5, out, points=dp, normals=dn, directional=directional, precision=_lib.FP64)
            ref = O.power_density(X, B, A, t.dt, pts, nrm, bool(directional), -O.QE, 0.5)
            got = out.cpu().numpy()
            assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


# Phases around the end of the fast reduction (2^50 rad is 7.4 MeV at 30 m) and far beyond it
@pytest.mark.parametrize("energies", [[7.0e6, 7.3e6, 7.5e6, 9.0e6], [1.0e5, 3.0e7, 1.0e9], [1.0e15, 2.0e20]])
def test_fp64_sums_at_extreme_phases(energies):
    import oracle as O
    import torch

    from srsoriginal_b200 import _lib, device as D

    t, (X, B, _) = _trajectory(1000)
    e = np.array(energies)
    de = torch.tensor(e, device="cuda")
    out = torch.empty(len(e), dtype=torch.float64, device="cuda")
    D.spectrum(t, -D.QE, 0.5, [1e-3, 2e-3, 30.0], de, out, precision=_lib.FP64)
    got = out.cpu().numpy()
    assert np.all(np.isfinite(got))
    if e.max() < 1e12:  # beyond, k of the reduction itself has no room in a double
        assert _normwise(got, O.spectrum(X, B, t.dt, [1e-3, 2e-3, 30.0], e, -O.QE, 0.5)) < TOL
    pts = np.array([[1e-3, -2e-3, 30.0], [0.0, 5e-3, 28.0]])
    D.flux(t, -D.QE, 0.5, float(e[-1]), out[:2], points=torch.tensor(pts.reshape(-1), device="cuda"), precision=_lib.FP64)
    got = out[:2].cpu().numpy()
    assert np.all(np.isfinite(got))
    if e.max() < 1e12:
        assert _normwise(got, O.flux(X, B, t.dt, pts, float(e[-1]), -O.QE, 0.5)) < TOL
