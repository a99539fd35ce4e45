"""The trajectory adjoint's scan at the edges of its chunks (16 steps) and blocks (128), and the sum adjoint
at the edges of its groups of energies, against long-double sums over the same stored points."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble
LIGHT = L(299792458.0)
PERIOD, NPERIODS, AMPLITUDE = 0.049, 31, (0.3, 1.0, 0.0)


def _shape(z):
    """Profile and z derivative of the undulator's field, in the library's doubles."""
    per = math.sqrt(PERIOD * PERIOD)
    length = per * (NPERIODS + 2)
    if z > length / 2 or z < -length / 2:
        return 0.0, 0.0
    a = 1.0
    if z < -length / 2 + per or z > length / 2 - per:
        a = 0.25 if z < -length / 2 + per / 2 or z > length / 2 - per / 2 else 0.75
    phase = 2 * math.pi * z / per
    return a * math.sin(phase), a * (math.cos(phase) * (2 * math.pi / per))


def _sweep(x, beta, gx, gb, chains, q):
    """Amplitude, initial-state and q gradients, and the sums of what the first and last add up in magnitude.
    The stages are formed in doubles as the library forms them (a zero crossing of the field would
    otherwise show the rounding of its phase), the adjoint in long double."""
    A = np.array(AMPLITUDE)
    amp, ic, qb = np.zeros(3, dtype=L), np.zeros(6, dtype=L), L(0)
    samp, sq = np.zeros(3, dtype=L), L(0)
    for n, h, base, direction, skip in chains:
        def g(j):
            if j == 0 and skip:
                return np.zeros(3, dtype=L), np.zeros(3, dtype=L)
            return gx[:, base + direction * j], gb[:, base + direction * j] / LIGHT
        lp, lv = (a.copy() for a in g(n - 1))
        weight, coef = (1, 2, 2, 1), (L(0), h / 2, h / 2, h)
        for j in range(n - 2, -1, -1):
            p, v = x[:, base + direction * j], beta[:, base + direction * j] * float(LIGHT)
            ps, vs, S, dS, a = [p], [v], [], [], None
            for s in range(4):
                if s:
                    ps.append(p + vs[s - 1] * float(coef[s]))
                    vs.append(v + a * float(coef[s]))
                sh = _shape(ps[s][2])
                S.append(sh[0])
                dS.append(sh[1])
                a = np.cross(vs[s], A * S[s]) * float(q)
            vbar = [lp * (h / 6 * w) for w in weight]
            abar = [lv * (h / 6 * w) for w in weight]
            nlp, nlv = lp.copy(), lv.copy()
            for s in (3, 2, 1, 0):
                vbar[s] = vbar[s] + np.cross(A * S[s], abar[s]) * q
                bbar = np.cross(abar[s], vs[s]) * q
                one = abar[s] * np.cross(vs[s], A * S[s])
                qb, sq = qb + one.sum(), sq + np.abs(one).sum()
                amp, samp = amp + bbar * S[s], samp + np.abs(bbar * S[s])
                pbar = np.array([0, 0, np.dot(bbar, A) * dS[s]], dtype=L)
                nlp, nlv = nlp + pbar, nlv + vbar[s]
                if s:
                    abar[s - 1] = abar[s - 1] + vbar[s] * coef[s]
                    vbar[s - 1] = vbar[s - 1] + pbar * coef[s]
            g0, g1 = g(j)
            lp, lv = g0 + nlp, g1 + nlv
        ic += np.concatenate([lp, lv * LIGHT])
    return amp, ic, qb, samp, sq


# A step's propagation is ~60 rounded operations on terms of the sizes added up here, and a gradient passes
# through at most all steps: 60 N eps of those sizes.
@pytest.mark.parametrize("npoints,start", [(2, 0.0), (3, 0.0), (17, 0.0), (18, 0.0), (128, 0.0), (129, 0.0), (130, 0.0),
                                           (257, -1.0), (260, -1.0), (385, -0.3)])
def test_trajectory_adjoint_against_a_serial_sweep(npoints, start):
    import torch

    from srsoriginal_b200 import _lib, device as D

    fields = (_lib.Field * 1)(D.undulator(list(AMPLITUDE), [0, 0, PERIOD], NPERIODS))
    part, _ = D.ideal_particle(3.0, [1e-5, -2e-5, -1.0 if start == 0.0 else 0.0], [1e-5, 2e-5, 1])
    tr = D.trajectory(list(fields), [part], start, start + 2.0, 0.0, npoints)
    n = tr.x.shape[-1]
    rng = np.random.default_rng(npoints)
    gx, gb = (torch.tensor(rng.normal(size=3 * n), device="cuda") for _ in range(2))
    amp, ic, none = (C.c_double * 3)(), (C.c_double * 7)(), (C.c_void_p * 1)()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    _lib.check(_lib.lib.srs_trajectory_adjoint(fields, 1, (_lib.Particle * 1)(part), start, start + 2.0, 0.0, npoints,
                                               ptr(tr.x), ptr(tr.beta), ptr(gx), ptr(gb), none, amp, ic, D._stream()))
    dt, nf, nb = D.counts(start, start + 2.0, 0.0, npoints)
    chains = [(nf, L(dt), nb, 1, False)] + ([(nb + 1, -L(dt), nb, -1, True)] if nb else [])
    host = lambda t: t.cpu().numpy().reshape(3, n).astype(L)
    q = L(part.qomg)
    ramp, ric, rq, samp, sq = _sweep(tr.x[0].cpu().numpy(), tr.beta[0].cpu().numpy(), host(gx), host(gb), chains, q)
    eps = 60 * n * 2.0 ** -53
    assert np.all(np.abs(np.array(amp[:]) - ramp) <= eps * samp.max())
    assert abs(ic[6] - rq) <= eps * sq
    span = 2.0 * max(nf, nb) * float(dt) * float(LIGHT)  # a position gradient's lever arm on a direction's
    sbeta = np.abs(gb.cpu().numpy()).sum() + span * np.abs(gx.cpu().numpy()).sum()
    turn = abs(float(q)) * 1.05 * span / float(LIGHT) * 2 * math.pi / PERIOD  # ... and back, through dB/dz
    sx = np.abs(gx.cpu().numpy()).sum() + turn * sbeta
    assert np.all(np.abs(np.array(ic[:3]) - ric[:3]) <= eps * sx)
    assert np.all(np.abs(np.array(ic[3:6]) - ric[3:]) <= eps * sbeta)


# The adjoint is linear in the energies: all at once against one energy at a time, summed in long double. An
# energy adds ~20 rounded operations and one addition to what is added up.
@pytest.mark.parametrize("npoints,ne", [(2, 1), (31, 3), (32, 4), (33, 5), (65, 127), (64, 128), (100, 129), (40, 260)])
def test_sum_adjoint_against_long_double(npoints, ne):
    import torch

    from srsoriginal_b200 import _lib, device as D

    part, _ = D.ideal_particle(3.0, [1e-5, -2e-5, -1.0], [1e-5, 2e-5, 1])
    tr = D.trajectory([D.undulator(list(AMPLITUDE), [0, 0, PERIOD], NPERIODS)], [part], 0.0, 2.0, 0.0, npoints)
    n = tr.x.shape[-1]
    rng = np.random.default_rng(ne)
    energies = np.linspace(100.0, 900.0, ne)
    e = torch.tensor(energies, device="cuda")
    e6, gf = torch.tensor(rng.normal(size=6 * ne), device="cuda"), torch.tensor(rng.normal(size=ne), device="cuda")
    gx, gb = torch.empty(3 * n, dtype=torch.float64, device="cuda"), torch.empty(3 * n, dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    args = (tr.view(), _lib.BeamConsts(-1.602176634e-19, 0.5), _lib.v3([0.0, 0.0, 30.0]), ptr(e))
    _lib.check(_lib.lib.srs_spectrum_adjoint(*args, ne, ptr(e6), ptr(gf), ptr(gx), ptr(gb), D._stream()))
    # linear in the energies; the terms of one energy are bounded by those of E's six real components
    sx, sb, mx, mb = (np.zeros(3 * n, dtype=L) for _ in range(4))
    hx, hb = torch.empty_like(gx), torch.empty_like(gb)
    for k in range(ne):
        for part in range(7):
            ek, ck, gk = e[k:k + 1].clone(), e6[6 * k:6 * k + 6].clone(), gf[k:k + 1].clone()
            if part:
                ck *= torch.arange(6, device="cuda") == part - 1
            _lib.check(_lib.lib.srs_spectrum_adjoint(*args[:3], ptr(ek), 1, ptr(ck), ptr(gk), ptr(hx), ptr(hb), D._stream()))
            x, b = hx.cpu().numpy().astype(L), hb.cpu().numpy().astype(L)
            if part:
                mx, mb = mx + np.abs(x), mb + np.abs(b)
            else:
                sx, sb = sx + x, sb + b
    eps = (20 + ne) * 2.0 ** -53
    # of the magnitudes per point: the three components share their terms (n Tt)
    top = lambda a: np.tile(a.reshape(3, n).sum(axis=0), 3)
    assert np.all(np.abs(gx.cpu().numpy() - sx) <= eps * top(mx))
    assert np.all(np.abs(gb.cpu().numpy() - sb) <= eps * top(mb))
