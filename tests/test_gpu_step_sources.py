"""2D forward steps that add their sources and record the step before, against the launch of its own that does both
for shots with more source points (a fifth, silent source): bitwise the same traces and gradients."""
import dataclasses

import numpy as np
import pytest

import cases as C
import vd_cases as V
from vd_cases import sw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,halo,nshots,nrec", [((150, 61), 12, 2, 300), ((33, 40), 0, 1, 1), ((517, 123), 9, 18, 130),
                                                    ((131, 411), 20, 16, 5), ((1100, 411), 9, 18, 40)])
@pytest.mark.parametrize("check_freq", [1, 7])
def test_sources_with_the_step(shape, halo, nshots, nrec, check_freq):
    h = (9.0, 8.0)
    vp = C.smooth_model(shape, 1700.0, 3100.0, 5)
    case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=halo, freetop=False)
    ex = [hh * (n - 1) for n, hh in zip(shape, h)]
    # source points in the first and last column and row that are advanced, in both x strips, twice on one point
    pos = [[h[0], h[1]], [ex[0] - h[0], ex[1] - h[1]], [0.5 * ex[0], 0.45 * ex[1]], [0.5 * ex[0], 0.45 * ex[1]],
           [ex[0] - 4 * h[0], 0.5 * ex[1]]]
    rec = [[x, 0.4 * ex[1]] for x in np.linspace(0.0, 1.0, nrec) * ex[0]]
    out = []
    for silent in (False, True):
        shots = []
        for k in range(nshots):
            s = C.make_shot(h, ex, 64 - (k % 5), case.dt, 25.0, pos + [[0.3 * ex[0], 0.6 * ex[1]]], rec)
            s.tf[:, 5] = 0.0
            s = s if silent else dataclasses.replace(s, src_pos=s.src_pos[:5], tf=np.asfortranarray(s.tf[:, :5]))
            s.observed = np.random.default_rng(k).standard_normal((s.nt, nrec)).astype(np.float32).astype(np.float64)
            shots.append(s)
        run = C.GpuRun(sw, case, gradient=True, check_freq=check_freq)
        g, m, t = run.gradient(shots)
        f = run.forward(shots)
        run.close()
        out.append([np.asarray(g), np.asarray(m)] + list(t) + list(f))
    assert np.abs(out[0][0]).max() > 0
    assert nrec == 1 or np.abs(out[0][2]).max() > 0  # the single receiver sits on the rigid boundary
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("nx,nz,halo,nshots,nrec", [(150, 61, 12, 2, 300), (33, 40, 0, 1, 1), (517, 62, 9, 18, 130)])
def test_vd_sources_with_the_step(nx, nz, halo, nshots, nrec):
    """Variable density: the pressure update adds the sources (the grid's corners included), the velocity launch
    records."""
    case = V.small_case(nt=50, nx=nx, nz=nz, halo=halo, f0=25.0)
    ex, ez = (nx - 1) * case.h, (nz - 1) * case.h
    pos = [[0.0, 0.0], [ex, ez], [0.5 * ex, 0.45 * ez], [0.5 * ex, 0.45 * ez], [ex - 2 * case.h, 0.5 * ez],
           [0.3 * ex, 0.6 * ez]]
    rec = np.array([[x, 0.4 * ez] for x in np.linspace(0.1, 0.9, nrec) * ex])
    t = np.arange(50) * case.dt
    tf = np.stack([V.ricker(t, 1.2 / 25.0 + 0.002 * k, 25.0) for k in range(6)], axis=1)
    tf[:, 5] = 0.0
    ctx = sw._lib.Context(0)
    out = []
    for n in (5, 6):
        shots = [V.VDShot(np.array(pos[:n]), rec, np.asfortranarray(tf[: 50 - k % 5, :n]), 25.0) for k in range(nshots)]
        obs = [np.random.default_rng(k).standard_normal((s.nt, nrec)) for k, s in enumerate(shots)]
        run = V.GpuVD(ctx, case, gradient=True, check_freq=7)
        g, m, tr = run.gradient(shots, obs)
        f = run.forward(shots)
        run.close()
        out.append([g["vp"], g["rho"], np.asarray(m)] + list(tr) + list(f))
    ctx.close()
    assert np.abs(out[0][0]).max() > 0 and np.abs(out[0][3]).max() > 0
    assert all(np.array_equal(a, b) for a, b in zip(*out))
