"""Explicit bands of small 2D launches, which take the kernel with the x strips in blocks of their own: bitwise the
default's single rows, in forward, recompute and adjoint steps, with sources in and beside the strips."""
import numpy as np
import pytest

import cases as C
from vd_cases import sw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,halo", [((201, 67), 12), ((37, 90), 3), ((130, 41), 0)])
@pytest.mark.parametrize("nsrc", [2, 5])
def test_explicit_bands_of_small_launches(shape, halo, nsrc):
    h = (9.0, 8.0)
    vp = C.smooth_model(shape, 1700.0, 3100.0, 5)
    case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=halo, freetop=bool(halo % 2))
    ex = [hh * (n - 1) for n, hh in zip(shape, h)]
    src = [[ex[0] - 2 * h[0], 0.5 * ex[1]], [0.4 * ex[0], 0.5 * ex[1]], [0.3 * ex[0], 0.6 * ex[1]],
           [0.5 * ex[0], 2 * h[1]], [0.6 * ex[0], 0.4 * ex[1]]][:nsrc]
    rec = [[x, 0.45 * ex[1]] for x in np.linspace(0.05, 0.95, 30) * ex[0]]
    shots = []
    for k in range(2):
        s = C.make_shot(h, ex, 64 - 5 * k, case.dt, 25.0, src, rec)
        s.observed = np.random.default_rng(k).standard_normal((s.nt, 30))
        shots.append(s)
    out = []
    for tz in (0, 1, 2, 8, 64):
        run = C.GpuRun(sw, case, gradient=True, check_freq=7, tz=tz)
        g, m, t = run.gradient(shots)
        f = run.forward(shots)
        run.close()
        out.append([np.asarray(g), np.asarray(m)] + list(t) + list(f))
    assert np.abs(out[0][0]).max() > 0 and np.abs(out[0][2]).max() > 0
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))
