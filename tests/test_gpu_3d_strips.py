"""The two launches of the 3D step (x-strip groups; all other rows) against the single launch (variant 65536), bit for
bit, in direct and replayed calls: 4 and 8 rows per block, every recompute buffer, grids of one and of two x tiles."""
import numpy as np
import pytest

import cases as C
from vd_cases import sw

pytestmark = pytest.mark.gpu

SINGLE = 65536


@pytest.mark.parametrize("shape,halo", [((58, 44, 40), 5), ((141, 27, 26), 6)])
@pytest.mark.parametrize("bf16", [0, 1, 3])
def test_two_launches_are_bitwise_the_single_one(shape, halo, bf16):
    h = (9.0, 8.0, 7.0)
    vp = C.smooth_model(shape, 1700.0, 3100.0, 3)
    case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=halo, freetop=True)
    ex = [hh * (n - 1) for n, hh in zip(shape, h)]
    src = [[0.45 * ex[0], 0.5 * ex[1], 0.4 * ex[2]], [ex[0] - 2 * h[0], 0.5 * ex[1], 0.5 * ex[2]]]
    rec = [[x, 0.5 * ex[1], 0.45 * ex[2]] for x in np.linspace(0.02, 0.98, 25) * ex[0]]
    shots = []
    for k in range(2):
        s = C.make_shot(h, ex, 70 - 9 * k, case.dt, 25.0, src, rec)
        s.observed = np.random.default_rng(k).standard_normal((s.nt, 25))
        shots.append(s)
    out = {}
    for variant in (SINGLE, 0, 2):
        run = C.GpuRun(sw, case, gradient=True, check_freq=7, variant=variant, bf16=bf16)
        for call in range(3):
            g, m, t = run.gradient(shots)
            out[variant, call] = [np.asarray(g), np.asarray(m)] + [np.array(x) for x in t]
        run.close()
    want = out[SINGLE, 0]
    assert np.abs(want[0]).max() > 0
    for key, got in out.items():
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), key
