"""Kernels that run beside the time loop's stream in captured loops (the x strips of the 3D step, the elastic gradient's
correlation): the replayed graph, the capturing call and the direct first call agree bit for bit, for steps that are
checkpointed, recomputed and follow shots that end, and for two simulations used in turn."""
import dataclasses

import numpy as np
import pytest

import cases as C
import elastic_cases as E
from vd_cases import sw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,halo", [((45, 30, 28), 6), ((133, 20, 18), 3), ((30, 28, 19), 0)])
@pytest.mark.parametrize("buffer", [0, 3])
def test_3d_strips_beside_the_main_rows(shape, halo, buffer):
    h = (9.0, 8.0, 7.0)
    vp = C.smooth_model(shape, 1700.0, 3100.0, 5)
    case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=halo, freetop=True)
    ex = [hh * (n - 1) for n, hh in zip(shape, h)]
    rec = [[x, 0.4 * ex[1], 0.3 * ex[2]] for x in np.linspace(0.1, 0.9, 7) * ex[0]]
    shots = [C.make_shot(h, ex, 60 - 7 * k, case.dt, 25.0, [[0.45 * e for e in ex]], rec) for k in range(2)]
    for k, s in enumerate(shots):
        s.observed = np.random.default_rng(k).standard_normal((s.nt, 7)).astype(np.float32).astype(np.float64)
    runs = [C.GpuRun(sw, case, gradient=True, check_freq=7, bf16=buffer) for _ in range(2)]
    out = []
    for call in range(4):
        for run in runs:
            g, m, t = run.gradient(shots)
            out.append([np.array(g), np.array(m)] + [np.array(x) for x in t] + [np.array(x) for x in run.forward(shots)])
    for run in runs:
        run.close()
    assert np.abs(out[0][0]).max() > 0
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))


@pytest.mark.parametrize("kind", ["mt", "force"])
def test_elastic_correlation_beside_the_stress_update(kind):
    ctx = sw._lib.Context(0)
    case = E.small_case(kind, nt=90, nx=150, nz=61, halo=8)
    shots = [dataclasses.replace(case.shots[0], nt=nt) for nt in (90, 89, 40)]
    obs = [np.random.default_rng(k).standard_normal((s.nt, 2, len(s.rec))) * 1e-12 for k, s in enumerate(shots)]
    runs = [E.GpuElastic(ctx, case, gradient=True, check_freq=7) for _ in range(2)]
    out = []
    for call in range(4):
        for run in runs:
            g, m, t = run.gradient(shots, obs)
            out.append([g["rho"].copy(), g["lambda"].copy(), g["mu"].copy(), np.array(m)] + [x.copy() for x in t])
    for run in runs:
        run.close()
    ctx.close()
    assert np.abs(out[0][1]).max() > 0
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))
