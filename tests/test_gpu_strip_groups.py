"""The x strips' memory variables of the variable-density and elastic kernels move in whole
groups of four columns: grids whose strips end inside a group, meet in one
group (nx = 2 halo + 3), or leave a partial last group, and band heights from
one row (the default on small grids) to more rows than the grid has."""
import numpy as np
import pytest

import cases as C
import elastic_cases as E
import vd_cases as V
from vd_cases import rel_l2, sw

pytestmark = pytest.mark.gpu

TOL = 1e-5  # traces and gradients against the FP64 oracle, relative L2 (FP32 state, a few hundred steps)
GRIDS = [(23, 26, 10), (43, 45, 20), (131, 40, 13), (150, 61, 8), (517, 33, 6), (60, 50, 1), (64, 40, 0)]


@pytest.fixture(scope="module")
def ctx():
    c = sw._lib.Context(0)
    yield c
    c.close()


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("nx,nz,halo", GRIDS)
@pytest.mark.parametrize("freetop", [False, True])
def test_vd_groups_and_bands(ctx, nx, nz, halo, freetop):
    case = V.small_case(nt=160, nx=nx, nz=nz, halo=halo, freetop=freetop, interp=int(freetop), nsrc=2, f0=25.0)
    shot = case.shots[0]
    obs = 0.5 * V.oracle_forward(case, shot).astype(np.float32).astype(np.float64)
    gref, _, tref = V.oracle_gradient(case, shot, obs, check_freq=7)
    out = {}
    for tz in (0, 8, 32):
        run = V.GpuVD(ctx, case, gradient=True, check_freq=7)
        ctx.check(ctx.lib.sw_acoustic_vd_set_tuning(run.h, tz), "set_tuning")
        g, m, t = run.gradient([shot], [obs])
        run.close()
        out[tz] = [g["vp"], g["rho"], t[0], np.array(m)]
    assert rel_l2(out[0][2], tref) < TOL
    assert rel_l2(out[0][0], gref["vp"]) < TOL and rel_l2(out[0][1], gref["rho"]) < TOL
    assert _same(out[8], out[0]) and _same(out[32], out[0])


@pytest.mark.parametrize("nx,nz,halo", GRIDS)
@pytest.mark.parametrize("kind,freetop", [("mt", False), ("force", True)])
def test_elastic_groups_and_bands(ctx, nx, nz, halo, kind, freetop):
    case = E.small_case(kind, nt=160, nx=nx, nz=nz, halo=halo, freetop=freetop)
    shot = case.shots[0]
    obs = 0.5 * E.oracle_forward(case, shot).astype(np.float32).astype(np.float64)
    gref, _, tref = E.oracle_gradient(case, shot, obs, check_freq=7)
    out = {}
    for tz in (0, 8, 32, 128):
        run = E.GpuElastic(ctx, case, gradient=True, check_freq=7)
        ctx.check(ctx.lib.sw_elastic_set_tuning(run.h, tz), "set_tuning")
        g, m, t = run.gradient([shot], [obs])
        run.close()
        out[tz] = [g["rho"], g["lambda"], g["mu"], t[0], np.array(m)]
    assert rel_l2(out[0][3], tref) < TOL
    for q, k in enumerate(("rho", "lambda", "mu")):
        assert rel_l2(out[0][q], gref[k]) < TOL, k
    for tz in (8, 32, 128):
        assert _same(out[tz], out[0]), tz


@pytest.mark.parametrize("shape,halo", [((23, 26), 10), ((131, 40), 13), ((517, 33), 6), ((60, 50), 1), ((64, 40), 0),
                                        ((23, 25, 24), 10), ((133, 20, 18), 3), ((30, 28, 19), 0)])
@pytest.mark.parametrize("freetop", [False, True])
def test_acoustic_groups(oracle, shape, halo, freetop):
    """Constant density, 2D and 3D: four points of an x strip at once, at the strips' ends inside a group and on
    the narrowest grid of a halo; gradient with checkpoints (the copies of the memory variables included)."""
    h = (9.0, 8.0, 7.0)[:len(shape)]
    vp = C.smooth_model(shape, 1700.0, 3100.0, 5)
    case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=halo, freetop=freetop)
    ex = [hh * (n - 1) for n, hh in zip(shape, h)]
    rec = [[x] + [0.4 * e for e in ex[1:-1]] + [0.3 * ex[-1]] for x in np.linspace(0.1, 0.9, 7) * ex[0]]
    shot = C.make_shot(h, ex, 90, case.dt, 25.0, [[0.45 * e for e in ex]], rec)
    shot.observed = 0.5 * C.oracle_forward(oracle, sw, case, shot).astype(np.float32).astype(np.float64)
    gref, _, tref = C.oracle_gradient(oracle, sw, case, shot, check_freq=7)
    run = C.GpuRun(sw, case, gradient=True, check_freq=7)
    g, _, t = run.gradient([shot])
    run.close()
    assert rel_l2(t[0], tref) < TOL and rel_l2(g, gref) < TOL


@pytest.mark.parametrize("shape,halo", [((23, 26), 10), ((131, 40), 13), ((517, 130), 6), ((60, 50), 1), ((64, 40), 0),
                                        ((23, 25, 24), 10), ((45, 20, 18), 3)])
@pytest.mark.parametrize("freetop", [False, True])
def test_compensated_groups(oracle, shape, halo, freetop):
    """The compensated forward at the same kinds of grids: within 1e-7 of the FP64 oracle (48-bit state, FP64 strips,
    traces rounded to FP32: 6e-8 of their largest value)."""
    h = (9.0, 8.0, 7.0)[:len(shape)]
    vp = C.smooth_model(shape, 1700.0, 3100.0, 5)
    case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=halo, freetop=freetop)
    ex = [hh * (n - 1) for n, hh in zip(shape, h)]
    rec = [[x] + [0.4 * e for e in ex[1:-1]] + [0.3 * ex[-1]] for x in np.linspace(0.1, 0.9, 7) * ex[0]]
    shots = [C.make_shot(h, ex, 120 - 11 * k, case.dt, 25.0, [[0.45 * e for e in ex]], rec) for k in range(2)]
    run = C.GpuRun(sw, case, precision=1)
    out = run.forward(shots)
    run.close()
    for s, t in zip(shots, out):
        # the source time function and the coefficients reach the oracle as the library gets them
        assert rel_l2(t, C.oracle_forward(oracle, sw, case, s)) < 1e-7
