"""The x strips' memory variables of the variable-density and elastic kernels move in whole
groups of four columns: grids whose strips end inside a group, meet in one
group (nx = 2 halo + 3), or leave a partial last group, and band heights from
one row (the default on small grids) to more rows than the grid has."""
import numpy as np
import pytest

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
