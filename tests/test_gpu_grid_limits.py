"""Launches at CUDA's limit of 65535 block rows: the default bands of very deep grids give the bits of explicit 8-row
bands, with and without a recording whose blocks no longer fit beside them; batches of very many shots."""
import numpy as np
import pytest

import cases as C
import elastic_cases as E
import vd_cases as V
from vd_cases import sw

pytestmark = pytest.mark.gpu


# the last depth at which 3- (4-) row bands fit by themselves, and depths beyond
@pytest.mark.parametrize("family,nz,nrec", [("vd", 196600, 600), ("vd", 200000, 2), ("el", 262136, 600), ("el", 270000, 2)])
def test_default_bands_of_deep_grids(family, nz, nrec):
    ctx = sw._lib.Context(0)
    nt, f0 = 30, 120.0
    if family == "vd":
        case = V.small_case(nt=nt, nx=16, nz=nz, halo=2)
    else:
        case = E.small_case("mt", nt=nt, nx=16, nz=nz, halo=2)
    ez = (nz - 1) * case.h
    src = np.array([[40.0, ez - 50.0]])
    rec = np.column_stack([np.linspace(30.0, 50.0, nrec), ez - 60.0 + 20.0 * np.cos(np.arange(nrec))])
    if family == "vd":
        shots = [V.VDShot(src, rec, V.ricker(np.arange(nt) * case.dt, 0.008, f0)[:, None], f0)]
        run = V.GpuVD(ctx, case)
        tune = ctx.lib.sw_acoustic_vd_set_tuning
    else:
        shots = [E.ElShot("mt", src, rec, nt, f0=f0)]
        run = E.GpuElastic(ctx, case)
        tune = ctx.lib.sw_elastic_set_tuning
    out = []
    for tz in (8, 0):
        ctx.check(tune(run.h, tz), "set_tuning")
        out.append(run.forward(shots)[0])
    run.close()
    ctx.close()
    assert np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1])


def _repeat(struct_type, template, n, last):
    return (struct_type * n)(last, *([template] * (n - 1)))


def test_elastic_recording_of_many_shots_that_end_together():
    """16500 shots end one step before the last shot, whose stress launch has no room for their recordings."""
    ctx = sw._lib.Context(0)
    case = E.small_case("mt", sinc=False, nt=30, nx=16, nz=16, halo=2)
    src, rec = np.array([[40.0, 40.0]]), np.column_stack([np.linspace(20.0, 60.0, 200), np.full(200, 45.0)])
    shots = [E.ElShot("mt", src, rec, n, f0=120.0) for n in (7, 6)]
    run = E.GpuElastic(ctx, case)
    want = run.forward(shots)
    structs, keep = run._structs(shots)
    many = _repeat(sw._lib.SwElasticShot, structs[1], 16500, structs[0])
    ctx.check(ctx.lib.sw_elastic_forward(run.h, len(many), many, 0), "forward")
    run.close()
    ctx.close()
    assert all(np.abs(w).max() > 0 and np.array_equal(k[0], w) for k, w in zip(keep, want))


def test_constant_density_recording_of_many_shots():
    """More shots than a grid has block rows (the last step's recording is a launch of its own)."""
    vp = C.smooth_model((33, 13), 1700.0, 3100.0, 5)
    case = C.Case(vp=vp, h=(8.0, 8.0), dt=C.stable_dt(vp, (8.0, 8.0)), halo=2, freetop=False)
    shots = [C.make_shot(case.h, None, n, case.dt, 120.0, [[128.0, 48.0]], [[128.0, 56.0]]) for n in (7, 7)]
    run = C.GpuRun(sw, case)
    want = [np.array(t) for t in run.forward(shots)]
    arr, keep, outs = run._structs(shots, False)
    many = _repeat(sw._lib.SwAcousticShot, arr[1], 66000, arr[0])
    run.ctx.check(run.ctx.lib.sw_acoustic_forward(run.h, len(many), many, 0), "forward")
    run.close()
    assert all(np.abs(w).max() > 0 and np.array_equal(o, w) for o, w in zip(outs, want))
