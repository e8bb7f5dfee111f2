"""Bands of the variable-density and elastic kernels in launches that fill the GPU, and the elastic recording that
rides on the next step's stress launch: shots that end at different steps, more receiver blocks than a row of the
launch holds."""
import dataclasses

import numpy as np
import pytest

import elastic_cases as E
import vd_cases as V
from vd_cases import sw

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sw._lib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("nz,halo", [(91, 7), (92, 10), (93, 2)])
def test_vd_default_bands_of_a_full_launch(ctx, nz, halo):
    """Bitwise the 8-row bands: last band of 1, 2 and 3 rows, last x tile of 5 points."""
    case = V.small_case(nt=40, nx=517, nz=nz, halo=halo, f0=25.0)
    shots = [dataclasses.replace(case.shots[0], tf=case.shots[0].tf[: 40 - k]) for k in range(18)]
    rng = np.random.default_rng(3)
    obs = [rng.standard_normal((s.nt, len(s.rec))) for s in shots]
    out = {}
    for tz in (0, 8):
        run = V.GpuVD(ctx, case, gradient=True, check_freq=6)
        ctx.check(ctx.lib.sw_acoustic_vd_set_tuning(run.h, tz), "set_tuning")
        g, m, t = run.gradient(shots, obs)
        run.close()
        out[tz] = [g["vp"], g["rho"], np.array(m)] + list(t)
    assert np.abs(out[0][0]).max() > 0
    assert all(np.array_equal(a, b) for a, b in zip(out[0], out[8]))


@pytest.mark.parametrize("kind", ["mt", "force"])
@pytest.mark.parametrize("nrec", [1, 65, 700])
def test_elastic_recording_of_shots_that_end_early(ctx, kind, nrec):
    """A batch's traces are bitwise those of each shot by itself, the last step's (a launch of its own) included."""
    case = E.small_case(kind, nt=60, nx=70, nz=50, halo=8)
    one = case.shots[0]
    ex, ez = (case.nx - 1) * case.h, (case.nz - 1) * case.h
    rec = np.column_stack([np.linspace(0.15, 0.85, nrec) * ex, np.linspace(0.3, 0.7, nrec) * ez])
    shots = [dataclasses.replace(one, rec=rec[: max(1, nrec // (k + 1))], nt=nt) for k, nt in enumerate((60, 59, 33, 1))]
    run = E.GpuElastic(ctx, case)
    batch = run.forward(shots)
    alone = [run.forward([s])[0] for s in shots]
    run.close()
    assert np.abs(batch[0]).max() > 0 and np.abs(batch[1]).max() > 0
    assert all(np.array_equal(a, b) for a, b in zip(batch, alone))
