"""The time loop's launches: a call that replays a captured graph gives, for
inputs the graph has not seen, what a fresh simulation's first call (plain
chained launches) gives, bit for bit; shots of different length in a batch
(the kernels of a step cover fewer shots towards the end of the loop)."""
import numpy as np
import pytest

import cases as C
import elastic_cases as E
import vd_cases as V
from vd_cases import sw

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sw._lib.Context(0)
    yield c
    c.close()


def _shots(kind, amp):
    """Two shots of different length; amp scales the source of the second call's inputs."""
    if kind == "vd":
        case = V.small_case(nt=140, nx=90, nz=70, halo=8, freetop=True, nsrc=2)
        a = case.shots[0]
        shots = [V.VDShot(a.src, a.rec, amp * a.tf[:n], a.f0) for n in (140, 101)]
        obs = [0.1 * amp * np.cos(np.outer(np.arange(s.nt), np.arange(1, 10))) for s in shots]
    else:
        case = E.small_case(kind, nt=140, nx=90, nz=70, halo=8, freetop=True)
        a = case.shots[0]
        shots = [E.ElShot(kind, amp * a.src, a.rec, n) for n in (140, 101)]
        obs = [1e-12 * amp * np.cos(np.arange(s.nt * 18).reshape(s.nt, 2, 9)) for s in shots]
    return case, shots, obs


def _run(ctx, kind, grad, amps):
    out = None
    case, _, _ = _shots(kind, 1.0)
    sim = (V.GpuVD if kind == "vd" else E.GpuElastic)(ctx, case, gradient=grad, check_freq=9)
    for amp in amps:
        _, shots, obs = _shots(kind, amp)
        out = sim.gradient(shots, obs) if grad else (sim.forward(shots),)
    sim.close()
    if not grad:
        return list(out[0])
    g, m, t = out
    return [g[k] for k in sorted(g)] + [np.array(m)] + list(t)


@pytest.mark.parametrize("kind", ["vd", "mt", "force"])
@pytest.mark.parametrize("grad", [False, True])
def test_replayed_time_loop_is_bitwise_a_first_call(ctx, kind, grad):
    want = _run(ctx, kind, grad, [0.9])
    got = _run(ctx, kind, grad, [1.0, 1.0, 1.1, 0.9])
    assert all(np.abs(w).max() > 0 for w in want)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("nx,nz,shots", [(45, 45, 1), (130, 90, 2), (700, 400, 1), (700, 410, 2), (257, 190, 9)])
def test_small_2d_launches_are_bitwise_the_split_ones(nx, nz, shots):
    """Constant density: one-row launches of small batches (below 16 rows of 128 points per SM; the sizes lie on
    both sides) against explicit 8-row bands with the x strips in the main blocks (variant bit 18)."""
    h = (9.0, 8.0)
    vp = C.smooth_model((nx, nz), 1700.0, 3200.0, nx)
    case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=9, freetop=bool(nx % 2))
    ex = [hh * (n - 1) for n, hh in zip(vp.shape, h)]
    sh = []
    for k in range(shots):  # receivers a few points off the source: 70 steps carry a wave about 25 points
        x, z = (0.2 + 0.06 * k) * ex[0], 0.3 * ex[1]
        sh.append(C.make_shot(h, ex, 70 - 5 * k, case.dt, 25.0, [[x, z]], [[x + 9.0 * q, z + 16.0] for q in range(9)]))
    for s in sh:
        s.observed = 1e-3 * np.cos(np.arange(s.nt * 9.0)).reshape(s.nt, 9)
    out = []
    for variant, bands in ((0, None), (262144, (8, 8, 8))):
        run = C.GpuRun(sw, case, gradient=True, check_freq=8, variant=variant)
        if bands:
            run.ctx.check(run.ctx.lib.sw_wavesim_set_band_heights(run.h, *bands), "band heights")
        g, m, t = run.gradient(sh)
        run.close()
        out.append([g, np.array(m)] + list(t))
    assert np.abs(out[0][0]).max() > 0
    assert all(np.array_equal(a, b) for a, b in zip(*out))
