"""The time loop's launches: a call that replays a captured graph gives, for
inputs the graph has not seen, what a fresh simulation's first call (plain
chained launches) gives, bit for bit; shots of different length in a batch
(the kernels of a step cover fewer shots towards the end of the loop)."""
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
