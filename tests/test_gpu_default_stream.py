"""Contexts on CUDA's default streams, which a caller may pass as handles: the legacy one (1), on which no capture can
begin, and the per-thread one (2).  Every call gives the bits of a context that owns its stream."""
import numpy as np
import pytest

import cases as C
import elastic_cases as E
import vd_cases as V
from vd_cases import sw

pytestmark = pytest.mark.gpu

NT = 60


def _calls(family, grad, stream, monkeypatch):
    """Outputs of four calls on one handle."""
    real = sw._lib.Context
    monkeypatch.setattr(sw._lib, "Context", lambda device=0: real(device, stream=stream))
    out = []
    if family in ("2d", "3d"):
        shape = (80, 60) if family == "2d" else (40, 30, 28)
        h = (8.0,) * len(shape)
        vp = C.smooth_model(shape, 1700.0, 3100.0, 5)
        case = C.Case(vp=vp, h=h, dt=C.stable_dt(vp, h), halo=6, freetop=True)
        mid = [0.5 * hh * (n - 1) for n, hh in zip(shape, h)]
        shot = C.make_shot(h, None, NT, case.dt, 25.0, [mid], [[mid[0] + 8.0 * q] + mid[1:] for q in range(5)])
        shot.observed = np.cos(np.arange(NT * 5.0)).reshape(NT, 5)
        run = C.GpuRun(sw, case, gradient=grad, check_freq=7)
        for _ in range(4):
            g = run.gradient([shot]) if grad else run.forward([shot])
            out.append([g[0], np.array(g[1])] + list(g[2]) if grad else list(g))
        run.close()
    else:
        ctx = sw._lib.Context(0)
        case = V.small_case(nt=NT, nx=90, nz=70, halo=8) if family == "vd" else E.small_case("mt", nt=NT, nx=90, nz=70, halo=8)
        sim = (V.GpuVD if family == "vd" else E.GpuElastic)(ctx, case, gradient=grad, check_freq=7)
        nrec = len(case.shots[0].rec)
        obs = 1e-6 * np.cos(np.arange(NT * 2.0 * nrec)).reshape(NT, 2, nrec)
        for _ in range(4):
            if not grad:
                out.append(list(sim.forward(case.shots)))
                continue
            g, m, t = sim.gradient(case.shots, [obs[:, 0] if family == "vd" else obs])
            out.append([g[k] for k in sorted(g)] + [np.array(m)] + list(t))
        sim.close()
        ctx.close()
    monkeypatch.undo()
    return out


@pytest.mark.parametrize("family", ["2d", "3d", "vd", "el"])
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("stream", [1, 2])
def test_default_stream_context(family, grad, stream, monkeypatch):
    want = _calls(family, grad, None, monkeypatch)[0]
    assert np.abs(want[0]).max() > 0
    for got in _calls(family, grad, stream, monkeypatch):
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
