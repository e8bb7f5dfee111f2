"""Gradients whose misfit, covariance, windows, receivers or muted balls change from call to call on one handle: every
call, replayed or not, gives what a fresh simulation's first call (plain launches) gives, bit for bit."""
import dataclasses

import numpy as np
import pytest

import cases as C
import elastic_cases as E
import vd_cases as V
from vd_cases import sw

pytestmark = pytest.mark.gpu

NT = 300


class GpuCD(C.GpuRun):
    """GpuRun whose shots take the CCTS misfit when ccts_dt is set."""
    ccts_dt = None

    def _structs(self, shots, grad):
        out = super()._structs(shots, grad)
        for st in out[0] if grad and self.ccts_dt else []:
            st.misfit_kind, st.misfit_dt = 1, self.ccts_dt
        return out


def _positions(nrec, shift):
    """Source and receivers of a 90 x 70 grid, spacing 5; `shift` moves them (and the muted balls)."""
    src = np.array([[205.0 + shift, 150.0]])
    return src, np.column_stack([np.linspace(120.0, 300.0, nrec) + shift, np.full(nrec, 110.0)])


class Sim:
    """One simulation handle of a family; `grad(call)` returns its gradients, misfit and traces."""

    def __init__(self, family, mute=0):
        self.family = family
        if family == "cd":
            vp = C.smooth_model((90, 70), 1800.0, 3000.0, 3)
            self.case = C.Case(vp=vp, h=(5.0, 5.0), dt=C.stable_dt(vp, (5.0, 5.0)), halo=8, freetop=False)
            self.sim = GpuCD(sw, self.case, gradient=True, check_freq=9, mute_src=mute, mute_rec=mute)
            self.ctx = None
            return
        self.ctx = sw._lib.Context(0)
        if family == "vd":
            self.case = V.small_case(nt=NT, nx=90, nz=70, halo=8)
            self.sim = V.GpuVD(self.ctx, self.case, gradient=True, check_freq=9, mute_src=mute, mute_rec=mute)
        else:
            self.case = E.small_case(family, nt=NT, nx=90, nz=70, halo=8)
            self.sim = E.GpuElastic(self.ctx, self.case, gradient=True, check_freq=9, mute_src=mute, mute_rec=mute)

    def close(self):
        self.sim.close()
        if self.ctx:
            self.ctx.close()

    def grad(self, kind="l2", nrec=9, seed=0, shift=0.0):
        rng = np.random.default_rng(seed)
        nts = (NT, NT - 31)
        src, rec = _positions(nrec, shift)
        amp = 1e-12 if self.family in ("mt", "force") else 0.1
        comp = (2,) if self.family in ("mt", "force") else ()
        obs = [np.cumsum(amp * rng.standard_normal((n, *comp, nrec)), axis=0) for n in nts]
        invcov = [None, None]
        if kind == "diag":
            invcov = [rng.uniform(0.5, 2.0, n) for n in nts]
        elif kind == "dense":
            invcov = [np.diag(rng.uniform(0.5, 2.0, n)) + 0.1 * np.eye(n, k=1) + 0.1 * np.eye(n, k=-1) for n in nts]
        windows = [[(20 + 10 * seed, 200)], [(60, 90), (120, 240 - 10 * seed)]] if kind == "windows" else [[], []]
        ccts_dt = self.case.dt if kind == "ccts" else None
        if self.family == "cd":
            shots = []
            for k, n in enumerate(nts):
                s = C.make_shot(self.case.h, None, n, self.case.dt, 25.0, src, rec)
                s.observed, s.invcov, s.windows = obs[k], invcov[k], windows[k]
                shots.append(s)
            self.sim.ccts_dt = ccts_dt
            g, m, t = self.sim.gradient(shots)
            return [g, np.array(m)] + list(t)
        one = self.case.shots[0]
        if self.family == "vd":
            shots = [V.VDShot(src, rec, one.tf[:n], one.f0) for n in nts]
        else:
            shots = [dataclasses.replace(one, src=src, rec=rec, nt=n) for n in nts]
        g, m, t = self.sim.gradient(shots, obs, invcov=invcov, windows=windows, ccts_dt=ccts_dt)
        return [g[k] for k in sorted(g)] + [np.array(m)] + list(t)


SEQUENCES = {
    "misfit": [("l2",), ("l2",), ("ccts",), ("ccts",), ("l2",), ("ccts",)],
    "receivers": [("ccts", 12), ("ccts", 3), ("ccts", 3), ("ccts", 5), ("ccts", 12), ("l2", 3), ("l2", 3), ("l2", 5)],
    "covariance": [("dense",), ("dense",), ("dense", 9, 1), ("l2",), ("l2",), ("diag",), ("dense", 9, 2), ("dense", 7, 2)],
    "windows": [("windows",), ("windows",), ("windows", 9, 1), ("l2",), ("windows", 9, 2)],
    "muting": [("l2",), ("l2",), ("l2", 9, 0, 40.0), ("l2", 4, 0, -20.0), ("ccts", 9, 0, 20.0)],
}


@pytest.mark.parametrize("family", ["cd", "vd", "mt", "force"])
@pytest.mark.parametrize("sequence", sorted(SEQUENCES))
def test_every_call_is_bitwise_a_first_call(family, sequence):
    mute = 3 if sequence == "muting" else 0
    sim = Sim(family, mute)
    first = {}
    for n, call in enumerate(SEQUENCES[sequence]):
        got = sim.grad(*call)
        if call not in first:
            fresh = Sim(family, mute)
            first[call] = fresh.grad(*call)
            fresh.close()
            assert np.abs(first[call][0]).max() > 0 and all(np.isfinite(a).all() for a in first[call]), call
        assert all(np.array_equal(a, b) for a, b in zip(got, first[call])), (n, call)
    sim.close()
