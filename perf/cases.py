"""Performance cases of the seismic modelling library.

What a user has it do: forward modelling and misfit gradients of a batch of
shots on one model, for the constant-density acoustic (2D and 3D), the
variable-density acoustic (2D) and the elastic (2D) simulations.  The two
smallest cases go through the Python mirror (swforward / swgradient, which set
the model first, as every call of a small script does).  The others go
through the C ABI of include/swgb300.h with device-resident data, as an
inversion driver does that runs many batches of shots on one model: the
simulation handle, its material, the shots' tables and the observed data are
in hand, one pass is one batched call.  Everything runs with the library's
default settings (no tuning calls).

Record lengths are shorter than a production run's (hundreds of steps instead
of thousands, with the same checkpoint periods), so that a pass stays below a
second; a time step costs the same whatever their number.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
DEV = "cuda"
VMIN, VMAX = 1500.0, 4500.0


def _package():
    name = "seismicwaves_gb300"
    if name not in sys.modules:
        pkg = ROOT / "seismicwaves.jl_gb300"
        spec = importlib.util.spec_from_file_location(name, pkg / "__init__.py", submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _case(name, family, mode, n, shots, nt, nt_min=None, recs=100, halo=20, freetop=False, K=50, h=10.0, f0=15.0,
          mirror=False, snap=0, compensated=False, harmonic=False, force=False):
    c = {"name": name, "family": family, "mode": mode, "nx": n[0], "ny": n[1] if len(n) == 3 else 0, "nz": n[-1],
         "shots": shots, "nt": nt, "nt_min": nt_min or nt, "recs": recs, "halo": halo, "freetop": freetop, "K": K,
         "h": h, "f0": f0, "mirror": mirror, "snap": snap, "compensated": compensated, "harmonic": harmonic,
         "force": force}
    return c


def listed():
    return [
        # a first script: one shot on the 201 x 201 model of the configurations, its whole record, through swforward
        _case("cd2d_forward_201", "cd", "forward", (201, 201), 1, 1000, recs=101, h=5.0, mirror=True),
        # a small teaching-size inversion step through swgradient: ragged grid, free surface, two shots of
        # different length, the default checkpoint period (1: every step kept)
        _case("cd2d_gradient_301x187", "cd", "gradient", (301, 187), 2, 500, 420, recs=57, freetop=True, K=1, mirror=True),
        # one shot of the 801 x 801 configuration (the shot loop of a program that does not batch)
        _case("cd2d_gradient_801", "cd", "gradient", (801, 801), 1, 1000, recs=401, h=5.0),
        # a batch of the headline survey: 2001 x 801, records of different length, checkpoint period 50
        _case("cd2d_gradient_2001x801", "cd", "gradient", (2001, 801), 16, 400, 200, recs=180),
        # modelling with the compensated arithmetic (misfits to 1e-8), a medium grid with a free surface
        _case("cd2d_compensated_901x455", "cd", "forward", (901, 455), 4, 400, recs=150, freetop=True, compensated=True),
        # 3D modelling, medium odd-sized model with a free surface
        _case("cd3d_forward_183", "cd", "forward", (183, 157, 141), 2, 300, recs=400, freetop=True),
        # 3D inversion step on the configuration's 400^3 model with the 2-byte recompute buffer
        _case("cd3d_gradient_400", "cd", "gradient", (400, 400, 400), 2, 60, recs=1600, K=20, snap=3),
        # variable density: one small shot modelled, harmonic averages of 1/rho
        _case("vd2d_forward_402x301", "vd", "forward", (402, 301), 1, 600, recs=80, freetop=True, harmonic=True),
        # variable density: a batch of the headline survey
        _case("vd2d_gradient_2001x801", "vd", "gradient", (2001, 801), 8, 300, 150, recs=180),
        # elastic: two vertical-force shots modelled below a free surface
        _case("el2d_forward_601x397", "elastic", "forward", (601, 397), 2, 500, recs=90, freetop=True, h=5.0, force=True),
        # elastic: a batch of the elastic configuration, 1200 x 600, explosive moment tensors, sinc-spread receivers
        _case("el2d_gradient_1200x600", "elastic", "gradient", (1200, 600), 8, 200, 150, recs=300, h=5.0),
        # elastic: one shot's gradient on a small model with a free surface
        _case("el2d_gradient_333x217", "elastic", "gradient", (333, 217), 1, 400, recs=60, freetop=True, K=20, h=5.0),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    family = rng.choice(["cd", "cd", "cd3", "vd", "elastic"])
    mode = rng.choice(["forward", "gradient"])
    freetop = rng.random() < 0.5
    if family == "cd3":
        n = tuple(log(70, 400) for _ in range(3))
        shots, nt, recs = rng.randint(1, 4), log(60, 300), log(20, 1600)
    else:
        n = (log(150, 2200), log(150, 900))
        shots, nt, recs = log(1, 16), log(150, 1000), log(10, 400)
    halo = rng.choice([10, 20, 20, 25])
    K = rng.choice([1, 10, 20, 50, 50]) if family != "cd3" else rng.choice([10, 20])
    c = _case("", family.rstrip("3"), mode, n, shots, nt, max(101, int(nt * rng.uniform(0.5, 1.0))) if nt > 101 else nt,
              recs, halo, freetop, K, rng.choice([5.0, 10.0]),
              mirror=family == "cd" and math.prod(n) * shots < 200000 and rng.random() < 0.5,
              snap=rng.choice([0, 3]) if family == "cd3" and mode == "gradient" else 0,
              compensated=family == "cd" and mode == "forward" and rng.random() < 0.2,
              harmonic=rng.random() < 0.3, force=rng.random() < 0.5)
    most = 0.3 * max(work(x)["bytes"] for x in listed())
    while work(c)["bytes"] > most and c["nt"] > 60:
        c["nt"] = max(60, int(c["nt"] * 0.8))
    while work(c)["bytes"] > most and c["shots"] > 1:
        c["shots"] -= 1
    # memory: a kept field per step between checkpoints, in a state that has to fit three times over
    while _points(c) * 4 * c["shots"] * (c["nt"] if c["K"] == 1 else c["K"]) * (4 if family == "elastic" else 1) > 25e9:
        if c["K"] == 1:
            c["K"] = 20
        elif c["shots"] > 1:
            c["shots"] -= 1
        else:
            break
    c["nt_min"] = min(c["nt_min"], c["nt"])
    del c["name"]
    return c


def _points(c):
    return c["nx"] * max(1, c["ny"]) * c["nz"]


def _nts(c):
    """Record lengths of the shots: spread evenly from nt_min to nt."""
    S = c["shots"]
    return [c["nt"] - (c["nt"] - c["nt_min"]) * k // max(1, S - 1) for k in range(S)]


def work(case):
    """Per grid point and time step: every state field read once and written once (constant density: p and its
    increment, 16 bytes; variable density: p, vx, vz, 24; elastic: u and its increment, 32), the same for the adjoint
    of a gradient, which also needs the forward history once (kept once, read once), and about 12, 26 or 60
    floating-point operations; plus the traces."""
    steps = sum(_nts(case)) * _points(case)
    state, hist, ops = {"cd": (16, 8 if case["snap"] == 0 else 4, 12 if not case["ny"] else 18), "vd": (24, 8, 26),
                        "elastic": (32, 16, 60)}[case["family"]]
    if case["compensated"]:
        state, ops = 32, 90
    grad = case["mode"] == "gradient"
    tr = sum(_nts(case)) * case["recs"] * (8 if case["family"] == "elastic" else 4)
    return {"bytes": steps * (2 * state + hist if grad else state) + tr * (2 if grad else 1),
            "flops": steps * ops * (2.2 if grad else 1)}


# ---------------------------------------------------------------------------
# Inputs: models, geometry, wavelets, observed data.  Arrays are (z, [y,] x),
# x fastest, i.e. the column-major (x, [y,] z) of the library.
# ---------------------------------------------------------------------------
def _spacing(c):
    return (c["h"],) * (3 if c["ny"] else 2)


def _dt(c):
    cfl = 0.6 / (VMAX * math.sqrt(sum(1.0 / h ** 2 for h in _spacing(c))))
    return cfl if c["family"] == "cd" else cfl * 6 / 7


def _smooth(shape, gen, step=14):
    """A smooth random field in [0, 1]."""
    coarse = torch.rand((1, 1) + tuple(s // step + 2 for s in shape), generator=gen, device=DEV)
    return torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear" if len(shape) == 3 else "bilinear",
                                           align_corners=True)[0, 0]


def _model(c, seed):
    """vp (and rho, or lambda, mu, rho): velocity rising with depth plus smooth heterogeneity, FP32 values."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 11)
    shape = (c["nz"], c["ny"], c["nx"]) if c["ny"] else (c["nz"], c["nx"])
    depth = torch.linspace(0, 1, c["nz"], device=DEV).reshape((-1,) + (1,) * (len(shape) - 1))
    vp = (1700.0 + 1800.0 * depth + 600.0 * _smooth(shape, gen)).clamp(VMIN, VMAX).float()
    if c["family"] == "cd":
        return {"vp": vp}
    rho = (310.0 * vp ** 0.25 * (0.95 + 0.1 * _smooth(shape, gen))).float()
    if c["family"] == "vd":
        return {"vp": vp, "rho": rho}
    vs = vp / math.sqrt(3.0) * (0.9 + 0.1 * _smooth(shape, gen))
    return {"lambda": (rho * (vp ** 2 - 2 * vs ** 2)).float(), "mu": (rho * vs ** 2).float(), "rho": rho}


def _geometry(c, seed):
    """Source and receiver grid nodes (1-based) of every shot, all outside the damping layers and off the outermost
    nodes: sources along a line near the top, each with a spread of receivers (a square patch in 3D) as wide as the
    waves of a record can travel."""
    rng = np.random.default_rng([int(seed), 3])
    lo = c["halo"] + 7
    top = 8 if c["freetop"] else lo
    span = [(lo, c["nx"] - lo)] + ([(lo, c["ny"] - lo)] if c["ny"] else [])
    reach = max(12, int(0.3 * c["nt"]))
    m = max(2, int(math.sqrt(c["recs"]))) if c["ny"] else c["recs"]
    src, rec = [], []
    for k in range(c["shots"]):
        at = [int(a + (b - a) * (k + rng.uniform(0.3, 0.7)) / c["shots"]) for a, b in span]
        lines = []
        for x, (a, b) in zip(at, span):  # a window of fixed width around x, moved inside the model
            width = min(2 * reach, b - a)
            lines.append(min(max(a, x - width // 2), b - width) + np.round(np.linspace(0, width, min(m, width + 1))))
        xy = np.stack([g.ravel() for g in np.meshgrid(*lines, indexing="ij")], 1)
        src.append(at + [top + 4])
        rec.append(np.concatenate([xy, np.full((len(xy), 1), top)], 1).astype(np.int32))
    return np.array(src, dtype=np.int32), rec


def _wavelet(c):
    t = np.arange(c["nt"]) * _dt(c)
    a = (np.pi * c["f0"] * (t - 1.2 / c["f0"])) ** 2
    return (1 - 2 * a) * np.exp(-a)


def _mean_velocity(seed):
    return 1900.0 + 200.0 * float(np.random.default_rng([int(seed), 5]).random())


def _observed(c, seed, k, nt, src, rec, amp):
    """Direct arrivals of a homogeneous medium with geometrical spreading: (nrec, nt), time fastest."""
    h, dt = c["h"], _dt(c)
    d = np.sqrt((((rec[k] - src[k]) * h).astype(np.float64) ** 2).sum(1)) + h
    t = torch.arange(nt, device=DEV, dtype=torch.float64) * dt
    delay = torch.from_numpy(d / _mean_velocity(seed) + 1.2 / c["f0"]).to(DEV)
    a = (math.pi * c["f0"] * (t[None, :] - delay[:, None])) ** 2
    return ((1 - 2 * a) * torch.exp(-a) * (amp / torch.from_numpy(np.sqrt(d / h)).to(DEV))[:, None]).float()


def _cpml(c, n, h, top):
    """The damping coefficients [a, a_h, b, b_h] of one axis, 64 bits (quadratic profile, rcoef 1e-4)."""
    H, dt = c["halo"], _dt(c)
    d0 = -3.0 * VMAX * math.log(1e-4) / (2.0 * H * h)
    out = []
    for count, off in ((H + 1, 0.0), (H, 0.5)):
        r = (off + np.arange(count)) / H
        r = np.concatenate([r[::-1], r])
        d, al = d0 * r * r, math.pi * c["f0"] * (1 - r)
        b = np.exp(-(d + al) * dt)
        a = d * (b - 1) / (d + al)
        if top:
            a[:count], b[:count] = 0.0, 1.0
        out.append((a, b))
    (a, b), (ah, bh) = out
    return a, ah, b, bh


def _cpml_axes(c):
    ns = [c["nx"]] + ([c["ny"]] if c["ny"] else []) + [c["nz"]]
    return [_cpml(c, n, c["h"], c["freetop"] and d == len(ns) - 1) for d, n in enumerate(ns)]


def _source_scale(c, model, src):
    """What the scaled source time function of each shot's source is multiplied with."""
    dt, h = _dt(c), _spacing(c)
    cell = math.prod(h)
    out = []
    for s in src:
        at = tuple(int(i) - 1 for i in s[::-1])
        if c["family"] == "cd":
            out.append(dt ** 2 * float(model["vp"][at]) ** 2 / cell)
        elif c["family"] == "vd":
            out.append(dt * float(model["vp"][at]) ** 2 * float(model["rho"][at]) / cell)
        else:
            out.append(1.0 / cell)
    return out


def _amplitude(c):
    """A typical amplitude of the recorded field per unit of scaled source."""
    dt, h = _dt(c), c["h"]
    if c["family"] == "cd":
        return 0.05 * dt ** 2 * 2000.0 ** 2 / math.prod(_spacing(c)) * 20
    if c["family"] == "vd":
        return 0.05 * dt * 2000.0 ** 2 * 2000.0 / h ** 2 * 5
    return dt ** 2 / (2000.0 * h ** 3) * (0.5 if not c["force"] else 5.0 * h)


# ---------------------------------------------------------------------------
# Elastic point tables: the windowed sinc of a node position on a grid whose
# points are shifted by (sx, sz) cells (Kaiser, radius 4, beta 6.31).
# ---------------------------------------------------------------------------
def _spread1(shift):
    k = np.arange(-4, 5) if shift == 0 else np.arange(-4, 4)
    x = k + shift
    w = np.i0(6.31 * np.sqrt(np.maximum(0.0, 1 - (x / 4.0) ** 2))) / np.i0(6.31) * np.sinc(x)
    keep = np.abs(w) > 1e-15
    return k[keep], w[keep]


def _spread(nodes, sx, sz):
    kx, wx = _spread1(sx)
    kz, wz = _spread1(sz)
    ij = np.stack([np.broadcast_to(kx[None, :], (len(kz), len(kx))), np.broadcast_to(kz[:, None], (len(kz), len(kx)))], -1)
    w = (wz[:, None] * wx[None, :]).reshape(-1)
    pts = np.asarray(nodes)[:, None, :] + ij.reshape(1, -1, 2)
    return pts.astype(np.int32), np.broadcast_to(w, pts.shape[:2]).astype(np.float32)


def _tables(c, nodes, kind):
    """kind: 'stress' (sigma_xx/zz nodes, sigma_xz nodes) or 'u' (ux nodes, uz nodes)."""
    shifts = [(0, 0), (0.5, 0.5)] if kind == "stress" else [(0.5, 0), (0, 0.5)]
    return [_spread(nodes, *s) for s in shifts]


def _momtens(c, seed):
    r = np.random.default_rng([int(seed), 9]).uniform(0.8, 1.2, 2)
    return np.array([r[0], r[1], 0.1], dtype=np.float32)


# ---------------------------------------------------------------------------
# Device-resident simulations through the C ABI
# ---------------------------------------------------------------------------
class _Sim:
    """A simulation handle with its material, shots and output buffers."""
    _ctx = None

    def __init__(self, c, seed):
        sw = _package()
        L = sw._lib
        if _Sim._ctx is None:
            _Sim._ctx = L.Context(0)
        self.ctx, self.lib, self.h, self.c = _Sim._ctx, _Sim._ctx.lib, ctypes.c_void_p(), c
        grad, fam = c["mode"] == "gradient", c["family"]
        model = _model(c, seed)
        src, rec = _geometry(c, seed)
        ns = [c["nx"]] + ([c["ny"]] if c["ny"] else []) + [c["nz"]]
        gp = L.SwGradParams(check_freq=c["K"], compute_misfit=1, snapshot_bf16=c["snap"])
        prm = L.SwElasticParams() if fam == "elastic" else L.SwAcousticParams()
        for d, n in enumerate(ns):
            prm.n[d], prm.h[d] = n, c["h"]
        prm.dt, prm.halo, prm.rcoef, prm.freetop = _dt(c), c["halo"], 1e-4, int(c["freetop"])
        host = {k: np.ascontiguousarray(v.cpu().numpy()) for k, v in model.items()} if fam != "cd" else {}
        if fam == "cd":
            prm.ndim = len(ns)
            self._ok(self.lib.sw_wavesim_create(self.ctx.h, ctypes.byref(prm), int(grad), ctypes.byref(gp), ctypes.byref(self.h)))
            self._free = self.lib.sw_wavesim_destroy
            if c["compensated"]:
                self._ok(self.lib.sw_wavesim_set_precision(self.h, 1))
                self.vp64 = model["vp"].double()
                torch.cuda.synchronize()
                self._ok(self.lib.sw_wavesim_set_vp64(self.h, self.vp64.data_ptr(), 1))
            else:
                self.vp = model["vp"]
                torch.cuda.synchronize()
                self._ok(self.lib.sw_wavesim_set_vp(self.h, self.vp.data_ptr(), 1))
        elif fam == "vd":
            prm.ndim, prm.n[2], prm.h[2] = 2, 1, 1.0
            self._ok(self.lib.sw_acoustic_vd_create(self.ctx.h, ctypes.byref(prm), int(c["harmonic"]), int(grad),
                                                    ctypes.byref(gp), ctypes.byref(self.h)))
            self._free = self.lib.sw_acoustic_vd_destroy
            self._ok(self.lib.sw_acoustic_vd_set_material(self.h, host["vp"].ctypes.data, host["rho"].ctypes.data))
        else:
            prm.interp_rho = prm.interp_mu = int(c["harmonic"])
            self._ok(self.lib.sw_elastic_create(self.ctx.h, ctypes.byref(prm), int(grad), ctypes.byref(gp), ctypes.byref(self.h)))
            self._free = self.lib.sw_elastic_destroy
            self._ok(self.lib.sw_elastic_set_material(self.h, *(host[k].ctypes.data for k in ("lambda", "mu", "rho"))))
        self._shots(L, c, seed, model, src, rec, grad)
        names = {"cd": ["vp"], "vd": ["vp", "rho"], "elastic": ["rho", "lambda", "mu"]}[fam] if grad else []
        shape = tuple(next(iter(model.values())).shape)
        self.grads = {k: torch.zeros(shape, dtype=torch.float64, device=DEV) for k in names}
        self.misfit = torch.zeros(1, dtype=torch.float64, device=DEV)
        fn = {"cd": "sw_acoustic_", "vd": "sw_acoustic_vd_", "elastic": "sw_elastic_"}[fam] + c["mode"]
        self.call = getattr(self.lib, fn)
        self.args = [self.h, c["shots"], self.structs, 1] + [g.data_ptr() for g in self.grads.values()]
        if grad:
            self.args.append(self.misfit.data_ptr())
        torch.cuda.synchronize()

    def _ok(self, rc):
        self.ctx.check(rc, "perf case")

    def _shots(self, L, c, seed, model, src, rec, grad):
        fam = c["family"]
        el = fam == "elastic"
        self.structs = ((L.SwElasticShot if el else L.SwAcousticShot) * c["shots"])()
        self.keep, self.traces = [], []
        axes = _cpml_axes(c)
        cp64 = np.concatenate([x for ax in axes for x in ax])
        cp = cp64.astype(np.float32)
        scale, stf = _source_scale(c, model, src), _wavelet(c)
        self.keep += [cp, cp64]
        for k, (st, nt) in enumerate(zip(self.structs, _nts(c))):
            tf = stf[:nt] * scale[k]
            if el and c["force"]:
                tf = np.stack([0.2 * tf, tf])
            tf = torch.from_numpy(np.ascontiguousarray(tf, dtype=np.float32)).to(DEV)
            tr = torch.zeros((len(rec[k]),) + ((2,) if el else ()) + (nt,), device=DEV)
            st.nt, st.nsrc, st.nrec = nt, 1, len(rec[k])
            st.srctf, st.traces, st.cpml = tf.data_ptr(), tr.data_ptr(), cp.ctypes.data
            self.keep.append(tf)
            self.traces.append(tr)
            if el:
                st.kind = int(c["force"])
                rec_tab = self._table_arrays(_tables(c, rec[k], "u"), len(rec[k]))
                src_tab = self._table_arrays(_tables(c, src[k:k + 1], "u" if c["force"] else "stress"), 1)
                mt = _momtens(c, seed)
                st.momtens = mt.ctypes.data
                self.keep += [mt]
                for t in range(2):
                    for tgt, tab in ((st.src[t], src_tab[t]), (st.rec[t], rec_tab[t])):
                        tgt.offsets, tgt.ij, tgt.coef = (x.ctypes.data for x in tab)
            else:
                si, ri = np.asfortranarray(src[k:k + 1]), np.asfortranarray(rec[k])
                st.src_idx, st.rec_idx, st.cpml64 = si.ctypes.data, ri.ctypes.data, cp64.ctypes.data
                self.keep += [si, ri]
            if grad:
                obs = _observed(c, seed, k, nt, src, rec, _amplitude(c))
                if el:
                    obs = torch.stack([0.4 * obs, obs], 1).contiguous()
                st.observed = obs.data_ptr()
                self.keep.append(obs)

    def _table_arrays(self, tables, count):
        out = []
        for ij, w in tables:
            off = np.arange(count + 1, dtype=np.int32) * w.shape[1]
            arrs = (off, np.ascontiguousarray(ij.reshape(-1, 2)), np.ascontiguousarray(w.reshape(-1)))
            self.keep += list(arrs)
            out.append(arrs)
        return out

    def run(self):
        self._ok(self.call(*self.args))
        out = {"traces": self.traces}
        if self.grads:
            out.update(gradient=self.grads, misfit=self.misfit)
        return out

    def __del__(self):
        if getattr(self, "_free", None) and self.h:
            self._free(self.h)
            self.h = ctypes.c_void_p()


class _Mirror:
    """The same through the package's swforward / swgradient, on host arrays."""

    def __init__(self, c, seed):
        sw = self.sw = _package()
        self.c = c
        model = _model(c, seed)
        src, rec = _geometry(c, seed)
        h, dt = c["h"], _dt(c)
        vp = np.asfortranarray(model["vp"].cpu().numpy().T.astype(np.float64))
        bc = sw.CPMLBoundaryConditionParameters(halo=c["halo"], rcoef=1e-4, freeboundtop=c["freetop"], vel_max=VMAX)
        prm = sw.InputParametersAcoustic(c["nt"], dt, vp.shape, _spacing(c), bc)
        stf, self.shots, self.misfits = _wavelet(c), [], []
        for k, nt in enumerate(_nts(c)):
            self.shots.append(sw.ScalarShot(sw.ScalarSources((src[k:k + 1] - 1) * h, stf[:nt], c["f0"]),
                                            sw.ScalarReceivers((rec[k] - 1) * h, nt)))
            self.misfits.append(sw.L2Misfit(observed=_observed(c, seed, k, nt, src, rec, _amplitude(c)).cpu().numpy().T))
        self.model = sw.VpAcousticCDMaterialProperties(vp)
        grad = c["mode"] == "gradient"
        gp = sw.GradParameters(compute_misfit=True, check_freq=c["K"]) if grad else None
        rp = sw.RunParameters(erroronPPW=False, minPPW=0, compensated=c["compensated"])
        self.ws = sw.build_wavesim(prm, self.model, runparams=rp, gradparams=gp, gradient=grad)
        self.gp = gp

    def run(self):
        if self.c["mode"] == "forward":
            self.sw.swforward(self.ws, self.model, self.shots)
            return {"traces": [s.recs.seismograms for s in self.shots]}
        g, m = self.sw.swgradient(self.ws, self.model, self.shots, self.misfits, gradparams=self.gp)
        return {"traces": [s.recs.seismograms for s in self.shots], "gradient": g, "misfit": m}


def prepare(case, seed):
    return (_Mirror if case["mirror"] else _Sim)(case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------
# The same results in 64 bits, plain torch: all shots of a case in one batch
# axis, the damping variables on the whole grid (their coefficients are 0
# outside the layers).
# ---------------------------------------------------------------------------
def _strip(vals, n, left, right, count):
    """Coefficients of `vals` on n points: the first `left` and from index n - right on, the rest 0."""
    out = torch.zeros(n, dtype=torch.float64)
    v = torch.from_numpy(vals)
    out[:left] = v[:left]
    out[n - right:] = v[count:count + right]
    return out.to(DEV)


def _on(v, dim, ndim):
    return v.reshape([-1 if d == dim else 1 for d in range(ndim)])


def _cut(x, dim, a, b):
    return x.narrow(dim, a, x.shape[dim] - a - b)


class _Points:
    """Weighted points of all shots: values at (shot, item) of a field, and scattered additions."""

    def __init__(self, shot, lin, w, item):
        self.shot, self.lin, self.w, self.item = (torch.as_tensor(x, device=DEV) for x in (shot, lin, w, item))
        self.w = self.w.double()

    def read(self, f, shots, items):
        v = f.reshape(f.shape[0], -1)[self.shot, self.lin] * self.w
        return torch.zeros(shots * items, dtype=torch.float64, device=DEV).index_add_(0, self.shot * items + self.item, v).reshape(shots, items)

    def weights(self, f, shots, items):
        """f at every (shot, item) of a table with one point per item."""
        out = torch.zeros((shots, items), dtype=torch.float64, device=DEV)
        out[self.shot, self.item] = f.reshape(-1)[self.lin]
        return out

    def add(self, f, values, scale=None):
        v = values[self.shot, self.item] * self.w
        if scale is not None:
            v = v * scale.reshape(-1)[self.lin]
        f.reshape(f.shape[0], -1).index_put_((self.shot, self.lin), v, accumulate=True)


def _nearest(c, nodes_per_shot):
    ns = [c["nx"]] + ([c["ny"]] if c["ny"] else []) + [c["nz"]]
    shot, lin, item = [], [], []
    for k, nodes in enumerate(nodes_per_shot):
        l = np.zeros(len(nodes), dtype=np.int64)
        for d in reversed(range(len(ns))):
            l = l * ns[d] + (nodes[:, d].astype(np.int64) - 1)
        shot.append(np.full(len(nodes), k))
        lin.append(l)
        item.append(np.arange(len(nodes)))
    lin = np.concatenate(lin)
    return _Points(np.concatenate(shot), lin, np.ones(len(lin)), np.concatenate(item))


def _spread_points(tables, nxs):
    """tables: per shot (ij, w) of one grid with nxs columns."""
    shot, lin, w, item = [], [], [], []
    for k, (ij, wt) in enumerate(tables):
        m, q = wt.shape
        shot.append(np.full(m * q, k))
        lin.append(((ij[..., 1].astype(np.int64) - 1) * nxs + ij[..., 0] - 1).reshape(-1))
        w.append(wt.astype(np.float64).reshape(-1))
        item.append(np.repeat(np.arange(m), q))
    return _Points(*(np.concatenate(x) for x in (shot, lin, w, item)))


class _CD:
    def __init__(self, c, model, src, rec):
        self.c, self.S = c, c["shots"]
        vp = model["vp"].double()
        self.vp, self.fact = vp, _dt(c) ** 2 * vp ** 2
        nd = vp.dim()
        self.axes = []
        for d, (a, ah, b, bh) in enumerate(_cpml_axes(c)):
            n, H, dim = vp.shape[nd - 1 - d], c["halo"], nd - d
            half = [_on(_strip(v, n - 1, H, H, H), dim, nd + 1) for v in (ah, bh)]
            # node i (1-based) takes entry i on the left, i - n + 2 halo + 1 on the right (from node n - halo + 1)
            node = [_on(_strip(v, n, H, H, H + 1)[1:-1], dim, nd + 1) for v in (a, b)]
            layer = _on(_strip(np.ones(2 * H + 2), n, H, H, H + 1)[1:-1], dim, nd + 1)
            self.axes.append((dim, half, node, layer))
        self.src, self.rec = _nearest(c, [s[None] for s in src]), _nearest(c, rec)
        self.recs = max(len(r) for r in rec)

    def zero(self):
        shape = (self.S,) + tuple(self.vp.shape)
        z = lambda s: torch.zeros(s, dtype=torch.float64, device=DEV)  # noqa: E731
        st = {"p": z(shape), "old": z(shape), "psi": [], "xi": []}
        for dim, _, _, _ in self.axes:
            s = list(shape)
            s[dim] -= 1
            st["psi"].append(z(s))
            st["xi"].append(z([shape[0]] + [x - 2 for x in shape[1:]]))
        return st

    def step(self, st, pts, values):
        p, h, lap = st["p"], self.c["h"], None
        for k, (dim, (ah, bh), (a, b), layer) in enumerate(self.axes):
            g = torch.diff(p, dim=dim) / h
            st["psi"][k].mul_(bh).add_(ah * g)
            # only the nodes in a layer see the half nodes' variables
            t = torch.diff(g, dim=dim) / h + layer * torch.diff(st["psi"][k], dim=dim) / h
            for other, _, _, _ in self.axes:
                if other != dim:
                    t = _cut(t, other, 1, 1)
            st["xi"][k].mul_(b).add_(a * t)
            t = t + st["xi"][k]
            lap = t if lap is None else lap + t
        new = torch.zeros_like(p)
        inner = tuple([slice(None)] + [slice(1, -1)] * (p.dim() - 1))
        new[inner] = 2 * p[inner] - st["old"][inner] + self.fact[inner[1:]] * lap
        pts.add(new, values)
        st["old"], st["p"] = p, new

    def forward(self, stf):
        st = self.zero()
        hist, tr = [st["old"], st["p"]], []
        for it in range(self.c["nt"]):
            self.step(st, self.src, stf[:, it:it + 1])
            tr.append(self.rec.read(st["p"], self.S, self.recs))
            if self.c["mode"] == "gradient":
                hist.append(st["p"])
        return torch.stack(tr, -1), hist

    def gradient(self, hist, res):
        st, g, dt = self.zero(), torch.zeros_like(self.vp), _dt(self.c)
        f = self.rec.weights(self.fact, self.S, self.recs)
        for it in range(self.c["nt"] - 1, -1, -1):
            self.step(st, self.rec, -res[..., it] * f)
            g += (st["p"] * (hist[it + 2] - 2 * hist[it + 1] + hist[it])).sum(0)
            del hist[it + 2]
        return {"vp": 2 / self.vp ** 3 * g / dt ** 2}


def _d4(f, dim, lo, hi, h):
    """(f[i-1] - 27 f[i] + 27 f[i+1] - f[i+2]) / 24 h with lo / hi points (tensors, or counts of zeros) put before and after."""
    parts = []
    for v in (lo, f, hi):
        if isinstance(v, int):
            if v == 0:
                continue
            s = list(f.shape)
            s[dim] = v
            v = torch.zeros(s, dtype=f.dtype, device=f.device)
        parts.append(v)
    x = torch.cat(parts, dim)
    m = x.shape[dim] - 3
    q = [x.narrow(dim, k, m) for k in range(4)]
    return ((q[0] - q[3]) + 27 * (q[2] - q[1])) / (24 * h)


def _half(m, dims, harmonic):
    v = 1 / m if harmonic else m
    for d in dims:
        v = (v.narrow(d, 0, v.shape[d] - 1) + v.narrow(d, 1, v.shape[d] - 1)) / 2
    return 1 / v if harmonic else v


def _back(m, g, dims, harmonic):
    """The chain rule of _half, added over the corners."""
    out = torch.zeros_like(m)
    w = g / 2 ** len(dims)
    if harmonic:
        w = w * _half(m, dims, True) ** 2
    for k in range(2 ** len(dims)):
        v = out
        for j, d in enumerate(dims):
            v = v.narrow(d, k >> j & 1, m.shape[d] - 1)
        v += w
    return out / m ** 2 if harmonic else out


class _VD:
    def __init__(self, c, model, src, rec):
        self.c, self.S, self.recs = c, c["shots"], max(len(r) for r in rec)
        self.vp, self.rho = model["vp"].double(), model["rho"].double()
        dt, H = _dt(c), c["halo"]
        self.m0 = self.vp ** 2 * self.rho * dt
        self.m = 1 / self.rho
        self.m1x, self.m1z = (_half(self.m, [d], c["harmonic"]) * dt for d in (1, 0))
        self.k = []
        for d, (a, ah, b, bh) in enumerate(_cpml_axes(c)):
            n = self.vp.shape[1 - d]
            half = [_on(_strip(v, n - 1, H, H, H), 2 - d, 3) for v in (ah, bh)]
            node = [_on(_strip(v, n, H + 1, H + 1, H + 1)[1:-1], 2 - d, 3) for v in (a, b)]
            self.k.append((half, node))
        self.src, self.rec = _nearest(c, [s[None] for s in src]), _nearest(c, rec)

    def zero(self):
        nz, nx = self.vp.shape
        z = lambda a, b: torch.zeros((self.S, a, b), dtype=torch.float64, device=DEV)  # noqa: E731
        return {"p": z(nz, nx), "vx": z(nz, nx - 1), "vz": z(nz - 1, nx), "psx": z(nz, nx - 1), "psz": z(nz - 1, nx),
                "xix": z(nz - 2, nx - 2), "xiz": z(nz - 2, nx - 2)}

    def update_p(self, s):
        h = self.c["h"]
        (_, (ax, bx)), (_, (az, bz)) = self.k
        dx = _d4(s["vx"][:, 1:-1], 2, 1, 1, h)
        s["xix"] = bx * s["xix"] + ax * dx
        dz = _d4(s["vz"][:, :, 1:-1], 1, 1, 1, h)
        s["xiz"] = bz * s["xiz"] + az * dz
        p = s["p"].clone()
        p[:, 1:-1, 1:-1] -= self.m0[1:-1, 1:-1] * (dx + s["xix"] + dz + s["xiz"])
        s["p"] = p

    def update_v(self, s):
        h = self.c["h"]
        ((ax, bx), _), ((az, bz), _) = self.k
        d = _d4(s["p"], 2, 1, 1, h)
        s["psx"] = bx * s["psx"] + ax * d
        s["vx"] = s["vx"] - self.m1x * (d + s["psx"])
        d = _d4(s["p"], 1, 1, 1, h)
        s["psz"] = bz * s["psz"] + az * d
        s["vz"] = s["vz"] - self.m1z * (d + s["psz"])

    def forward(self, stf):
        s = self.zero()
        hist, tr = [s["p"]], []
        for it in range(self.c["nt"]):
            self.update_p(s)
            self.src.add(s["p"], stf[:, it:it + 1])
            self.update_v(s)
            tr.append(self.rec.read(s["p"], self.S, self.recs))
            if self.c["mode"] == "gradient":
                hist.append(s["p"])
        return torch.stack(tr, -1), hist

    def gradient(self, hist, res):
        s, h, dt = self.zero(), self.c["h"], _dt(self.c)
        g0, gx, gz = torch.zeros_like(self.m0), torch.zeros_like(self.m1x), torch.zeros_like(self.m1z)
        f = self.rec.weights(self.m0, self.S, self.recs)
        for it in range(self.c["nt"] - 1, -1, -1):
            self.update_v(s)
            self.update_p(s)
            self.rec.add(s["p"], -res[..., it] * f)
            pc = hist[it + 1]
            g0 -= (s["p"] * (pc - hist[it])).sum(0) / dt
            gx += (s["vx"] * _d4(pc, 2, 1, 1, h)).sum(0)
            gz += (s["vz"] * _d4(pc, 1, 1, 1, h)).sum(0)
            del hist[it + 1]
        hm = self.c["harmonic"]
        g1 = _back(self.m, gx, [1], hm) + _back(self.m, gz, [0], hm)
        vp, rho = self.vp, self.rho
        return {"vp": -2 * g0 / (vp ** 3 * rho), "rho": -g0 / (vp ** 2 * rho ** 2) - g1 / rho}


class _Elastic:
    def __init__(self, c, model, src, rec, seed):
        self.c, self.S, self.recs = c, c["shots"], max(len(r) for r in rec)
        self.lam, self.mu, self.rho = (model[k].double() for k in ("lambda", "mu", "rho"))
        hm, dt, H = c["harmonic"], _dt(c), c["halo"]
        self.bx, self.bz = dt ** 2 / _half(self.rho, [1], hm), dt ** 2 / _half(self.rho, [0], hm)
        self.muxz = _half(self.mu, [0, 1], hm)
        self.k = []
        for d, (a, ah, b, bh) in enumerate(_cpml_axes(c)):
            n = self.lam.shape[1 - d]
            half = [_on(_strip(v, n - 1, H, H, H), 2 - d, 3) for v in (ah, bh)]
            # node i takes entry i up to halo + 1 and i - n + 2 halo + 2 from node n - halo on
            node = [_on(_strip(v, n, H + 1, H + 1, H + 1), 2 - d, 3) for v in (a, b)]
            self.k.append((half, node))
        nx = c["nx"]
        ts = [_tables(c, s[None], "u" if c["force"] else "stress") for s in src]
        self.src = [_spread_points([t[q] for t in ts], (nx - 1, nx)[q] if c["force"] else (nx, nx - 1)[q]) for q in range(2)]
        tr = [_tables(c, r, "u") for r in rec]
        self.rec = [_spread_points([t[q] for t in tr], (nx - 1, nx)[q]) for q in range(2)]
        self.mt = _momtens(c, seed).astype(np.float64)

    def zero(self):
        nz, nx = self.lam.shape
        z = lambda a, b: torch.zeros((self.S, a, b), dtype=torch.float64, device=DEV)  # noqa: E731
        s = {k: z(nz, nx - 1) for k in ("ux", "uxo", "p_sxx_x", "p_sxz_z")}
        s.update({k: z(nz - 1, nx) for k in ("uz", "uzo", "p_sxz_x", "p_szz_z")})
        s.update({k: z(nz, nx) for k in ("p_ux_x", "p_uz_z")})
        s.update({k: z(nz - 1, nx - 1) for k in ("p_uz_x", "p_ux_z")})
        return s

    # derivatives, with the mirror rules of the free surface at the top
    def dux_dx(self, ux):  # on the nodes
        return _d4(ux, 2, 2, 2, self.c["h"])

    def duz_dz(self, ux, uz, dxx):
        if not self.c["freetop"]:
            return _d4(uz, 1, 2, 2, self.c["h"])
        d = _d4(uz, 1, torch.cat([uz[:, 1:2], uz[:, :1]], 1), 2, self.c["h"])  # row 2 reads uz(1) twice
        d[:, 0] = -(self.lam[0] / (self.lam[0] + 2 * self.mu[0])) * dxx[:, 0]
        return d

    def duz_dx(self, uz):
        return _d4(uz, 2, 1, 1, self.c["h"])

    def dux_dz(self, ux):
        return _d4(ux, 1, ux[:, 1:2] if self.c["freetop"] else 1, 1, self.c["h"])

    def step(self, s, pts, values, force, stress=None):
        c, h, lam, mu = self.c, self.c["h"], self.lam, self.mu
        ((axh, bxh), (ax, bx)), ((azh, bzh), (az, bz)) = self.k

        def damp(key, d, a, b):
            s[key] = b * s[key] + a * d
            return d + s[key]

        dxx = self.dux_dx(s["ux"])
        dzz = self.duz_dz(s["ux"], s["uz"], dxx)
        dxx, dzz = damp("p_ux_x", dxx, ax, bx), damp("p_uz_z", dzz, az, bz)
        sxx, szz = (lam + 2 * mu) * dxx + lam * dzz, lam * dxx + (lam + 2 * mu) * dzz
        for q in (sxx, szz):  # never updated there
            q[:, -1] = 0
            q[:, :, 0] = 0
            q[:, :, -1] = 0
        szz[:, 0] = 0
        if not c["freetop"]:
            sxx[:, 0] = 0
        sxz = self.muxz * (damp("p_uz_x", self.duz_dx(s["uz"]), axh, bxh) + damp("p_ux_z", self.dux_dz(s["ux"]), azh, bzh))
        if stress is not None:
            self.src[0].add(sxx, self.mt[0] * stress)
            self.src[0].add(szz, self.mt[1] * stress)
            self.src[1].add(sxz, self.mt[2] * stress)
        ft = c["freetop"]
        d1 = damp("p_sxx_x", _d4(sxx, 2, 1, 1, h), axh, bxh)
        d2 = damp("p_sxz_z", _d4(sxz, 1, -sxz[:, :2].flip(1) if ft else 2, 2, h), az, bz)
        uxn = 2 * s["ux"] - s["uxo"] + self.bx * (d1 + d2)
        d1 = damp("p_sxz_x", _d4(sxz, 2, 2, 2, h), ax, bx)
        d2 = damp("p_szz_z", _d4(szz, 1, -szz[:, 1:2] if ft else 1, 1, h), azh, bzh)
        uzn = 2 * s["uz"] - s["uzo"] + self.bz * (d1 + d2)
        if force:
            pts[0].add(uxn, values[0], self.bx)
            pts[1].add(uzn, values[1], self.bz)
        s["uxo"], s["uzo"], s["ux"], s["uz"] = s["ux"], s["uz"], uxn, uzn

    def forward(self, stf):
        c, s = self.c, self.zero()
        hist, tr = [(s["uxo"], s["uzo"]), (s["ux"], s["uz"])], []
        for it in range(c["nt"]):
            f = stf[:, it:it + 1]
            if c["force"]:
                self.step(s, self.src, (0.2 * f, f), True)
            else:
                self.step(s, None, None, False, f)
            tr.append(torch.stack([r.read(s[k], self.S, self.recs) for r, k in zip(self.rec, ("ux", "uz"))], 2))
            if c["mode"] == "gradient":
                hist.append((s["ux"], s["uz"]))
        return torch.stack(tr, -1), hist

    def gradient(self, hist, res):
        s, ft, dt = self.zero(), self.c["freetop"], _dt(self.c)
        gl, gm = torch.zeros_like(self.lam), torch.zeros_like(self.lam)
        gx, gz, gxz = torch.zeros_like(self.bx), torch.zeros_like(self.bz), torch.zeros_like(self.muxz)
        w = torch.ones_like(self.lam)
        w[-1], w[:, 0], w[:, -1] = 0, 0, 0
        w[0] = 0.5 if ft else 0
        wx = torch.ones_like(self.bx)
        if ft:
            wx[0] = 0.5
        for it in range(self.c["nt"] - 1, -1, -1):
            self.step(s, self.rec, (-res[..., 0, it], -res[..., 1, it]), True)
            (ux0, uz0), (ux, uz), (ux2, uz2) = hist[it], hist[it + 1], hist[it + 2]
            gx += wx * (s["ux"] * (ux0 - 2 * ux + ux2)).sum(0) / dt ** 2
            gz += (s["uz"] * (uz0 - 2 * uz + uz2)).sum(0) / dt ** 2
            exx, axx = self.dux_dx(ux), self.dux_dx(s["ux"])
            ezz, azz = self.duz_dz(ux, uz, exx), self.duz_dz(s["ux"], s["uz"], axx)
            gl += w * ((exx + ezz) * (axx + azz)).sum(0)
            gm += w * 2 * (exx * axx + ezz * azz).sum(0)
            gxz += ((self.duz_dx(uz) + self.dux_dz(ux)) * (self.duz_dx(s["uz"]) + self.dux_dz(s["ux"]))).sum(0)
            del hist[it + 2]
        hm = self.c["harmonic"]
        return {"rho": _back(self.rho, gx, [1], hm) + _back(self.rho, gz, [0], hm), "lambda": gl,
                "mu": gm + _back(self.mu, gxz, [0, 1], hm)}


def exact(case, seed):
    c = case
    model = _model(c, seed)
    src, rec = _geometry(c, seed)
    S, nts, grad, el = c["shots"], _nts(c), c["mode"] == "gradient", c["family"] == "elastic"
    sim = (_Elastic(c, model, src, rec, seed) if el else {"cd": _CD, "vd": _VD}[c["family"]](c, model, src, rec))
    scale = torch.tensor(_source_scale(c, model, src), dtype=torch.float64, device=DEV)
    stf = torch.from_numpy(_wavelet(c)).to(DEV)[None, :] * scale[:, None]
    tr, hist = sim.forward(stf)
    traces = [tr[k, :len(rec[k]), ..., :nts[k]] for k in range(S)]
    if c["mirror"]:
        traces = [t.transpose(-1, -2) for t in traces]
    out = {"traces": traces}
    if grad:
        res, misfit = torch.zeros_like(tr), 0.0
        for k in range(S):
            obs = _observed(c, seed, k, nts[k], src, rec, _amplitude(c)).double()
            if el:
                obs = torch.stack([(0.4 * obs.float()).double(), obs], 1)
            res[k, :len(rec[k]), ..., :nts[k]] = tr[k, :len(rec[k]), ..., :nts[k]] - obs
            misfit = misfit + (res[k] ** 2).sum() / 2
        g = sim.gradient(hist, res)
        if c["mirror"]:
            g = {k: v.transpose(-1, -2) for k, v in g.items()}
        out.update(gradient=g, misfit=misfit if c["mirror"] else misfit.reshape(1))
    return out
