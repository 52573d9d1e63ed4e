"""Timed cases of the framework's public entry points.

A case is a dict of plain values. `kind` says which call it stands for:

  columns   moist_implicit_correction_noalloc on device arrays of a host with its own memory pool
  oneshot   model.rk3_step(s, p): the reference's calling convention on a host State
  steps     model.Model kept by the program: upload a State, advance it, download it
  ensemble  model.Ensemble kept by the program: upload, advance and download every member
  adjoint   Model.adjoint: a forward run and the gradient of rain and condensed water
  adjoint_ensemble  Ensemble.adjoint: the same, packed over members

and `workload` which simulation it runs: "bubble" (warm moist bubble on 100 m cells), "sounding"
(bubbles on an analytic sounding, 250 m x 125 m cells) or "default" (the reference's default
Params: stretched grid, surface fluxes and radiation on). States are advanced `spin` large steps
when they are prepared, so that the timed steps meet developed flow, clouds and rain; `prec` is
the State's precision, `native` the literal Float32 elimination of the w-p columns.
"""
import ctypes as C
import math

import numpy as np
import torch

from moist2d_b200 import abi, init, model
from moist2d_b200._lib import lib
from moist2d_b200.params import Params, State, exchange_halo

FIELDS = ("rho", "rho_u", "rho_w", "rho_theta", "rho_qv", "rho_qc", "rho_qr")


def _case(name, kind, workload, nx, nz, prec="f32", ns=8, steps=1, spin=0, native=False, members=0, ckpt=0):
    c = {"kind": kind, "workload": workload, "nx": nx, "nz": nz, "prec": prec, "ns": ns, "steps": steps,
         "spin": spin, "native": native, "members": members, "ckpt": ckpt}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the column solve alone, from a host with its own device memory pool: one domain's columns
        _case("columns-2048x128", "columns", "sounding", 2048, 128),
        # a script or a unit test of a host program: one step of a small State, nothing kept
        _case("oneshot-64x40", "oneshot", "bubble", 64, 40, ns=6),
        # the warm bubble in both precisions, mid-run: the small domain where latency counts
        _case("bubble-200x100", "steps", "bubble", 200, 100, ns=6, steps=8, spin=300),
        _case("bubble-200x100-f64", "steps", "bubble", 200, 100, prec="f64", ns=6, steps=4, spin=200),
        # the command-line program's default simulation: 640 x 250, all physics on
        _case("default-640x250", "steps", "default", 640, 250, ns=3, steps=4, spin=30),
        # the benchmark domain, the early minutes of the simulation
        _case("sounding-2048x128", "steps", "sounding", 2048, 128, steps=5, spin=40),
        _case("sounding-2048x128-f64", "steps", "sounding", 2048, 128, prec="f64", steps=3, spin=15),
        # sizes that divide by nothing, the reference's literal Float32 elimination
        _case("ragged-733x77", "steps", "sounding", 733, 77, ns=5, steps=6, spin=60, native=True),
        # the largest single domain: four times the benchmark's
        _case("large-4096x256", "steps", "sounding", 4096, 256, steps=2, spin=6),
        # uneven members advanced together
        _case("ensemble-64", "ensemble", "sounding", 2048, 128, steps=6, spin=20, members=64),
        # gradients of the surface rain: one domain, and a few members packed
        _case("adjoint-512x96", "adjoint", "sounding", 512, 96, steps=8, spin=120, ckpt=4),
        _case("adjoint-ensemble-6", "adjoint_ensemble", "sounding", 1024, 128, steps=4, spin=80, members=6, ckpt=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "oneshot", "columns", "ensemble", "adjoint"])
    prec = rng.choice(["f32", "f32", "f32", "f64"])
    native = prec == "f32" and rng.random() < 0.2
    ns = rng.randint(2, 8)
    if kind == "columns":
        nz = _log(rng, 16, 500)
        return _case("", kind, "sounding", min(_log(rng, 33, 4000), 4 * 1024 * 1024 // (16 * nz)), nz, prec, native=native)
    if kind == "oneshot":
        return _case("", kind, "bubble", _log(rng, 24, 400), rng.randint(30, 100), prec, 6, native=native)
    if kind == "ensemble":
        return _case("", kind, "sounding", 256 * rng.randint(1, 8), 32 * rng.randint(1, 4), "f32", 8, rng.randint(2, 5),
                     rng.randint(4, 16), native, rng.randint(4, 56))
    if kind == "adjoint":
        steps = rng.randint(2, 6)
        return _case("", kind, "sounding", _log(rng, 64, 900), rng.randint(40, 128), prec, 8, steps, rng.randint(10, 60),
                     ckpt=rng.randint(1, steps))
    workload = rng.choice(["sounding", "sounding", "bubble", "default"])
    nx, nz = _log(rng, 48, 4096), _log(rng, 24, 250)
    if prec == "f64":
        nx = min(nx, 2048)
    if workload == "default":
        nz = max(nz, 150)  # the stretched grid has to reach the model top
    if workload == "bubble":
        nx, nz, ns = min(nx, 600), min(max(nz, 50), 120), max(ns, 6)
    if workload == "sounding":
        ns = max(ns, 5)
    if workload == "default":
        ns = 3
    return _case("", "steps", workload, nx, nz, prec, ns, rng.randint(1, 3), rng.randint(4, 12), native)


# ---------------------------------------------------------------- inputs

def _type(case):
    return np.float64 if case["prec"] == "f64" else np.float32


def _flags(case):
    return abi.MOIST_FLAG_TRI_NATIVE if case["native"] else 0


def _sounding(T, nx, nz, ns, seed, nbub):
    """Bubbles of a seeded amplitude and radius on the analytic sounding, spread over the domain:
    the environment column everywhere, the columns of one bubble at nbub places."""
    w = 40
    p0, b = init.sounding_bubbles_lib(T, seed=seed, nx=w, nz=nz, nbub=1, rad=(1.5e3, 3e3))
    p = p0.replace(Nx=nx, Lx=250.0 * nx, ns=ns)
    s = State(p)
    s.theta_ref[:] = b.theta_ref
    shift = int(np.random.RandomState(seed).randint(nx))
    h = p.halo
    for f in FIELDS:
        a, src = getattr(s, f)[:, h:h + nx], getattr(b, f)[:, h:h + w]
        a[:] = src[:, :1]
        for j in range(nbub):
            at = np.arange(w) + int((j + 0.5) * nx / nbub) - w // 2 + shift
            a[:, at % nx] = src
        exchange_halo(getattr(s, f), p)
    return p, s


def _initial(case, seed):
    T, nx, nz, ns = _type(case), case["nx"], case["nz"], case["ns"]
    if case["workload"] == "bubble":
        p, s = init.warm_bubble_lib(T, seed=seed % 100000, nx=nx, nz=nz)
        return (p, s) if ns == p.ns else (p.replace(ns=ns), s)
    if case["workload"] == "default":
        p = Params(T, Nx=nx, Nz=nz, Lx=250.0 * nx, ns=ns)
        s = State(p)
        init.init_state_lib(s, p, seed=seed % 100000)
        return p, s
    return _sounding(T, nx, nz, ns, seed % 100000, max(1, nx // 400))


def _members(case, seed):
    """Uneven members: sizes of the case alone, bubbles of the seed."""
    r = np.random.RandomState(17)
    out = []
    for m in range(case["members"]):
        nx = 256 * int(r.randint(max(1, case["nx"] // 1024), case["nx"] // 256 + 1))
        nz = 32 * int(r.randint(max(1, case["nz"] // 64), case["nz"] // 32 + 1))
        out.append(_sounding(_type(case), nx, nz, case["ns"], seed % 100000 + 7 * m, 1))
    return out


def _pinned(states, T):
    """The States with their fields in page-locked memory, the members' fields side by side:
    the States, and one flat array for each field."""
    flat = {}
    out = [State.__new__(State) for _ in states]
    for f in abi.STATE_FIELDS:
        n = sum(getattr(s, f).size for s in states)
        a = torch.empty(n, dtype=torch.float64 if T is np.float64 else torch.float32, pin_memory=True).numpy()
        at = 0
        for s, o in zip(states, out):
            v = getattr(s, f)
            w = a[at:at + v.size].reshape(v.shape, order="F")
            w[...] = v
            setattr(o, f, w)
            at += v.size
        flat[f] = a
    return out, flat


def _spun_up(case, seed):
    p, s = _initial(case, seed)
    m = model.Model(p, _flags(case))
    m.upload(s)
    if case["spin"]:
        m.step(case["spin"])
        m.download(s)
    return p, s, m


def _rain_weights(p):
    w = np.zeros(p.ia)
    w[p.is_ - 1:p.ie] = float(p.dx)
    return w


def _water_seed(p):
    """The condensed water of the final State counts as well: cloud, and rain that is falling."""
    return {f: np.asfortranarray(np.full((p.ka, p.ia), 100.0)) for f in ("rho_qc", "rho_qr")}


def _column_inputs(case, seed):
    """(ncols, nz) arrays, z fastest: rho_w, drho_w, theta, rt2pres of the sounding's columns."""
    T, nz, ncols = _type(case), case["nz"], case["nx"]
    p = Params(T, Nx=2, Nz=nz, Lx=500.0, H=125.0 * nz, dz0=125.0, z_fact=1.0, ns=8, dt=2.0)
    r = np.random.RandomState(seed % 100000)
    z = p.z.astype(np.float64)
    theta = 300.0 + 4e-3 * z[None, :] + r.uniform(-1, 1, (ncols, nz))
    rt2pres = 340.0 - 5e-3 * np.minimum(z, 12e3)[None, :] + r.uniform(-5, 5, (ncols, nz))
    rho_w = r.uniform(-0.5, 0.5, (ncols, nz))
    rho_w[:, -1] = 0.0
    drho_w = r.uniform(-1e-2, 1e-2, (ncols, nz))
    return p, [np.ascontiguousarray(a.astype(T)) for a in (rho_w, drho_w, theta, rt2pres)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "columns":
        p, arrays = _column_inputs(case, seed)
        dev = [torch.from_numpy(a).cuda() for a in arrays]
        return {"case": case, "p": p, "cp": p.to_c(), "dev": dev, "out": torch.empty_like(dev[0])}
    if kind == "oneshot":
        p, s = _initial(case, seed)
        return {"case": case, "p": p, "s": s}
    if kind in ("ensemble", "adjoint_ensemble"):
        mem = _members(case, seed)
        ps = [p for p, _ in mem]
        e = model.Ensemble(ps, _flags(case))
        for i, (_, s) in enumerate(mem):
            e.upload(i, s)
        e.step(case["spin"])
        for i, (_, s) in enumerate(mem):
            e.download(i, s)
        start, _ = _pinned([s for _, s in mem], _type(case))
        st = {"case": case, "e": e, "start": start}
        if kind == "ensemble":
            st["out"], st["flat"] = _pinned([s for _, s in mem], _type(case))
        else:
            st["weights"] = [_rain_weights(p) for p in ps]
            st["seeds"] = [_water_seed(p) for p in ps]
        return st
    p, s, m = _spun_up(case, seed)
    start, _ = _pinned([s], _type(case))
    st = {"case": case, "p": p, "m": m, "start": start[0]}
    if kind == "adjoint":
        st["weights"] = _rain_weights(p)
        st["seed"] = _water_seed(p)
    else:
        out, _ = _pinned([s], _type(case))
        st["out"] = out[0]
    return st


# ---------------------------------------------------------------- one pass

GRADS = FIELDS + ("prec", "k_auto", "qc_threshold", "objective")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "columns":
        p, dev, out = state["p"], state["dev"], state["out"]
        out.copy_(dev[0])
        err = C.create_string_buffer(256)
        rc = lib().moist_implicit_correction_noalloc(
            C.byref(state["cp"]), p.precision, _flags(case), case["nx"], out.data_ptr(), dev[1].data_ptr(),
            dev[2].data_ptr(), dev[3].data_ptr(), 0.25, C.c_void_p(torch.cuda.current_stream().cuda_stream), err, 256)
        if rc != abi.MOIST_OK:
            raise RuntimeError(err.value.decode())
        return out
    if kind == "oneshot":
        s = state["s"].copy()
        model.rk3_step(s, state["p"], 1, flags=_flags(case))
        return {f: getattr(s, f) for f in FIELDS + ("prec",)}
    if kind == "steps":
        m = state["m"]
        m.upload(state["start"])
        m.step(case["steps"])
        s = m.download(state["out"])
        return {f: getattr(s, f) for f in FIELDS + ("prec",)}
    if kind == "adjoint":
        m = state["m"]
        m.upload(state["start"])
        g = m.adjoint(case["steps"], case["ckpt"], prec_weight=state["weights"], state_seed=state["seed"])
        return {k: g[k] for k in GRADS}
    e = state["e"]
    for i, s in enumerate(state["start"]):
        e.upload(i, s)
    if kind == "adjoint_ensemble":
        grads = e.adjoint(case["steps"], case["ckpt"], prec_weights=state["weights"], state_seeds=state["seeds"])
        return [[g[k] for k in FIELDS + ("objective",)] for g in grads]
    e.step(case["steps"])
    for i, s in enumerate(state["out"]):
        e.download(i, s)
    return {f: state["flat"][f] for f in FIELDS + ("prec",)}


# ---------------------------------------------------------------- work

def work(case):
    """Bytes: the State (7 fields) read and written once a pass; with the adjoint the gradients
    too. Flops: about 75 a cell and acoustic substep, 250 + 150 a cell and stage of tendencies and
    diagnostics, 170 a cell, stage and tracer of transport, 1200 a cell of microphysics; the
    adjoint counted as four forward runs."""
    b = 8 if case["prec"] == "f64" else 4
    cells = case["nx"] * case["nz"]
    if case["kind"] == "columns":
        return {"bytes": 5 * cells * b, "flops": 45 * cells}
    if case["members"]:
        r = np.random.RandomState(17)
        cells = 0
        for _ in range(case["members"]):
            nx = 256 * int(r.randint(max(1, case["nx"] // 1024), case["nx"] // 256 + 1))
            cells += nx * 32 * int(r.randint(max(1, case["nz"] // 64), case["nz"] // 32 + 1))
    ns = case["ns"]
    sub = max(1, -(-ns // 3)) + max(1, -(-ns // 2)) + ns
    per = 75 * sub + 3 * 400 + 9 * 170 + 1200
    if case["kind"].startswith("adjoint"):
        return {"bytes": cells * (7 * b + 7 * 8), "flops": 4 * per * cells * case["steps"]}
    return {"bytes": 14 * cells * b, "flops": per * cells * case["steps"]}


# ---------------------------------------------------------------- the same step in 64 bits

class _Step64:
    """The large time step (Wicker-Skamarock RK3, split-explicit acoustic substeps, Koren-limited
    in-place tracer transport, Kessler microphysics) on (nz, nx) float64 arrays."""

    def __init__(self, p, s):
        f = lambda a: np.array(a, dtype=np.float64)  # noqa: E731
        self.p, self.c = p, p.c
        for k in ("GRAV", "Rd", "Rv", "Cpd", "Cpv", "Cpl", "P0", "Lv", "SIGMA", "K_auto", "Qc_threshold", "K_accr",
                  "K_evap", "A_term", "B_term", "T0", "ES0", "A_SAT", "B_SAT", "EPS", "EPSvap"):
            setattr(self, k, float(getattr(p.c, k)))
        self.dz, self.z, self.zf = f(p.dz), f(p.z), f(p.zf)
        self.dx, self.dt, self.nx, self.nz = float(p.dx), float(p.dt), p.Nx, p.Nz
        h = p.halo
        self.q = [f(getattr(s, x)[:, h:h + p.Nx]) for x in FIELDS]
        self.prec = f(s.prec[h:h + p.Nx])
        self.theta_ref = f(s.theta_ref)
        self.ru_left, self.rho_right = float(s.rho_u[0, h - 1]), float(s.rho[0, p.Nx + h])

    @staticmethod
    def sh(a, d):
        return np.roll(a, -d, axis=-1)  # a at i + d

    def gas(self, qv, qc, qr):
        qd = 1.0 - qv - qc - qr
        r = self.Rd * qd + self.Rv * qv
        cp = self.Cpd * qd + self.Cpv * qv + self.Cpl * (qc + qr)
        return qd, r, cp

    def sat(self, Tk, pr):
        tc = Tk - self.T0
        t = self.B_SAT + tc
        es = self.ES0 * np.exp(self.A_SAT * tc / t)
        des = es * self.A_SAT * (t - tc) / (t * t)
        t = pr - (1.0 - self.EPSvap) * es
        ok = t > self.EPS
        return np.where(ok, self.EPSvap * es / t, 0.0), np.where(ok, self.EPSvap * pr / (t * t), 1.0) * des

    def surface(self):
        p, (rho, ru, _, rt, qv, qc, qr) = self.p, [a[0] for a in self.q]
        qv, qc, qr = qv / rho, qc / rho, qr / rho
        _, r, cp = self.gas(qv, qc, qr)
        rum, rhop = np.roll(ru, 1), np.roll(rho, -1)
        rum[0], rhop[-1] = self.ru_left, self.rho_right
        uabs = np.maximum(np.abs(rum + ru) * 0.5 / rho, float(p.uabs_min))
        th = rt / rho
        pi = (r * rt / self.P0) ** (r / (cp - r))
        pis = pi + self.dz[0] * 0.5 * self.GRAV / (cp * th)
        ps = self.P0 * pis ** (cp / r)
        ts = float(p.temp_surf)
        rs = ps / (r * ts)
        u = ru / (rho + rhop) * 2.0
        d_u = -rs * float(p.Cd) * u * np.abs(u) / self.dz[0]
        d_th = rs * float(p.Ch) * uabs * (ts / pis - th) * pis / (pi * self.dz[0])
        qs, _ = self.sat(np.full_like(ps, ts), ps)
        return d_u, d_th, rs * float(p.Ce) * uabs * (qs - qv) / self.dz[0]

    def radiation(self):
        p, (rho, _, _, rt, rqv, rqc, rqr) = self.p, self.q
        _, r, cp = self.gas(rqv / rho, rqc / rho, rqr / rho)
        pi = (r * rt / self.P0) ** (r / (cp - r))
        T = rt / rho * pi
        dz = self.dz[:, None]
        eps = 1.0 - np.exp(-(float(p.k_abs_qv) * rqv + float(p.k_abs_qc) * rqc + float(p.k_abs_qr) * rqr) * dz)
        up, dn = np.zeros((self.nz + 1, self.nx)), np.zeros((self.nz + 1, self.nx))
        up[0] = float(p.surf_emissivity) * self.SIGMA * float(p.temp_surf) ** 4
        for k in range(self.nz):
            up[k + 1] = up[k] * (1.0 - eps[k]) + eps[k] * self.SIGMA * T[k] ** 4
        for k in range(self.nz - 1, -1, -1):
            dn[k] = dn[k + 1] * (1.0 - eps[k]) + eps[k] * self.SIGMA * T[k] ** 4
        hr = -(((up[1:] - dn[1:]) - (up[:-1] - dn[:-1])) / dz) / (cp * pi)
        al = 0.5 * (1.0 + np.tanh((self.z - (float(p.z_tropopose) + 1e3)) / 2e3)) / float(p.tau_cooling)
        return hr - (rt - rho * self.theta_ref[:, None]) * al[:, None]

    def physics(self):
        p, dt = self.p, self.dt
        rho, _, _, rt, rqv, rqc, rqr = self.q
        z2 = np.zeros_like(rho)
        d_u, d_th_s, d_qv_s = self.surface() if p.do_sf else (np.zeros(self.nx),) * 3
        th_rd = self.radiation() if p.do_rd else z2
        dqv, dqc, dqr, dth = z2.copy(), z2.copy(), z2.copy(), z2.copy()
        sed = z2.copy()
        d_prec = np.zeros(self.nx)
        if p.do_mp:
            th, qv, qc, qr = rt / rho, rqv / rho, rqc / rho, rqr / rho
            qd, r, cp = self.gas(qv, qc, qr)
            pi = (r * rt / self.P0) ** (r / (cp - r))
            lat, qv0 = self.Lv / (cp * pi), qv
            for _ in range(3):
                T, pr = th * pi, self.P0 * pi ** (cp / r)
                qs, dqs = self.sat(T, pr)
                ce = np.maximum(np.minimum((qv - qs) / (1.0 + (self.Lv / cp) * dqs), qv), -qc)
                qv, qc, th = qv - ce, qc + ce, th + ce * lat
                r = self.Rd * qd + self.Rv * qv
                cp = self.Cpd * qd + self.Cpv * qv + self.Cpl * (qc + qr)
                pi = (r * rho * th / self.P0) ** (r / (cp - r))
                lat = self.Lv / (cp * pi)
            ce = (qv0 - qv) * rho / dt
            dqv, dqc, dth = dqv - ce, dqc + ce, dth + ce * lat
            if p.do_auto:
                a = np.minimum(self.K_auto * np.maximum(0.0, qc - self.Qc_threshold), qc / dt)
                qc, qr, dqc, dqr = qc - a * dt, qr + a * dt, dqc - a * rho, dqr + a * rho
            if p.do_accr:
                a = np.where((qr > 1e-12) & (qc > 1e-12), np.minimum(self.K_accr * qc * qr, qc / dt), 0.0)
                qc, qr, dqc, dqr = qc - a * dt, qr + a * dt, dqc - a * rho, dqr + a * rho
            if p.do_revap:
                a = self.K_evap * (qs - qv) * np.sqrt(np.maximum(rho * qr, 0.0))
                a = np.where((qr > 1e-12) & (qv < qs), np.minimum(a, qr) / dt, 0.0) * rho
                dqr, dqv = dqr - a, dqv + a
                cp = self.Cpd * qd + self.Cpv * qv + self.Cpl * (qc + qr)
                r = self.Rd * qd + self.Rv * qv
                pi = (r * rho * th / self.P0) ** (r / (cp - r))
                dth = dth - a * self.Lv / (cp * pi)
            if p.do_sed:
                eff = np.maximum(0.0, rqr)
                vt = np.where(eff > 1e-12, self.A_term * (eff / rho) ** self.B_term, 0.0)
                fl = np.vstack([rqr * vt, np.zeros((1, self.nx))])
                sed = (fl[1:] - fl[:-1]) / self.dz[:, None]
                d_prec = fl[0]
        d_rho = sed.copy()
        d_rho[0] += d_qv_s
        du = z2.copy()
        du[0] += d_u
        d_th = dth + th_rd + d_rho * rt / rho
        d_th[0] += d_th_s
        dqv[0] += d_qv_s
        return (d_rho, du, d_th, dqv, dqc, dqr + sed), d_prec

    def faces_x(self, flux, a):
        """Third-order upwind flux at i + 1/2 of a face velocity / mass flux and the values a."""
        m1, p1, p2 = self.sh(a, -1), self.sh(a, 1), self.sh(a, 2)
        up, dn = flux * (-m1 + 5.0 * a + 2.0 * p1) / 6.0, flux * (-p2 + 5.0 * p1 + 2.0 * a) / 6.0
        return np.where(flux > self.EPS, up, np.where(flux < -self.EPS, dn, flux * (a + p1) * 0.5))

    def faces_z(self, flux, a, top, pos=None, neg=None):
        """The same at k + 1/2 for k = 0 .. len - 2 (rows of a): centred where an upwind row is
        missing (upward in the lowest row, downward from row `top` on)."""
        n = a.shape[0] - 1
        dz = self.dz[:n + 1, None]
        cen = flux * (a[:-1] * dz[1:] + a[1:] * dz[:-1]) / (dz[:-1] + dz[1:])
        up, dn = cen.copy(), cen.copy()
        up[1:] = flux[1:] * (-a[:-2] + 5.0 * a[1:-1] + 2.0 * a[2:]) / 6.0
        dn[:-1] = flux[:-1] * (-a[2:] + 5.0 * a[1:-1] + 2.0 * a[:-2]) / 6.0
        k = np.arange(n)[:, None]
        pos = (flux if pos is None else pos) > self.EPS
        neg = (flux if neg is None else neg) < -self.EPS
        return np.where(pos & (k > 0), up, np.where(neg & (k < top), dn, cen))

    def tendencies(self, s, ph):
        rho, ru, rw, rt, pres, th = s
        sh, dx, nz = self.sh, self.dx, self.nz
        ke = nz - 1
        dz, z, zero = self.dz[:, None], self.z[:, None], np.zeros((1, self.nx))
        nu, eps = float(self.p.nu), self.EPS
        uf = ru * 2.0 / (rho + sh(rho, 1))
        half = lambda a, d: (a[:-1] * d[1:] + a[1:] * d[:-1]) / (d[:-1] + d[1:])  # noqa: E731
        wf = np.zeros_like(rw)
        wf[:-1] = rw[:-1] / half(rho, dz)
        R_rho = -((ru - sh(ru, -1)) / dx + np.diff(np.vstack([zero, rw[:-1], zero]), axis=0) / dz) + ph[0]
        # rho u at i + 1/2: fluxes at the cell centres i + 1 and at the corners
        fx = self.faces_x(0.5 * (ru + sh(ru, 1)), uf)
        fz = self.faces_z((0.5 * (rw + sh(rw, 1)))[:-1], uf, ke - 1)
        adv = -(fx - sh(fx, -1)) / dx - np.diff(np.vstack([zero, fz, zero]), axis=0) / dz
        uxx = ((sh(uf, 1) - uf) / dx * sh(rho, 1) - (uf - sh(uf, -1)) / dx * rho) / dx
        rc = 0.25 * (rho[:-1] + rho[1:] + sh(rho, 1)[:-1] + sh(rho, 1)[1:])
        g = np.diff(uf, axis=0) / np.diff(z, axis=0) * rc
        uzz = np.diff(np.vstack([zero, g, zero]), axis=0) / dz
        R_ru = adv - (sh(pres, 1) - pres) / dx + nu * (uxx + uzz) + ph[1]
        # rho w at k + 1/2, k < ke
        w, zd = wf[:-1], np.diff(z, axis=0)
        r_ip = half(ru, z)                      # z weights at i + 1/2, dz weights at i - 1/2
        r_im = sh(half(ru, dz), -1)

        def xface(f, m1, c, p1, p2):
            return np.where(f > eps, f * (-m1 + 5.0 * c + 2.0 * p1) / 6.0,
                            np.where(f < -eps, f * (-p2 + 5.0 * p1 + 2.0 * c) / 6.0, f * (c + p1) * 0.5))

        f_ip = xface(r_ip, sh(w, -1), w, sh(w, 1), sh(w, 2))
        f_im = xface(r_im, sh(w, -2), sh(w, -1), w, sh(w, 1))
        fz = self.faces_z(half(rw, dz)[:ke - 1], w, ke - 2)   # at k + 1 between w faces k and k + 1
        adv = -(f_ip - f_im) / dx - np.diff(np.vstack([zero, fz, zero]), axis=0) / zd
        wxx = ((sh(w, 1) - w) / dx * rc - (w - sh(w, -1)) / dx * sh(rc, -1)) / dx
        g = np.vstack([zero, np.diff(w, axis=0) / dz[1:-1] * rho[1:-1], zero])
        wzz = np.diff(g, axis=0) / zd
        H, zs = float(self.p.H), float(self.p.zf_sponge)
        zf = self.zf[:-1, None]
        sig = np.where(zf > (1.0 - zs) * H, (self.GRAV / 30.0) * ((zf - (1.0 - zs) * H) / (zs * H)), 0.0)
        R_rw = (adv - np.diff(pres, axis=0) / zd - self.GRAV * (rho[:-1] + rho[1:]) * 0.5 + nu * (wxx + wzz)
                - sig * rw[:-1])
        fx = self.faces_x(ru, th)
        fz = self.faces_z(rw[:-1], th, ke - 1)
        R_rt = -((fx - sh(fx, -1)) / dx + np.diff(np.vstack([zero, fz, zero]), axis=0) / dz) + ph[2]
        return R_rho, R_ru, R_rw, R_rt

    def tracers(self, qs, q0, dph, rho, mfx, mfz, dt):
        """The in-place sweep: cells of one anti-diagonal together, from the lower left."""
        nx, nz = self.nx, self.nz
        ke, eps = nz - 1, self.EPS
        kap, dx = float(self.p.kappa), self.dx
        q = np.stack(qs)
        s0 = q / rho
        lin = q[:, :, nx - 2]
        dz, z = self.dz, self.z
        up = lambda a, n: np.concatenate([a[..., n:, :], np.zeros(a.shape[:-2] + (n, nx))], axis=-2)  # noqa: E731
        rface = np.zeros((nz + 1, nx))            # density at k - 1/2
        rface[1:nz] = (rho[:-1] * dz[1:, None] + rho[1:] * dz[:-1, None]) / (dz[:-1] + dz[1:])[:, None]
        zd = np.ones(nz + 1)
        zd[1:nz] = np.diff(z)
        mz = np.zeros((nz + 1, nx))               # vertical flux at k - 1/2
        mz[1:nz] = mfz[:-1]
        sc1, sk1 = self.sh(s0, 1), up(s0, 1)
        old_x = (self.sh(rho, 1) + rho) * 0.5 * (sc1 - s0) / dx
        rx = (rho + self.sh(rho, -1)) * 0.5
        old_z = rface[1:] * (sk1 - s0) / zd[1:, None]
        old_z[:, ke] = 0.0
        col = {"c": s0, "x1": sc1, "x2": self.sh(s0, 2), "z1": sk1, "z2": up(s0, 2), "ox": old_x, "oz": old_z,
               "q0": np.stack(q0), "dp": np.stack(dph)}
        one = {"m": mfx, "mm": self.sh(mfx, -1), "wp": mz[1:], "wm": mz[:-1], "rx": rx, "rz": rface[:-1], "r": rho}
        K = np.arange(nz)
        new_q = np.empty_like(q)
        p1, p2 = s0[:, :, nx - 1].copy(), s0[:, :, nx - 2].copy()

        def koren(num, den):
            r = np.where(np.abs(den) < eps, 1.0, num / den)
            return np.maximum(0.0, np.minimum(2.0 * r, np.minimum((1.0 + 2.0 * r) / 3.0, 2.0)))

        def flux_x(v, m1, c, q1, q2):
            pos = v > eps
            num, den = np.where(pos, q1 - c, c - q1), np.where(pos, c - m1, q1 - q2)
            lim = np.where(pos, c, q1) + 0.5 * koren(num, den) * den
            return np.where(np.abs(v) > eps, lim, 0.5 * (c + q1)) * v

        def flux_z(v, m1, c, q1, q2, k):          # face k + 1/2
            pos, neg = v > eps, v < -eps
            kp = np.minimum(k + 1, ke)
            a, b = dz[np.maximum(k, 0)], dz[kp]
            f2 = (c * b + q1 * a) / (a + b)
            cl = np.minimum(f2, np.where(pos, lin[:, np.maximum(k, 0)], lin[:, kp]) / (np.abs(v) * self.dt))
            num, den = np.where(pos, q1 - c, c - q1), np.where(pos, c - m1, q1 - q2)
            hf = 0.5 * koren(num, den) * den
            face = np.where(pos, np.where(k == 0, cl, c + hf), np.where(neg, np.where(k == nz - 2, cl, q1 - hf), f2))
            return face * v

        for step in range(nx + nz - 1):
            lo, hi = max(0, step - nx + 1), min(nz, step + 1)
            k = K[lo:hi]
            i = step - k
            g = {n: a[:, k, i] for n, a in col.items()}
            o = {n: a[k, i] for n, a in one.items()}
            z0 = np.zeros((3, hi - lo))
            km1, km2 = z0.copy(), z0.copy()
            for n, to, of in ((1, km1, p1), (2, km2, p2)):  # rows k - 1 and k - 2 at this column
                a = max(lo, n)
                if hi > a:
                    to[:, a - lo:] = of[:, a - n:hi - n]
            x1, x2 = p1[:, lo:hi].copy(), p2[:, lo:hi].copy()
            fip = flux_x(o["m"], x1, g["c"], g["x1"], g["x2"])
            fim = flux_x(o["mm"], x2, x1, g["c"], g["x1"])
            fkp = np.where(k == ke, 0.0, flux_z(o["wp"], km1, g["c"], g["z1"], g["z2"], k))
            fkm = np.where(k == 0, 0.0, flux_z(o["wm"], km2, km1, g["c"], g["z1"], k - 1))
            adv = -((fip - fim) / dx + (fkp - fkm) / dz[k])
            dif = kap * (g["ox"] - o["rx"] * (g["c"] - x1) / dx) / dx
            dif = dif + kap * (g["oz"] - np.where(k == 0, 0.0, o["rz"] * (g["c"] - km1) / zd[k])) / dz[k]
            v = g["q0"] + dt * (adv + dif + g["dp"])
            new_q[:, k, i] = v
            p2[:, lo:hi] = x1
            p1[:, lo:hi] = v / o["r"]
            p2[:, :lo] = p1[:, :lo]               # finished rows: their last column is what row k + 2 reads next
        return list(new_q)

    def stage(self, s, s0, ph, dt, m):
        sh, dx, dz, z = self.sh, self.dx, self.dz[:, None], self.z[:, None]
        nz, ke = self.nz, self.nz - 1
        n = ke
        rho, ru, rw, rt, rqv, rqc, rqr = s
        self.ru_left, self.rho_right = float(ru[0, -1]), float(rho[0, 0])
        _, r, cp = self.gas(rqv / rho, rqc / rho, rqr / rho)
        pres = self.P0 * (r * rt / self.P0) ** (cp / (cp - r))
        th, r2 = rt / rho, cp / (cp - r) * pres / rt
        R_rho, R_ru, R_rw, R_rt = self.tendencies((rho, ru, rw, rt, pres, th), ph)
        rp, up, wp, tp = s0[0] - rho, s0[1] - ru, s0[2] - rw, s0[3] - rt
        mfx, mfz = ru.copy(), rw.copy()
        ds = dt / m
        beta, gd = float(self.p.beta_offcenter), float(self.p.gamma_d)
        ftp, ftm = 0.5 * (1.0 + beta), 0.5 * (1.0 - beta)
        d2, fact = (ds * ftp) ** 2, ftm / ftp
        thh = (th[:-1] * dz[1:] + th[1:] * dz[:-1]) / (dz[:-1] + dz[1:])
        zd, gz = np.diff(z, axis=0), self.GRAV / (dz[:-1] + dz[1:])
        b = d2 * (r2[:-1] / dz[:-1] + r2[1:] / dz[1:]) * thh / zd
        a, c = np.zeros_like(b), np.zeros_like(b)
        a[1:] = -d2 * (r2[1:-1] * thh[:-1] / (zd[1:] * dz[1:-1]) - gz[1:])
        c[:-1] = -d2 * (r2[1:-1] * thh[1:] / (zd[:-1] * dz[1:-1]) + gz[:-1])
        old = tp
        zero = np.zeros((1, self.nx))
        for _ in range(m):
            gx, go = (sh(tp, 1) - tp) / dx, (sh(old, 1) - old) / dx
            old = tp
            up = up + ds * (R_ru - (r2 + sh(r2, 1)) * 0.5 * (gx + gd * (gx - go)))
            mfx = mfx + up / m
            inc = ds * (R_rho - (up - sh(up, -1)) / dx)
            rtp = rp + ftp * inc
            rp = rp + inc
            f = (sh(th, 1) + th) * 0.5 * up
            inc = ds * (R_rt - (f - sh(f, -1)) / dx)
            ttp = tp + ftp * inc
            tp = tp + inc
            w = wp[:-1]
            d = w + ds * (R_rw - (r2[:-1] + r2[1:]) * 0.5 * np.diff(ttp, axis=0) / zd
                          - self.GRAV * 0.5 * (rtp[1:] + rtp[:-1]))
            d = d - a * fact * w - b * fact * w
            d[:-1] -= c[:-1] * fact * w[1:]
            x = _thomas(a, b + 1.0, c, d)
            wp = np.vstack([x, wp[-1:]])
            rp = rp - ds * np.diff(np.vstack([zero, x, zero]), axis=0) / dz
            # the upper face of a cell selects upward on the new w and downward on the stage's,
            # its lower face selects on the stage's alone, as the model is written
            hi = self.faces_z(x, th, ke - 1, pos=x, neg=rw[:-1])
            lo = self.faces_z(x, th, ke - 1, pos=rw[:-1], neg=rw[:-1])
            tp = tp - ds * (np.vstack([hi, zero]) - np.vstack([zero, lo])) / dz
            mfz = np.vstack([mfz[:-1] + x / m, mfz[-1:]])
        qs = self.tracers(s[4:], s0[4:], ph[3:], rho, mfx, mfz, dt)
        out = [rho + rp, ru + up, np.vstack([rw[:-1] + wp[:-1], rw[-1:]]), rt + tp]
        return out + qs

    def step(self):
        ph, d_prec = self.physics()
        s0, ns, dt = self.q, self.p.ns, self.dt
        s = self.stage(s0, s0, ph, dt / 3.0, max(1, -(-ns // 3)))
        s = self.stage(s, s0, ph, dt / 2.0, max(1, -(-ns // 2)))
        self.q = self.stage(s, s0, ph, dt, ns)
        self.prec = self.prec + d_prec * dt


def _thomas(a, b, c, d):
    n = b.shape[0]
    cp, dp, x = np.empty_like(b), np.empty_like(b), np.empty_like(b)
    cp[0], dp[0] = c[0] / b[0], d[0] / b[0]
    for j in range(1, n):
        piv = b[j] - a[j] * cp[j - 1]
        cp[j], dp[j] = c[j] / piv, (d[j] - a[j] * dp[j - 1]) / piv
    x[n - 1] = dp[n - 1]
    for j in range(n - 2, -1, -1):
        x[j] = dp[j] - cp[j] * x[j + 1]
    return x


def _exact_steps(p, s, steps):
    with np.errstate(all="ignore"):
        m = _Step64(p, s)
        for _ in range(steps):
            m.step()
    out = {}
    for f, a in zip(FIELDS, m.q):
        v = np.zeros((p.ka, p.ia), order="F")
        v[:, p.halo:p.halo + p.Nx] = a
        exchange_halo(v, p)
        out[f] = v
    out["prec"] = np.array(s.prec, dtype=np.float64)
    out["prec"][p.halo:p.halo + p.Nx] = m.prec
    return out


def _exact_columns(case, seed):
    p, (w, dw, th, r2) = _column_inputs(case, seed)
    w, dw, th, r2 = (a.astype(np.float64).T for a in (w, dw, th, r2))
    dz, z = p.dz.astype(np.float64)[:, None], p.z.astype(np.float64)[:, None]
    beta, grav = float(p.beta_offcenter), float(p.c.GRAV)
    ftp, ftm = 0.5 * (1.0 + beta), 0.5 * (1.0 - beta)
    d2, fact = (0.25 * ftp) ** 2, ftm / ftp
    thh = (th[:-1] * dz[1:] + th[1:] * dz[:-1]) / (dz[:-1] + dz[1:])
    zd, gz = np.diff(z, axis=0), grav / (dz[:-1] + dz[1:])
    b = d2 * (r2[:-1] / dz[:-1] + r2[1:] / dz[1:]) * thh / zd
    a, c = np.zeros_like(b), np.zeros_like(b)
    a[1:] = -d2 * (r2[1:-1] * thh[:-1] / (zd[1:] * dz[1:-1]) - gz[1:])
    c[:-1] = -d2 * (r2[1:-1] * thh[1:] / (zd[:-1] * dz[1:-1]) + gz[:-1])
    d = w[:-1] + dw[:-1] - a * fact * w[:-1] - b * fact * w[:-1]
    d[:-1] -= c[:-1] * fact * w[1:-1]
    return np.ascontiguousarray(np.vstack([_thomas(a, b + 1.0, c, d), w[-1:]]).T)


def exact(case, seed):
    """What run() returns, in 64 bits with numpy; None for ensembles and gradients, and where it
    would take too long (the anti-diagonals of the sweep, and the cells)."""
    if case["kind"] == "columns":
        return _exact_columns(case, seed)
    if case["kind"] not in ("steps", "oneshot"):
        return None
    cells, diag = case["nx"] * case["nz"], case["nx"] + case["nz"]
    if case["steps"] * (1e-3 * diag + 4e-6 * cells) > 17.0:
        return None
    if case["kind"] == "oneshot":
        p, s = _initial(case, seed)
    else:
        p, s, m = _spun_up(case, seed)
        m.close()
    return _exact_steps(p, s, case["steps"])
