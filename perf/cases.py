"""Workloads of the dynamical core, through the entry points a program calls.

listed() and draw() give the cases, prepare() builds what a program holds before the call (a Dycore handle with
its state uploaded, a projected source), run() makes one pass, work() states what a pass cannot do without, and
exact() restates the pass in plain FP64 torch (none of this repository's kernels) for the same inputs.

Kinds of case:
  iterate     atsat_dyn_iterate: two resident iterations (pressure call on the even one, RK4 step, boundary
              conditions, restoreVar); `glue` adds the driver's filter, species floor and turbulence closure
  replay      the same two iterations as a replay of the captured CUDA graph, as a long resident run does
  step        one drop-in step on host arrays: upload, density, pressure call, RK4 step, download
  pressure    one pressure call with the radial line pass and the barotropic correction switched on
  turbulence  one run of the closure (k-omega SST)
  poisson     one standalone solve of the pressure equation: `refine` to a relative residual of 1e-10 by FP64
              defect correction around FP32 direct solves, or the FP64 direct solve

Inputs are the seeded jet state of atsat_gb300/synth.py with every source term non-zero, drawn on the GPU.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from atsat_gb300 import abi, dyn, fields as F, synth

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
PROJECTION = [F.RHS_U, F.RHS_V, F.RHS_W, F.AUX_U, F.AUX_V, F.AUX_W]
CLOSURE = [F.NUE, F.TKE_SOURCE, F.DIS_SOURCE]
SPECIES = list(range(F.H2O, F.NH4SH + 1))


# ---- the cases ----

def listed():
    def c(name, kind, im, jm, km, **kw):
        return dict({"name": name, "kind": kind, "im": im, "jm": jm, "km": km}, **kw)

    return [
        # the default 1-degree shell in mixed precision, a long resident run: graph replays
        c("mixed_41x181x361_replay", "replay", 41, 181, 361, precision="mixed", glue=False),
        # the half-degree shell (21 M cells), the largest grid the model is run on
        c("mixed_81x361x721_replay", "replay", 81, 361, 721, precision="mixed", glue=False),
        # a coarse 2-degree ensemble member, stepped by plain calls
        c("mixed_21x91x181", "iterate", 21, 91, 181, precision="mixed", glue=False),
        # the smallest calls: a test-sized shell with an odd periodic ring, where launches count
        c("mixed_10x20x36", "iterate", 10, 20, 36, precision="mixed", glue=False),
        # the plain FP64 drop-in on the default shell
        c("fp64_41x181x361", "iterate", 41, 181, 361, precision="fp64", glue=False),
        # FP64 on an odd ring and sizes that fill no tile evenly
        c("fp64_27x118x222", "iterate", 27, 118, 222, precision="fp64", glue=False),
        # the whole driver loop resident: filter, species floor and turbulence closure in every iteration, in FP64
        # (the closure amplifies the mixed path's FP32 rounding of k* beyond any comparison of omega*'s source)
        c("fp64_41x181x361_glue", "iterate", 41, 181, 361, precision="fp64", glue=True),
        # the CPU model calling the library as a drop-in: host arrays in, host arrays out
        c("host_step_21x91x181", "step", 21, 91, 181, precision="mixed"),
        # the pressure call with both of its optional passes
        c("press_line_baro_41x181x361", "pressure", 41, 181, 361, line=True, baro=True),
        # the turbulence closure alone
        c("turbulence_41x181x361", "turbulence", 41, 181, 361),
        # the standalone pressure equation to 1e-10, and its FP64 direct solve on the coarse shell
        c("poisson_refine_41x181x361", "poisson", 41, 181, 361, method="refine"),
        c("poisson_direct_21x91x181", "poisson", 21, 91, 181, method="direct"),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate", "iterate", "iterate", "replay", "replay", "step", "pressure", "turbulence",
                       "poisson", "poisson"])
    if kind == "poisson":                       # the factored solver is held for each grid: up to the default shell
        case = {"kind": kind, "im": _size(rng, 9, 41), "jm": _size(rng, 21, 181), "km": _size(rng, 33, 361),
                "method": rng.choice(["refine", "direct"])}
        return case
    case = {"kind": kind, "im": _size(rng, 9, 61), "jm": _size(rng, 17, 271), "km": _size(rng, 25, 541)}
    if kind in ("iterate", "replay"):
        case["glue"] = kind == "iterate" and rng.random() < 0.25
        case["precision"] = "fp64" if case["glue"] else rng.choice(["mixed", "mixed", "fp64"])
    elif kind == "step":
        case["precision"] = rng.choice(["mixed", "fp64"])
        case["im"], case["jm"], case["km"] = min(case["im"], 41), min(case["jm"], 121), min(case["km"], 241)
    elif kind == "pressure":
        case["line"] = rng.random() < 0.6
        case["baro"] = (not case["line"]) or rng.random() < 0.5
        case["im"], case["jm"], case["km"] = min(case["im"], 41), min(case["jm"], 181), min(case["km"], 361)
    return case


def _params(case):
    p = abi.default_params()
    if case["kind"] in ("iterate", "replay"):   # without the host physics the jet state outgrows FP64 after some
        p["dt"] = 0.001                         # hundred steps of 0.01: a tenth of it lasts for thousands of passes
    p["precision"] = 1 if case.get("precision") == "mixed" else 0
    p["driver_glue"] = int(bool(case.get("glue")))
    p["press_line"] = int(bool(case.get("line")))
    p["press_baro"] = int(bool(case.get("baro")))
    return p


# ---- inputs, made on the GPU from the seed alone ----

def _fields(case, seed):
    """field id -> (im, jm, km) FP64 tensor, and the cell-hold tables: the state of synth.saturn_state with its
    `exercise` noise, from torch's generator."""
    g, P = synth.make_grid(case["im"], case["jm"], case["km"]), _params(case)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 17)
    shp = g.shape

    def nz(s):
        return torch.randn(shp, generator=gen, dtype=torch.float64, device=DEV) * s

    def un():
        return torch.rand(shp, generator=gen, dtype=torch.float64, device=DEV)

    u_0, t_ref = P["u_0"], P["t_ref"]
    the = torch.tensor(g.the_z, device=DEV)[None, :, None]
    lat = 90.0 - the * (180.0 / math.pi)
    z = (torch.arange(g.im, dtype=torch.float64, device=DEV) * (g.L_atm * g.dr))[:, None, None]
    a = {}
    a[F.W] = ((400.0 * torch.exp(-(lat / 15.0) ** 2) + 60.0 * torch.cos(6.0 * lat * (math.pi / 180.0))) / u_0
              ).expand(shp).clone()
    a[F.V] = nz(0.5 / u_0)
    a[F.U] = nz(0.01 / u_0)
    T = torch.clamp(134.0 - 0.7 * z + 10.0 * (1.0 - (2.0 * the / math.pi - 1.0) ** 2) + nz(0.1), min=0.4064 * t_ref)
    a[F.T] = T / t_ref
    ps = torch.empty(shp, dtype=torch.float64, device=DEV)
    ps[0] = a[F.T][0] ** (P["g"] / (0.7 * 3.89))
    for i in range(1, g.im):
        ps[i] = ps[i - 1] * torch.exp(-P["g"] * g.L_atm * g.dr * 1.0e3 / (P["R_mix"] * 0.5 * (T[i - 1] + T[i])))
    a[F.P_STAT] = ps
    rho = ps * 1.0e5 / (P["R_mix"] * T)
    a[F.RHO_MIX] = rho
    decay = torch.exp(-z / 100.0)
    a[F.H2O] = 1.0e-3 * (0.5 + 0.5 * un()) * decay * rho
    a[F.NH3] = 1.0e-4 * (0.5 + 0.5 * un()) * decay * rho
    for f in (F.H2O_CLOUD, F.H2O_ICE, F.NH3_CLOUD, F.NH3_ICE, F.CH4_CLOUD, F.CH4_ICE):
        a[f] = nz(1.0e-6).abs() * decay
    a[F.H2S] = nz(1.0e-5).abs() * decay * rho
    a[F.CH4] = nz(1.0e-4).abs() * rho
    a[F.NH4SH] = nz(1.0e-6).abs()
    a[F.TKE] = (1.0e-3 / (u_0 * u_0)) * (1.0 + nz(0.1))
    a[F.DIS] = (1.0e-4 * (g.L_atm * 1.0e3) / u_0) * (1.0 + nz(0.1))
    a[F.P_DYN] = nz(1.0e-3)
    a[F.NUE] = nz(1.0e-5)
    for f in (F.Q_PRECIP, F.Q_RAD):
        a[f] = nz(1.0e-2)
    for f in [F.TKE_SOURCE, F.DIS_SOURCE] + F.S_PRECIP_FIELDS + [F.MASSFLUX_H2S, F.MASSFLUX_NH3, F.MASSFLUX_NH4SH,
                                                               F.FLUXLIM_NH4SH, F.THERMALMASSFLUX]:
        a[f] = nz(1.0e-6)
    for f in PROJECTION:                        # the tendencies a previous step left for the projection
        a[f] = nz(1.0e-3)
    hold = [a[f][:, :, :-1].mean(dim=2) for f in (F.V, F.U)]
    return g, P, a, hold


def _source(case, seed):
    """The standalone equation's source: N(0, 1), 3-point box filter in theta and phi, zero interior mean."""
    g = synth.make_grid(case["im"], case["jm"], case["km"])
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 29)
    s = torch.randn(g.shape, generator=gen, dtype=torch.float64, device=DEV)
    s[:, 1:-1] = (s[:, :-2] + s[:, 1:-1] + s[:, 2:]) / 3.0
    r = s[1:-1, 1:-1, :-1]
    r = (torch.roll(r, 1, 2) + r + torch.roll(r, -1, 2)) / 3.0
    out = torch.zeros_like(s)
    out[1:-1, 1:-1, :-1] = r - r.mean()
    return g, out


class _Device:
    """A device field as torch sees it: no copy, the row pitch in the strides. It keeps the handle, which owns the
    memory, as long as the tensor lives."""

    def __init__(self, owner, ptr, shape, pitch):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": (shape[1] * pitch * 8, pitch * 8, 8)}


def _views(d, fids):
    out = {}
    for f in fids:
        ptr, pitch = C.POINTER(C.c_double)(), C.c_int64()
        rc = dyn.lib().atsat_dyn_device_field(d.h, f, C.byref(ptr), C.byref(pitch))
        assert rc == 0
        out[F.NAMES[f]] = torch.as_tensor(_Device(d, C.cast(ptr, C.c_void_p).value, d.grid.shape, pitch.value),
                                          device="cuda")
    return out


def _pinned(x):
    h = torch.empty(x.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(x)
    return h


def prepare(case, seed):
    if case["kind"] == "poisson":
        g, src = _source(case, seed)
        d = dyn.Dycore(g, abi.default_params())
        return {"kind": "poisson", "d": d, "src": d.poisson_project(src.cpu().numpy()),
                "method": {"refine": abi.POISSON_METHODS[5], "direct": abi.POISSON_METHODS[3]}[case["method"]]}
    g, P, a, hold = _fields(case, seed)
    d = dyn.Dycore(g, P)
    st = {"kind": case["kind"], "d": d}
    host = {}
    if case["kind"] == "step":                  # the CPU model's own arrays, page-locked, bound once
        for f in F.STEP_INPUTS + PROJECTION:
            host[f] = _pinned(a[f - F.N_BASE] if F.N_BASE <= f < F.N_BASE + F.NPROG else a[f])
            d.bind(f, host[f].numpy())
        d.upload(list(host))
        st["out"] = {F.NAMES[f]: host[f].numpy() for f in F.STEP_OUTPUTS + [F.P_DYN]}
        d.set_async(True)
    else:
        buf = torch.empty(g.shape, dtype=torch.float64, pin_memory=True)
        for f, x in a.items():
            buf.copy_(x)
            for fid in ([f, F.N_BASE + f] if f < F.NPROG else [f]):
                d.bind(fid, buf.numpy())
                d.upload([fid])
        st["buf"] = buf
    d.set_tables(*[h.cpu().numpy() for h in hold])
    st["host"] = host
    if case["kind"] == "turbulence":
        st["out"] = _views(d, [F.TKE, F.DIS] + CLOSURE)
    elif case["kind"] == "pressure":
        st["out"] = _views(d, [F.P_DYN])
    elif case["kind"] in ("iterate", "replay"):
        st["out"] = _views(d, F.PROG + [F.P_DYN] + PROJECTION + (CLOSURE if case["glue"] else []))
        if case["kind"] == "replay":
            d.iterate(0, 2)
            d.graph_capture(2, 2)
    return st


def run(st):
    d, kind = st["d"], st["kind"]
    if kind == "poisson":
        return d.poisson_solve(st["method"], st["src"], tol=1e-10, max_iter=40)[0]
    if kind == "iterate":
        d.iterate(0, 2)
    elif kind == "replay":
        d.graph_launch(1)
    elif kind == "pressure":
        d.PressureSolver_run(stats=False)
    elif kind == "turbulence":
        d.TurbulenceSat_run()
    else:
        d.upload(F.STEP_INPUTS)
        d.computeMixtureDensity()
        d.PressureSolver_run(stats=False)
        d.RungeKuttaSat()
        d.download([F.P_DYN])
        d.download(F.STEP_OUTPUTS)
        d.sync()
    return st["out"]


def work(case):
    n = case["im"] * case["jm"] * case["km"]
    kind = case["kind"]
    if kind == "poisson":                       # source in, pressure out; the spectral solve's transforms
        ring = case["km"] - 1
        return {"bytes": 16 * n, "flops": n * (2 * 5 * math.log2(ring) + 8 * (case["im"] - 2))}
    if kind == "turbulence":                    # 14 fields in, 5 out
        return {"bytes": 19 * 8 * n, "flops": 250 * n}
    if kind == "pressure":                      # the projection's tendencies and p_dyn in, p_dyn out
        return {"bytes": (3 + 1 + 1) * 8 * n, "flops": (60 + 30 * case["line"] + 20 * case["baro"]) * n}
    # y_n, p_dyn, p_stat, rho_mix and the point inputs in; y_{n+1}, p_dyn and the tendencies out
    io = (F.NPROG + 3 + len(F.POINT_INPUTS) + F.NPROG + 1 + len(PROJECTION)) * 8 * n
    if kind == "step":
        return {"bytes": io + (len(F.STEP_INPUTS) + len(F.STEP_OUTPUTS) + 1) * 8 * n, "flops": 4 * 600 * n}
    glue = 2 if case["glue"] else 0
    return {"bytes": 2 * io + glue * 19 * 8 * n, "flops": (2 * 4 * 600 + glue * 250) * n}


# ---- exact(): the same pass in plain FP64 torch ----
# Arrays are (im, jm, km); formulas follow the reference's sources named in include/atsat_dyn.h.

C43, C13 = 4.0 / 3.0, 1.0 / 3.0


class _Model:
    def __init__(self, g, P, a, hold):
        self.g, self.P, self.a = g, P, a
        self.nl = {q: a[q].clone() for q in F.PROG}
        self.hold = hold
        t = lambda x: torch.tensor(x, dtype=torch.float64, device=DEV)  # noqa: E731
        self.rm = t(g.rad_z) + (P["metric_radius_km"] / P["L_atm"] - 1.0)
        self.the = t(g.the_z)
        self.sin, self.cos = torch.sin(self.the), torch.cos(self.the)
        sp = self.sin.clone()
        sp[sp == 0.0] = 1.0e-5
        self.sinp = sp
        self.i2 = (1.0 / (2.0 * g.dr), 1.0 / (2.0 * g.dthe), 1.0 / (2.0 * g.dphi))
        self.id2 = (1.0 / g.dr ** 2, 1.0 / g.dthe ** 2, 1.0 / g.dphi ** 2)

    # computeMixtureDensity, computeBuoyancyRefLevel, computeMetricPressure
    def density(self):
        self.a[F.RHO_MIX] = self.a[F.P_STAT] * 1.0e5 / (self.P["R_mix"] * (self.a[F.T] * self.P["t_ref"]))

    def level_and_metric(self):
        P, a, g = self.P, self.a, self.g
        b = P["g"] * a[F.P_STAT] / (P["r_mix"] * P["R_mix"] * a[F.T] * P["t_ref"])
        w = self.sin[None, :, None]
        self.buoy = (b * w).sum(dim=(1, 2)) / (self.sin.sum() * g.km)
        cor = P["Coriolis"] * (P["L_atm"] * 1.0e3 / P["u_0"]) * 2.0 * P["omega"] * self.sin.abs()
        f = (a[F.V] ** 2 + a[F.W] ** 2) / self.rm[:, None, None] + cor[None, :, None] * a[F.W]
        pm = torch.zeros_like(f)
        pm[1:] = torch.cumsum(0.5 * g.dr * (f[:-1] + f[1:]), dim=0)
        self.pm = pm

    def _d(self, f):
        """First and second differences on the RK interior (j = 2..jm-3, ring k = 0..km-2), unscaled."""
        f = f[:, :, :-1]
        c = f[1:-1, 2:-2]
        rp, rn, tp, tn = f[2:, 2:-2], f[:-2, 2:-2], f[1:-1, 3:-1], f[1:-1, 1:-3]
        e, w = torch.roll(c, -1, 2), torch.roll(c, 1, 2)
        (ir, it, ip), (ir2, it2, ip2) = self.i2, self.id2
        return ((rp - rn) * ir, (rp - 2.0 * c + rn) * ir2, (tp - tn) * it, (tp - 2.0 * c + tn) * it2,
                (e - w) * ip, (e - 2.0 * c + w) * ip2)

    # RHSSat on the RK interior with the default knobs
    def rhs(self, y):
        P, a = self.P, self.a
        I = (slice(1, -1), slice(2, -2), slice(0, -1))  # noqa: E741
        rm = self.rm[1:-1, None, None]
        st, ct = self.sin[None, 2:-2, None], self.cos[None, 2:-2, None]
        cot = ct / st
        irm, irm2, irs = 1.0 / rm, 1.0 / (rm * rm), 1.0 / (rm * st)
        irm2s, irm2s2 = irm2 / st, irm2 / (st * st)
        u, v, w, t = (y[q][I] for q in (F.U, F.V, F.W, F.T))
        du, dv, dw = (self._d(y[q]) for q in (F.U, F.V, F.W))
        dp, dpm, dps = self._d(a[F.P_DYN]), self._d(self.pm), self._d(a[F.P_STAT])

        def adv(d):
            return u * d[0] + v * d[2] * irm + w * d[4] * irs

        def dif(d):
            return d[1] + d[0] * 2.0 * irm + d[3] * irm2 + d[2] * ct * irm2s + d[5] * irm2s2

        nd = P["L_atm"] * 1.0e3 / P["u_0"]
        nue = a[F.NUE][I]
        nut = P["turb_coupling"] * torch.clamp(nue, min=0.0)
        nuts = nut / 0.9
        visc = 1.0 / P["re"] + nut
        r, strue = {}, torch.sqrt(torch.clamp(1.0 - ct * ct, min=0.0))
        vb, ub = (h[1:-1, 2:-2, None] for h in self.hold)
        buoy = -P["buoy_scale"] * P["buoyancy"] * (
            P["g"] * a[F.P_STAT][I] / (P["r_mix"] * P["R_mix"] * t * P["t_ref"]) - self.buoy[1:-1, None, None])
        vm = (1.0 + ct / (st * st)) * irm2
        om = P["omega"]
        cent = om * om * rm * strue * P["centrifugal"]
        r[F.U] = (-dp[0] + buoy - adv(du) + (dif(du) + du[0] * 2.0 * irm + 2.0 * u * irm2) * visc + cent * strue)
        r[F.V] = (-(dp[2] + dpm[2]) * irm - adv(dv) - (u * v - w * w * cot) * irm
                  + (dif(dv) - vm * v + 2.0 * du[2] * irm2 - 2.0 * dw[4] * ct * irm2s2) * visc
                  + nd * 2.0 * om * ct * w * P["Coriolis"] + cent * ct)
        r[F.W] = (-(dp[4] + dpm[4]) * irs - adv(dw) - (w * u + v * w * cot) * irm
                  + (dif(dw) - vm * w + 2.0 * du[4] * irm2s + 2.0 * dv[4] * ct * irm2s2) * visc
                  - nd * 2.0 * om * (ct * (v - vb) + strue * (u - ub)) * P["Coriolis"])
        dps_r = dps[0] / (P["r_mix"] * P["u_0"] ** 2 * 1.0e-5) * (P["r_mix"] / a[F.RHO_MIX][I])
        ce = P["u_0"] ** 2 / (P["cp_mix"] * P["t_ref"])
        pre = P["precip_coupling"] * a[F.Q_PRECIP][I] * P["L_atm"] * 1.0e3 / (
            P["r_mix"] * P["cp_mix"] * P["u_0"] * P["t_ref"])
        dt = self._d(y[F.T])
        r[F.T] = (ce * (u * (dp[0] + dps_r) + v * dp[2] * irm + w * dp[4] * irs) - adv(dt)
                  + dif(dt) * (1.0 / (P["re"] * P["pr"]) + nuts) + torch.clamp(pre, -0.5, 0.5))
        pc, ch = P["precip_coupling"], P["chemical_reaction"]
        for q in SPECIES:
            d = self._d(y[q])
            n = F.NAMES[q].split("_")[0]
            r[q] = -adv(d) + dif(d) * (1.0 / (P["sc_" + n] * P["re"]) + nuts)
        for s, q in enumerate((F.H2O, F.H2O_CLOUD, F.H2O_ICE, F.NH3, F.NH3_CLOUD, F.NH3_ICE, F.CH4, F.CH4_CLOUD,
                               F.CH4_ICE)):
            r[q] = r[q] + pc * a[F.S_PRECIP_H2O + s][I]
        r[F.H2S] = r[F.H2S] + ch * a[F.MASSFLUX_H2S][I]
        r[F.NH3] = r[F.NH3] + ch * a[F.MASSFLUX_NH3][I]
        r[F.NH4SH] = r[F.NH4SH] + a[F.FLUXLIM_NH4SH][I] + ch * a[F.MASSFLUX_NH4SH][I]
        for q, sig, s in ((F.TKE, 0.85, F.TKE_SOURCE), (F.DIS, 0.5, F.DIS_SOURCE)):
            d = self._d(y[q])
            r[q] = -adv(d) + dif(d) * (1.0 / P["re"] + nue / sig) + a[s][I]
        self.grad_p = (dp[0], dp[2] * irm, dp[4] * irs)
        return r

    def rk4(self):
        P, a, I = self.P, self.a, (slice(1, -1), slice(2, -2), slice(0, -1))  # noqa: E741
        self.level_and_metric()
        y = {q: a[q].clone() for q in F.PROG}
        acc = {}

        def bounded(q, x):
            if q == F.TKE:
                return torch.clamp(x, 0.0, 1000.0 / P["u_0"] ** 2)
            return torch.clamp(x, min=1.0e-10) if q == F.DIS else x

        for c, wgt in ((0.5, 1.0), (0.5, 2.0), (1.0, 2.0), (0.0, 1.0)):
            r = self.rhs(y)
            for q in F.PROG:
                acc[q] = wgt * r[q] + (acc[q] if q in acc else 0.0)
                if c:
                    y[q][I] = bounded(q, self.nl[q][I] + c * P["dt"] * r[q])
        for q in F.PROG:
            a[q] = y[q]
            a[q][I] = bounded(q, self.nl[q][I] + P["dt"] / 6.0 * acc[q])
        for n, q in enumerate((F.U, F.V, F.W)):
            a[F.RHS_U + n][I] = r[q]
            a[F.AUX_U + n][I] = r[q] + self.grad_p[n]

    # PressureSolver::run with prepareProjectionBoundaries (increment form, one sweep)
    def pressure(self):
        P, a, g = self.P, self.a, self.g
        K = slice(0, -1)
        for f in PROJECTION:
            x, lid = a[f], f == F.AUX_U
            J = slice(1, -1)
            x[0, J, K] = 0.0 if lid else x[3, J, K] - 3.0 * x[2, J, K] + 3.0 * x[1, J, K]
            x[-1, J, K] = 0.0 if lid else x[-4, J, K] - 3.0 * x[-3, J, K] + 3.0 * x[-2, J, K]
            radial = f in (F.AUX_U, F.RHS_U)
            i = slice(1, -1)
            x[i, 0, K] = x[i, 3, K] - 3.0 * x[i, 2, K] + 3.0 * x[i, 1, K] if radial else 0.0
            x[i, -1, K] = x[i, -4, K] - 3.0 * x[i, -3, K] + 3.0 * x[i, -2, K] if radial else 0.0
            x[:, :, -1] = x[:, :, 0]
        p, n = a[F.P_DYN], g.km - 1
        rm = self.rm[1:-1, None, None]
        s = self.sinp[None, 1:-1, None]
        n1 = torch.full_like(rm, self.id2[0])
        n2, n3 = self.id2[1] / (rm * rm), self.id2[2] / (rm * rm * s * s)
        den = 2.0 * (n1 + n2 + n3)

        def parts():
            c = p[1:-1, 1:-1, :n]
            return (c, n1 * (p[2:, 1:-1, :n] + p[:-2, 1:-1, :n]) + n2 * (p[1:-1, 2:, :n] + p[1:-1, :-2, :n]),
                    n3 * (torch.roll(c, -1, 2) + torch.roll(c, 1, 2)))

        c, h, k3 = parts()
        lc = h + k3 - den * c
        su = a[F.RHS_U][:, 1:-1, :n].clone()
        su[0], su[-1] = 0.0, 0.0
        sv, sw = a[F.RHS_V][1:-1, :, :n], a[F.RHS_W][1:-1, 1:-1, :n]
        div = ((su[2:] - su[:-2]) * self.i2[0] + (sv[:, 2:] - sv[:, :-2]) * self.i2[1] / rm
               + (torch.roll(sw, -1, 2) - torch.roll(sw, 1, 2)) * self.i2[2] / (rm * s))
        cap = den * P["pdyn_cap"]
        src = torch.minimum(torch.maximum(div, -cap), cap) + lc
        ijk = sum(torch.meshgrid(*[torch.arange(1, m - 1, device=DEV) for m in (g.im, g.jm)],
                                 torch.arange(n, device=DEV), indexing="ij"))
        jk = ijk[0] - 1
        partner = torch.zeros(n, dtype=torch.bool, device=DEV)
        partner[-1] = n % 2 == 1                # visited after k = 0, whose colour it shares
        mean0 = p[1:-1, 1:-1, :n].mean()
        for colour in (0, 1):
            for late in (False, True):
                mask = ((ijk & 1) == colour) & (partner == late)
                c, h, k3 = parts()
                p[1:-1, 1:-1, :n] = torch.where(mask, (h + k3 - src) / den, c)
        if P["press_line"]:
            self._line(src, n1, n2, n3, jk, partner)
        if P["press_baro"]:
            self._baro(src, n1, n2, n3)
        p[0], p[-1] = C43 * p[1] - C13 * p[2], C43 * p[-2] - C13 * p[-3]
        p[:, 0], p[:, -1] = C43 * p[:, 1] - C13 * p[:, 2], C43 * p[:, -2] - C13 * p[:, -3]
        p[:, :, -1] = p[:, :, 0]
        if P["press_line"]:
            p -= p[1:-1, 1:-1, :n].mean() - mean0

    def _line(self, src, n1, n2, n3, jk, partner):
        p, n = self.a[F.P_DYN], self.g.km - 1
        for colour in (0, 1):
            for late in (False, True):
                c = p[1:-1, 1:-1, :n]
                d = (n2 * (p[1:-1, 2:, :n] + p[1:-1, :-2, :n]) + n3 * (torch.roll(c, -1, 2) + torch.roll(c, 1, 2)) - src)
                b = (2.0 * (n1 + n2 + n3)).expand_as(src).clone()
                lo, up = (-n1).expand_as(src).clone(), (-n1).expand_as(src).clone()
                b[0] += lo[0] * C43
                up[0] -= lo[0] * C13
                b[-1] += up[-1] * C43
                lo[-1] -= up[-1] * C13
                x = _thomas(lo, b, up, d)
                mask = ((jk & 1) == colour) & (partner == late)
                p[1:-1, 1:-1, :n] = torch.where(mask, x, c)

    def _baro(self, src, n1, n2, n3):
        p, n, g = self.a[F.P_DYN], self.g.km - 1, self.g
        q = p[:, :, :n].clone()
        q[0], q[-1] = C43 * q[1] - C13 * q[2], C43 * q[-2] - C13 * q[-3]
        q[:, 0], q[:, -1] = C43 * q[:, 1] - C13 * q[:, 2], C43 * q[:, -2] - C13 * q[:, -3]
        c = q[1:-1, 1:-1]
        lc = (n1 * (q[2:, 1:-1] + q[:-2, 1:-1] - 2.0 * c) + n2 * (q[1:-1, 2:] + q[1:-1, :-2] - 2.0 * c)
              + n3 * (torch.roll(c, -1, 2) + torch.roll(c, 1, 2) - 2.0 * c))
        R = (src - lc).sum(dim=0) / (1.0 / self.rm[1:-1] ** 2).sum()        # (J, n)
        S = torch.fft.rfft(R, dim=1)
        tol = 1.0e-12 * R.abs().sum(dim=1, keepdim=True)
        re, im = S.real.clone(), S.imag.clone()
        re[:, 1:] = torch.where(re[:, 1:].abs() < tol, torch.zeros_like(re[:, 1:]), re[:, 1:])
        im[:, 1:] = torch.where(im[:, 1:].abs() < tol, torch.zeros_like(im[:, 1:]), im[:, 1:])
        ws = self.sin[1:-1].abs()
        yw = torch.ones_like(ws)
        yw[0] = yw[-1] = 1.5
        re[:, 0] -= (yw * re[:, 0]).sum() / (yw * ws).sum() * ws
        e = self.id2[1]
        lam = 4.0 * torch.sin(math.pi * torch.arange(S.shape[1], dtype=torch.float64, device=DEV) / n) ** 2 * self.id2[2]
        b = -2.0 * e - lam[None, :] / self.sinp[1:-1, None] ** 2
        lo, up = torch.full_like(b, e), torch.full_like(b, e)
        b[0] += C43 * e
        up[0] -= C13 * e
        b[-1] += C43 * e
        lo[-1] -= C13 * e
        b[0, 0], up[0, 0], re[0, 0] = 1.0, 0.0, 0.0
        re, im = _thomas(lo, b, up, re), _thomas(lo, b, up, im)
        re[:, 0] -= (ws * re[:, 0]).sum() / ws.sum()
        p[:, 1:-1, :n] += torch.fft.irfft(torch.complex(re, im), n=n, dim=1)[None]

    # BC_Sat's bcTheta, bcPhi, bcRadius on the dycore's fields (default forms)
    def boundaries(self):
        a = self.a
        turb = {F.TKE: 0.0, F.DIS: 1.0e-10, F.NUE: 0.0}
        zero = (F.V, F.W, F.FLUXLIM_NH4SH)
        rest = [F.T, F.U] + SPECIES + [F.MASSFLUX_H2S, F.MASSFLUX_NH3, F.MASSFLUX_NH4SH, F.THERMALMASSFLUX]
        i, K, J = slice(1, -1), slice(0, -1), slice(1, -1)
        for f in list(zero) + rest + list(turb):
            x = a[f]
            for j0, j1, j2 in ((0, 1, 2), (-1, -2, -3)):
                if f in zero:
                    x[i, j1, K] = 0.5 * x[i, j2, K]
                    x[i, j0, K] = 0.0
                elif f in turb:
                    x[i, j1, K] = torch.clamp(x[i, j2, K], min=turb[f])
                    x[i, j0, K] = torch.clamp(C43 * x[i, j1, K] - C13 * x[i, j2, K], min=turb[f])
                else:
                    x[i, j1, K] = x[i, j2, K]
                    x[i, j0, K] = x[i, j1, K]
            if f in turb:
                x[:, :, 0] = torch.clamp(x[:, :, 0], min=turb[f])
            x[:, :, -1] = x[:, :, 0]
            top = C43 * x[-2, J, K] - C13 * x[-3, J, K]
            low = C43 * x[1, J, K] - C13 * x[2, J, K]
            if f in turb:
                top, low = torch.clamp(top, min=turb[f]), torch.clamp(low, min=turb[f])
            elif f != F.U:
                low = x[3, J, K] - 3.0 * x[2, J, K] + 3.0 * x[1, J, K]
            x[0, J, K], x[-1, J, K] = low, top
        a[F.U][0], a[F.U][-1] = 0.0, 0.0
        for f in (F.V, F.W):
            x = a[f]
            x[-1] = 0.0
            x[-2], x[-3] = (1.0 / 3.0) * x[-4], (2.0 / 3.0) * x[-4]
        fr = a[F.RHO_MIX][0] / a[F.RHO_MIX][1]
        for f in SPECIES:
            a[f][-1] = a[f][-2]
            a[f][0] = a[f][1] * fr

    # the driver's glue: damp_wiggles along k and i, clampNegativeSpecies, the k-omega SST closure
    def damp(self):
        p, n = self.a[F.P_DYN], self.g.km - 1
        r = p[:, :, :n]
        p[:, :, :n] = r + 0.25 * (torch.roll(r, 1, 2) - 2.0 * r + torch.roll(r, -1, 2))
        p[:, :, n] = p[:, :, 0]
        e = torch.cat([p[:1], p, p[-1:]])
        self.a[F.P_DYN] = p + 0.25 * (e[:-2] - 2.0 * p + e[2:])

    def turbulence(self):
        P, a, g, n = self.P, self.a, self.g, self.g.km - 1
        I = (slice(1, -1), slice(1, -1), slice(0, n))  # noqa: E741
        h = float(np.float32(P["L_atm"] * g.dr))
        hm = np.array([float(np.float32(np.float32(i) * np.float32(h))) * 1.0e3 for i in range(g.im)])
        L_m, u_0 = P["L_atm"] * 1.0e3, P["u_0"]
        for f, lo in ((F.TKE, 0.0), (F.DIS, 1.0e-10)):
            a[f][I] = torch.clamp(a[f][I], min=lo)
        rm = self.rm[1:-1, None, None]
        s = self.sinp[None, 1:-1, None]
        cot = self.cos[None, 1:-1, None] / s

        def grad(f):
            f = f[:, :, :n]
            c = f[1:-1, 1:-1]
            return ((f[2:, 1:-1] - f[:-2, 1:-1]) * self.i2[0], (f[1:-1, 2:] - f[1:-1, :-2]) * self.i2[1] / rm,
                    (torch.roll(c, -1, 2) - torch.roll(c, 1, 2)) * self.i2[2] / (rm * s))

        gu, gv, gw, gk, gd = (grad(a[f]) for f in (F.U, F.V, F.W, F.TKE, F.DIS))
        k, d = a[F.TKE][I], a[F.DIS][I]
        nue_max = 1.0e5 / (u_0 * L_m)
        cn = torch.clamp(k / d, max=nue_max)
        ur, vr, wr = (a[f][I] / rm for f in (F.U, F.V, F.W))
        rr, rt, rp = gu[0], gu[1] - vr, gu[2] - wr
        tr, tt, tp = gv[0], gv[1] + ur, gv[2] - wr * cot
        pr, pt, pp = gw[0], gw[1], gw[2] + ur + vr * cot
        der = 0.66667 * (rr + tt + pp)
        prod = torch.clamp((cn * (2.0 * rr - der) - 0.66667 * k) * rr + cn * (rt + tr) * (rt + tr)
                           + cn * (rp + pr) * (rp + pr) + (cn * (2.0 * tt - der) - 0.66667 * k) * tt
                           + cn * (tp + pt) * (tp + pt) + (cn * (2.0 * pp - der) - 0.66667 * k) * pp, min=0.0)
        om = torch.sqrt((rt - tr) ** 2 + (rp - pr) ** 2 + (tp - pt) ** 2)
        bs, sw2 = 0.09, 1.168
        nu_nd, ys = 1.8e-5 / (u_0 * L_m), 1.0e20 / L_m
        gdot = gk[0] * gd[0] + gk[1] * gd[1] + gk[2] * gd[2]
        cd = torch.clamp(2.0 * sw2 / d * gdot, min=1.0e-20)
        ta, tb = torch.sqrt(k) / (bs * d * ys), 500.0 * nu_nd / (ys * ys * d)
        F1 = torch.tanh(torch.minimum(torch.maximum(ta, tb), 4.0 * sw2 * k / (cd * ys * ys)) ** 4)
        F2 = torch.tanh(torch.maximum(2.0 * ta, tb) ** 2)
        nue = 0.31 * k / torch.maximum(0.31 * d, om * F2)
        ks = torch.clamp(k, min=1.0e-20)
        yk = bs * ks * d
        pk = torch.minimum(prod, 20.0 * yk)
        tks = pk - yk
        dss = ((F1 * 0.413 + (1.0 - F1) * 0.2) * pk * d / ks - (F1 * 0.0333 + (1.0 - F1) * 0.0368) * d * d
               + 2.0 * (1.0 - F1) * sw2 / d * gdot)
        T = a[F.T][I] * P["t_ref"]
        dz = torch.tensor(hm[2:] - hm[:-2], device=DEV)[:, None, None]
        dTdz = (a[F.T][2:, 1:-1, :n] - a[F.T][:-2, 1:-1, :n]) * P["t_ref"] / dz
        rho = a[F.RHO_MIX][I]
        A, B = torch.zeros_like(T), torch.zeros_like(T)
        tp_ = abi.make_turb_params()
        for m, (v, c, ic) in enumerate(((F.H2O, F.H2O_CLOUD, F.H2O_ICE), (F.NH3, F.NH3_CLOUD, F.NH3_ICE),
                                        (F.CH4, F.CH4_CLOUD, F.CH4_ICE))):
            sat = (torch.clamp(a[c][I], min=0.0) + torch.clamp(a[ic][I], min=0.0)) / rho > 1.0e-9
            qv = torch.where(sat, torch.clamp(a[v][I], min=0.0) / rho, torch.zeros_like(T))
            L = torch.where(T >= tp_.t_0[m], torch.full_like(T, tp_.lv[m]), torch.full_like(T, tp_.ls[m]))
            A += L * qv / (P["R_mix"] * T)
            B += tp_.ep[m] * L * L * qv / (P["cp_mix"] * P["R_mix"] * T * T)
        N2 = P["g"] / T * (dTdz + P["g"] / P["cp_mix"] * (1.0 + A) / (1.0 + B)) * (1.0 + A)
        tks = tks - torch.clamp(nue, min=0.0) * torch.clamp(N2, min=0.0) * (L_m / u_0) ** 2 / 0.9
        k, d = torch.clamp(k, min=1.0 / (u_0 * u_0)), torch.clamp(d, min=1.0e-10)
        a[F.TKE][I], a[F.DIS][I] = k, d
        a[F.NUE][I] = nue
        lim_d, lim_k = 20.0 * d * d, 20.0 * k * d
        a[F.DIS_SOURCE][I] = torch.minimum(torch.maximum(dss, -lim_d), lim_d)
        a[F.TKE_SOURCE][I] = torch.minimum(torch.maximum(tks, -lim_k), lim_k)
        for f in (F.TKE, F.DIS, F.NUE):
            a[f][0] = a[f][1]
        a[F.NUE].clamp_(0.0, nue_max)
        for x in [a[f] for f in [F.TKE, F.DIS] + CLOSURE] + [self.nl[F.TKE], self.nl[F.DIS]]:
            x[:, :, -1] = x[:, :, 0]
            x[-1, 0] = 0.5 * (x[-1, 1] + x[-2, 0])
            x[-1, -1] = 0.5 * (x[-1, -2] + x[-2, -1])

    def iterate(self, n):
        for it in range(n):
            if it % 2 == 0:
                self.density()
                self.pressure()
                if self.P["driver_glue"]:
                    self.damp()
            self.rk4()
            self.boundaries()
            if self.P["driver_glue"]:
                for q in SPECIES:
                    self.a[q].clamp_(min=0.0)
            self.nl = {q: self.a[q].clone() for q in F.PROG}
            if self.P["driver_glue"]:
                self.turbulence()


def _thomas(lo, b, up, d):
    """Tridiagonal solves along the first axis."""
    cp, dp = [up[0] / b[0]], [d[0] / b[0]]
    for q in range(1, b.shape[0]):
        dn = b[q] - lo[q] * cp[-1]
        cp.append(up[q] / dn)
        dp.append((d[q] - lo[q] * dp[-1]) / dn)
    x = [dp[-1]]
    for q in range(b.shape[0] - 2, -1, -1):
        x.append(dp[q] - cp[q] * x[-1])
    return torch.stack(x[::-1])


def _poisson(case, seed):
    """The zero-mean solution for the compatible part of the source: a real FFT over phi, a block-tridiagonal
    solve in theta per mode (dense radial blocks), corrected once with the FP64 residual."""
    g, f = _source(case, seed)
    m = _Model(g, abi.default_params(), {q: torch.zeros(1, device=DEV) for q in F.PROG}, None)
    n, NI, NJ = g.km - 1, g.im - 2, g.jm - 2
    rm = m.rm[1:-1]
    n1 = m.id2[0]
    n2 = (m.id2[1] / (rm * rm))[:, None].expand(NI, NJ)
    n3 = m.id2[2] / (rm[:, None] ** 2 * m.sinp[None, 1:-1] ** 2)
    den = 2.0 * (n1 + n2 + n3)
    yi, yj = (torch.ones(s, dtype=torch.float64, device=DEV) for s in (NI, NJ))
    yi[0] = yi[-1] = yj[0] = yj[-1] = 1.5       # the operator's left null vector is yi yj on every meridian
    y = (yi[:, None] * yj[None, :])[:, :, None].expand(NI, NJ, n)
    f = f[1:-1, 1:-1, :n]
    f = f - (y * f).sum() / (y * y).sum() * y

    def apply(p):
        e = torch.zeros((NI + 2, NJ + 2, n), dtype=torch.float64, device=DEV)
        e[1:-1, 1:-1] = p
        e[0], e[-1] = C43 * e[1] - C13 * e[2], C43 * e[-2] - C13 * e[-3]
        e[:, 0], e[:, -1] = C43 * e[:, 1] - C13 * e[:, 2], C43 * e[:, -2] - C13 * e[:, -3]
        return (n1 * (e[2:, 1:-1] + e[:-2, 1:-1]) + n2[:, :, None] * (e[1:-1, 2:] + e[1:-1, :-2])
                + n3[:, :, None] * (torch.roll(p, 1, 2) + torch.roll(p, -1, 2)) - den[:, :, None] * p)

    cth = torch.cos(2.0 * math.pi * torch.arange(n // 2 + 1, dtype=torch.float64, device=DEV) / n)
    M = cth.shape[0]
    W, low, upp = [], n2.clone(), n2.clone()
    low[:, -1] *= 1.0 - C13
    upp[:, 0] *= 1.0 - C13
    eye = torch.eye(NI, dtype=torch.float64, device=DEV).expand(M, NI, NI)
    for j in range(NJ):
        D = torch.zeros((M, NI, NI), dtype=torch.float64, device=DEV)
        dg = -den[None, :, j] + 2.0 * n3[None, :, j] * cth[:, None]
        if j in (0, NJ - 1):
            dg = dg + C43 * n2[None, :, j]
        dg[:, 0] += C43 * n1
        dg[:, -1] += C43 * n1
        D.diagonal(dim1=1, dim2=2).copy_(dg)
        up1, lo1 = torch.full((NI - 1,), n1, dtype=torch.float64, device=DEV), torch.full(
            (NI - 1,), n1, dtype=torch.float64, device=DEV)
        up1[0] *= 1.0 - C13
        lo1[-1] *= 1.0 - C13
        D.diagonal(1, 1, 2).copy_(up1.expand(M, -1))
        D.diagonal(-1, 1, 2).copy_(lo1.expand(M, -1))
        if j == 0:
            D[0, 0] = 0.0
            D[0, 0, 0] = 1.0
        else:
            cc = upp[:, j - 1].expand(M, NI).clone()
            if j == 1:
                cc[0, 0] = 0.0
            D = D - low[None, :, j, None] * W[-1] * cc[:, None, :]
        W.append(torch.linalg.solve(D, eye))

    def solve(r):
        S = torch.view_as_real(torch.fft.rfft(r, dim=2)).permute(1, 2, 0, 3).contiguous()    # NJ, M, NI, 2
        S[0, 0, 0] = 0.0
        z = [S[0]]
        for j in range(1, NJ):
            z.append(S[j] - low[None, :, j, None] * (W[j - 1] @ z[-1]))
        x = [W[-1] @ z[-1]]
        for j in range(NJ - 2, -1, -1):
            cc = upp[:, j].expand(M, NI).clone()
            if j == 0:
                cc[0, 0] = 0.0
            x.append(W[j] @ (z[j] - cc[:, :, None] * x[-1]))
        X = torch.view_as_complex(torch.stack(x[::-1]).permute(2, 0, 1, 3).contiguous())
        return torch.fft.irfft(X, n=n, dim=2)

    p = solve(f)
    p = p + solve(f - apply(p))
    p = p - p.mean()
    out = torch.zeros(g.shape, dtype=torch.float64, device=DEV)
    out[1:-1, 1:-1, :n] = p
    out[0], out[-1] = C43 * out[1] - C13 * out[2], C43 * out[-2] - C13 * out[-3]
    out[:, 0], out[:, -1] = C43 * out[:, 1] - C13 * out[:, 2], C43 * out[:, -2] - C13 * out[:, -3]
    out[:, :, n] = out[:, :, 0]
    return out.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        return _poisson(case, seed)
    g, P, a, hold = _fields(case, seed)
    m = _Model(g, P, a, hold)
    if kind == "pressure":
        m.pressure()
        return {"p_dyn": a[F.P_DYN]}
    if kind == "turbulence":
        m.turbulence()
        return {F.NAMES[f]: a[f] for f in [F.TKE, F.DIS] + CLOSURE}
    if kind == "step":
        m.density()
        m.pressure()
        m.rk4()
        return {F.NAMES[f]: a[f].cpu().numpy() for f in F.STEP_OUTPUTS + [F.P_DYN]}
    m.iterate(4 if kind == "replay" else 2)
    return {F.NAMES[f]: a[f] for f in F.PROG + [F.P_DYN] + PROJECTION + (CLOSURE if case["glue"] else [])}
