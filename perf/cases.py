"""Timed cases of the library: tracer advection steps, barotropic steps, whole baroclinic steps and ensembles.

Every case drives the public entry points (`mom5_gb300.capi`) on a seeded synthetic domain of `mom5_gb300.grid`, from
time level 1 to time level 2.  The outputs are views of the library's own device fields, whole data domains unless a
field's halo is documented as not maintained.  `exact` restates the same equations in plain torch, in 64 bits.
"""
import dataclasses
import math
import random

import torch

from mom5_gb300 import capi, grid, harness, serving
from mom5_gb300.capi import F

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
SCHEMES = {"mdfl_sweby": capi.ADVECT_MDFL_SWEBY, "dst_linear": capi.ADVECT_DST_LINEAR, "mdppm": capi.ADVECT_MDPPM,
           "psom": capi.ADVECT_PSOM}
BARO_OUT = {"eta_t_bar": (F.ETA_T_BAR, 2), "udrho_u": (F.UDRHO_U, 2), "udrho_v": (F.UDRHO_V, 2),
            "conv_rho_ud_t": (F.CONV_RHO_UD_T, 2), "eta_u": (F.ETA_U, 2), "ps": (F.PS, 0),
            "grad_ps_x": (F.GRAD_PS_X, 0), "grad_ps_y": (F.GRAD_PS_Y, 0)}
MOMENTS = ("S0", "SX", "SXX", "SY", "SYY", "SZ", "SZZ", "SXY", "SXZ", "SYZ")


def _case(name, kind, ni, nj, nk, ntr, **kw):
    c = {"name": name, "kind": kind, "ni": ni, "nj": nj, "nk": nk, "ntr": ntr, "cyclic_x": False, "cyclic_y": False,
         "lon": 0.25 * ni, "lat": min(75.0, 0.125 * nj), "dt": 600.0, "nts": 60, "mixed": False,
         "scheme": "mdfl_sweby", "cgrid": False, "step_b": True, "autotune": False}
    return {**c, **kw}


def listed():
    return [
        # a test-sized basin: a developer's first run, launches only
        _case("advect_basin_37x29x12", "advect", 37, 29, 12, 2, lon=37.0, lat=20.0, dt=1800.0),
        # the regional box of the benchmark (C0): temperature and salinity, one-hour step
        _case("advect_regional_120x80x30", "advect", 120, 80, 30, 2, lon=60.0, lat=40.0, dt=3600.0),
        # one rank's block of the quarter-degree grid with a biogeochemical tracer set
        _case("advect_block_360x270x50", "advect", 360, 270, 50, 10),
        # the headline workload: the global quarter-degree grid, drop-in arithmetic, advection and barotropic step
        _case("step_global_1440x1080x50", "step", 1440, 1080, 50, 10, cyclic_x=True, lon=360.0, lat=80.0),
        # the same step in the precision form, with the launch shape a program tunes once and keeps
        _case("step_global_mixed", "step", 1440, 1080, 50, 10, cyclic_x=True, lon=360.0, lat=80.0, mixed=True,
              autotune=True),
        # a periodic channel of odd extents in the precision form, launch shape left at its default
        _case("advect_mixed_255x181x40", "advect", 255, 181, 40, 4, cyclic_x=True, mixed=True),
        # the one-degree barotropic workload (C1): 80 subcycles of 67.5 s
        _case("barotropic_360x300", "baro", 360, 300, 1, 0, cyclic_x=True, lon=360.0, lat=75.0, dt=2700.0, nts=80),
        # a C-grid model of odd extents with the other time stepping
        _case("barotropic_cgrid_361x243", "baro", 361, 243, 1, 0, cyclic_x=True, lon=361 * 0.5, lat=60.0, dt=900.0,
              nts=48, cgrid=True, step_b=False),
        # temperature and salinity with the piecewise-parabolic scheme
        _case("mdppm_180x135x50", "advect", 180, 135, 50, 2, scheme="mdppm"),
        # temperature and salinity with second-order moments in a narrow periodic channel
        _case("psom_channel_121x30x30", "advect", 121, 30, 30, 2, cyclic_x=True, scheme="psom"),
        # an ensemble of uneven regional domains stepped as one batch: drop-in and precision form
        {"name": "batch_8_domains", "kind": "batch", "count": 8, "sizes": 3, "ntr": 4, "dt": 400.0, "nts": 40,
         "mixed": False},
        {"name": "batch_8_domains_mixed", "kind": "batch", "count": 8, "sizes": 3, "ntr": 4, "dt": 400.0, "nts": 40,
         "mixed": True},
    ]


def draw(rng):
    kind = rng.choice(["advect", "advect", "advect", "step", "baro", "scheme", "batch"])
    mixed = kind != "scheme" and rng.random() < 0.35
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(2, 8), "sizes": rng.randint(10, 99999), "ntr": rng.randint(1, 4),
                "dt": 400.0, "nts": 40, "mixed": mixed}
    lo, hi = (math.log(24), math.log(700)) if kind != "scheme" else (math.log(24), math.log(200))
    ni, nj = (int(math.exp(rng.uniform(lo, hi))) for _ in range(2))
    nk = 1 if kind == "baro" else rng.randint(8, 50)
    ntr = 0 if kind == "baro" else rng.randint(1, 2 if kind == "scheme" else 10)
    scheme = rng.choice(["mdppm", "psom"]) if kind == "scheme" else rng.choice(["mdfl_sweby"] * 3 + ["dst_linear"])
    if scheme == "psom":
        ni, nj, nk = min(ni, 126), min(nj, 30), min(nk, 30)
    if mixed or kind == "step":
        scheme = "mdfl_sweby"
    cgrid = kind == "baro" and not mixed and rng.random() < 0.4
    c = _case("", "advect" if kind == "scheme" else kind, ni, nj, nk, ntr, cyclic_x=rng.random() < 0.5,
              cyclic_y=rng.random() < 0.2, mixed=mixed, scheme=scheme, cgrid=cgrid, step_b=rng.random() < 0.7,
              nts=rng.choice([40, 48, 60]))
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ inputs
def _tracers(dom, ntr, seed):
    """The tracers grid.make_domain draws, drawn on the device: temperature, salinity, then passive tracers."""
    s, tmask = dom.spec, dom["tmask"]
    g = torch.Generator(device=tmask.device)
    g.manual_seed(seed * 7919 + 17)
    zt = (dom.zw - 0.5 * dom.dzt).to(tmask.device)
    lat = s.lat0 + (torch.arange(s.nyd, dtype=torch.float64, device=tmask.device) - 0.5) * (s.lat1 - s.lat0) / s.nj
    T = torch.empty((ntr, *tmask.shape), dtype=torch.float64, device=tmask.device)
    for n in range(ntr):
        if n == 0:
            T[n].normal_(generator=g).mul_(0.1).add_(25.0 * torch.exp(-zt / 800.0)[:, None, None])
        elif n == 1:
            T[n] = 35.0 + 0.5 * torch.tanh(lat / 20.0)[None, :, None]
        else:
            T[n].uniform_(generator=g)
        T[n] *= tmask
    return _halo(T, s.cyclic_x, s.cyclic_y)


def _domain(spec, ntr, seed):
    dom = grid.make_domain(dataclasses.replace(spec, ntracers=0, seed=seed), device=DEVICE)
    dom.spec = dataclasses.replace(dom.spec, ntracers=ntr)
    if ntr:
        dom.f["T"] = _tracers(dom, ntr, seed)
    return dom


def _domains(case, seed):
    """The seeded input domains of a case, one for all kinds but "batch"."""
    if case["kind"] == "batch":
        for i, spec in enumerate(serving.ensemble_specs(case["count"], seed=case["sizes"])):
            yield _domain(spec, case["ntr"], seed * 131 + i)
        return
    c = case
    ni, nj = c["ni"], c["nj"]
    spec = grid.DomainSpec(ni=ni, nj=nj, nk=c["nk"], lon0=0.0, lon1=c["lon"], lat0=-c["lat"], lat1=c["lat"],
                           cyclic_x=c["cyclic_x"], cyclic_y=c["cyclic_y"])
    if c["kind"] == "baro":  # a ridge under one layer, as the one-degree barotropic workload has it
        spec = dataclasses.replace(spec, hmin=None, ridge_amp=1500.0)
    else:
        spec = dataclasses.replace(spec, continent=(5 * ni // 12, 3 * nj // 8, max(2, ni // 9), max(2, nj // 9)))
    yield _domain(spec, c["ntr"], seed)


def prepare(case, seed):
    batch = case["kind"] == "batch"
    opts = capi.default_options(
        precision=capi.PRECISION_MIXED if case["mixed"] else capi.PRECISION_FP64,
        barotropic_time_stepping_B=int(batch or case["step_b"]),
        barotropic_time_stepping_A=int(not (batch or case["step_b"])))
    doms = []
    for dom in _domains(case, seed):
        torch.cuda.synchronize()
        d = harness.load(dom, options=opts, horz_grid=capi.CGRID if case.get("cgrid") else capi.BGRID,
                         scheme=SCHEMES[case.get("scheme", "mdfl_sweby")])
        for n in range(1, case["ntr"] + 1):
            if case.get("scheme") == "psom":
                d.set_psom_limit(n, True)
        if case["kind"] != "advect":
            d.barotropic_init(dtuv=case["dt"], dtbt=2.0 * case["dt"] / case["nts"])
        d.synchronize()
        if case.get("autotune"):
            d.autotune(case["dt"])
        doms.append(d)
    state = {"case": case, "domains": doms, "batch": capi.Batch(doms) if batch else None}
    state["out"] = _views(state)
    return state


class _Field:
    """One device field of a domain; it holds the domain for as long as a tensor looks at it."""

    def __init__(self, d, fid, n, level, levels):
        shape = (levels, d.dims.nj + 2, d.dims.ni + 2) if levels else (d.dims.nj + 2, d.dims.ni + 2)
        self.domain = d
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "version": 3, "strides": None,
                                         "data": (d.device_ptr(fid, n=n, level=level), False)}


def _view(d, fid, n=0, level=0, levels=0):
    return torch.as_tensor(_Field(d, fid, n, level, levels), device="cuda")


def _views(state):
    c, out = state["case"], {}
    for i, d in enumerate(state["domains"]):
        o, nk, ntr = {}, d.dims.nk, c["ntr"]
        if c["kind"] != "baro":
            o["tracer"] = [_view(d, F.TRACER, n, 2, nk) for n in range(1, ntr + 1)]
            if c["kind"] == "advect" and not c["mixed"]:
                o["tendency"] = [_view(d, F.TH_TENDENCY, n, 0, nk) for n in range(1, ntr + 1)]
            if c.get("scheme") == "psom":  # their halos are not maintained
                o["moments"] = [[_view(d, getattr(F, "PSOM_" + m), n, 0, nk)[:, 1:-1, 1:-1] for m in MOMENTS]
                                for n in range(1, ntr + 1)]
        if c["kind"] != "advect":
            names = ("eta_t_bar", "udrho_u", "udrho_v") if c["kind"] == "batch" else BARO_OUT
            o["baro"] = {k: _view(d, BARO_OUT[k][0], 0, BARO_OUT[k][1]) for k in names}
        out["domain%d" % i] = o
    return out


def run(state):
    c = state["case"]
    if state["batch"] is not None:
        state["batch"].step(c["dt"], parity=0)
        return state["out"]
    d = state["domains"][0]
    if c["kind"] != "baro":
        d.tracer_advection_step(1, 1, 2, c["dt"])
    if c["kind"] != "advect":
        d.update_ocean_barotropic(1, 2)
    return state["out"]


def _work(ni, nj, nk, ntr, nts, scheme, advect, baro):
    """Advection: T read and written per tracer, u, v, w, rho_dzt and its reciprocal per cell, seven metrics; the
    tendency too where it is an output.  Barotropic: 18 planes read and 8 written once (the state and the metrics of a
    step; its subcycles need no memory traffic).  Operations: those of one evaluation of the equations."""
    bytes_, flops = 0, 0
    if advect:
        per = {"mdppm": 320, "psom": 640}.get(scheme, 75)
        planes = 2 * ntr + 5 + (20 * ntr if scheme == "psom" else 0)
        bytes_ += 8 * ni * nj * (nk * planes + 7)
        flops += per * ni * nj * nk * ntr
    if baro:
        bytes_ += 8 * ni * nj * 26
        flops += 51 * ni * nj * nts
    return bytes_, flops


def work(case):
    c = case
    if c["kind"] == "batch":
        parts = [_work(s.ni, s.nj, s.nk, c["ntr"], c["nts"], "", True, True)
                 for s in serving.ensemble_specs(c["count"], seed=c["sizes"])]
    else:
        parts = [_work(c["ni"], c["nj"], c["nk"], c["ntr"], c["nts"], c["scheme"], c["kind"] != "baro",
                       c["kind"] != "advect")]
        if c["kind"] == "advect" and not c["mixed"]:
            parts.append((8 * c["ni"] * c["nj"] * c["nk"] * c["ntr"], 0))
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


# ------------------------------------------------------------------------------------------------ 64-bit restatement
def _halo(a, cx, cy):
    """Periodic images in the halo of the last two dimensions; corners where both directions are periodic."""
    if cx:
        a[..., 1:-1, 0], a[..., 1:-1, -1] = a[..., 1:-1, -2], a[..., 1:-1, 1]
    if cy:
        a[..., 0, 1:-1], a[..., -1, 1:-1] = a[..., -2, 1:-1], a[..., 1, 1:-1]
    if cx and cy:
        a[..., 0, 0], a[..., 0, -1], a[..., -1, 0], a[..., -1, -1] = (
            a[..., -2, -2], a[..., -2, 1], a[..., 1, -2], a[..., 1, 1])
    return a


def _shift(a, n, dim, cyclic):
    """b[i] = a[i + n] along dim, zero beyond a closed end."""
    if n == 0:
        return a
    b = torch.roll(a, -n, dim)
    if not cyclic:
        m = min(abs(n), b.shape[dim])
        b.narrow(dim, b.shape[dim] - m if n > 0 else 0, m).zero_()
    return b


def _clamped(a, n):
    """b[k] = a[min(max(k + n, 0), nk - 1)]."""
    k = (torch.arange(a.shape[0], device=a.device) + n).clamp(0, a.shape[0] - 1)
    return a[k]


class _Grid:
    """The compute-domain arrays an advection scheme reads."""

    def __init__(self, dom):
        s = dom.spec
        self.cx, self.cy, self.nk = s.cyclic_x, s.cyclic_y, s.nk
        c = lambda name: dom[name][..., 1:-1, 1:-1]  # noqa: E731
        self.m, self.rdz, self.rdzr, self.dat, self.datr = c("tmask"), c("rho_dzt"), c("rho_dztr"), c("dat"), c("datr")
        self.w = dom["wrho_bt"][1:, 1:-1, 1:-1]  # bottom face of each level
        self.wtop = torch.cat([torch.zeros_like(self.w[:1]), self.w[:-1]])
        self.u, self.v = c("uhrho_et"), c("vhrho_nt")
        uf, vf = dom["dyte"] * dom["uhrho_et"], dom["dxtn"] * dom["vhrho_nt"]
        self.ue, self.uw, self.vn = uf[:, 1:-1, 1:-1], uf[:, 1:-1, :-2], vf[:, 1:-1, 1:-1]
        self.dxte, self.dytn = c("dxte"), c("dytn")
        self.dyte, self.dxtn = c("dyte"), c("dxtn")
        rd = dom["rho_dzt"]
        self.rde, self.rdn = rd[:, 1:-1, 2:], rd[:, 2:, 1:-1]  # rho_dzt of the eastern and northern neighbour

    def x(self, a, n):
        return _shift(a, n, -1, self.cx)

    def y(self, a, n):
        return _shift(a, n, -2, self.cy)


def _face(mf, cfl, rjm, rj, rjp, tp, tm, sweby):
    """Flux of the direct-space-time scheme through a face whose flow comes from tp (mf > 0) or tm."""
    d0, d1 = (2.0 - cfl) * (1.0 - cfl) / 6.0, (1.0 - cfl * cfl) / 6.0
    pos = mf > 0
    theta = torch.where(pos, rjm, rjp) / (1.0e-30 + rj)
    psi = d0 + d1 * theta
    if sweby:
        psi = psi.clamp_max(1.0).minimum((1.0 - cfl) / (1.0e-30 + cfl) * theta).clamp_min(0.0)
    return mf * torch.where(pos, tp + psi * rj, tm - psi * rj)


def _mdfl(g, T, dt, sweby):
    m, m1 = g.m, _clamped(g.m, 1)
    R = (T - _clamped(T, 1)) * m * m1
    Rup = (_clamped(T, -1) - T) * _clamped(g.m, -1) * m
    fb = _face(g.dat * g.w, (g.w * dt / g.rdz).abs(), _clamped(R, 1), R, Rup, _clamped(T, 1), T, sweby) * m * m1
    del R, Rup
    ft = torch.cat([torch.zeros_like(fb[:1]), fb[:-1]])
    t = T + dt / g.rdz * (g.datr * (fb - ft) + T * (g.wtop - g.w))
    for s, vel, dl, rn, f2 in ((g.x, g.u, g.dxte, g.rde, g.ue), (g.y, g.v, g.dytn, g.rdn, g.vn)):
        mp = s(m, 1) * m
        R = (s(t, 1) - t) * mp
        cfl = (2.0 * vel * dt / ((g.rdz + rn) * dl)).abs()
        fe = _face(f2, cfl, s(R, -1), R, s(R, 1), t, s(t, 1), sweby) * mp
        div = s(fe, -1) - fe
        if s == g.x:
            div = div + T * (g.ue - g.uw)
        t = t + dt * m * g.datr / g.rdz * div
    t = t + dt * T / g.rdz * (g.w - g.wtop + g.datr * (g.uw - g.ue))
    return g.rdz * (t - T) / dt * m


def _slopes(s, m, at):
    """Limited slope of the parabola and the masked differences; at(a, n) is a at offset n, m the five masks."""
    s0, s1, s2, sm1, sm2 = s, at(s, 1), at(s, 2), at(s, -1), at(s, -2)
    mm2, mm1, m0, mp1, mp2 = m
    a3m = (2 * sm2 - 12 * sm1 + 6 * s0 + 4 * s1) / 12.0
    a3p = (-4 * sm1 - 6 * s0 + 12 * s1 - 2 * s2) / 12.0
    a = (mm2 * (1 - 0.5 * mp2) * a3m + mp2 * (1 - 0.5 * mm2) * a3p) + (1 - mm2) * (1 - mp2) * 0.5 * (s1 - sm1)
    hi, lo = torch.maximum(torch.maximum(s1, sm1), s0) - s0, s0 - torch.minimum(torch.minimum(s1, sm1), s0)
    da = torch.copysign(torch.minimum(a.abs(), 2 * torch.minimum(hi, lo)), a) * mm1 * mp1 * m0
    return da, (s0 - sm1) * mm1, (s1 - s0) * mp1


def _parabola(s, da, dm, dp, at):
    """Edge values under the improved full constraint, and the curvature."""
    al = 0.5 * ((s - dm) + s) + (at(da, -1) - da) / 6.0
    ar = 0.5 * (s + (s + dp)) + (da - at(da, 1)) / 6.0
    sg = torch.copysign(torch.ones_like(da), da)
    al, ar = (s - sg * torch.minimum(da.abs(), (al - s).abs()), s + sg * torch.minimum(da.abs(), (ar - s).abs()))
    return al, ar, 6 * s - 3 * (ar + al)


def _mdppm(g, T, dt):
    nk, third2 = g.nk, 2.0 / 3.0
    k = torch.arange(nk, device=T.device)
    inner = lambda n, frm: ((k + n).clamp(0, nk - 1) - (k + frm).clamp(0, nk - 1)).abs()[:, None, None]  # noqa: E731
    m = (_clamped(g.m, -2) * inner(-2, -1), _clamped(g.m, -1) * inner(-1, 0), g.m, _clamped(g.m, 1) * inner(1, 0),
         _clamped(g.m, 2) * inner(2, 1))
    da, dm, dp = _slopes(T, m, _clamped)
    al, ar, c6 = _parabola(T, da, dm, dp, _clamped)
    cfl = (g.w * dt / g.rdz).abs()
    mf = g.dat * g.w * m[2] * m[3]
    down = mf * (ar + 0.5 * cfl * ((al - ar) + (1 - third2 * cfl) * c6))
    cup = (g.wtop * dt / torch.cat([g.rdz[:1], g.rdz[:-1]])).abs()
    mu = g.dat * g.wtop * m[2] * m[1]
    up = mu * (al + 0.5 * cup * ((ar - al) + (1 - third2 * cup) * c6))  # through the top face, from below
    up = torch.cat([up[1:], torch.zeros_like(up[:1])])
    fz = torch.where(mf <= 0, down, up)
    ft = torch.cat([torch.zeros_like(fz[:1]), fz[:-1]])
    t = T + dt / g.rdz * (g.datr * (fz - ft) + T * (g.wtop - g.w))
    for s, vel, dl, rn, f2 in ((g.x, g.u, g.dxte, g.rde, g.ue), (g.y, g.v, g.dytn, g.rdn, g.vn)):
        m = tuple(s(g.m, n) for n in (-2, -1, 0, 1, 2))
        da, dm, dp = _slopes(t, m, s)
        al, ar, c6 = _parabola(t, da, dm, dp, s)
        cfl = 2.0 * vel * dt / ((g.rdz + rn) * dl)
        pos = ar + 0.5 * cfl * ((al - ar) + (1 - third2 * cfl) * c6)
        ale, are, c6e = s(al, 1), s(ar, 1), s(c6, 1)
        neg = ale - 0.5 * cfl * ((are - ale) + (1 + third2 * cfl) * c6e)
        fe = f2 * m[2] * m[3] * torch.where(f2 >= 0, pos, neg)
        div = s(fe, -1) - fe
        if s == g.x:
            div = div + T * (g.ue - g.uw)
        t = t + dt * g.m * g.datr / g.rdz * div
    t = t + dt * T / g.rdz * (g.w - g.wtop + g.datr * (g.uw - g.ue))
    return g.rdz * (t - T) / dt * g.m


# moments along a direction: first, second; the other firsts; the crosses with them; the other seconds; the other cross
_ROLES = {"x": "SX SXX SY SZ SXY SXZ SYY SZZ SYZ", "y": "SY SYY SX SZ SXY SYZ SXX SZZ SXZ",
          "z": "SZ SZZ SX SY SXZ SYZ SXX SYY SXY"}


def _psom_limit(g, st, T, axis, nb):
    a, aa, _, _, c1, c2 = _ROLES[axis].split()[:6]
    cl = lambda x, lo, hi: torch.minimum(hi, torch.maximum(lo, x))  # noqa: E731
    for sgn, pick in ((-1.0, torch.maximum), (1.0, torch.minimum)):
        ext = T * g.m
        for n in (-1, 1):
            ext = torch.where(nb(g.m, n) > 0, pick(nb(T, n), ext), ext)
        slp = sgn * (st["S0"] - ext * st["SM"])
        s1 = cl(sgn * st[a], -1.5 * slp, 1.5 * slp)
        s2 = cl(sgn * st[aa], s1.abs() - slp, 2 * slp - 0.3334 * s1.abs())
        for c in (c1, c2):
            st[c] = sgn * cl(sgn * st[c], -slp, slp)
        st[a], st[aa] = sgn * s1, sgn * s2


def _psom_sweep(g, st, axis, vel, dv, dt, to_b, from_b, to_a, from_a):
    """Both transport sweeps of a direction.  A face joins cell a (upstream for vel >= 0) and cell b: to_b/to_a bring a
    face's values to its cell b/a, from_b/from_a a cell's values to the face it is b/a of."""
    a, aa, b1, b2, c1, c2, bb1, bb2, bc = _ROLES[axis].split()
    moved = {}
    for sgn in (-1.0, 1.0):  # a cell gives through its face as b first
        to, frm = (to_b, from_b) if sgn < 0 else (to_a, from_a)
        on = to((vel < 0).double()) > 0 if sgn < 0 else to((vel > 0).double()) > 0
        fm = torch.where(on, sgn * to(vel * dt * dv), torch.zeros_like(st["SM"]))
        al = fm / (st["SM"] + 1.0e-20)
        q, r = al * al, 1.0 - al
        f = {"S0": al * (st["S0"] + sgn * r * (st[a] + sgn * (r - al) * st[aa])),
             a: q * (st[a] + sgn * 3.0 * r * st[aa]), aa: al * q * st[aa], b1: al * (st[b1] + sgn * r * st[c1]),
             b2: al * (st[b2] + sgn * r * st[c2]), c1: q * st[c1], c2: q * st[c2], bb1: al * st[bb1],
             bb2: al * st[bb2], bc: al * st[bc], "SM": fm}
        st[a] = r * r * (st[a] - sgn * 3.0 * al * st[aa])
        st[aa] = r * r * r * st[aa]
        st[c1], st[c2] = r * r * st[c1], r * r * st[c2]
        for k in ("SM", "S0", b1, b2, bb1, bb2, bc):
            st[k] = st[k] - f[k]
        moved[sgn] = {k: frm(v) for k, v in f.items()}
    flux = (moved[1.0]["S0"] - moved[-1.0]["S0"]) / dt
    for sgn in (1.0, -1.0):  # and receives as b first
        f = {k: (to_b if sgn > 0 else to_a)(v) for k, v in moved[sgn].items()}
        st["SM"] = st["SM"] + f["SM"]
        al = f["SM"] / (st["SM"] + 1.0e-20)
        r = 1.0 - al
        tt = sgn * (al * st["S0"] - r * f["S0"])
        st["S0"] = st["S0"] + f["S0"]
        st[aa] = al * al * f[aa] + r * r * st[aa] + 5.0 * (sgn * al * r * (st[a] - f[a]) - sgn * (r - al) * tt)
        st[a] = al * f[a] + r * st[a] + 3.0 * tt
        st[c1] = al * f[c1] + r * st[c1] + 3.0 * sgn * (al * st[b1] - r * f[b1])
        st[c2] = al * f[c2] + r * st[c2] + 3.0 * sgn * (al * st[b2] - r * f[b2])
        for k in (b1, b2, bb1, bb2, bc):
            st[k] = st[k] + f[k]
    return flux


def _psom(g, T, dt):
    """One call from zero moments with the Merryfield-Holloway limiter, sweeps in the order x, y, z."""
    st = {k: torch.zeros_like(T) for k in MOMENTS}
    st["SM"] = g.rdz * g.dat
    st["S0"] = T * st["SM"] * g.m
    div = 0.0
    for axis in "xyz":
        if axis == "z":
            nb = _clamped
            up = lambda x, n=1: _shift(x, n, 0, False)  # noqa: E731
            vel = g.w * up(g.m)
            to_b, from_b, to_a, from_a = (lambda x: x), (lambda x: x), (lambda x: _shift(x, -1, 0, False)), up
            dv = g.dat.expand_as(vel)
        else:
            s, vel, dv = (g.x, g.u, g.dyte) if axis == "x" else (g.y, g.v, g.dxtn)
            nb = s
            vel, dv = vel * torch.minimum(g.m, s(g.m, 1)), dv.expand_as(vel)
            to_b, from_b = (lambda x, s=s: s(x, -1)), (lambda x, s=s: s(x, 1))
            to_a, from_a = (lambda x: x), (lambda x: x)
        _psom_limit(g, st, T, axis, nb)
        f = _psom_sweep(g, st, axis, vel, dv, dt, to_b, from_b, to_a, from_a)
        if axis == "z":
            div = div + _shift(f, -1, 0, False) - f
        else:
            div = div + f - nb(f, -1)
    return -g.m * div * g.datr, [st[k] for k in MOMENTS]


def _advect(dom, case):
    s, dt, g = dom.spec, case["dt"], _Grid(dom)
    out = {"tracer": [], "tendency": [], "moments": []}
    scheme = case.get("scheme", "mdfl_sweby")
    full = lambda a: torch.nn.functional.pad(a, (1, 1, 1, 1))  # noqa: E731
    for n in range(s.ntracers):
        T = dom["T"][n][:, 1:-1, 1:-1]
        if scheme == "psom":
            th, mom = _psom(g, T, dt)
            out["moments"].append(mom)
        else:
            th = _mdppm(g, T, dt) if scheme == "mdppm" else _mdfl(g, T, dt, scheme == "mdfl_sweby")
        out["tracer"].append(_halo(full((g.rdz * T + dt * th) * g.rdzr), s.cyclic_x, s.cyclic_y))
        out["tendency"].append(full(th) if case["kind"] == "advect" and not case["mixed"] else None)
    return out


def _divergence(dom, u, v, cgrid):
    """Divergence of a transport on the whole data domain, zero in its first row and column."""
    out = torch.zeros_like(u)
    if cgrid:
        a, b = u * dom["dat"] * dom["dxter"], v * dom["dat"] * dom["dytnr"]
        out[1:, 1:] = (a[1:, 1:] - a[1:, :-1]) + (b[1:, 1:] - b[:-1, 1:])
    else:
        a, b = u * dom["dyu"], v * dom["dxu"]
        a = 0.5 * (a[1:] + a[:-1])
        b = 0.5 * (b[:, 1:] + b[:, :-1])
        out[1:, 1:] = (a[:, 1:] - a[:, :-1]) + (b[1:] - b[:-1])
    return out * dom["datr"]


def _gradient(dom, p, cgrid):
    gx, gy = torch.zeros_like(p), torch.zeros_like(p)
    if cgrid:
        gx[:-1, :-1] = (p[:-1, 1:] - p[:-1, :-1])
        gy[:-1, :-1] = (p[1:, :-1] - p[:-1, :-1])
        return gx * dom["dxter"] * dom["tmasken_e1"], gy * dom["dytnr"] * dom["tmasken_n1"]
    fay, fax = 0.5 * (p[:-1] + p[1:]), 0.5 * (p[:, :-1] + p[:, 1:])
    gx[:-1, :-1], gy[:-1, :-1] = fay[:, 1:] - fay[:, :-1], fax[1:] - fax[:-1]
    return gx * dom["dxur"] * dom["umask1"], gy * dom["dyur"] * dom["umask1"]


def _coriolis(f, u, v):
    c0, c1 = torch.zeros_like(u), torch.zeros_like(u)
    c0[1:-1, 1:-1] = 0.25 * (f[1:-1, 1:-1] * (v[1:-1, 1:-1] + v[1:-1, 2:])
                             + f[:-2, 1:-1] * (v[:-2, 1:-1] + v[:-2, 2:]))
    c1[1:-1, 1:-1] = -0.25 * (f[1:-1, 1:-1] * (u[1:-1, 1:-1] + u[2:, 1:-1])
                              + f[1:-1, :-2] * (u[1:-1, :-2] + u[2:, :-2]))
    return c0, c1


def _barotropic(dom, case):
    s, nts, cgrid = dom.spec, case["nts"], case.get("cgrid", False)
    step_b = case.get("step_b", True)
    dt, rho0, gamma = 2.0 * case["dt"] / nts, grid.RHO0, 0.2
    fill = lambda a: _halo(a, s.cyclic_x, s.cyclic_y)  # noqa: E731
    f, tm = dom["f"], dom["tmask1"]
    me, mn = dom["tmasken_e1"], dom["tmasken_n1"]
    c1 = 0.5 * dt * f
    c2 = 1.0 / (1.0 + c1 * c1)
    bar, us, vs = dom["eta_t_bar"].clone(), torch.zeros_like(f), torch.zeros_like(f)
    eta, u, v = dom["eta_t_bar"].clone(), dom["udrho_u"].clone(), dom["udrho_v"].clone()
    steady = tm * (dom["pme"] + dom["river"] + dom["source"] - dom["eta_smooth"])
    hist = [_coriolis(f, u, v)] * 2 if cgrid else None
    for it in range(1, nts + 1):
        pred = eta + dt * gamma / rho0 * (-_divergence(dom, u, v, cgrid) * tm + steady)
        ps = dom["rho_g"] * (pred if cgrid else fill(pred)) + dom["patm"]
        gx, gy = _gradient(dom, ps, cgrid)
        if cgrid:
            now = _coriolis(f, u, v)
            a0, a1 = ((23.0 * now[i] - 16.0 * hist[0][i] + 5.0 * hist[1][i]) / 12.0 for i in (0, 1))
            hist = [now, hist[0]]
            u, v = (fill(u + dt * me * (a0 - dom["thicken_e"] * gx + dom["forcing_u"])),
                    fill(v + dt * mn * (a1 - dom["thicken_n"] * gy + dom["forcing_v"])))
        else:
            t1 = u + dt * (0.5 * f * v - dom["thicku"] * gx + dom["forcing_u"])
            t2 = v + dt * (-0.5 * f * u - dom["thicku"] * gy + dom["forcing_v"])
            u, v = c2 * (t1 + c1 * t2), c2 * (t2 - c1 * t1)
        eta = eta + dt / rho0 * (-_divergence(dom, u, v, cgrid) * tm + steady)
        w = float(nts - it + 1) if step_b else 1.0
        bar, us, vs = bar + eta, us + w * u, vs + w * v
    bar = fill(bar / (nts + 1.0))
    r = 2.0 / (nts * (nts + 1.0)) if step_b else 1.0 / nts
    us, vs = fill(us * r), fill(vs * r)
    eu = torch.zeros_like(bar)
    e, w_ = bar * dom["dte"], bar * dom["dtw"]
    eu[:-1, :-1] = ((e[:-1, :-1] + w_[:-1, 1:]) * dom["dus"][:-1, :-1]
                    + (e[1:, :-1] + w_[1:, 1:]) * dom["dun"][:-1, :-1]) * dom["daur"][:-1, :-1]
    ps = dom["rho_g"] * bar + dom["patm"]
    gx, gy = _gradient(dom, ps, cgrid)
    return {"eta_t_bar": bar, "udrho_u": us, "udrho_v": vs, "conv_rho_ud_t": fill(-_divergence(dom, us, vs, cgrid)),
            "eta_u": fill(dom["umask1"] * eu), "ps": ps, "grad_ps_x": gx, "grad_ps_y": gy}


def exact(case, seed):
    out = {}
    for i, dom in enumerate(_domains(case, seed)):
        o = {}
        if case["kind"] != "baro":
            a = _advect(dom, case)
            o["tracer"] = a["tracer"]
            if case["kind"] == "advect" and not case["mixed"]:
                o["tendency"] = a["tendency"]
            if case.get("scheme") == "psom":
                o["moments"] = a["moments"]
        if case["kind"] != "advect":
            b = _barotropic(dom, case)
            o["baro"] = {k: b[k] for k in ("eta_t_bar", "udrho_u", "udrho_v")} if case["kind"] == "batch" else b
        out["domain%d" % i] = o
    return out
