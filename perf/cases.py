"""Measured workloads of the tracer framework.

Each case is one pass through the package's public entry points, as a model's
host program makes it: a few tracer steps of a resident domain and the reading
of its new state, a coupled step with host forcing, an ensemble step, or one of
the kernels that run beside the tracer step (turbulence closure, momentum
friction).  Inputs come from the package's seeded generator; ``exact`` gives
the same results from plain torch in 64 bits.

A case is a dict of plain values:

* ``kind``: "step", "coupled", "ensemble", "turb" or "del4u";
* ``nx, ny, km``: physical sizes; ``steps``: tracer steps of one pass;
* ``mixed``: the mixed-precision form (else FP64); ``diag``: FP64 diagnostics;
* ``deep``: ocean depths from the global area-depth curve (else the shallow
  map that is linear in the land field);
* ``cyclic, tripole``: the boundaries; ``members, uneven``: of an ensemble.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

lt = importlib.import_module("licom3-hip_b200")

DAY = 86400.0


def _case(name, kind, nx, ny, km, steps=1, mixed=False, diag=False, deep=False, cyclic=True, tripole=True, members=0,
          uneven=False):
    c = dict(kind=kind, nx=nx, ny=ny, km=km, steps=steps, mixed=mixed, diag=diag, deep=deep, cyclic=cyclic,
             tripole=tripole, members=members, uneven=uneven)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's own compiled block size: latency and launches
        _case("block_fp64", "step", 36, 40, 55, steps=5),
        # the 1-degree global model in the bit-exact form and in the fast one
        _case("deg1_fp64", "step", 360, 218, 30, steps=5),
        _case("deg1_mixed", "step", 360, 218, 30, steps=5, mixed=True),
        # a regional model of odd sizes and closed boundaries (no TMA row pitch)
        _case("regional_odd_mixed", "step", 397, 251, 47, steps=5, mixed=True, deep=True, cyclic=False, tripole=False),
        # quarter-degree global ocean on realistic depths: production resolution
        _case("quarter_deep_mixed", "step", 1440, 921, 55, steps=4, mixed=True, deep=True),
        _case("quarter_deep_fp64", "step", 1440, 920, 55, steps=2, deep=True),
        # eddying grid on the shallow depth map of the headline configuration
        _case("eddy_shallow_mixed", "step", 1800, 1151, 55, steps=4, mixed=True),
        # the bit-exact form with the diagnostics the reference always writes
        _case("half_diag_fp64", "step", 720, 460, 55, steps=2, diag=True, deep=True),
        # stepon: forcing from the host each step, sea ice, convection
        _case("half_coupled_mixed", "coupled", 720, 460, 55, steps=4, mixed=True, deep=True),
        # an ensemble of 1-degree members in one batch
        _case("ensemble_deg1_mixed", "ensemble", 360, 218, 30, steps=5, mixed=True, members=32),
        # the closure that produces the mixing coefficients, once per step
        _case("half_turb", "turb", 720, 460, 55, deep=True),
        # the momentum equations' biharmonic friction, once per step
        _case("half_del4u", "del4u", 720, 460, 55, deep=True),
    ]


def draw(rng):
    kind = rng.choices(["step", "coupled", "ensemble", "turb", "del4u"], [10, 3, 3, 2, 2])[0]
    top = {"step": 1440, "coupled": 900, "ensemble": 360, "turb": 720, "del4u": 720}[kind]
    nx = int(round(math.exp(rng.uniform(math.log(36), math.log(top)))))
    bounds = rng.choice([(True, True), (True, True), (True, False), (False, False)])
    if bounds[1]:
        nx += nx % 2                       # the fold pairs columns
    ny = max(24, int(nx * rng.uniform(0.55, 0.64)))
    km = rng.randint(20, 55)
    mixed = kind == "ensemble" or (kind in ("step", "coupled") and rng.random() < 0.6)
    diag = kind == "step" and not mixed and nx <= 720 and rng.random() < 0.3
    steps = {"step": rng.randint(1, 5), "coupled": rng.randint(1, 4), "ensemble": rng.randint(1, 5)}.get(kind, 1)
    members = rng.randint(2, 24) if kind == "ensemble" else 0
    return _case(None, kind, nx, ny, km, steps=steps, mixed=mixed, diag=diag, deep=rng.random() < 0.6,
                 cyclic=bounds[0], tripole=bounds[1], members=members, uneven=members > 0 and rng.random() < 0.5)


# ------------------------------------------------------------------ states
FORCING = ("SWV", "NSWV", "SST", "SSS", "FRESH", "SEAICE")
DIAGNOSTICS = ("AX", "AY", "AZ", "DZ", "PENETRATE", "TEND", "DT_DIFF")
AM_BIHAR, C0F = -1.0e17, 2.6e-3
NCC, DFRICMX = 4, 0.1


def _synth(case, seed, member=0):
    nx, ny = case["nx"], case["ny"]
    if case["uneven"]:
        nx, ny = _uneven(case, member)
    fine = nx >= 1000
    return lt.Synth(nx, ny, case["km"], seed=seed, member=member, tpert=0.01 if member else 0.0, forced=1,
                    hypsometry=int(case["deep"]), umax=0.3 if fine else 0.1, dz_top=5.0 if case["km"] > 40 else 10.0,
                    dz_bot=300.0 if case["km"] > 40 else 250.0, cap_north=0 if case["tripole"] else 3,
                    ew_cyclic=int(case["cyclic"]), tripole=int(case["tripole"]))


def _domain(case, seed, member=0):
    syn = _synth(case, seed, member)
    return syn, syn.domain(precision=lt.PREC_MIXED if case["mixed"] else lt.PREC_FP64, diagnostics=case["diag"])


def _buffer(dom, name):
    return torch.empty(dom.shape(name), dtype=torch.int32 if name in lt.INT_FIELDS else torch.float64, device="cuda")


def _get(dom, name, buf):
    """A field of the domain into a device tensor of the caller's."""
    rc = lt.lib.lt_get_field_device(dom.h, lt.FIELD_ID[name], buf.data_ptr(), buf.numel() * buf.element_size())
    if rc != lt.LT_OK:
        raise lt.LtError(rc, "lt_get_field_device(%s)" % name)
    return buf


def _set(dom, name, x):
    x = x.contiguous()
    torch.cuda.synchronize()               # the library copies on the domain's own stream
    dom.set_device(name, x.data_ptr(), x.numel() * x.element_size())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        pairs = [_domain(case, seed, m + 1) for m in range(case["members"])]
        doms = [d for _, d in pairs]
        return {"case": case, "doms": doms, "batch": lt.Batch(doms), "at": [_buffer(d, "AT") for d in doms]}
    syn, dom = _domain(case, seed)
    s = {"case": case, "dom": dom}
    if kind in ("step", "coupled"):
        s["out"] = {n: _buffer(dom, n) for n in ("AT", "NET") + (DIAGNOSTICS if case["diag"] else ())}
    if kind == "coupled":
        s["forcing"] = [torch.from_numpy(syn.field(n)).pin_memory() for n in FORCING]
        s["fw"] = torch.zeros(case["steps"], dtype=torch.float64).pin_memory()
    if kind == "turb":
        s["tab"] = lt.TurbTab(_turb_tables())
        for n, x in _turb_inputs(dom, seed).items():
            _set(dom, n, x)
        s["out"] = {n: _buffer(dom, n) for n in ("AKT", "AKMT", "AK_TIDE", "AMLD")}
    if kind == "del4u":
        for n, x in {**_del4u_stencil(dom), **_del4u_velocities(dom, seed)}.items():
            _set(dom, n, x)
        s["am"] = AM_BIHAR * (36.0 / case["nx"]) ** 4
        s["out"] = {n: _buffer(dom, n) for n in ("DLU", "DLV", "WKA_DRAG")}
    return s


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "ensemble":
        state["batch"].step(case["steps"])
        state["batch"].sync()
        return [_get(d, "AT", b) for d, b in zip(state["doms"], state["at"])]
    dom = state["dom"]
    if kind == "step":
        dom.step(case["steps"])
    elif kind == "coupled":
        ptrs = [f.data_ptr() for f in state["forcing"]]
        for k in range(case["steps"]):
            dom.step_host_async_ptrs(ptrs, state["fw"].data_ptr() + 8 * k)
            dom.icesnow()
            dom.convadj()
        dom.sync()
    elif kind == "turb":
        dom.turb(state["tab"], ncc=NCC, dfricmx=DFRICMX)
    else:
        dom.hdiffu_del4(state["am"], C0F)
    out = {n: _get(dom, n, b) for n, b in state["out"].items()}
    if "AT" in out:
        at = out.pop("AT")
        out["T"], out["S"] = at[0], at[1]
    if kind == "coupled":
        out["FW"] = state["fw"]
    return out


# -------------------------------------------------------- work, tolerances
def work(case):
    kind = case["kind"]
    cells = case["nx"] * case["ny"] * case["km"]
    if kind == "turb":      # T, density, four interface inputs, tidal structure; AKT x 2, AKMT, AK_TIDE, 3 diagnostics
        return {"bytes": 8.0 * (7 + 7) * cells, "flops": 250.0 * cells}
    if kind == "del4u":     # velocities, tendencies in and out, drag
        return {"bytes": 56.0 * cells, "flops": 110.0 * cells}
    # per cell and step: state and previous state in and out (both tracers),
    # velocities, mixing and the continuity's fields
    per = 100.0 if case["mixed"] else 240.0 if case["diag"] else 136.0
    if case["uneven"]:
        cells = sum((lambda g: g[0] * g[1])(_uneven(case, m + 1)) for m in range(case["members"])) * case["km"]
    elif case["members"]:
        cells *= case["members"]
    extra = 64.0 if kind == "coupled" else 0.0     # convection and sea ice: the state in and out once more
    return {"bytes": (per + extra) * cells * case["steps"], "flops": 400.0 * cells * case["steps"]}


def _uneven(case, member):
    """Size of one of an uneven ensemble's regional members."""
    shrink = 0.55 + 0.45 * ((member * 0.6180339887) % 1.0)
    return max(16, int(case["nx"] * shrink) // 2 * 2), max(16, int(case["ny"] * shrink))


def tolerance(case):
    if case["kind"] == "turb":
        return {"rel": 1e-9, "max": 1e-6}
    if case["kind"] == "del4u":
        return {"rel": 1e-11, "max": 1e-8}
    if case["kind"] == "coupled" and case["mixed"]:      # a nearly neutral pair of levels may mix or not
        return {"rel": 1e-6, "max": 2e-2}
    if case["mixed"]:       # f32 fluxes, and limiter decisions at near-ties (S: up to 1.4e-8 from 64 bits)
        return {"rel": 1e-7, "max": 1e-4}
    return {"rel": 1e-11, "max": 1e-8}


# ------------------------------------------- inputs of the other two kernels
MT, MT0, NTH = 1462, 400, 75     # table sizes of the closure


def _turb_tables():
    """Closure tables on the reference's grids (linear to |i| = MT0, geometric
    beyond) with smooth positive stability functions."""
    dri = 4.0 / MT0
    i = np.arange(-MT, MT + 1)
    rib = i * dri
    ratio = MT0 / (MT0 - 1.0)
    far = np.abs(i) > MT0
    rib[far] = np.sign(i[far]) * (MT0 * dri) * ratio ** (np.abs(i[far]) - MT0)
    rimax = 0.2 + 0.1 * np.tanh(0.5 * rib)
    irimax = np.clip(np.searchsorted(rib, rimax, side="right") - 1 - MT, -MT, MT).astype(np.int32)
    ri, rid = rib[None, :], rib[:, None]
    pos, neg = np.maximum(ri, 0.0), np.sqrt(np.maximum(-ri, 0.0))
    tid = np.tanh(rid)
    dth = (math.pi / 4.0) / NTH
    th = np.arange(-NTH, 3 * NTH + 1) * dth
    wrap = lambda x: x + math.pi if x < -math.pi / 4 else x  # noqa: E731
    c = np.ascontiguousarray
    tx = np.tanh(rib)
    return dict(
        rib=c(rib), irimax=c(irimax), and2on2a1=c(rib.copy()),
        slq2b=c(0.01 * np.sqrt(np.maximum(1.0 - pos / (rimax[:, None] + 1e-3), 0.0)) + 1e-4 + 0.01 * neg / (1 + 0.1 * neg)),
        smb=c(0.10 / (1 + 8 * pos) * (1 + 0.1 * tid) * (1 + 0.5 * neg / (1 + neg))),
        shb=c(0.12 / (1 + 12 * pos) * (1 + 0.2 * tid) * (1 + 0.6 * neg / (1 + neg))),
        ssb=c(0.11 / (1 + 10 * pos) * (1 - 0.1 * tid) * (1 + 0.6 * neg / (1 + neg))),
        amtaun2a1=c(0.5 + 0.1 * tx), sma1=c(0.08 + 0.01 * tx), sha1=c(0.10 + 0.02 * tx), ssa1=c(0.09 - 0.01 * tx),
        back_ra_r=c(0.3 + 0.1 * np.cos(2 * th)), sm_r1=c(0.05 + 0.01 * np.sin(th)), sh_r1=c(0.06 + 0.01 * np.cos(th)),
        ss_r1=c(0.055 + 0.01 * np.sin(2 * th)), slq2_r1=c(0.005 + 0.001 * np.cos(th)),
        rri=ratio, rnd2on2=ratio, dri=dri, dand2on2=dri, deltheta_r=dth, b1=16.6,
        theta_rcrp=wrap(math.atan(-0.5)), theta_rcrn=wrap(math.atan(-2.0)))


def _fields(dom, names):
    return {n: _get(dom, n, _buffer(dom, n)) for n in names}


def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    normal = lambda shape: torch.randn(shape, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    uniform = lambda shape: torch.rand(shape, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    return normal, uniform


def _turb_inputs(dom, seed):
    """Density of a linear equation of state, log-normal shear, Ri = N^2 / S^2,
    tidal structure decaying from the bottom: what the closure meets."""
    normal, uniform = _rng(seed)
    f = _fields(dom, ("AT", "KMT", "DZP"))
    t, s, kmt, dzp = f["AT"][0], f["AT"][1] * 1000.0 + 35.0, f["KMT"].long(), f["DZP"]
    km, jmt, imt = t.shape
    zkp = torch.zeros(km + 1, dtype=torch.float64, device="cuda")
    zkp[1:] = -torch.cumsum(dzp, 0)
    depth = -0.5 * (zkp[:-1] + zkp[1:])
    pd = torch.empty((km + 1, jmt, imt), dtype=torch.float64, device="cuda")
    pd[:km] = 1025.0 + 0.78 * (s - 35.0) - 0.17 * (t - 10.0) + 0.0006 * depth[:, None, None]
    pd[km] = pd[km - 1]
    n2 = 9.806 / 1025.0 * (pd[1:km] - pd[:km - 1]) / (0.5 * (dzp[:-1] + dzp[1:]))[:, None, None]
    n2 += 2e-6 * normal(n2.shape)
    n2[0] = n2[0].abs() + 1e-7                       # the top interface is stable
    s2 = torch.exp(math.log(5e-5) + 1.5 * normal(n2.shape))
    weak = uniform(n2.shape) < 0.01                  # strongly unstable, hardly sheared
    weak[0] = False
    n2 = torch.where(weak, -n2.abs() - 1e-5, n2)
    s2 = torch.where(weak, torch.full_like(s2, 1e-9), s2)
    rit = n2 / (s2 + 1e-25)
    lat = torch.deg2rad(88.0 - 166.0 * (torch.arange(jmt, device="cuda", dtype=torch.float64) - 2) / (jmt - 5))
    hcol = torch.where(kmt > 0, -zkp[kmt], torch.ones_like(zkp[kmt]))
    fz = torch.exp((depth[:, None, None] - hcol[None]) / 500.0)
    fz = fz / fz.sum(0, keepdim=True).clamp_min(1e-30)
    return dict(ZKP=zkp, PDENSITY=pd, RICT=n2, S2T=s2, RIT=rit, RICDTTMS=rit * (3.0 * uniform(rit.shape) - 1.5),
                FCORT=(2.0 * 7.292e-5 * torch.sin(lat))[:, None].repeat(1, imt), FZ_TIDE=fz,
                BUOYTUR=1e-8 * normal((jmt, imt)), BUOYSOL=(3e-9 * normal((jmt, imt))).abs(),
                WAVE_DIS=torch.exp(math.log(3e-3) + normal((jmt, imt))))


def _next(x, axis):
    """x(i+1) along an axis, zero beyond the end."""
    y = torch.zeros_like(x)
    n = x.shape[axis]
    y.narrow(axis, 0, n - 1).copy_(x.narrow(axis, 1, n - 1))
    return y


def _prev(x, axis):
    y = torch.zeros_like(x)
    n = x.shape[axis]
    y.narrow(axis, 1, n - 1).copy_(x.narrow(axis, 0, n - 1))
    return y


def _over(a, b):
    return torch.where(b != 0, a / torch.where(b != 0, b, torch.ones_like(b)), torch.zeros_like(b))


def _del4u_stencil(dom):
    """The friction's del4 coefficients from the grid metrics (init_del4u,
    hmix_del4.F90:88-288)."""
    f = _fields(dom, ("HUN", "HUE", "HTW", "HTS", "DXU", "DYU", "TAREA_R"))
    hun, hue, htw, hts, dxu, dyu, tr = (f[n] for n in ("HUN", "HUE", "HTW", "HTS", "DXU", "DYU", "TAREA_R"))
    one = torch.ones_like(dxu)
    uarea = dxu * dyu
    ur, dxur, dyur = _over(one, uarea), _over(one, dxu), _over(one, dyu)
    w = _over(hun, htw)
    dun, dus = w * ur, _next(w, 0) * ur
    w = _over(hue, hts)
    due, duw = w * ur, _prev(w, 1) * ur
    kxu, kyu = (hue - _prev(hue, 1)) * ur, (_next(hun, 0) - hun) * ur
    w = (_next(htw, 1) - htw) * tr
    v = 0.5 * (w + _next(w, 0))
    dxkx = (v - _prev(v, 1)) * dxur
    v = 0.5 * (w + _prev(w, 1))
    dykx = (_next(v, 0) - v) * dyur
    w = (hts - _prev(hts, 0)) * tr
    v = 0.5 * (w + _prev(w, 1))
    dyky = (_next(v, 0) - v) * dyur
    v = 0.5 * (w + _next(w, 0))
    dxky = (v - _prev(v, 1)) * dxur
    dme = _over(2.0 * kyu, hts + _prev(hts, 1))
    dms = _over(-2.0 * kxu, htw + _next(htw, 0))
    mean = uarea[uarea > 0].mean()
    return dict(DUC=-(dun + dus + due + duw), DUM=-(dxkx + dyky + 2.0 * (kxu ** 2 + kyu ** 2)), DUN=dun, DUS=dus,
                DUE=due, DUW=duw, DMC=dxky - dykx, DMN=-dms, DMS=dms, DME=dme, DMW=-dme,
                AMF=(uarea.abs() / mean) ** 1.5, UAREA_R=ur, DXUR=dxur, DYUR=dyur)


def _del4u_velocities(dom, seed, umax=0.5):
    """Gyres with small-scale noise, zero below the bottom; small tendencies."""
    normal, _ = _rng(seed)
    kmu = _fields(dom, ("KMU",))["KMU"]
    km, (jmt, imt) = dom.km, kmu.shape
    ar = lambda n: torch.arange(n, dtype=torch.float64, device="cuda")  # noqa: E731
    k = ar(km)[:, None, None]
    wet = (k < kmu[None]).double()
    decay = umax * torch.exp(-k / max(km / 3.0, 1.0))
    y, x = (2 * math.pi / jmt * ar(jmt))[None, :, None], (2 * math.pi / imt * ar(imt))[None, None, :]
    shape = (km, jmt, imt)
    up = decay * torch.sin(y) * torch.cos(2 * x) + 0.05 * umax * normal(shape)
    vp = decay * torch.cos(y) * torch.sin(x) + 0.05 * umax * normal(shape)
    return dict(UP=up * wet, VP=vp * wet, DLU=1e-6 * normal(shape) * wet, DLV=1e-6 * normal(shape) * wet)


# ------------------------------------------------------- 64-bit restatement
def _w(x):
    return torch.roll(x, 1, -1)      # the value at i-1


def _e(x):
    return torch.roll(x, -1, -1)     # at i+1


def _n(x):
    return torch.roll(x, 1, -2)      # at j-1 (north)


def _s(x):
    return torch.roll(x, -1, -2)     # at j+1


def _up(x):
    """The level above (itself at the top); [km][...]."""
    return torch.cat([x[:1], x[:-1]])


def _dn(x):
    return torch.cat([x[1:], x[-1:]])


def _halo(x, cyclic, tripole):
    """Ghost cells of [...][jmt][imt] in place: east-west copies, then the fold
    of the top rows with its averaged first row."""
    imt, jmt = x.shape[-1], x.shape[-2]
    nx = imt - 4
    if cyclic:
        x[..., 2:jmt - 2, 0:2] = x[..., 2:jmt - 2, nx:nx + 2].clone()
        x[..., 2:jmt - 2, nx + 2:nx + 4] = x[..., 2:jmt - 2, 2:4].clone()
    if not tripole:
        return x
    buf = x[..., 2:5, 2:2 + nx].clone()               # columns g = 1 .. nx at index g - 1
    g = torch.arange(1, nx // 2, device=x.device)
    mean = 0.5 * (buf[..., 0, g - 1] + buf[..., 0, nx - g - 1])
    buf[..., 0, g - 1] = mean
    buf[..., 0, nx - g - 1] = mean
    i = torch.arange(1, imt + 1, device=x.device) - 2  # global column of each local one
    src = nx - torch.where(i < 1, i + nx if cyclic else 0 * i, torch.where(i > nx, i - nx if cyclic else 0 * i, i))
    src = torch.where(src == 0, torch.full_like(src, nx), src)
    for jf in (1, 2, 3):
        x[..., jf - 1, :] = buf[..., 3 - jf, :][..., src - 1]
    return x


def _col(v):
    return v[:, None, None]


class _Exact:
    """The tracer step on plain f64 tensors (tracer.cpp:1701-1903, tspas)."""

    def __init__(self, dom, case, forcing=None):
        names = ["AT", "ATB", "UTF", "VTF", "UTL", "VTL", "AKT", "H0F", "H0L", "NET", "KMT", "TAREA", "TAREA_R", "HTW",
                 "HTS", "HUN", "HUE", "AHF", "DTN", "DTS", "DTE", "DTW", "OHBT", "OHBU", "AU0", "AUS", "AUW", "AUSW",
                 "DZP", "ODZP", "ODZT", "PEN", "TO", "SO", "C", "QICE", "WS", "KMTN", "KMTS", "KMTE", "KMTW"]
        self.f = _fields(dom, names + list(FORCING))
        self.p, self.case = dom.params, case
        self.at = self.f["AT"]
        self.atb = self.f["ATB"][:, 1:].clone()
        self.net = self.f["NET"]
        self.kmt = self.f["KMT"].long()
        km = dom.km
        lev = torch.arange(km, device="cuda")[:, None, None]
        self.lev = lev
        self.vit = (lev < self.kmt[None]).double()
        self.wet = lev < self.kmt[None]
        self._dynamics()

    def _dynamics(self):
        f, p = self.f, self.p
        ssh = 0.5 * f["H0F"] * p.onbc + 0.5 * f["H0L"]
        wkd = 0.5 * f["UTF"] * p.oncc + 0.5 * f["UTL"]
        wkb = 0.5 * f["VTF"] * p.oncc + 0.5 * f["VTL"]
        for n in ("UTF", "UTL", "VTF", "VTL"):
            del f[n]
        fac = 1.0 + f["OHBU"] * (f["AU0"] * ssh + f["AUS"] * _s(ssh) + f["AUW"] * _w(ssh) + f["AUSW"] * _s(_w(ssh)))
        fac[-1, :] = 0.0
        fac[:, 0] = 0.0
        uk, vk = wkd * fac, wkb * fac
        fx, fy = (uk + _n(uk)) * f["HTW"], (vk + _e(vk)) * f["HTS"]
        del uk, vk
        div = 0.5 * (_e(fx) - fx + fy - _n(fy)) * f["TAREA_R"] * self.vit
        del fx, fy
        inner = torch.zeros_like(f["TAREA"], dtype=torch.bool)
        inner[1:-1, 1:-1] = True
        wsum = -(f["DZP"][:, None, None] * div).sum(0)
        ws = f["WS"]
        for k in range(1, div.shape[0]):
            nw = self.vit[k] * (ws[k - 1] + f["DZP"][k - 1] * (wsum * f["OHBT"] + div[k - 1]))
            ws[k] = torch.where(inner, nw, ws[k])
        ws[1:-1] = torch.where(inner, ws[1:-1] / (1.0 + ssh * f["OHBT"]), ws[1:-1])
        self.ws = ws[:-1]
        self.wsd = torch.cat([ws[1:-1], torch.zeros_like(ws[:1])])
        self.uw, self.vs = (wkd + _n(wkd)) * f["HTW"] * 0.25, (wkb + _e(wkb)) * f["HTS"] * 0.25
        self.ssh = ssh

    def step(self):
        f, p, dts = self.f, self.p, self.p.dts
        tr, odzp, odzt = f["TAREA_R"], _col(f["ODZP"]), _col(f["ODZT"])
        odzt_d = torch.cat([odzt[1:], torch.zeros_like(odzt[:1])])
        hor = 2.0 * dts * tr
        uw, vs, ws, wsd, vit = self.uw, self.vs, self.ws, self.wsd, self.vit
        jmt, imt = tr.shape
        ring = torch.zeros_like(tr, dtype=torch.bool)
        ring[1:-1, 1:-1] = True
        inner = torch.zeros_like(ring)
        inner[2:-2, 2:-2] = True
        kmt, wet = self.kmt, self.wet
        # surface forcing from the previous state
        top = self.atb[:, 0]
        ocean = kmt > 0
        o0 = f["ODZP"][0]
        salt = f["FRESH"] * 34.7 * p.od0 / 1000.0 + p.gamma * (f["SSS"] - top[1]) * f["SEAICE"] / o0 \
            + p.gamma * 30.0 / 365.0 / 4.0 * 50.0 * (f["SSS"] - top[1]) / o0 * (1.0 - f["SEAICE"])
        heat = (f["SWV"] + f["NSWV"]) * p.od0cp + f["SEAICE"] * p.gamma * (f["SST"] - top[0]) / o0
        stf = [torch.where(ocean, x, torch.zeros_like(x)) for x in (heat, salt)]
        self.net[0] = torch.where(ocean, heat * o0, self.net[0])
        self.net[1] = torch.where(ocean, salt * o0, self.net[1])
        self.fw = -float((f["TAREA"] * self.net[1] * vit[0])[2:-2, 2:-2].sum()) / p.area_t
        _halo(self.net, self.case["cyclic"], self.case["tripole"])
        surf = f["AKT"][0, 0]
        f["AKT"][0, 0, 1:-1, 1:-1] = surf[1:-1, 1:-1].clamp_min(p.dwndmix)
        # masks of the Laplacian's neighbours
        near = [wet & (self.lev < f[m].long()[None]) for m in ("KMTN", "KMTS", "KMTE", "KMTW")]

        def lap(x):
            h = torch.zeros_like(x)
            for m, c, nb in zip(near, ("DTN", "DTS", "DTE", "DTW"), (_n, _s, _e, _w)):
                h += torch.where(m, f[c] * (nb(x) - x), torch.zeros_like(x))
            return h

        self.diag = {}
        for tracer in range(2):
            a = self.at[tracer]
            de, dw, ds, dn = _e(a) - a, a - _w(a), _s(a) - a, a - _n(a)
            du, dd = _up(a) - a, a - _dn(a)           # above minus here, here minus below
            lw = [hor * _e(uw) ** 2 / _e(f["HTW"] * f["HUN"]) * de, hor * uw ** 2 / (f["HTW"] * f["HUN"]) * dw,
                  hor * vs ** 2 / (f["HTS"] * f["HUE"]) * ds, hor * _n(vs) ** 2 / _n(f["HTS"] * f["HUE"]) * dn]
            lw = [torch.where(ring, x, torch.zeros_like(x)) for x in lw]
            zu, zd = 0.5 * odzp * dts * ws ** 2 * odzt * du, 0.5 * odzp * dts * wsd ** 2 * odzt_d * dd
            cx, cy = -tr * (_e(uw) * de + uw * dw), -tr * (vs * ds + _n(vs) * dn)
            cz = -0.5 * odzp * (ws * du + wsd * dd)
            pred = a + dts * (cx + lw[0] - lw[1] + cy + lw[2] - lw[3] + cz + zu - zd)
            big = torch.where(wet, a, torch.full_like(a, -1.0e10))
            small = torch.where(wet, a, torch.full_like(a, 1.0e10))
            hi, lo = big, small
            for nb in (_n, _s, _w, _e, _up, _dn):
                hi, lo = torch.maximum(hi, nb(big)), torch.minimum(lo, nb(small))
            out = ((pred > hi) | (pred < lo)) & ring
            del pred, big, small, hi, lo
            # between the top and bottom level a face on the region's rim keeps its form
            i, j = torch.arange(imt, device="cuda")[None, :], torch.arange(jmt, device="cuda")[:, None]
            edge = (self.lev == 0) | (self.lev == a.shape[0] - 1)
            rim = [edge | m for m in (i <= imt - 3, i >= 2, j <= jmt - 3, j >= 2)]
            fl = [torch.where((out | nb(out)) & g, tr * u.abs() * d, x) for nb, u, d, x, g in
                  zip((_e, _w, _s, _n), (_e(uw), uw, vs, _n(vs)), (de, dw, ds, dn), lw, rim)]
            zu = torch.where(out | _up(out), 0.5 * odzp * ws.abs() * du, zu)
            zd = torch.where(out | _dn(out), 0.5 * odzp * wsd.abs() * dd, zd)
            ax, ay, az = cx + fl[0] - fl[1], cy + fl[2] - fl[3], cz + zu - zd
            del lw, fl, zu, zd, cx, cy, cz, out, de, dw, ds, dn, du, dd
            tf = (ax + ay + az) * vit
            b = self.atb[tracer]
            d2 = torch.where(ring, f["AHF"] * lap(b), torch.zeros_like(b))
            tf += p.ah * lap(d2)
            del d2
            akt = f["AKT"][tracer]
            below = torch.cat([vit[1:], torch.zeros_like(vit[:1])])
            if tracer == 0:
                pen = _col(f["PEN"])
                sw = f["SWV"] * (torch.cat([torch.zeros_like(pen[:1]), pen[:-1]]) * vit - pen * below)
                sw[0] = -f["SWV"] * pen[0] * vit[1]
                tf += sw * odzp
                self.diag["PENETRATE"] = sw * odzp * inner
            w1 = torch.zeros_like(b)
            w1[1:] = akt[:-1] * (b[:-1] - b[1:]) * odzt[1:] * vit[1:]
            mix = 0.5 * odzp * (w1 - torch.cat([w1[1:], torch.zeros_like(w1[:1])]))
            tf += mix
            tf[0] += stf[tracer] * 0.5 * o0
            if tracer == 1:
                tf[0] += self.fw * vit[0]
            new = a.clone()
            new[:, 2:-2, 2:-2] = (a + dts * tf)[:, 2:-2, 2:-2]
            # implicit half of the vertical mixing, from the bottom up
            km = a.shape[0]
            e, g = torch.zeros_like(tr), torch.zeros_like(tr)
            es, fs = torch.empty_like(a), torch.empty_like(a)
            for k in range(km - 1, -1, -1):
                last = kmt == k + 1
                a8 = akt[k - 1] * odzt[k] * odzp[k] * dts * 0.5 if k else odzp[0] * dts * 0.5 + 0 * tr
                c8 = torch.where(last, odzp[k] * dts * 0.5 + 0 * tr,
                                 akt[k] * odzt[k + 1] * odzp[k] * dts * 0.5 if k < km - 1 else 0 * tr)
                b8 = torch.where(last, 1.0 + a8, 1.0 + c8 + (a8 if k else 0.0))
                here = k < kmt
                r = 1.0 / (b8 - c8 * e)
                g = torch.where(here, (new[k] + c8 * g) * r, torch.zeros_like(tr))
                e = torch.where(here, a8 * r, torch.zeros_like(tr))
                es[k], fs[k] = e, g
            x = stf[tracer]
            for k in range(km):
                x = es[k] * x + fs[k]
                new[k] = torch.where(inner & (k < kmt), x, new[k])
            del es, fs
            _halo(new, self.case["cyclic"], self.case["tripole"])
            if self.case["diag"]:
                for n, v in (("AX", ax * ring), ("AY", ay * ring), ("AZ", az * ring), ("DZ", mix * inner),
                             ("TEND", (new - a) / dts * vit)):
                    self.diag.setdefault(n, [None, None])[tracer] = v
            del ax, ay, az, tf, mix, w1
            self.at[tracer] = new
            self.atb[tracer] = new

    def icesnow(self):
        f, at = self.f, self.at
        t, s = at[0, 0], at[1, 0]
        brine = (34.7 - 4.0) * 3996.0 / 3.337e5 * 0.001
        cold = (t < -1.8) & (self.kmt > 0)
        d = torch.where(cold, -1.8 - t, torch.zeros_like(t))
        s += d * brine
        t.copy_(torch.where(cold, torch.full_like(t, -1.8), t))
        at[0].clamp_min_(-1.8)

    def convadj(self):
        """Convective adjustment (convadj.cpp:29-288), every column at once:
        mix the shallowest unstable pair, grow it down and up, go on below."""
        f = self.f
        km = self.at.shape[1]
        cols = (self.kmt.reshape(-1) > 1).nonzero()[:, 0]
        x = [self.at[n].reshape(km, -1)[:, cols].clone() for n in range(2)]
        kcon = self.kmt.reshape(-1)[cols]
        to, so, dz, cc = f["TO"], f["SO"], f["DZP"], f["C"].reshape(9, km)

        def rho(t, s, l):
            t, s, c = t - to[l], s - so[l], cc[:, l]
            return (c[0] + (c[3] + c[6] * s) * s + (c[2] + c[7] * s + c[5] * t) * t) * t + (c[1] + (c[4] + c[8] * s) * s) * s

        lv = torch.arange(km, device="cuda")[:, None]
        up, lo = torch.zeros_like(x[0]), torch.zeros_like(x[0])
        for l in range(km - 1):
            up[l + 1] = rho(x[0][l + 1], x[1][l + 1], l + 1)
            lo[l] = rho(x[0][l], x[1][l], l + 1)
        bad = torch.zeros_like(lo, dtype=torch.bool)
        bad[:-1] = (lo[:-1] > up[1:]) & (lv[:-1] + 1 < kcon)
        some = bad.any(0).nonzero()[:, 0]
        if some.numel():
            y, kc = [v[:, some] for v in x], kcon[some]
            up, lo = up[:, some], lo[:, some]
            n = torch.arange(some.numel(), device="cuda")
            at_ = lambda v, l: v[l, n]  # noqa: E731
            l_a = bad[:, some].long().argmax(0)       # 0-based top and bottom of the mixed stretch
            l_b = l_a + 1
            live = torch.ones_like(l_a, dtype=torch.bool)
            dzs = dz[l_a] + dz[l_b]
            tot = [at_(v, l_a) * dz[l_a] + at_(v, l_b) * dz[l_b] for v in y]

            def spread(where):
                inside = (lv >= l_a) & (lv <= l_b) & where
                for v, q in zip(y, tot):
                    v.copy_(torch.where(inside, (q / dzs).expand_as(v), v))

            spread(live)
            while bool(live.any()):
                can = live & (l_b + 1 != kc)
                nb = torch.where(can, l_b + 1, l_b)
                r = rho(at_(y[0], l_b), at_(y[1], l_b), nb)
                lo[l_b, n] = torch.where(can, r, lo[l_b, n])
                down = can & (r > at_(up, nb))
                look = live & ~down & (l_a > 0)
                na = torch.where(look, l_a - 1, l_a)
                r = rho(at_(y[0], na), at_(y[1], na), l_a)
                q = rho(at_(y[0], l_a), at_(y[1], l_a), l_a)
                lo[na, n] = torch.where(look, r, lo[na, n])
                up[l_a, n] = torch.where(look, q, up[l_a, n])
                rise = look & (r > q)
                grow = down | rise
                l_b = torch.where(down, nb, l_b)
                l_a = torch.where(rise, na, l_a)
                new = torch.where(down, l_b, l_a)
                dzs = torch.where(grow, dzs + dz[new], dzs)
                tot = [torch.where(grow, q + at_(v, new) * dz[new], q) for v, q in zip(y, tot)]
                spread(grow)
                # neither way: the next unstable pair below, or done
                stop = live & ~grow
                pair = torch.zeros_like(lo, dtype=torch.bool)
                pair[:-1] = (lo[:-1] > up[1:]) & (lv[:-1] + 1 < kc) & (lv[:-1] > l_b) & stop
                again = pair.any(0)
                nl = pair.long().argmax(0)
                l_a = torch.where(again, nl, l_a)
                l_b = torch.where(again, nl + 1, l_b)
                dzs = torch.where(again, dz[l_a] + dz[l_b], dzs)
                tot = [torch.where(again, at_(v, l_a) * dz[l_a] + at_(v, l_b) * dz[l_b], q) for v, q in zip(y, tot)]
                spread(again)
                live = live & (grow | again)
            for v, w in zip(x, y):
                v[:, some] = w
        for n_, v in enumerate(x):
            flat = self.at[n_].reshape(km, -1)
            flat[:, cols] = v
        self.atb.copy_(self.at)


def _exact_del4u(dom, am):
    f = _fields(dom, ("UP", "VP", "DLU", "DLV", "KMT", "KMU", "HTW", "HTS", "TAREA_R", "DXU", "DYU", "DUC", "DUM", "DUN",
                      "DUS", "DUE", "DUW", "DMC", "DMN", "DMS", "DME", "DMW", "AMF", "UAREA_R", "DXUR", "DYUR"))
    u, v = f["UP"], f["VP"]
    km, jmt, imt = u.shape
    lev = torch.arange(km, device="cuda")[:, None, None]
    wet_t, wet_u = lev < f["KMT"], lev < f["KMU"]
    j, i = torch.arange(jmt, device="cuda")[:, None], torch.arange(imt, device="cuda")[None, :]
    zero = torch.zeros_like(u)
    fx, fy = (u + _n(u)) * f["HTW"], (v + _e(v)) * f["HTS"]
    div = torch.where(wet_t & (i < imt - 1) & (j >= 1), 0.5 * (_e(fx) - fx + fy - _n(fy)) * f["TAREA_R"], zero)
    cx, cy = u * f["DXU"], v * f["DYU"]
    cy, cx = cy + _n(cy), cx + _w(cx)
    curl = torch.where(wet_t & (i >= 1) & (j >= 1), 0.5 * (cy - _w(cy) - cx + _n(cx)), zero)
    fac = torch.zeros_like(u)
    for q in (div, curl):
        gx = f["DXUR"] * 0.5 * (_s(q) - _w(q) - _s(_w(q)) + q)
        gy = f["DYUR"] * 0.5 * (_s(q) - _w(q) + _s(_w(q)) - q)
        fac += torch.where(wet_u & (i >= 1) & (j < jmt - 1), gx ** 2 + gy ** 2, zero)
    area = torch.sqrt(1.0 / f["UAREA_R"])
    here = wet_u & (j >= 1) & (j <= jmt - 2) & (i >= 1) & (i <= imt - 2)
    amf = (torch.sqrt(fac) * area ** 5 * 45.0 / (am * f["AMF"]).abs()).clamp(1.0, 40.0)

    def lap(a, b, sign):
        c = f["DUC"] + f["DUM"]
        return (c * a + f["DUN"] * _n(a) + f["DUS"] * _s(a) + f["DUE"] * _e(a) + f["DUW"] * _w(a)) + sign * (
            f["DMC"] * b + f["DMN"] * _n(b) + f["DMS"] * _s(b) + f["DME"] * _e(b) + f["DMW"] * _w(b))

    pu = torch.where(here, amf * f["AMF"] * lap(u, v, 1.0), zero)
    pv = torch.where(here, amf * f["AMF"] * lap(v, u, -1.0), zero)
    own = wet_u & (j >= 2) & (j < jmt - 2) & (i >= 2) & (i < imt - 2)
    return {"DLU": f["DLU"] + torch.where(own, am * lap(pu, pv, 1.0), zero),
            "DLV": f["DLV"] + torch.where(own, am * lap(pv, pu, -1.0), zero), "WKA_DRAG": C0F * torch.sqrt(u ** 2 + v ** 2)}


def _exact_turb(dom):
    """The tidal mixing and the mixed-layer depth; the closure's own values
    hang on table look-ups that have no plain form."""
    f = _fields(dom, ("AT", "PDENSITY", "DZP", "ZKP", "KMT", "WAVE_DIS", "FZ_TIDE", "RICT"))
    t, pd, dz, n = f["AT"][0], f["PDENSITY"], f["DZP"], f["KMT"].long() - 1
    km, jmt, imt = t.shape
    part = (dz[:-1] / (dz[:-1] + dz[1:]))[:, None, None]
    ti, rh = t[:-1] - (t[:-1] - t[1:]) * part, pd[:km - 1] + (pd[1:km] - pd[:km - 1]) * part
    lev = torch.arange(km - 1, device="cuda")[:, None, None]
    tide = 1.0e-6 + 0.2 * 0.33 * f["WAVE_DIS"] * f["FZ_TIDE"][:-1] / (f["RICT"].clamp_min(1.0e-8) * rh)
    tide = tide.clamp_max(1.0e-2)
    tide = torch.where(lev < n, tide, torch.full_like(tide, 1.0e-2))
    tide = torch.flip(torch.cummin(torch.flip(tide, (0,)), 0).values, (0,))
    inside = torch.zeros((jmt, imt), dtype=torch.bool, device="cuda")
    inside[1:-1, 1:-1] = True
    col = inside & (n >= 0)
    out = torch.zeros_like(t)
    out[:-1] = torch.where(col & (lev < n), tide, torch.zeros_like(tide))
    z = -f["ZKP"][1:] * 100.0
    far = ((ti - ti[:1]).abs() > 0.1) & (lev < n) & (lev >= 1)
    k = far.long().argmax(0)
    k1 = k.clamp_min(1)
    take = lambda v, q: torch.gather(v, 0, q[None])[0]  # noqa: E731
    t0, tk, tp = ti[0], take(ti, k1), take(ti, k1 - 1)
    tm = t0 - torch.where(t0 - tk >= 0, 0.1 + 0 * t0, -0.1 + 0 * t0)
    depth = z[k1] + (z[k1 - 1] - z[k1]) * (tm - tk) / (tp - tk + 1.0e-20)
    depth = torch.where(far.any(0), depth, torch.where(n > 0, z[(n - 1).clamp_min(0)], torch.zeros_like(depth)))
    return {"AKT": None, "AKMT": None, "AK_TIDE": out, "AMLD": torch.where(col, depth * 0.01, torch.zeros_like(depth))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for m in range(case["members"]):
            _, dom = _domain(case, seed, m + 1)
            x = _Exact(dom, case)
            for _k in range(case["steps"]):
                x.step()
            out.append(x.at)
        return out
    if kind in ("turb", "del4u"):
        s = prepare(case, seed)
        return _exact_turb(s["dom"]) if kind == "turb" else _exact_del4u(s["dom"], s["am"])
    _, dom = _domain(case, seed)
    x, fw = _Exact(dom, case), []
    dom.close()
    for _k in range(case["steps"]):
        x.step()
        fw.append(x.fw)
        if kind == "coupled":
            x.icesnow()
            x.convadj()
    out = {"T": x.at[0], "S": x.at[1], "NET": x.net}
    if kind == "coupled":
        out["FW"] = torch.tensor(fw, dtype=torch.float64)
    if case["diag"]:
        out.update({n: torch.stack(v) if isinstance(v, list) else v for n, v in x.diag.items()})
        out["DT_DIFF"] = None
    return out
