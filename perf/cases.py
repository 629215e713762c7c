"""Workloads of the dynamical core, from a 64 x 64 x 65 boundary layer to a 1024 x 1024 x 200 moist layer.

Each case is a model restarted from a turbulent state (as from a checkpoint, so that its steps are
centred) and one pass is a call a host program makes between two looks at the fields: some whole
timesteps, or the adjoint of a window of them, and the fields it then reads on the GPU.  FP64
models return FP64 fields, FP32-mixed ones the FP32 values they hold.

`exact` restates the timestep in plain torch in FP64, whole fields at a time.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from monc_b200 import api, config as cf

ADJ_OUT = ("u", "v", "w", "th", "zu", "zv", "zw", "zth")


def _case(name, **kw):
    c = {"physics": "dry", "kind": "step", "precision": "fp64", "nx": 64, "ny": 64, "nz": 65, "dx": 50.0, "dz": 25.0,
         "dt": 1.0, "wind": 5.0, "steps": 10, "tracers": 0, "flow": "pw", "solver": "fft", "forcing": False,
         "watch": False}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a teaching-size convective boundary layer whose host program looks at the mean profiles
        # after every step: launches and latency
        _case("dry_64x64x65_watched", wind=0.0, steps=12, watch=True),
        # the dry boundary layer the throughput figures are quoted on, in both precisions
        _case("dry_256x256x128_fp64", nx=256, ny=256, nz=128, dx=25.0, dz=15.0, dt=0.5),
        _case("dry_256x256x128_fp32", nx=256, ny=256, nz=128, dx=25.0, dz=15.0, dt=0.5, precision="fp32"),
        # the stratocumulus-like layer of the precision comparison
        _case("moist_512x512x160_fp64", physics="moist", nx=512, ny=512, nz=160, dx=35.0, dz=5.0, dt=0.3, steps=4),
        _case("moist_512x512x160_fp32", physics="moist", nx=512, ny=512, nz=160, dx=35.0, dz=5.0, dt=0.3, steps=4,
              precision="fp32"),
        # the largest single-GPU run: a deep moist layer with three tracers
        _case("tracers_1024x1024x200_fp32", physics="moist", nx=1024, ny=1024, nz=200, dx=25.0, dz=10.0, dt=0.5,
              steps=2, tracers=3, precision="fp32"),
        # a domain of another shape: lengths with factors 3 and 5, an odd number of levels, sizes that
        # no tile divides
        _case("dry_360x300x81_fp64", nx=360, ny=300, nz=81, dx=25.0, dz=15.0, dt=0.5),
        # the flow advected by TVD instead of Piacsek-Williams
        _case("tvdflow_256x256x128_fp64", nx=256, ny=256, nz=128, dx=25.0, dz=15.0, dt=0.5, steps=6, flow="tvd"),
        # the options most test cases of the reference switch on: damping layer, subsidence, adaptive
        # timestep and the Galilean frame, with the profile diagnostics read once a pass
        _case("forced_128x128x96_fp64", nx=128, ny=128, nz=96, dz=20.0, steps=12, forcing=True),
        # the iterative pressure solver at the reference's default tolerance
        _case("bicgstab_256x256x64_fp64", physics="moist", nx=256, ny=256, nz=64, dx=35.0, dz=10.0, dt=0.3, steps=3,
              solver="bicgstab"),
        # the reference's own driver calling the drop-in components one at a time
        _case("components_128x128x96_fp64", kind="components", nx=128, ny=128, nz=96, dz=20.0, steps=4),
        # the gradient of a window of steps with respect to its initial state
        _case("adjoint_128x128x96_fp64", kind="adjoint", nx=128, ny=128, nz=96, dz=20.0, wind=0.0, steps=30),
    ]


def _lengths(lo, hi):
    """Even lengths lo .. hi with no prime factor above 5."""
    out = []
    for n in range(lo + lo % 2, hi + 1, 2):
        m = n
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        if m == 1:
            out.append(n)
    return out


def draw(rng):
    """A case of the listed kinds on a grid drawn over the logarithm of its size."""
    kind = rng.choices(("step", "components", "adjoint"), (10, 1, 2))[0]
    small = kind != "step"
    physics = "moist" if kind == "step" and rng.random() < 0.45 else "dry"
    solver = rng.choices(("fft", "bicgstab", "cg"), (7, 1, 1))[0] if kind == "step" else "fft"
    small = small or solver != "fft"
    sizes = _lengths(32, 160 if small else 640)
    pick = lambda: min(sizes, key=lambda n, t=math.log(sizes[0]) + rng.random() * math.log(sizes[-1] / sizes[0]):
                       abs(math.log(n) - t))  # noqa: E731
    # half of the drawn grids have power-of-two lengths, as most runs do
    nx, ny = (1 << rng.randint(5, 7 if small else 9), 1 << rng.randint(5, 7 if small else 9)) if rng.random() < 0.5 \
        else (pick(), pick())
    nz = int(round(math.exp(rng.uniform(math.log(24), math.log(160)))))
    forcing = kind == "step" and physics == "dry" and solver == "fft" and rng.random() < 0.3
    tvd = kind == "step" and physics == "dry" and not forcing and rng.random() < 0.3
    return _case(None, kind=kind, physics=physics, solver=solver, nx=nx, ny=ny, nz=nz, forcing=forcing,
                 precision="fp32" if kind == "step" and not forcing and rng.random() < 0.4 else "fp64",
                 dx=rng.choice((25.0, 35.0, 50.0)), dz=rng.choice((5.0, 10.0)) if physics == "moist" else 1600.0 / nz,
                 dt=rng.choice((0.3, 0.5)), wind=rng.choice((0.0, 5.0)),
                 steps={"step": 4, "components": 2, "adjoint": rng.randint(6, 20)}[kind],
                 tracers=rng.randint(1, 3) if physics == "moist" and rng.random() < 0.3 else 0,
                 flow="tvd" if tvd else "pw",
                 watch=kind == "step" and rng.random() < 0.2)


# ---- configuration and initial state ------------------------------------------------------------
def _levels(case):
    """w-level heights: uniform for the dry layers, stretched up to 20 or 50 m for the moist ones."""
    nz = case["nz"]
    if case["physics"] == "dry":
        return case["dz"] * np.arange(nz)
    if case["tracers"]:
        return cf.stretched_levels(nz, case["dz"], 50.0, ztop=30.0 * nz)
    return cf.stretched_levels(nz, case["dz"], 20.0)


def _config(case):
    prec = cf.FP32_MIXED if case["precision"] == "fp32" else cf.FP64
    solver = cf.SOLVER_FFT if case["solver"] == "fft" else cf.SOLVER_ITERATIVE
    nx, ny, nz, dx, dt = case["nx"], case["ny"], case["nz"], case["dx"], case["dt"]
    if case["physics"] == "dry":
        c = cf.dry_cbl_config(nx, ny, nz, dx, case["dz"], dt, ug=case["wind"], fcoriol=1e-4 if case["wind"] else 0.0,
                              precision=prec, solver=solver)
    else:
        deep = case["tracers"] > 0
        c = cf.moist_config(nx, ny, _levels(case), dx, dt, shf_wm2=150.0 if deep else 0.0,
                            lhf_wm2=200.0 if deep else 0.0, max_height_cloud=5000.0 if deep else 20000.0,
                            n_tracers=case["tracers"], precision=prec, solver=solver)
    if case["solver"] == "cg":
        c.solver_type = cf.ITER_CG
    if case["flow"] == "tvd":
        c.advection_flow_fields = cf.ADVECT_TVD
    if case["forcing"]:
        top = float(_levels(case)[-1])
        cf.enable_damping(c, 0.001, 0.75 * top, 0.2 * top)
        cf.enable_subsidence(c, [0.0, 0.5 * top, top], [0.0, -0.005, -0.005])
        cf.enable_cfl(c, dtmmax=2.0 * dt)
        cf.enable_galilean(c)
        c.profile_diagnostics_enabled = 1
    return c


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _eddies(shape, gen):
    """Random eddies of unit variance: noise with a k^(-4/3) horizontal amplitude spectrum, smooth in z."""
    nz, ny, nx = shape
    dev = gen.device
    a = torch.randn(shape, generator=gen, device=dev, dtype=torch.float32)
    ky = torch.fft.fftfreq(ny, device=dev)[:, None] * ny
    kx = torch.fft.rfftfreq(nx, device=dev)[None, :] * nx
    spectrum = (9.0 + kx * kx + ky * ky) ** (-2.0 / 3.0)
    for k in range(0, nz, 16):  # a few levels at a time: the largest grids' spectra are as large as the fields
        a[k:k + 16] = torch.fft.irfft2(torch.fft.rfft2(a[k:k + 16]) * spectrum, s=(ny, nx))
    for _ in range(2):
        lo, hi = torch.cat([a[:1], a[:-1]]), torch.cat([a[1:], a[-1:]])
        a = 0.25 * lo + 0.5 * a + 0.25 * hi
    return a / a.std()


def _state(case, seed):
    """(name, field) pairs of a turbulent boundary layer under an inversion, each [nz][ny][nx] FP64,
    the fields of the previous time level (z...) a little behind.  One field at a time, so that
    the largest state need not be held twice."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * (int(seed) % 1000000007) + 17)
    z = torch.tensor(_levels(case), device=dev, dtype=torch.float32)[:, None, None]
    shape = (case["nz"], case["ny"], case["nx"])
    moist = case["physics"] == "moist"
    top = float(z[-1])
    zi = min(840.0, 0.6 * top) if moist else min(800.0, 0.6 * top)
    env = 0.05 + 0.95 * torch.sigmoid((zi - z) / (0.06 * zi))
    hill = env * (4.0 * z / top * (1.0 - z / top)).clamp(min=0.0)
    above = (z > zi).float()
    fields = [("u", lambda e: case["wind"] + 0.8 * env * e), ("v", lambda e: 0.8 * env * e), ("w", lambda e: 0.6 * hill * e)]
    if moist:
        fields.append(("th", lambda e: above * (8.5 + 0.00365 * (z - zi)) + 0.15 * env * e))
        fields.append(("q0", lambda e: 9e-3 - 7.5e-3 * above + 1.5e-4 * env * e))
    else:
        fields.append(("th", lambda e: above * 0.003 * (z - zi) + 0.15 * env * e))
    for name, make in fields:
        f = make(_eddies(shape, gen))
        if name == "w":  # rigid lid and ground
            f[0] = 0.0
            f[-1] = 0.0
        yield name, f.double()
        yield "z" + name, (0.97 * f + 0.03 * torch.roll(f, 1, 2)).double()
    if moist:
        zero = torch.zeros(shape, device=dev, dtype=torch.float64)
        yield "q1", zero
        yield "zq1", zero
        for t in range(case["tracers"]):
            f = torch.exp(0.5 * _eddies(shape, gen)) * torch.exp(-z / 200.0)
            yield f"q{2 + t}", f.double()
            yield f"zq{2 + t}", (0.97 * f + 0.03 * torch.roll(f, 1, 2)).double()


def _seeds(case, seed):
    """Gradients of an objective with respect to the window's final u, v, w, th."""
    gen = torch.Generator(device=_device())
    gen.manual_seed(1000003 * (int(seed) % 1000000007) + 29)
    shape = (case["nz"], case["ny"], case["nx"])
    out = {}
    for n in ("u", "v", "w", "th"):
        g = _eddies(shape, gen).double()
        if n == "w":
            g[0] = 0.0
            g[-1] = 0.0
        out[n] = g
    return out


def _mean_rows(case, fields):
    """The mean profiles a checkpoint carries (dry models): olz*bar, then ol*bar."""
    return np.stack([fields[n].mean(dim=(1, 2)).cpu().numpy() for n in ("zu", "zv", "zth", "u", "v", "th")])


def _outputs(case):
    q = [] if case["physics"] == "dry" else [f"q{n}" for n in range(2 + case["tracers"])]
    return ["u", "v", "w", "th"] + q + (["p"] if case["precision"] == "fp64" else [])


# ---- the measured program -------------------------------------------------------------------------
def prepare(case, seed):
    cfg = _config(case)
    model = api.Model(cfg)
    keep = case["kind"] == "adjoint" or case["forcing"]
    fields = {}
    for name, f in _state(case, seed):
        model.upload_tensor(name, f)
        if keep:
            fields[name] = f
    meta = api.CheckpointMeta(timestep=2, last_cfl_timestep=2, time=2.0 * case["dt"], dtm=case["dt"],
                              dtm_new=case["dt"], absolute_new_dtm=case["dt"])
    model.restore_state(meta, _mean_rows(case, fields) if case["forcing"] else None)
    st = {"case": case, "model": model, "meta": meta}
    if case["kind"] == "adjoint":
        st["fields"] = fields
        st["seeds"] = _seeds(case, seed)
        st["zero"] = torch.zeros_like(fields["u"])
    return st


def run(state):
    case, m = state["case"], state["model"]
    dev = torch.device("cuda")
    if case["kind"] == "adjoint":
        # the gradient at the current iterate: its state in, the adjoint of the window out
        for name, f in state["fields"].items():
            m.upload_tensor(name, f)
        m.restore_state(state["meta"])
        for name in ADJ_OUT:
            m.upload_tensor("adj:" + name, state["seeds"].get(name, state["zero"]))
        mixing = m.adjoint_run(case["steps"], 10)
        out = {name: m.download_tensor("adj:" + name, dev) for name in ADJ_OUT}
        out["mixing"] = mixing
        return out
    out = {}
    if case["kind"] == "components":
        for _ in range(case["steps"]):
            api.run_groups(m)
    elif case["watch"]:
        seen = []
        for _ in range(case["steps"]):
            m.step(1)
            seen += m.diagnostics()
        out["profiles"] = np.stack(seen)
    else:
        m.step(case["steps"])
    for name in _outputs(case):
        f = m.download_tensor(name, dev)
        out[name] = f if case["precision"] == "fp64" else f.float()
    if case["forcing"]:
        out["mean"] = m.mean_profile_rows()
        out["sums"] = np.stack(list(m.profile_diagnostics().values()))
    return out


def work(case):
    """Per step: the state read and written once, and a count of the step's arithmetic; per pass, the
    fields handed back."""
    n = float(case["nx"] * case["ny"] * case["nz"])
    es = 8 if case["precision"] == "fp64" else 4
    nq = 0 if case["physics"] == "dry" else 2 + case["tracers"]
    fft = 10.0 * math.log2(case["nx"] * case["ny"])
    step_flops = n * (250 + 120 + 300 * (1 + nq) + (700 if case["flow"] == "tvd" else 0) + fft + 40)
    step_bytes = 2.0 * (8 + 2 * nq) * n * es
    if case["kind"] == "adjoint":  # the window forward and back: the state once more, the adjoints in and out
        return {"bytes": case["steps"] * (step_bytes + 24.0 * n * es) + 16.0 * n * es, "flops": 3.5 * case["steps"] * step_flops}
    return {"bytes": case["steps"] * step_bytes + len(_outputs(case)) * n * es, "flops": case["steps"] * step_flops}


# ---- the timestep in plain torch -------------------------------------------------------------------
# Levels are the first axis, element k-1 MONC's level k.  xm(f) is the value at i-1, xp at i+1, and
# so on; up(f) is level k+1 and dn(f) level k-1, the end levels repeated.
def xm(f):
    return torch.roll(f, 1, 2)


def xp(f):
    return torch.roll(f, -1, 2)


def ym(f):
    return torch.roll(f, 1, 1)


def yp(f):
    return torch.roll(f, -1, 1)


def up(f):
    return torch.cat([f[1:], f[-1:]])


def dn(f):
    return torch.cat([f[:1], f[:-1]])


def _lower(a, b):
    return torch.where(a < b, a, b)


def _upper(a, b):
    return torch.where(a > b, a, b)


def _pos(f):
    return torch.where(f > 0, f, torch.zeros_like(f))


def _neg(f):
    return torch.where(f < 0, -f, torch.zeros_like(f))


def _inner(f, first=None, last=None):
    """f with its first and last levels replaced (by 0 where nothing is given and asked for)."""
    parts = [f]
    if first is not None:
        parts = [torch.zeros_like(f[:1]) if isinstance(first, int) else first, f[1:]]
    if last is not None:
        parts[-1] = parts[-1][:-1]
        parts.append(torch.zeros_like(f[:1]) if isinstance(last, int) else last)
    return torch.cat(parts)


class _Core:
    """The centred timestep of a case: grid, reference state and the passes in MONC's order."""

    def __init__(self, case, rmlmax=None):
        self.case = case
        c = self.cfg = _config(case)
        dev = self.dev = _device()
        nz = case["nz"]
        self.moist = case["physics"] == "moist"
        self.nq = 2 + case["tracers"] if self.moist else 0
        z = np.asarray(_levels(case), dtype=np.float64)
        zn = np.zeros(nz)
        zn[2:nz - 1] = 0.0625 * (9.0 * (z[1:nz - 2] + z[2:nz - 1]) - z[3:] - z[:nz - 3])
        zn[1] = 0.5 * (z[0] + z[1])
        zn[0] = -zn[1]
        zn[-1] = 0.5 * (z[-2] + z[-1])
        dz, dzn = np.zeros(nz), np.zeros(nz)
        dz[1:], dzn[1:] = np.diff(z), np.diff(zn)
        rdz, rdzn = np.zeros(nz), np.zeros(nz)
        rdz[1:], rdzn[1:] = 1.0 / dz[1:], 1.0 / dzn[1:]
        rdzn_up = np.append(rdzn[1:], 0.0)
        czb, cza = rdz * rdzn, rdz * rdzn_up
        tzd = 0.25 * rdzn_up
        self.z, self.zn = z, zn

        def col(a):
            return torch.tensor(a, device=dev, dtype=torch.float64)[:, None, None]

        self.rdz, self.rdzn, self.dz, self.dzn = col(rdz), col(rdzn), col(dz), col(dzn)
        self.rdzn_up = col(rdzn_up)
        self.czb, self.cza, self.tz, self.tzd = col(czb), col(cza), col(0.25 * rdz), col(tzd)
        self.np_czb, self.np_cza = czb, cza
        dx = float(np.float32(c.dxx))
        self.cx = self.cy = 1.0 / dx
        self.thref = c.thref0
        # pressure and Exner function of the reference state, its saturation humidity
        kappa = c.r / c.cp
        p0, ps = c.surface_reference_pressure, c.surface_pressure
        step = np.append(c.G * dzn[1:] / (c.cp * self.thref), 0.0)
        ptop = 0.0
        for n in range(2):
            ex = (ptop / p0) ** kappa + np.cumsum(step[::-1])[::-1]
            pref = p0 * ex ** (1.0 / kappa)
            if n == 0:
                ptop = (ps ** kappa + ptop ** kappa - (0.5 * (pref[0] + pref[1])) ** kappa) ** (1.0 / kappa)
        exner = (pref / p0) ** kappa
        tref = self.thref * exner
        sat = lambda t: 3.8 / (0.01 * pref * np.exp(17.2693882 * (t - 273.15) / (t - 35.86)) ** -1.0 - 6.109)  # noqa: E731
        dq = 0.5 * (sat(tref + 1.0) - sat(tref - 1.0))
        self.rl = c.rlvap / c.cp
        self.exner, self.pmb, self.tref, self.qsat, self.dqsat = col(exner), col(pref / 100.0), col(tref), col(sat(tref)), col(dq)
        self.qfac = col(1.0 / (1.0 + self.rl * dq))
        rml = torch.tensor(c.rmlmax, device=dev, dtype=torch.float64) if rmlmax is None else rmlmax
        self.rneut_sq = 1.0 / (1.0 / (c.von_karman_constant * col(z + c.z0)) ** 2 + 1.0 / rml ** 2)
        self.buoy = c.G / c.thref0
        self.cq = [c.ratio_mol_wts - 1.0, -1.0] + [0.0] * case["tracers"]
        self.k_cloud = max([k for k in range(2, nz) if zn[k - 1] <= c.max_height_cloud and (zn[1:k] <= c.max_height_cloud).all()] or [1])
        self._surface()
        self._options()
        # frame velocities, timestep and cfltest state
        self.ugal = self.vgal = 0.0
        self.dt = self.dt_new = self.dt_abs = case["dt"]
        self.timestep, self.last_cfl = 3, 2

    def _surface(self):
        c, zn2 = self.cfg, self.zn[1]
        self.zlogm = math.log(1.0 + zn2 / c.z0)
        self.zlogth = math.log((zn2 + c.z0) / c.z0th)
        self.tflux = c.surface_sensible_heat_flux / (c.rhobous * c.cp)
        self.qflux = c.surface_latent_heat_flux / (c.rhobous * c.rlvap)
        self.fbuoy = self.buoy * self.tflux + (self.cq[0] * self.qflux * c.G if self.moist else 0.0)
        if self.fbuoy <= 0.0:
            return
        e = (np.arange(80, dtype=np.float32) / np.float32(79)).astype(np.float64)
        vel = 0.1 * 1000.0 ** e
        ustr = vel * c.von_karman_constant / self.zlogm
        for _ in range(30):
            ob = -ustr ** 3 / (c.von_karman_constant * self.fbuoy)
            x1 = (1.0 - c.gammam * (zn2 + c.z0) / ob) ** 0.25
            x0 = (1.0 - c.gammam * c.z0 / ob) ** 0.25
            psi = 2.0 * np.log((x1 + 1) / (x0 + 1)) + np.log((x1 * x1 + 1) / (x0 * x0 + 1)) + 2.0 * (np.arctan(x0) - np.arctan(x1))
            ustr = 0.9 * ustr + 0.1 * c.von_karman_constant * vel / (self.zlogm - psi)
        self.table = torch.tensor(ustr, device=self.dev)
        self.cneut, self.cfc = ustr[-1] / vel[-1], ustr[0] * vel[0] ** c.convective_limit

    def _options(self):
        c = self.cfg
        col = lambda a: torch.tensor(a, device=self.dev)[:, None, None]  # noqa: E731
        if not self.case["forcing"]:
            return
        damp = lambda h: np.where(h >= c.zdmp, c.dmptim * (np.exp((h - c.zdmp) / c.hdmp) - 1.0), 0.0)  # noqa: E731
        kmin = np.nonzero(self.zn < c.zdmp)[0].max()  # the level below the layer is the lowest one touched
        mask = np.arange(len(self.zn)) >= kmin
        self.dmp, self.dmpz = col(damp(self.zn) * mask), col(damp(self.z) * mask)
        nodes = range(c.n_subs_pl)
        self.wsubs = col(np.interp(self.z, [c.z_subs_pl[n] for n in nodes], [c.f_subs_pl[n] for n in nodes]))

    # -- lower_bc: eddy coefficients of level 1 and the scalars' ghost level
    def lower_bc(self, s):
        c, vk, czn, zn2 = self.cfg, self.cfg.von_karman_constant, 0.5 * self.zn_dz2(), self.zn[1]
        zu, zv = s["zu"][1:2], s["zv"][1:2]
        hv = torch.sqrt((0.5 * (zu + xm(zu)) + self.ugal) ** 2 + (0.5 * (zv + ym(zv)) + self.vgal) ** 2) + float(np.float32(1e-14))
        if self.fbuoy > 0.0:
            posn = 1.0 + 79.0 * torch.log(hv / 0.1) / math.log(1000.0)
            ip = posn.detach().floor().clamp(1, 79).long()
            a, b = self.table[ip - 1], self.table[ip]
            ustr = torch.where(posn < 1.0, hv ** (-c.convective_limit) * self.cfc,
                               torch.where(posn >= 80.0, hv * self.cneut, a + (posn - ip) * (b - a)))
            x = c.gammah * vk * self.fbuoy / ustr ** 3
            diff = (vk * czn * ustr / c.alphah) / (self.zlogth - 2.0 * torch.log(
                (1.0 + torch.sqrt(1.0 + x * (zn2 + c.z0))) / (1.0 + torch.sqrt(1.0 + x * c.z0th))))
            vis = czn * ustr ** 2 / hv
        else:
            vis = czn * (hv * vk / self.zlogm) ** 2 / hv
            diff = vis * self.zlogm / (c.alphah * self.zlogth)
        s["zth"] = _inner(s["zth"], first=self.tflux * self.zn_dz2() / diff + s["zth"][1:2])
        if self.moist:
            s["zq0"] = _inner(s["zq0"], first=self.qflux * self.zn_dz2() / diff + s["zq0"][1:2])
        return vis, diff

    def zn_dz2(self):
        return float(self.zn[1] - self.zn[0])

    # -- smagorinsky, levels 2 .. nz-1
    def subgrid(self, s):
        vis1, diff1 = self.lower_bc(s)
        c, cx, cy, r1 = self.cfg, self.cx, self.cy, self.rdzn_up
        u, v, w = s["zu"], s["zv"], s["zw"]
        a11, a22 = (u - xm(u)) ** 2, (v - ym(v)) ** 2
        a33 = ((w - dn(w)) * self.rdz) ** 2
        sh = ((yp(u) - u) * cy + (xp(v) - v) * cx) ** 2  # at the corner (i+1/2, j+1/2)
        g12 = (ym(xm(sh)) + xm(sh)) + (ym(sh) + sh)
        s13 = ((up(u) - u) * r1 + (xp(w) - w) * cx) ** 2
        s23 = ((yp(w) - w) * cy + (up(v) - v) * r1) ** 2
        ssq = (cx * cx * (up(a11) + a11) + cy * cy * (up(a22) + a22) + (up(a33) + a33) + 0.5 * (s13 + xm(s13))
               + 0.5 * (ym(s23) + s23) + 0.125 * (g12 + up(g12)) + float(np.float32(1e-14)))
        if self.moist:
            num = self.moist_ri(s)
        else:
            num = (up(s["th"]) - s["th"]) * r1 * self.buoy
        ri = num / ssq
        rn = _lower(ri, torch.zeros_like(ri))
        t4 = (1.0 - ri / 0.25) ** 4
        zero = torch.zeros_like(ri)
        fv = torch.where(ri <= 0, torch.sqrt(1.0 - c.smag_subc * rn), torch.where(ri < 0.25, t4, zero))
        fd = torch.where(ri <= 0, torch.sqrt(1.0 - c.smag_subb * rn), torch.where(ri < 0.25, t4 * (1.0 - 1.2 * ri), zero)) / 0.7
        mix = self.rneut_sq * torch.sqrt(ssq)
        return _inner(fv * mix, vis1, 0), _inner(fd * mix, diff1, 0)

    def moist_ri(self, s):
        th, qv, ql = s["zth"], s["zq0"], s["zq1"]
        eps, rl, pr, ex = 0.01, self.rl, 1.0 / self.exner, self.exner
        thcona = self.cfg.ratio_mol_wts * self.thref
        qt = qv + ql
        thl = th - rl * ql * pr
        qt1, thl1 = up(qt), up(th) - rl * up(ql) * pr
        dqt, dth = qt1 - qt, thl1 - thl

        def liquid(q, t, off):
            return _upper(torch.zeros_like(q), (q - (self.qsat + self.dqsat * (ex * t + off))) * self.qfac)

        hi = ex * self.thref - self.tref
        # the level's own value and the neighbour's, mixed a little way towards each other
        dl = eps * dth + (rl * pr - thcona) * (liquid(qt + eps * dqt, thl + eps * dth, 0.0) - liquid(qt, thl, 0.0))
        du = -eps * dth + (rl * pr - thcona) * (liquid(qt1 - eps * dqt, thl1 - eps * dth, hi) - liquid(qt1, thl1, hi))
        return self.rdzn_up * self.buoy * ((thcona - self.thref) * dqt + (dl - du) * 0.5 / eps)

    # -- the momentum sources
    def momentum(self, s, vis):
        c, cx, cy = self.cfg, self.cx, self.cy
        u, v, w, zu, zv, zw = (s[n] for n in ("u", "v", "w", "zu", "zv", "zw"))
        if self.case["flow"] == "tvd":
            su, sv, sw = self.tvd_flow(s)
        else:
            tx, ty, t1, d1 = 0.25 * cx, 0.25 * cy, self.tz, self.tzd
            su = (tx * (xm(u) * (u + xm(u)) - xp(u) * (u + xp(u))) + ty * (ym(u) * (ym(v) + xp(ym(v))) - yp(u) * (v + xp(v)))
                  + t1 * (dn(u) * (dn(w) + xp(dn(w))) - up(u) * (w + xp(w))))
            sv = (ty * (ym(v) * (v + ym(v)) - yp(v) * (v + yp(v))) + tx * (xm(v) * (xm(u) + yp(xm(u))) - xp(v) * (u + yp(u)))
                  + t1 * (dn(v) * (dn(w) + yp(dn(w))) - up(v) * (w + yp(w))))
            sw = (d1 * (dn(w) * (w + dn(w)) - up(w) * (w + up(w))) + tx * (xm(w) * (xm(u) + up(xm(u))) - xp(w) * (u + up(u)))
                  + ty * (ym(w) * (ym(v) + up(ym(v))) - yp(w) * (v + up(v))))
        # viscosity: the stresses where they sit on the staggered grid, then their differences
        vk = vis + dn(vis)
        v4 = vk + yp(vk)
        t12 = 0.125 * (v4 + xp(v4)) * ((yp(zu) - zu) * cy + (xp(zv) - zv) * cx)
        t11 = vk * (zu - xm(zu)) * cx
        t22 = vk * (zv - ym(zv)) * cy
        t33 = _inner(vk * (zw - dn(zw)) * self.rdz, first=0)
        t13 = _inner(0.5 * (vis + xp(vis)) * ((up(zu) - zu) * self.rdzn_up + (xp(zw) - zw) * cx), last=0)
        t23 = _inner(0.5 * (vis + yp(vis)) * ((yp(zw) - zw) * cy + (up(zv) - zv) * self.rdzn_up), last=0)
        su = su + (xp(t11) - t11) * cx + (t12 - ym(t12)) * cy + (t13 - dn(t13)) * self.rdz
        sv = sv + (t12 - xm(t12)) * cx + (yp(t22) - t22) * cy + (t23 - dn(t23)) * self.rdz
        sw = sw + (t13 - xm(t13)) * cx + (t23 - ym(t23)) * cy + (up(t33) - t33) * self.rdzn_up
        if c.coriolis_enabled:
            su = su + c.fcoriol * (0.25 * (v + xp(v) + ym(v) + xp(ym(v))) + self.vgal - c.surface_geostrophic_wind_y)
            sv = sv - c.fcoriol * (0.25 * (u + xm(u) + yp(u) + xm(yp(u))) + self.ugal - c.surface_geostrophic_wind_x)
        sw = sw + 0.5 * self.buoy * (s["th"] + up(s["th"]))
        for n in range(self.nq):
            sw = sw + 0.5 * c.G * self.cq[n] * (s[f"q{n}"] + up(s[f"q{n}"]))
        if self.case["forcing"]:
            su = su - self.dmp * (zu - (s["mean"][0] - self.ugal)) - self.subsidence(s["mean"][0])
            sv = sv - self.dmp * (zv - (s["mean"][1] - self.vgal)) - self.subsidence(s["mean"][1])
            sw = sw - self.dmpz * zw
        return _inner(su, first=0), _inner(sv, first=0), _inner(sw, first=0, last=0)

    def subsidence(self, prof):
        """2 (w(k-1) tzc1 (f(k) - f(k-1)) + w(k) tzc2 (f(k+1) - f(k))) of a mean profile."""
        return 2.0 * self.tz * (dn(self.wsubs) * (prof - dn(prof)) + self.wsubs * (up(prof) - prof))

    # -- ULTIMATE-QUICKEST advection of f by u, v, w; vertical metrics (rdz, rdzn, dzn, tz) and, for
    #    w on its dual grid, rdz of the gradients one level up and a face above level 1
    def tvd(self, u, v, w, f, dual_w=False):
        cx, cy, dt = self.cx, self.cy, 2.0 * self.dt
        if dual_w:
            rdz, rdzn, dzn, tz = self.rdzn, self.rdz, self.dz, self.tzd
            rdz_g, top_rdz = up(rdz), rdz[-1:]
        else:
            rdz, rdzn, dzn, tz = self.rdz, self.rdzn, self.dzn, self.tz
            rdz_g, top_rdz = rdz, rdz[-1:]
        wd = _inner(dn(w), first=0)
        horizontal = cy * (_pos(v) + _neg(ym(v))) + cx * (_pos(u) + _neg(xm(u)))
        cfl = rdz * (_pos(w) + _neg(wd)) + horizontal

        def limited(ffs, fc, fu, fd, outflow):
            fdels = fd - fu
            flat = torch.abs(fd - 2.0 * fc + fu) >= torch.abs(fdels)
            safe = torch.where(flat, torch.ones_like(fdels), fdels) + 1e-30
            ncs, nfs = (fc - fu) / safe, (ffs - fu) / safe
            ref = ncs / (outflow * dt + 1e-30)
            lim = _upper(ncs, _lower(_lower(nfs, ref), torch.ones_like(ref)))
            return torch.where(flat, fc, lim * fdels + fu)

        def quickest(c, fd, fc, fu, curv, grad, scale=1.0):
            cm = torch.abs(c * dt)
            return 0.5 * (fd + fc) - 0.5 * cm * (fd - fc) - (1.0 - cm * cm) / 6.0 * scale * curv - grad

        sel = torch.where
        zlo, zhi = f - dn(f), _inner(f, last=dn(f)[-1:]) - _inner(up(f), last=f[-1:])

        def vertical(sf):
            return torch.abs(sf) * rdz_g * dt

        def upwind(sf, ahead, behind, ps, g):
            """The face's central value (of f or, against the flow, of g) one point upwind across it."""
            return sel(torch.signbit(sf), sel(ps, ahead(f), ahead(g)), sel(ps, behind(f), behind(g)))

        # x faces
        ps = ~torch.signbit(u)
        fu, fc, fd = sel(ps, xm(f), xp(xp(f))), sel(ps, f, xp(f)), sel(ps, xp(f), f)
        sf = 0.125 * (w + wd + xp(w) + xp(wd))
        pz = ~torch.signbit(sf)
        g1 = vertical(sf) * sel(pz, sel(ps, zlo, xp(zlo)), sel(ps, zhi, xp(zhi)))
        sf = 0.125 * (xp(v) + v + xp(ym(v)) + ym(v))
        g2 = torch.abs(sf) * cy * dt * (fc - upwind(sf, yp, ym, ps, xp(f)))
        fx = limited(quickest(u * cx, fd, fc, fu, fd - 2.0 * fc + fu, g1 + g2), fc, fu, fd, sel(u > 0, cfl, xp(cfl)))
        # y faces
        ps = ~torch.signbit(v)
        fu, fc, fd = sel(ps, ym(f), yp(yp(f))), sel(ps, f, yp(f)), sel(ps, yp(f), f)
        sf = 0.125 * (w + wd + yp(w) + yp(wd))
        pz = ~torch.signbit(sf)
        g1 = vertical(sf) * sel(pz, sel(ps, zlo, yp(zlo)), sel(ps, zhi, yp(zhi)))
        sf = 0.125 * (xm(u) + u + yp(xm(u)) + yp(u))
        g2 = torch.abs(sf) * cx * dt * (fc - upwind(sf, xp, xm, ps, yp(f)))
        fy = limited(quickest(v * cy, fd, fc, fu, fd - 2.0 * fc + fu, g1 + g2), fc, fu, fd, sel(ps, cfl, yp(cfl)))
        # z faces, above each level; beyond the top the field is extrapolated linearly
        ps = ~torch.signbit(w)
        above2 = torch.cat([f[2:], (2.0 * f[-1:] - f[-2:-1]), f[-1:]])
        fu, fc, fd = sel(ps, dn(f), above2), sel(ps, f, up(f)), sel(ps, up(f), f)
        # the outflow of the upwind cell; the end faces of w's dual grid take the shifted rdz
        lo, hi = cfl, up(cfl)
        if dual_w:
            lo_top = (top_rdz * (_pos(w) + _neg(wd)) + horizontal)[-2:-1]
            lo = _inner(torch.cat([lo[:-2], lo_top, lo[-1:]]), first=(rdz_g * _pos(w) + horizontal)[:1])
            bottom = (rdz[2:3] * (_pos(w[1:2]) + _neg(w[:1])) + horizontal[1:2])
            hi = torch.cat([bottom, hi[1:]])
        sf = 0.125 * (ym(v) + v + up(ym(v)) + up(v))
        grad = torch.abs(sf) * cy * dt * (fc - upwind(sf, yp, ym, ps, up(f)))
        sf = 0.125 * (xm(u) + u + up(xm(u)) + up(u))
        grad = grad + torch.abs(sf) * cx * dt * (fc - upwind(sf, xp, xm, ps, up(f)))
        rdd, dd = up(rdzn), up(dzn)
        rdu = sel(ps, _inner(rdzn, first=rdzn[1:2]), torch.cat([rdzn[2:], rdzn[-1:], rdzn[-1:]]))
        rdc = sel(ps, rdz_g, up(rdz_g))
        fz = limited(quickest(w * rdd, fd, fc, fu, (fd - fc) * rdd - (fc - fu) * rdu, grad, dd * dd * rdc), fc, fu, fd,
                     sel(ps, lo, hi))
        flux = 4.0 * w * fz
        if not dual_w:
            flux = _inner(flux, first=0, last=0)
        return ((ym(v * fy) - v * fy) * cy + (dn(flux) - flux) * tz + (xm(u * fx) - u * fx) * cx)

    def tvd_flow(self, s):
        u, v, w = s["u"], s["v"], s["w"]
        mid_x, mid_y = lambda a: 0.5 * (a + xp(a)), lambda a: 0.5 * (a + yp(a))  # noqa: E731
        mid_z = lambda a: 0.5 * (a + up(a))  # noqa: E731
        return (self.tvd(mid_x(u), mid_x(v), mid_x(w), s["zu"]), self.tvd(mid_y(u), mid_y(v), mid_y(w), s["zv"]),
                self.tvd(mid_z(u), mid_z(v), mid_z(w), s["zw"], dual_w=True))

    def diffusion(self, f, d):
        d2 = d + dn(d)
        ax, ay = d2 + xp(d2), d2 + yp(d2)
        gx, gy = ax * (xp(f) - f), ay * (yp(f) - f)
        term = 0.25 * (self.cx ** 2 * (gx - xm(gx)) + self.cy ** 2 * (gy - ym(gy))) + self.czb * dn(d) * (dn(f) - f)
        return term + _inner(self.cza * d * (up(f) - f), last=0)

    # -- scalar sources of theta and the q fields, then the saturation adjustment
    def scalars(self, s, diff):
        out = {}
        for n in ["th"] + [f"q{m}" for m in range(self.nq)]:
            f = s["z" + n]
            src = self.tvd(s["u"], s["v"], s["w"], f) + self.diffusion(f, diff)
            if self.case["forcing"]:  # dry
                m = s["mean"][2]
                src = src - self.dmp * (f - m)
                grad = up(m) - m
                src = src - self.wsubs * _inner(grad, last=dn(grad)[-1:]) * _inner(self.rdzn_up, last=self.rdzn[-1:])
            out[n] = _inner(src, first=0)
        if self.moist:
            self.cloud(s, out)
        return out

    def cloud(self, s, src):
        dtm, pr = 2.0 * self.dt, 1.0 / self.exner
        th, qv, ql = s["zth"], s["zq0"], s["zq1"]
        t = (th + src["th"] * dtm + self.thref) * self.exner
        v, l = qv + src["q0"] * dtm, ql + src["q1"] * dtm
        qs = 3.8 / (self.pmb * torch.exp(-17.2693882 * (t - 273.15) / (t - 35.86)) - 6.109)
        dqs = 17.2693882 * (273.15 - 35.86) * (1.0 + 6.109 * qs / 3.8) * qs / (t - 35.86) ** 2
        wet = (v > qs) | (l > 0)
        dm = torch.where(wet, _upper(-l, (v - qs) / (1.0 + self.rl * dqs)) / dtm, torch.zeros_like(l))
        kc = self.k_cloud
        high = torch.where(l > 0, -l / dtm, torch.zeros_like(l))
        dm = torch.cat([torch.zeros_like(dm[:1]), dm[1:kc], high[kc:]])
        warm = torch.cat([pr[:kc], pr[kc - 1:kc].expand(len(self.z) - kc, 1, 1)])
        src["q0"] = src["q0"] - dm
        src["q1"] = src["q1"] + dm
        src["th"] = src["th"] + self.rl * dm * warm

    # -- the pressure from its source: horizontal transforms and a tridiagonal solve per wavenumber
    def pressure(self, p):
        nz, ny, nx = p.shape
        b = torch.fft.rfft2(p)
        lam = lambda n, c, m: 2.0 * c * c * (torch.cos(2.0 * math.pi * torch.arange(m, device=p.device, dtype=torch.float64) / n) - 1.0)  # noqa: E731
        cij = lam(ny, self.cy, ny)[:, None] + lam(nx, self.cx, nx // 2 + 1)[None, :]
        lo, hi = self.np_czb, self.np_cza
        cij = torch.cat([(cij.flatten() * 0.0 - 1.0)[:1], cij.flatten()[1:]]).reshape(cij.shape)  # mean mode: below
        piv, val = [None, 1.0 / (cij - hi[1])], [None, b[1]]
        for k in range(2, nz):
            val.append(b[k] - lo[k] * val[k - 1] * piv[k - 1])
            piv.append(1.0 / (cij - lo[k] - (hi[k] if k < nz - 1 else 0.0) - lo[k] * hi[k - 1] * piv[k - 1]))
        x = [None] * nz
        x[nz - 1] = val[-1] * piv[-1]
        for k in range(nz - 2, 0, -1):
            x[k] = (val[k] - hi[k] * x[k + 1]) * piv[k]
        x[0] = b[0]
        # the horizontal mean, integrated upwards from zero at the lowest two levels
        mean = [torch.zeros_like(b[0, 0, 0])] * 2
        for k in range(2, nz):
            mean.append((b[k - 1, 0, 0] + (lo[k - 1] + hi[k - 1]) * mean[k - 1] - lo[k - 1] * mean[k - 2]) / hi[k - 1])
        q = torch.stack(x)
        q = torch.cat([torch.stack(mean)[:, None], q.reshape(nz, -1)[:, 1:]], dim=1).reshape(q.shape)
        return torch.fft.irfft2(q, s=(ny, nx))

    # -- one centred step of the state s (a dict of fields), in place of it a new dict
    def step(self, s):
        s = dict(s)
        forcing = self.case["forcing"]
        if forcing:
            self.dt = self.dt_new
        dt2, tm, ug, vg = 2.0 * self.dt, 1e-2, self.ugal, self.vgal
        vis, diff = self.subgrid(s)
        frame = (ug, vg)
        if forcing:
            frame = self.cfltest(s, vis, diff)
        su, sv, sw = self.momentum(s, vis)
        src = self.scalars(s, diff)
        nu, nv, nw = ug + s["zu"] + dt2 * su, vg + s["zv"] + dt2 * sv, s["zw"] + dt2 * sw
        new = {}
        for n, f in src.items():
            smooth = (1.0 - 2.0 * tm) * s[n] + tm * s["z" + n]
            fn = s["z" + n] + dt2 * f
            if n != "th":
                fn = _upper(fn, torch.zeros_like(fn))
            new[n], new["z" + n] = fn, smooth + tm * fn
            if forcing:
                thbar = smooth
        if forcing:
            mean = [f.mean(dim=(1, 2), keepdim=True) for f in (nu, nv, new["th"], ug + s["u"], vg + s["v"], thbar)]
            new["mean"] = torch.stack(mean)
        p = (self.cx * (nu - xm(nu)) + self.cy * (nv - ym(nv)) + (nw - dn(nw)) * self.rdz) / dt2
        p = self.pressure(_inner(p, first=0))
        pu, pv = nu - frame[0] + dt2 * self.cx * (p - xp(p)), nv - frame[1] + dt2 * self.cy * (p - yp(p))
        pu = _inner(pu, first=-pu[1:2] - 2.0 * frame[0])
        pv = _inner(pv, first=-pv[1:2] - 2.0 * frame[1])
        pw = nw + _inner(dt2 * self.rdzn_up * (p - up(p)), first=0, last=0)
        for n, f, g, h in (("u", pu, ug, frame[0]), ("v", pv, vg, frame[1]), ("w", pw, 0.0, 0.0)):
            new["z" + n] = (1.0 - 2.0 * tm) * (g + s[n] - h) + tm * (f + s["z" + n] + g - h)
            new[n] = f
        new["p"] = p
        self.ugal, self.vgal = frame
        self.timestep += 1
        return new

    def cfltest(self, s, vis, diff):
        """The frame velocity after this step and, for the next one, its timestep."""
        c, n, f = self.cfg, self.timestep, self.cfg.cfl_frequency
        frame = (self.ugal, self.vgal)
        if n % f == 1 or n - 1 <= f or n >= self.last_cfl + f:
            self.last_cfl = n
            ext = []
            for a, g in ((s["zu"], self.ugal), (s["zv"], self.vgal)):
                lo, hi = float(a[1:].min()) + g, float(a[1:].max()) + g
                mid = 0.5 * (lo + hi)
                ext.append((mid, max(abs(hi - mid), abs(lo - mid))))
            frame = (ext[0][0], ext[1][0])
            r = self.rdzn_up[1:-1]
            cz = float((s["zw"][1:-1].abs() * r).max())
            cv = float((_upper(vis, diff)[1:-1] * (r * r + self.cx ** 2 + self.cy ** 2)).max())
            number = cv * 4.0 * self.dt / c.cfl_cvismax + (ext[0][1] * self.cx + ext[1][1] * self.cy + cz) * self.dt / c.cfl_cvelmax
            self.dt_abs = self.dt
            if number > 0 and abs(number - 1.0) > c.cfl_tollerance:
                self.dt_abs = self.dt / number
        self.dt_new = self.dt
        if self.dt != self.dt_abs and (self.dt != c.cfl_dtmmax or self.dt_abs < c.cfl_dtmmax):
            self.dt_new = min(self.dt * (1.0 + c.cfl_rincmax), self.dt_abs, c.cfl_dtmmax)
        return frame

    def sums(self, s):
        """profile_diagnostics' sums over the columns, dry."""
        u, v, w, th = s["u"] + self.ugal, s["v"] + self.vgal, s["w"], s["th"]
        ub, vb, tb = s["mean"][3], s["mean"][4], s["mean"][5]
        wu = _inner(w, first=0)
        low = lambda a: _inner(a, last=0)  # noqa: E731
        uw = low(0.25 * (u + xm(u) + up(u) + up(xm(u))) - 0.5 * (ub + up(ub))) * w
        vw = low(0.25 * (v + ym(v) + up(v) + up(ym(v))) - 0.5 * (vb + up(vb))) * w
        rows = [u, v, wu, w * w, wu ** 3, wu ** 4, th + self.thref, (th - tb) ** 2, low(wu * 0.5 * (th + up(th))), uw, vw]
        return torch.stack([r.sum(dim=(1, 2)) for r in rows])


def exact(case, seed):
    """The pass in FP64.  None where the answer depends on where an iteration stops, and for grids
    on which this takes too long."""
    if case["solver"] != "fft" or case["nx"] * case["ny"] * case["nz"] * case["steps"] > 200e6:
        return None
    s = dict(_state(case, seed))
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, s)
    with torch.no_grad():
        core = _Core(case)
        if case["forcing"]:
            s["mean"] = torch.tensor(_mean_rows(case, s), device=core.dev)[:, :, None, None]
        out, seen = {}, []
        for _ in range(case["steps"]):
            s = core.step(s)
            if case["watch"]:
                seen += [s["th"].mean(dim=(1, 2)) + core.thref, (s["w"] ** 2).mean(dim=(1, 2))]
        if case["watch"]:
            out["profiles"] = torch.stack(seen)
        out.update({n: s[n] for n in _outputs(case)})
        if case["forcing"]:
            out["mean"] = s["mean"][:, :, 0, 0]
            out["sums"] = core.sums(s)
        return out


def _exact_adjoint(case, seed, s):
    seeds = _seeds(case, seed)
    leaves = {n: s[n].clone().requires_grad_() for n in ADJ_OUT}
    rml = torch.tensor(_config(case).rmlmax, device=_device(), dtype=torch.float64, requires_grad=True)

    def one(rmlmax, *f):
        new = _Core(case, rmlmax).step(dict(zip(ADJ_OUT, f)))
        return tuple(new[n] for n in ADJ_OUT)

    f = tuple(leaves[n] for n in ADJ_OUT)
    for _ in range(case["steps"]):
        f = checkpoint(one, rml, *f, use_reentrant=False)
    objective = sum((a * seeds[n]).sum() for n, a in zip(ADJ_OUT, f) if n in seeds)
    grads = torch.autograd.grad(objective, [rml] + [leaves[n] for n in ADJ_OUT])
    out = dict(zip(ADJ_OUT, grads[1:]))
    # w and zw are exactly 0 on the lowest and the top level, on the kinks of the upwind choices, where
    # the derivative is a convention
    out["w"] = out["zw"] = None
    out["mixing"] = float(grads[0])
    return out
