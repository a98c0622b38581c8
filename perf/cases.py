"""Timing cases of the split step: what a program has the library do, at the sizes it does it.

Kinds of cases, and what each stands for in use:

* ``hooks``: one transport RHS and one chemistry RHS of a host state (rs_rhs_transport,
  rs_rhs_chem), the calls a host integrator or a parity check makes; the smallest ones.
* ``window``: one window of the drop-in driver (lie_trotter_solve), host state in and out, from
  a cold start; on the 36x18x10 grid the launches and the controller's latency decide.
* ``step``: one macro step on the resident state in mid-run (one earlier macro step is done in
  the preparation): the production loop.  FP64 or mixed precision, global grids or a regional
  one with open walls, PBL mixing and the pressure fixer.
* ``transport``: the SSPRK43 half alone, 12 tracers or the 30 of the synthetic mechanism.
* ``attempt``: one Rosenbrock23 attempt on the caller's device buffers
  (rs_ros23_attempt_noalloc), with the specialised (SuperFast) or the table kernels (synthetic).
* ``cells``: per-cell adaptive chemistry of independent cells over one window.
* ``adjoint``: macro steps recorded, then swept back: gradients with respect to the state and
  to the emissions.

Sizes are those of the repository's workloads (36x18x10, 72x46x47, 144x91x47, 360x181x72 and
2^18 cells of the 2^20-cell batch) and odd ones in between.  Long runs tune once
(``tuned``: rs_autotune in the preparation), short ones take the defaults.
"""
import ctypes
import math

import numpy as np
import torch

from reseact.esm_gb300 import Solver, abi, lie_trotter_solve, mechanism, workloads

DAY = 86400.0


# ------------------------------------------------------------------------------- the cases
def listed():
    def case(name, kind, nlon, nlat, nlev, **kw):
        c = dict(name=name, kind=kind, nlon=nlon, nlat=nlat, nlev=nlev, mech="superfast",
                 mixed=False, regional=False, tuned=False, dt=600.0)
        c.update(kw)
        return c

    return [
        # a host integrator's two RHS calls on the 10-degree grid
        case("hooks-36x18x10", "hooks", 36, 18, 10),
        # the drop-in call of a small run: latency of launches and of the device controller
        case("window-36x18x10", "window", 36, 18, 10),
        # the headline run: 2.5 x 2 degrees, FP64
        case("step-144x91x47", "step", 144, 91, 47, tuned=True),
        # the same run with compensated FP32 transport
        case("step-mixed-144x91x47", "step", 144, 91, 47, mixed=True, tuned=True),
        # a regional run: open walls, PBL mixing, pressure fixer, emissions, ragged sizes
        case("step-regional-67x45x37", "step", 67, 45, 37, regional=True),
        # tracer transport alone, FP64, at 2 degrees with 72 levels and 30 tracers
        case("transport-180x91x72", "transport", 180, 91, 72, mech="synthetic", tuned=True,
             dt=300.0),
        # and at full size, 1 degree, in the precision that configuration runs in
        case("transport-mixed-360x181x72", "transport", 360, 181, 72, mech="synthetic",
             mixed=True, tuned=True, dt=300.0),
        # one chemistry attempt of a caller that owns the buffers: specialised kernels
        case("attempt-144x91x47", "attempt", 144, 91, 47, dt=20.0),
        # and of a mechanism too large for them
        case("attempt-synthetic-72x46x47", "attempt", 72, 46, 47, mech="synthetic", dt=0.05),
        # independent stiff cells, uneven step counts
        case("cells-2^18", "cells", 1024, 256, 1, mech="synthetic", tuned=True),
        # gradient of a two-step window with respect to the state and the emissions
        case("adjoint-72x46x47", "adjoint", 72, 46, 47),
    ]


def draw(rng):
    """One more case: a kind, and a grid drawn over the logarithm of the sizes."""
    kind = rng.choice(["hooks", "window", "step", "step", "step", "transport", "transport",
                       "attempt", "cells", "adjoint"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = dict(kind=kind, mech="superfast", mixed=False, regional=False,
             tuned=rng.random() < 0.5, dt=600.0)
    if kind == "cells":
        c.update(nlon=1024, nlat=size(16, 256), nlev=1, mech="synthetic")
        return c
    top = dict(hooks=(72, 46, 30), window=(72, 46, 30), step=(150, 92, 48),
               transport=(240, 121, 72), attempt=(160, 100, 60), adjoint=(80, 50, 47))[kind]
    c.update(nlon=size(24, top[0]), nlat=size(15, top[1]), nlev=size(8, top[2]))
    if kind in ("step", "transport"):
        c["mixed"] = rng.random() < 0.5
    if kind == "step":
        c["regional"] = rng.random() < 0.3
    if kind in ("transport", "attempt") and rng.random() < 0.5:
        c["mech"] = "synthetic"
        c["dt"] = 300.0
    if kind == "attempt":
        c["dt"] = 0.05 if c["mech"] == "synthetic" else rng.choice([5.0, 20.0, 60.0])
    return c


# ------------------------------------------------------------------------------- the inputs
def _mech(case):
    return mechanism.superfast() if case["mech"] == "superfast" else mechanism.synthetic()


def _regional(nlon, nlat, nlev, dp, seed):
    """Fluxes of a divergent inflow / outflow on a 1 x 1 degree regional grid."""
    g = workloads.latlon_grid(nlon, nlat, nlev, lon_bc=abi.RS_BC_OPEN, lat_bc=abi.RS_BC_OPEN,
                              lon0=-120.0, dlon=60.0 / nlon, lat0=25.0, dlat=25.0 / nlat,
                              pole_centred=False)
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(0.0, 2 * math.pi, 2)
    x = np.arange(nlon + 1) / nlon
    y = np.arange(nlat + 1) / nlat
    xm, ym = 0.5 * (x[1:] + x[:-1]), 0.5 * (y[1:] + y[:-1])
    u = 12.0 + 6.0 * np.sin(2 * math.pi * x[None, :] + a) * np.cos(math.pi * ym[:, None])
    v = 5.0 * np.cos(2 * math.pi * xm[None, :] + b) * np.sin(math.pi * y[:, None] + 0.4)
    mx = dp[:, None, None] * u[None] / workloads.A_EARTH
    my = dp[:, None, None] * v[None] / workloads.A_EARTH
    return g, np.ascontiguousarray(mx), np.ascontiguousarray(my)


def _workload(case, seed):
    """The repository's workload object of a case, without its initial state."""
    mech = _mech(case)
    nlon, nlat, nlev = case["nlon"], case["nlat"], case["nlev"]
    precision = abi.RS_PREC_MIXED if case["mixed"] else abi.RS_PREC_FP64
    rng = np.random.default_rng(seed + 1000)
    if case["kind"] == "cells":
        g = workloads.latlon_grid(nlon, nlat, 1, pole_centred=False)
        shape = (1, nlat, nlon)
        forcing = dict(temperature=rng.uniform(200.0, 310.0, size=shape),
                       pressure=np.full(shape, 101325.0), dp=np.ones(shape))
        return workloads.Workload("cells", g, mech, forcing, None, 600.0, 1, has_air_mass=False,
                                  do_transport=False, chem_mode=abi.RS_CHEM_PER_CELL,
                                  dt0_C=1e-3)
    if nlev == 72:
        dp, pm = workloads.hybrid72()
    else:
        dp, pm = workloads.pressure_levels(nlev)
    if case["regional"]:
        g, mx, my = _regional(nlon, nlat, nlev, dp, seed + 100)
        mz = np.zeros((nlev + 1, nlat, nlon))
    else:
        g = workloads.latlon_grid(nlon, nlat, nlev, lon0=0.0, dlon=360.0 / nlon)
        mx, my, mz = workloads.winds_deformational(g, dp, seed=seed + 100, w_shape="sine")
    dp3, p3, t3 = workloads._column_fields(g, dp, pm)
    forcing = dict(mx=mx, my=my, mz=mz, dp=dp3, temperature=t3, pressure=p3,
                   flux_omega=0.0 if case["regional"] else math.pi / DAY)
    if case["regional"] or case["kind"] == "adjoint":  # surface NO emissions
        e = np.zeros((mech.ns, nlev, nlat, nlon))
        e[mech.species.index("NO"), 0] = 1e-4 * np.exp(0.5 * rng.standard_normal((nlat, nlon)))
        forcing["emission"] = e
    if case["regional"]:  # lognormal inflow about the defaults
        med = np.array([mech.defaults[s] for s in mech.species])[:, None, None]
        for key, n in (("qbc_w", nlat), ("qbc_e", nlat), ("qbc_s", nlon), ("qbc_n", nlon)):
            forcing[key] = med * np.exp(0.3 * rng.standard_normal((mech.ns, nlev, n)))
    w = workloads.Workload(case["kind"], g, mech, forcing, None, case["dt"], 1,
                           precision=precision,
                           do_chemistry=case["kind"] != "transport")
    if case["regional"]:
        workloads.with_pbl(w, seed=seed + 11)
        workloads.with_pressure_fixer(w, seed=seed + 12)
    return w


def _device():
    return torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")


def _planes(w, seed):
    """The initial state on the device, species-major planes [species][nlev][nlat][nlon]:
    lognormal about the mechanism's defaults, log-uniform for the synthetic one."""
    gen = torch.Generator(device=_device()).manual_seed(int(seed) + 7)
    g = w.grid
    u = torch.empty((w.nsp, g["nlev"], g["nlat"], g["nlon"]), dtype=torch.float64,
                    device=_device())
    for s, name in enumerate(w.mech.species):
        if w.mech.name.startswith("Synthetic"):
            u[s].uniform_(-12.0, -6.0, generator=gen)
            u[s] = torch.pow(10.0, u[s])
        else:
            u[s].normal_(0.0, 0.5, generator=gen)
            u[s] = w.mech.defaults[name] * torch.exp(u[s])
    if w.has_air_mass:
        u[-1] = torch.as_tensor(w.forcing["dp"], device=u.device)
    return u


def _cellmajor(u):
    return u.permute(3, 2, 1, 0).contiguous().reshape(-1).cpu().numpy()


def _by_species(u, nsp):
    """A state as one output per species (their sizes differ by many orders): planes of a
    species-major tensor, columns of a cell-major host array."""
    return list(u.unbind(0)) if isinstance(u, torch.Tensor) else list(u.reshape(-1, nsp).T)


def _lambda(case, w, seed):
    """dJ/du at the end: a seeded misfit of surface ozone."""
    rng = np.random.default_rng(seed + 44)
    g = w.grid
    lam = np.zeros((w.nsp, g["nlev"], g["nlat"], g["nlon"]))
    lam[w.mech.species.index("O3"), 0] = rng.standard_normal((g["nlat"], g["nlon"]))
    return lam


class _DeviceArray:
    """A raw device pointer as something torch can view."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False),
                                             version=3)


class State:
    """What a program keeps: the handle, its stream and the inputs of the next call."""

    def __init__(self, case, seed):
        self.case = case
        self.w = w = _workload(case, seed)
        self.solver = Solver.for_workload(w)
        self.shape = (w.nsp, w.grid["nlev"], w.grid["nlat"], w.grid["nlon"])
        self.stream = torch.cuda.ExternalStream(self.solver.stream())
        self.u = _planes(w, seed)
        self.t, self.dtT, self.dtC = 0.0, w.dt0_T, w.dt0_C
        torch.cuda.synchronize()
        kind = case["kind"]
        if kind in ("hooks", "window"):
            self.u = _cellmajor(self.u)
            if case["tuned"]:
                self.solver.set_state(self.u)
                self.solver.autotune()
            return
        self.load()
        if case["tuned"]:
            self.solver.autotune()
        if kind in ("step", "adjoint"):  # one macro step from the cold start
            _, self.dtT, self.dtC, _ = self.solver.macro_step(0.0, 600.0, self.dtT, self.dtC)
            self.t = 600.0
            self.u = self.take()
        if kind == "attempt":
            self.out = torch.empty_like(self.u)
        if kind == "adjoint":
            self.lam = workloads.soa_to_cellmajor(_lambda(case, w, seed), w.grid["nlon"],
                                                  w.grid["nlat"], w.grid["nlev"])
            self.solver.set_adjoint_tape(6 << 30)
        torch.cuda.synchronize()

    def view(self):
        p = ctypes.c_void_p()
        self.solver.L.rs_state_device_ptr(self.solver.h, ctypes.byref(p))
        return torch.as_tensor(_DeviceArray(p.value, self.shape), device="cuda")

    def load(self):
        """The resident state <- self.u, on the handle's stream."""
        with torch.cuda.stream(self.stream):
            self.view().copy_(self.u)

    def take(self):
        with torch.cuda.stream(self.stream):
            return self.view().clone()


def prepare(case, seed):
    return State(case, seed)


def run(s):
    kind, sv, dt, nsp = s.case["kind"], s.solver, s.case["dt"], s.w.nsp
    if kind == "hooks":
        return {"transport": _by_species(sv.rhs_transport(s.u, 300.0), nsp),
                "chemistry": _by_species(sv.rhs_chem(s.u, 300.0), nsp)}
    if kind == "window":
        r = lie_trotter_solve(sv, s.u, (0.0, dt), macro_dt=dt, dtT=s.dtT, dtC=s.dtC)
        return {"u": _by_species(r.u, nsp), "dtT": r.dtT, "dtC": r.dtC,
                "counts": [r.naT, r.nrT, r.naC, r.nrC, r.nmacro]}
    if kind == "attempt":
        eest = ctypes.c_double()
        rc = sv.L.rs_ros23_attempt_noalloc(sv.h, dt, s.u.data_ptr(), s.out.data_ptr(),
                                           ctypes.byref(eest))
        if rc != abi.RS_OK:
            raise RuntimeError("attempt failed: %d" % rc)
        return {"u": _by_species(s.out, nsp), "eest": eest.value}
    s.load()
    if kind == "adjoint":
        sv.record(True)
        t, a, b = s.t, s.dtT, s.dtC
        for _ in range(2):
            _, a, b, _ = sv.macro_step(t, t + dt, a, b)
            t += dt
        sv.record(False)
        lam0, grad = sv.adjoint_backward(s.lam)
        return {"lambda": _by_species(lam0, nsp), "emission": list(grad), "dtC": b}
    _, a, b, st = sv.macro_step(s.t, s.t + dt, s.dtT, s.dtC)
    out = {"u": _by_species(s.take(), nsp)}
    if kind == "cells":
        return out
    if kind == "step" or kind == "transport":
        out["dtT"] = a
        out["counts"] = [int(st.naT), int(st.nrT), int(st.naC), int(st.nrC)]
    if kind == "step":
        out["dtC"] = b
    return out


def work(case):
    """Inputs read and outputs written once, and the arithmetic of the attempts a pass takes:
    transport attempts of 4 stages of ~45 FP64 operations (about 75 flops) per cell and tracer,
    chemistry attempts of ~1,450 (SuperFast) or ~4,500 (synthetic) flops per cell.  The numbers of
    attempts are those of the controllers on these inputs, to within a few."""
    mech = _mech(case)
    nc = case["nlon"] * case["nlat"] * case["nlev"]
    ntr = mech.ns
    state = 8.0 * (ntr + 1) * nc
    rates, fluxes = 8.0 * mech.nr * nc, 3 * 8.0 * nc
    tr, ch = 4 * 75.0 * ntr * nc, (1450.0 if case["mech"] == "superfast" else 4500.0) * nc
    kind = case["kind"]
    if kind == "hooks":
        return {"bytes": 4 * state + rates + fluxes, "flops": tr / 4 + ch / 10}
    if kind == "attempt":
        return {"bytes": 2 * state + rates, "flops": ch}
    if kind == "cells":
        return {"bytes": 2 * state + rates, "flops": 40 * ch}
    if kind == "transport":
        return {"bytes": 2 * state + fluxes, "flops": 3 * tr}
    if kind == "window":
        return {"bytes": 2 * state + rates + fluxes, "flops": 5 * tr + 150 * ch}
    if kind == "step":
        return {"bytes": 2 * state + rates + fluxes, "flops": 4 * tr + 35 * ch}
    return {"bytes": 2 * (3 * state + rates + fluxes), "flops": 2 * 3 * (4 * tr + 25 * ch)}


# ------------------------------------------------------------------------------- in 64 bits
class _Math:
    """The split step in plain torch, FP64: the PPM transport tendency with optional PBL mixing
    and pressure fixer, SSPRK43, mass-action chemistry, Rosenbrock23 and the PI controller."""

    def __init__(self, w):
        self.w, self.dev = w, _device()
        g, f = w.grid, w.forcing
        self.nlon, self.nlat, self.nlev = g["nlon"], g["nlat"], g["nlev"]
        self.ntr, self.nsp = w.mech.ns, w.nsp
        self.ten = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64,
                                             device=self.dev)
        if w.do_transport:
            self._geometry(g, f)
        self._chemistry(w.mech, f)

    # ---- transport
    def _geometry(self, g, f):
        d2r = 0.017453292519943295
        phi = np.clip(g["lat0_deg"] + (np.arange(self.nlat + 1) - 0.5) * g["dlat_deg"], -90, 90)
        cos = np.where(np.abs(phi) >= 90.0, 0.0, np.cos(phi * d2r))
        ds = np.sin(phi[1:] * d2r) - np.sin(phi[:-1] * d2r)
        dphi = (phi[1:] - phi[:-1]) * d2r
        self.gx = self.ten((dphi / (g["dlon_deg"] * d2r * ds))[:, None])
        self.glo, self.ghi = self.ten((cos[:-1] / ds)[:, None]), self.ten((cos[1:] / ds)[:, None])
        self.open = g["lon_bc"] == abi.RS_BC_OPEN
        mx, my, mz = self.ten(f["mx"]), self.ten(f["my"]).clone(), self.ten(f["mz"]).clone()
        if g["lat_bc"] != abi.RS_BC_OPEN:
            my[:, 0] = 0.0
            my[:, -1] = 0.0
        self.omega = float(f.get("flux_omega", 0.0))
        self.corr = None
        if "dps_dt" in f:
            b, dps, dp = self.ten(f["hyb_b"]), self.ten(f["dps_dt"]), self.ten(f["dp"])
            divh = (mx[..., 1:] - mx[..., :-1]) * self.gx + (my[:, 1:] * self.ghi - my[:, :-1] * self.glo)
            self.corr = (-dps - divh.sum(0)) * (dp / dp.sum(0))
            mz = torch.zeros_like(mz)
            mz[1:] = torch.cumsum(-((b[:-1] - b[1:])[:, None, None] * dps + (divh + self.corr)), 0)
        mz[0] = 0.0
        mz[-1] = 0.0
        self.mx, self.my, self.mz = mx, my, mz
        if self.open:
            self.bc = {k: self.ten(f[k]) for k in ("qbc_w", "qbc_e", "qbc_s", "qbc_n")}
        dp = self.ten(f["dp"])
        d = torch.cat([dp[:3].flip(0), dp, dp[-3:].flip(0)], 0)  # cells -3 .. nlev+2
        n = self.nlev
        lo, mid, hi = d[1:n + 3], d[2:n + 4], d[3:n + 5]         # around cells -1 .. n
        c = mid / (lo + mid + hi)
        self.sA = c * (2.0 * lo + mid) / (hi + mid)
        self.sB = c * (mid + 2.0 * hi) / (lo + mid)
        dm, d0, d1, d2 = d[1:n + 2], d[2:n + 3], d[3:n + 4], d[4:n + 5]  # edges 0 .. n
        tot = dm + d0 + d1 + d2
        t1, t2 = (dm + d0) / (2.0 * d0 + d1), (d2 + d1) / (2.0 * d1 + d0)
        self.eAB = d0 / (d0 + d1) + (2.0 * d1 * d0 / (d0 + d1)) * (t1 - t2) / tot
        self.eC, self.eD = -(d0 * t1) / tot, d1 * (d1 + d2) / (d0 + 2.0 * d1) / tot
        self.pbl = None
        if f.get("tau_pblmix"):
            a, b, ps = self.ten(f["hyb_a"]), self.ten(f["hyb_b"]), self.ten(f["ps"])
            top = ps * torch.exp(-(self.ten(f["pblh"]) * 9.80665) / (287.05 * self.ten(f["temperature"])[0]))
            p = a[:, None, None] + b[:, None, None] * ps
            fr = ((torch.minimum(ps, p[:-1]) - torch.maximum(top, p[1:])) / dp).clamp(0.0, 1.0)
            wt = dp * fr
            self.pbl = (fr, wt, wt.sum(0).clamp(min=1.0), float(f["tau_pblmix"]))

    def factor(self, t):
        return math.cos(self.omega * t) if self.omega else 1.0

    @staticmethod
    def _slope(d0, d1, da):
        m = torch.minimum(da.abs(), 2.0 * torch.minimum(d0.abs(), d1.abs()))
        return torch.where(d1 * d0 > 0.0, torch.where(da > 0.0, m, -m), torch.zeros_like(m))

    @staticmethod
    def _face(a, left, right, pick_right):
        flat = (right - a) * (a - left) <= 0.0
        d, a6 = right - left, 6.0 * (a - 0.5 * (left + right))
        over, under = d * a6 > d * d, -(d * d) > d * a6
        lo = torch.where(over, 3.0 * a - 2.0 * right, left)
        hi = torch.where(under & ~over, 3.0 * a - 2.0 * left, right)
        return torch.where(flat, a, hi if pick_right else lo)

    def _fluxes(self, v, m, dim, edges, off):
        """Face fluxes from padded values v (cell p at p + 3 along dim), edge values (edge e at
        e + off) and the air-mass fluxes m: the upwind cell's limited edge."""
        n = m.shape[dim] - 1
        cut = lambda x, i: x.narrow(dim, i, n + 1)  # noqa: E731
        fr = self._face(cut(v, 2), cut(edges, off - 1), cut(edges, off), True)
        fl = self._face(cut(v, 3), cut(edges, off), cut(edges, off + 1), False)
        return m * torch.where(m > 0.0, fr, fl)

    def _uniform(self, v, m, dim):
        n = m.shape[dim] - 1
        d = torch.diff(v, dim=dim)                      # between p and p + 1, p from -3
        d0, d1 = d.narrow(dim, 0, n + 4), d.narrow(dim, 1, n + 4)
        s = self._slope(d0, d1, 0.5 * (d0 + d1))        # cells -2 .. n+1
        e = v.narrow(dim, 1, n + 3) + 0.5 * d.narrow(dim, 1, n + 3) \
            - torch.diff(s, dim=dim) / 6.0              # edges -1 .. n+1
        return self._fluxes(v, m, dim, e, 1)

    def _vertical(self, v, m):
        n = self.nlev
        d = torch.diff(v, dim=0)
        d0, d1 = d[1:n + 3], d[2:n + 4]                 # around cells -1 .. n
        s = self._slope(d0, d1, self.sA * d1 + self.sB * d0)
        e = v[2:n + 3] + self.eAB * d[2:n + 3] + self.eC * s[1:] + self.eD * s[:-1]  # edges 0 .. n
        e = torch.cat([e[:1], e, e[-1:]], 0)            # the walls' outer edges carry no flux
        return self._fluxes(v, m, 0, e, 1)

    def rhs_transport(self, u, t):
        g = self.factor(t)
        mx, my, mz, m = g * self.mx, g * self.my, g * self.mz, u[-1]
        div = lambda x, y, z: ((x[..., 1:] - x[..., :-1]) * self.gx  # noqa: E731
                               + (y[:, 1:] * self.ghi - y[:, :-1] * self.glo)) + (z[1:] - z[:-1])
        divm = div(mx, my, mz)
        rows = []
        for s in range(self.ntr):
            q = u[s]
            if self.open:
                one = lambda k: self.bc[k][s]  # noqa: E731
                wst, est = one("qbc_w")[..., None].expand(-1, -1, 3), one("qbc_e")[..., None].expand(-1, -1, 3)
                sth, nth = one("qbc_s")[:, None].expand(-1, 3, -1), one("qbc_n")[:, None].expand(-1, 3, -1)
            else:
                wst, est = q[..., -3:], q[..., :3]
                sth, nth = q[:, :3].flip(1), q[:, -3:].flip(1)
            fx = self._uniform(torch.cat([wst, q, est], 2), mx, 2)
            fy = self._uniform(torch.cat([sth, q, nth], 1), my, 1)
            fz = self._vertical(torch.cat([q[:3].flip(0), q, q[-3:].flip(0)], 0), mz)
            du = (-div(fx, fy, fz) + q * divm) / m
            if self.pbl:
                fr, wt, den, tau = self.pbl
                du = du + fr * ((wt * q).sum(0) / den - q) / tau
            rows.append(du)
        rows.append(-divm - self.corr if self.corr is not None else -divm)
        return torch.stack(rows)

    def transport_step(self, u, t, dt):
        """(new state, embedded error) of one SSPRK43 step."""
        h = dt / 2
        s = u + h * self.rhs_transport(u, t)
        s = s + h * self.rhs_transport(s, t + h)
        s = s + h * self.rhs_transport(s, t + dt)
        v = (2.0 / 3.0) * u + (1.0 / 3.0) * s
        new = v + h * self.rhs_transport(v, t + h)
        return new, 0.5 * ((1.0 / 3.0) * u + (2.0 / 3.0) * s - new)

    # ---- chemistry
    def _chemistry(self, mech, f):
        T, P = self.ten(f["temperature"]), self.ten(f["pressure"])
        self.k, self.reac = [], [rx.reactants for rx in mech.reactions]
        self.net = mech.net_stoich()
        for rx in mech.reactions:
            st = []
            for op, v in zip(rx.prog_ops, rx.prog_vals):
                if op == mechanism.OP_CONST:
                    st.append(torch.full_like(T, v))
                elif op == mechanism.OP_TEMP:
                    st.append(T)
                elif op == mechanism.OP_PRES:
                    st.append(P)
                elif op == mechanism.OP_PARAM:
                    st.append(torch.full_like(T, mech.param_values[int(v)]))
                elif op in (mechanism.OP_NEG, mechanism.OP_EXP, mechanism.OP_LOG,
                            mechanism.OP_LOG10, mechanism.OP_SQRT):
                    fn = {mechanism.OP_NEG: torch.neg, mechanism.OP_EXP: torch.exp,
                          mechanism.OP_LOG: torch.log, mechanism.OP_LOG10: torch.log10,
                          mechanism.OP_SQRT: torch.sqrt}[op]
                    st.append(fn(st.pop()))
                else:
                    b, a = st.pop(), st.pop()
                    fn = {mechanism.OP_ADD: torch.add, mechanism.OP_SUB: torch.sub,
                          mechanism.OP_MUL: torch.mul, mechanism.OP_DIV: torch.div,
                          mechanism.OP_POW: torch.pow}[op]
                    st.append(fn(a, b))
            self.k.append(st[0])
        self.em = None if f.get("emission") is None else self.ten(f["emission"])

    def _combine(self, terms, like):
        acc = None
        for c, x in terms:
            y = x if c == 1.0 else c * x
            acc = y if acc is None else acc + y
        return torch.zeros_like(like) if acc is None else acc

    def rhs_chem(self, x, em):
        v = []
        for k, reac in zip(self.k, self.reac):
            for s, nu in reac:
                k = k * x[s] ** nu if nu > 1 else k * x[s]
            v.append(k)
        out = []
        for s in range(self.ntr):
            r = self._combine([(self.net[q, s], v[q]) for q in range(len(v)) if self.net[q, s]], x[s])
            out.append(r if em is None else r + em[s])
        return out

    def _factor(self, x, hd):
        """Sparse pivot-free LU of I - hd J(x), rows of the matrix as dicts of planes."""
        jac = {}
        for r, reac in enumerate(self.reac):
            for q, _ in reac:
                p = self.k[r]
                for s, nu in reac:
                    if s == q:
                        p = p * (nu * x[s] ** (nu - 1)) if nu > 1 else p
                    else:
                        p = p * x[s] ** nu if nu > 1 else p * x[s]
                for s in range(self.ntr):
                    if self.net[r, s]:
                        y = self.net[r, s] * p
                        jac[s, q] = jac[s, q] + y if (s, q) in jac else y
        one = torch.ones_like(x[0])
        a = {e: -hd * v for e, v in jac.items()}
        for i in range(self.ntr):
            a[i, i] = a[i, i] + 1.0 if (i, i) in a else one
        # few-entries-first order keeps the fill small
        left, order = set(range(self.ntr)), []
        pat = set(a)
        while left:
            cost = lambda k: (sum((i, k) in pat for i in left if i != k)  # noqa: E731
                              * sum((k, j) in pat for j in left if j != k), k)
            k = min(left, key=cost)
            left.discard(k)
            order.append(k)
            pat |= {(i, j) for i in left if (i, k) in pat for j in left if (k, j) in pat}
        for n, k in enumerate(order):
            rest = order[n + 1:]
            for i in rest:
                if (i, k) in a:
                    a[i, k] = a[i, k] / a[k, k]
                    for j in rest:
                        if (k, j) in a:
                            y = a[i, k] * a[k, j]
                            a[i, j] = a[i, j] - y if (i, j) in a else -y
        return a, order

    @staticmethod
    def _solve(lu, b):
        a, order = lu
        x = list(b)
        for n, k in enumerate(order):
            for i in order[n + 1:]:
                if (i, k) in a:
                    x[i] = x[i] - a[i, k] * x[k]
        for n in range(len(order) - 1, -1, -1):
            k = order[n]
            for j in order[n + 1:]:
                if (k, j) in a:
                    x[k] = x[k] - a[k, j] * x[j]
            x[k] = x[k] / a[k, k]
        return x

    def chem_step(self, x, dt, em, error=True):
        """(new species planes, error estimate planes) of one Rosenbrock23 step."""
        d, c32 = 1.0 / (2.0 + math.sqrt(2.0)), 6.0 + math.sqrt(2.0)
        f0 = self.rhs_chem(x, em)
        lu = self._factor(x, dt * d)
        k1 = self._solve(lu, f0)
        f1 = self.rhs_chem([a + (dt / 2) * b for a, b in zip(x, k1)], em)
        z = self._solve(lu, [a - b for a, b in zip(f1, k1)])
        k2 = [a + b for a, b in zip(z, k1)]
        new = [a + dt * b for a, b in zip(x, k2)]
        if not error:
            return new, None
        f2 = self.rhs_chem(new, em)
        k3 = self._solve(lu, [c - c32 * (b - e) - 2.0 * (a - f)
                              for a, b, c, e, f in zip(k1, k2, f2, f1, f0)])
        return new, [(dt / 6) * (a - 2.0 * b + c) for a, b, c in zip(k1, k2, k3)]

    # ---- the adaptive loop of one half
    def _attempt(self, half, u, t, dt):
        if half == "T":
            new, err = self.transport_step(u, t, dt)
            atol = 1e-6
        else:
            x, e = self.chem_step(list(u[:self.ntr]), dt, self.em)
            atol = 1e-9
            new = torch.cat([torch.stack(x), u[self.ntr:]])
            err = torch.cat([torch.stack(e), torch.zeros_like(u[self.ntr:])])
        den = torch.maximum(u.abs(), new.abs()) * 1e-4 + atol
        return new, math.sqrt(float(((err / den) ** 2).sum()) / u.numel())

    def adaptive(self, half, u, t, tend, dt, seq=None):
        b1, b2, qs = (7 / 30, 2 / 15, 1.0) if half == "T" else (7 / 20, 1 / 5, 6 / 5)
        qold, na, nr = 1e-4, 0, 0
        while t < tend - 1e-9:
            h = min(dt, tend - t)
            new, e = self._attempt(half, u, t, h)
            q11 = max(e, 1e-35) ** b1
            q = max(0.1, min(5.0, (q11 / qold ** b2) / 0.9))
            if e <= 1.0:
                if seq is not None:
                    seq.append((half, t, h, u))
                u, t = new.clamp(min=0.0), t + h
                dt, qold, na = h / (1.0 if 1.0 <= q <= qs else q), max(e, 1e-4), na + 1
            else:
                dt, nr = h / min(5.0, q11 / 0.9), nr + 1
        return u, dt, na, nr

    def macro(self, u, t, dt, dtT, dtC, seq=None):
        counts = [0, 0, 0, 0]
        if self.w.do_transport:
            u, dtT, counts[0], counts[1] = self.adaptive("T", u, t, t + dt, dtT, seq)
        if self.w.do_chemistry:
            u, dtC, counts[2], counts[3] = self.adaptive("C", u, t, t + dt, dtC, seq)
        return u, dtT, dtC, counts

    def backward(self, seq, uend, lam):
        """Reverse sweep along the accepted steps: (dJ/du at the start, dJ/d emission)."""
        grad = torch.zeros_like(self.em)
        out = uend
        for half, t, h, u in reversed(seq):
            lam = lam * (out > 0.0)
            with torch.enable_grad():
                if half == "T":
                    v = u.detach().requires_grad_(True)
                    new, _ = self.transport_step(v, t, h)
                    lam = torch.autograd.grad(new, v, lam)[0]
                else:
                    v = u[:self.ntr].detach().requires_grad_(True)
                    e = self.em.detach().requires_grad_(True)
                    new, _ = self.chem_step(list(v), h, e, error=False)
                    gv, ge = torch.autograd.grad(torch.stack(new), (v, e), lam[:self.ntr])
                    grad += ge
                    lam = torch.cat([gv, lam[self.ntr:]])
            out = u
        return lam, grad


def exact(case, seed):
    kind, dt = case["kind"], case["dt"]
    if kind == "cells":  # thousands of steps in the stiffest cells
        return None
    w = _workload(case, seed)
    m, u = _Math(w), _planes(w, seed)
    with torch.no_grad():
        if kind == "hooks":
            tr = m.rhs_transport(u, 300.0)
            ch = torch.cat([torch.stack(m.rhs_chem(list(u[:-1]), m.em)), torch.zeros_like(u[-1:])])
            return {"transport": _by_species(_cellmajor(tr), w.nsp),
                    "chemistry": _by_species(_cellmajor(ch), w.nsp)}
        if kind == "attempt":
            new, e = m._attempt("C", u, 0.0, dt)
            return {"u": _by_species(new, w.nsp), "eest": e}
        t, dtT, dtC = 0.0, w.dt0_T, w.dt0_C
        if kind in ("step", "adjoint"):
            u, dtT, dtC, _ = m.macro(u, 0.0, 600.0, dtT, dtC)
            t = 600.0
        if kind == "adjoint":
            seq = []
            for _ in range(2):
                u, dtT, dtC, _ = m.macro(u, t, dt, dtT, dtC, seq)
                t += dt
            lam = torch.as_tensor(_lambda(case, w, seed), device=u.device)
            lam, grad = m.backward(seq, u, lam)
            return {"lambda": _by_species(_cellmajor(lam), w.nsp), "emission": list(grad),
                    "dtC": dtC}
        u, dtT, dtC, counts = m.macro(u, t, dt, dtT, dtC)
    if kind == "window":
        return {"u": _by_species(_cellmajor(u), w.nsp), "dtT": dtT, "dtC": dtC,
                "counts": counts + [1]}
    out = {"u": _by_species(u, w.nsp), "dtT": dtT, "counts": counts}
    if kind == "step":
        out["dtC"] = dtC
    return out
