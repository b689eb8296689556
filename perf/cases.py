"""Cases of the work that a program has this library do, with their inputs,
their results in 64 bits and the bytes and operations they cannot do without.

Each case goes through the public entry points (``BarotropicSolver``,
``Ensemble``, ``MLP``) as the host model or a standalone run calls them.
Geometry (coastline, depth, metrics, masks) belongs to a case's sizes and is
built once; the state, the forcing and the 3-D fields come from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from inmsom_elfs_b200 import basins
from inmsom_elfs_b200.closure import ClosureConfig, closure_basins, make_norm
from inmsom_elfs_b200.grid import FORCING, MEANS, SCRATCH, STATE, Basin
from inmsom_elfs_b200.mlp import HID, KIN, MLP, NOUT
from inmsom_elfs_b200.solver import BarotropicSolver, Ensemble, GpuBackend

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # a small idealised basin stepped on its own, then read for output:
        # launches and latency count (the 256 x 256 beta-plane workload)
        dict(name="run beta 256", kind="run", basin="beta", nx=256, ny=256, steps=400, fp32=False),
        # the regional benchmark basin: 40 % land, 6-hour wind cycle, the
        # state read every 800 s of model time
        dict(name="run regional 2048x1536", kind="run", basin="regional", nx=2048, ny=1536, steps=400, fp32=False),
        # the largest basin, with FP32 velocity storage
        dict(name="run ridge 4096 fp32", kind="run", basin="ridge", nx=4096, ny=4096, steps=200, fp32=True),
        # a lat-lon basin of odd sizes: metrics that vary along y
        dict(name="run spherical 701x487", kind="run", basin="spherical", nx=701, ny=487, steps=200, fp32=False),
        # a zonally periodic band on the sphere (Williamson's test 2 on
        # 1.25 x 1 degrees, perturbed, with viscosity)
        dict(name="run periodic 288x160", kind="run", basin="sphere", nx=288, ny=160, steps=100, fp32=False),
        # the coupled model's call: wind forcing in, 100 substeps, time means out
        dict(name="call regional 2048x1536", kind="call", basin="regional", nx=2048, ny=1536, nstep=50, ksw4=0,
             resident=True),
        # the smallest call: every array in and out, biharmonic viscosity,
        # coefficients that vary in space, odd sizes
        dict(name="call biharmonic 93x71", kind="call", basin="regional", nx=93, ny=71, nstep=5, ksw4=1,
             resident=False),
        # an ensemble of regional basins of mixed sizes
        dict(name="ensemble of 10", kind="ens", members=10, lo=192, hi=704, steps=200, persistent=False),
        # a coarse run with the learned closure, evaluated every 10 steps
        dict(name="closure 512", kind="closure", n=512, steps=200, every=10),
        # one training step of that network at the study's batch
        dict(name="train 65536", kind="train", batch=65536, rows=1 << 20),
        # the 3-D velocity of the mode-split step, host arrays in and out
        dict(name="baroclinic 512x384x20", kind="baroclinic", nx=512, ny=384, nz=20),
        # one tracer's step, odd sizes and levels
        dict(name="tracer 301x203x33", kind="tracer", nx=301, ny=203, nz=33),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.randrange(10)
    if k == 0:
        return dict(kind="run", basin="beta", nx=_log(rng, 40, 640), ny=_log(rng, 40, 640), steps=_log(rng, 50, 500),
                    fp32=rng.random() < 0.3)
    if k == 1:
        return dict(kind="run", basin="regional", nx=_log(rng, 150, 2048), ny=_log(rng, 150, 1536),
                    steps=_log(rng, 20, 400), fp32=rng.random() < 0.3)
    if k == 2:
        n = _log(rng, 256, 4096)
        return dict(kind="run", basin="ridge", nx=n, ny=n, steps=_log(rng, 20, 100), fp32=rng.random() < 0.6)
    if k == 3:
        return dict(kind="run", basin="spherical", nx=_log(rng, 60, 1400), ny=_log(rng, 60, 900),
                    steps=_log(rng, 20, 300), fp32=False)
    if k == 4:
        ny = _log(rng, 40, 640)
        return dict(kind="run", basin="sphere", nx=int(1.8 * ny), ny=ny, steps=_log(rng, 10, 200), fp32=False)
    if k == 5:
        return dict(kind="call", basin=rng.choice(("regional", "spherical")), nx=_log(rng, 150, 2048),
                    ny=_log(rng, 150, 1536), nstep=_log(rng, 5, 60), ksw4=0, resident=rng.random() < 0.7)
    if k == 6:
        return dict(kind="call", basin="regional", nx=_log(rng, 60, 900), ny=_log(rng, 60, 700),
                    nstep=_log(rng, 2, 20), ksw4=1, resident=rng.random() < 0.5)
    if k == 7:
        return dict(kind="ens", members=rng.randrange(2, 11), lo=64 * rng.randrange(2, 5),
                    hi=64 * rng.randrange(6, 17), steps=10 * rng.randrange(2, 21), persistent=rng.random() < 0.3)
    if k == 8:
        if rng.random() < 0.5:
            return dict(kind="train", batch=128 * _log(rng, 4, 1024), rows=_log(rng, 1 << 17, 1 << 21))
        every = 2 * rng.randrange(2, 11)
        return dict(kind="closure", n=_log(rng, 96, 1024), steps=every * rng.randrange(2, 16), every=every)
    return dict(kind=rng.choice(("baroclinic", "tracer")), nx=_log(rng, 40, 700), ny=_log(rng, 40, 500),
                nz=rng.randrange(5, 51))


# ------------------------------------------------------------------ geometry
@functools.lru_cache(maxsize=32)
def _geometry(kind, nx, ny):
    """Masks, metrics, Coriolis, depth and coefficients of a basin."""
    if kind == "beta":
        b = basins.beta_plane_basin(n=nx, ny=ny)
    elif kind == "regional":
        b = basins.regional_basin(nx=nx, ny=ny)
    elif kind == "ridge":
        b = basins.ridge_basin(n=nx)
    elif kind == "spherical":
        # 20 degrees of latitude whatever the size; a stable step
        b = basins.spherical_basin(nx=nx, ny=ny, dxst=25.0 / ny, dyst=20.0 / ny, dt=120.0 * 20.0 / ny)
    elif kind == "closure":
        return closure_basins(ClosureConfig(n_coarse=nx), GpuBackend(), which=("base",))["base"]
    else:
        b = basins.williamson2_basin(dlon=360.0 / nx, dlat=160.0 / ny, dt=40.0 * 160.0 / ny)
        b.forcing["mu"][...] = 1.0e4
        b.forcing["rdis"][...] = 1.0e-6
    b.masks.update(GpuBackend().gridcon(b.bounds, b.masks["lu"]))
    return b


def _modes(rng, shape, amp, n=4):
    """A smooth field: n products of sinusoids."""
    x, y = np.linspace(0.0, 1.0, shape[0]), np.linspace(0.0, 1.0, shape[1])
    fx = np.stack([np.sin(2 * math.pi * (rng.integers(1, 7) * x + rng.random())) for _ in range(n)])
    fy = np.stack([np.sin(2 * math.pi * (rng.integers(1, 7) * y + rng.random())) for _ in range(n)])
    return np.asfortranarray((amp / math.sqrt(n)) * (fy.T @ fx).T)


def _host(shape, fill=None):
    """A Fortran-ordered array in pinned memory, as a host model keeps the
    arrays that it exchanges with the device."""
    t = torch.empty(tuple(reversed(shape)), dtype=F64, pin_memory=True)
    if fill is None:
        t.zero_()
    else:
        t.copy_(torch.from_numpy(np.ascontiguousarray(fill.T)))
    return t.numpy().T


def _wrap_x(b, a):
    if b.periodicity_x:
        i0, i1 = b.mmm - b.bnd_x1, b.mm - b.bnd_x1
        a[i0 - 1], a[i1 + 1] = a[i1].copy(), a[i0].copy()


def _basin(kind, nx, ny, seed, varied=False):
    """A basin with the case's geometry and the seed's state and forcing."""
    g = _geometry(kind, nx, ny)
    rng = np.random.default_rng([int(seed) & 0xFFFFFFFF, nx, ny])
    b = Basin(g.bounds, g.consts, g.masks, g.metrics, g.rlh_s, g.hhq_rest, dt=g.dt, info=g.info)
    m, mt, shp = g.masks, g.metrics, g.bounds.shape
    vel, lev = (0.05, 0.05) if kind == "regional" else (0.02, 0.2)
    now = {"ubrtr_e": _modes(rng, shp, vel) * m["lcu"], "vbrtr_e": _modes(rng, shp, vel) * m["lcv"],
           "ssh_e": _modes(rng, shp, lev) * m["lu"]}
    if kind == "sphere":
        eta, u = basins.williamson2_fields(g)
        now["ssh_e"] += eta
        now["ubrtr_e"] += u
    for k, v in now.items():
        _wrap_x(g.bounds, v)
        b.state[k] = _host(shp, v)
        b.state[{"ubrtr_e": "ubrtrp_e", "vbrtr_e": "vbrtrp_e", "ssh_e": "sshp_e"}[k]] = _host(shp, v)
    b.state = {k: b.state[k] for k in STATE}
    b.means = {k: _host(shp) for k in MEANS}
    rho = b.consts.ref_den
    b.forcing = {"RHSx": _host(shp, _modes(rng, shp, 0.1 / rho) * mt["dxt"] * mt["dyh"] * m["lcu"]),
                 "RHSy": _host(shp, _modes(rng, shp, 0.1 / rho) * mt["dyt"] * mt["dxh"] * m["lcv"]),
                 "wflux": _host(shp), "mu": _host(shp, g.forcing["mu"]), "mu4": _host(shp),
                 "rdis": _host(shp, g.forcing["rdis"])}
    if varied:
        b.forcing["mu"] = _host(shp, 500.0 + 1000.0 * rng.random(shp))
        b.forcing["mu4"] = _host(shp, np.full(shp, 3.0e4))
        b.forcing["rdis"] = _host(shp, 1.0e-6 * (1.0 + rng.random(shp)))
        b.forcing["wflux"] = _host(shp, 1.0e-2 * rng.standard_normal(shp))
    b.scratch = {k: _host(shp) for k in SCRATCH}
    return b


def _sides(c):
    rng = np.random.default_rng(c["members"] * 1000 + c["lo"] + c["hi"])
    return [tuple(int(64 * x) for x in rng.integers(c["lo"] // 64, c["hi"] // 64 + 1, 2)) for _ in range(c["members"])]


def _scale(c, dt):
    return basins.wind_cycle(c["steps"], dt) if c.get("basin") == "regional" else None


# ------------------------------------------------------------------ the cases
def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "run":
        b = _basin(c["basin"], c["nx"], c["ny"], seed)
        s = BarotropicSolver(b, register_depths=False, fp32_velocity=c["fp32"])
        s.load_state()
        return dict(kind=kind, solver=s, steps=c["steps"], scale=_scale(c, b.dt))
    if kind == "call":
        b = _basin(c["basin"], c["nx"], c["ny"], seed, varied=c["ksw4"] > 0)
        s = BarotropicSolver(b, register_depths=False, resident=c["resident"], static_coeffs=c["resident"])
        if c["resident"]:
            s.load_state()
        return dict(kind=kind, solver=s, nstep=c["nstep"], ksw4=c["ksw4"], resident=c["resident"])
    if kind == "ens":
        ms = []
        for k, (nx, ny) in enumerate(_sides(c)):
            ms.append(BarotropicSolver(_basin("regional", nx, ny, seed * 64 + k), register_depths=False))
            ms[-1].load_state()
        return dict(kind=kind, ens=Ensemble(ms, persistent=c["persistent"]), steps=c["steps"],
                    dt=[m.basin.dt for m in ms])
    if kind == "closure":
        b = _basin("closure", c["n"], c["n"], seed)
        s = BarotropicSolver(b, register_depths=False)
        s.load_state()
        st = b.state
        norm = make_norm(b, st["ubrtr_e"], st["vbrtr_e"], st["ssh_e"], (1.0e-7, 1.0e-7))
        return dict(kind=kind, solver=s, net=MLP(seed=seed), norm=norm, steps=c["steps"], every=c["every"])
    if kind == "train":
        x, t, idx, m, v = _batch(c, seed)
        net = MLP(seed=seed)
        net.m, net.v, net.step = m, v, 1000        # a training under way
        return dict(kind=kind, net=net, x=x, t=t, idx=idx)
    b = _basin("regional", c["nx"], c["ny"], seed)
    dz, hzt = basins.vertical_grid(c["nz"], 0)
    f = (_column_fields if kind == "baroclinic" else _tracer_fields)(b, c["nz"], seed)
    f = {k: _host_of(v) if isinstance(v, torch.Tensor) else v for k, v in f.items()}
    s = BarotropicSolver(b, register_depths=False)
    out = dict(kind=kind, solver=s, dz=dz, hzt=hzt, f=f)
    if kind == "tracer":
        out["flux"] = [_host((*b.bounds.shape, 4)) for _ in range(2)]
    else:
        f.pop("wflux")
    return out


def run(state):
    kind = state["kind"]
    if kind == "run":
        s = state["solver"]
        s.run_substeps(state["steps"], s.basin.dt, state["scale"])
        s.sync_to_host()
        return s.basin.state
    if kind == "call":
        s = state["solver"]
        b = s.basin
        s.barotropic_dynamics(state["nstep"] * b.dt, state["nstep"], state["ksw4"])
        return b.means if state["resident"] else {"state": b.state, "means": b.means, "scratch": b.scratch}
    if kind == "ens":
        e = state["ens"]
        e.run(state["steps"], state["dt"])
        for m in e.members:
            m.sync_to_host()
        return [m.basin.state for m in e.members]
    if kind == "closure":
        s, net = state["solver"], state["net"]
        s.run_closure(state["steps"], s.basin.dt, state["every"], net.params.data_ptr(), net.wbf16.data_ptr(),
                      state["norm"])
        s.sync_to_host()
        return s.basin.state
    if kind == "train":
        net = state["net"]
        net.loss_grad(state["x"], state["t"], state["idx"])
        net.adam()
        return {"grad": net.grad, "params": net.params, "m": net.m, "v": net.v}
    s, f = state["solver"], state["f"]
    if kind == "baroclinic":
        fields = {k: v for k, v in f.items() if k not in ("uu", "uup", "vv", "vvp")}
        return list(s.baroclinic_dynamics(state["dz"], state["hzt"], TAU, f["uu"], f["uup"], f["vv"], f["vvp"], **fields))
    return list(s.tracer_tran_diff(state["dz"], state["hzt"], TAU, f["ff"], f["ffp"], *state["flux"], f))


def work(case):
    """A substep reads two levels of three fields, the depth and the forcing
    and writes two levels; 3-D calls read and write each field once."""
    c = dict(case)
    kind = c["kind"]

    def ocean(k, nx, ny):
        return float(_geometry(k, nx, ny).masks["lu"].sum())

    if kind == "run":
        n, pts = ocean(c["basin"], c["nx"], c["ny"]) * c["steps"], (c["nx"] + 4) * (c["ny"] + 4)
        return {"bytes": n * (80 if c["fp32"] else 120) + 48.0 * pts, "flops": 110.0 * n}
    if kind == "call":
        n, pts = ocean(c["basin"], c["nx"], c["ny"]) * 2 * c["nstep"], (c["nx"] + 4) * (c["ny"] + 4)
        per = 240 if c["ksw4"] else 152
        return {"bytes": n * per + 8.0 * pts * (6 if c["resident"] else 44), "flops": (250.0 if c["ksw4"] else 120.0) * n}
    if kind == "ens":
        n = sum(ocean("regional", nx, ny) for nx, ny in _sides(c)) * c["steps"]
        pts = sum((nx + 4) * (ny + 4) for nx, ny in _sides(c))
        return {"bytes": n * 120 + 48.0 * pts, "flops": 110.0 * n}
    if kind == "closure":
        n, ev = float(c["n"] ** 2), c["steps"] // c["every"]
        return {"bytes": n * (120 * c["steps"] + 88 * ev + 48),
                "flops": n * (110.0 * c["steps"] + 2.0 * (KIN * HID + HID * HID + 2 * HID) * ev)}
    if kind == "train":
        return {"bytes": c["batch"] * (2.0 * KIN + 4 + 4 * NOUT) + 7816 * 40,
                "flops": c["batch"] * 6.0 * (KIN * HID + HID * HID + NOUT * HID)}
    pts, nz = float((c["nx"] + 4) * (c["ny"] + 4)), c["nz"]
    if kind == "baroclinic":
        return {"bytes": pts * (112 * nz + 200), "flops": pts * nz * 120}
    return {"bytes": pts * (112 * nz + 240), "flops": pts * nz * 200}


# ------------------------------------------------------------------ inputs
TAU = 60.0        # s, the model step of the 3-D calls


def _batch(c, seed):
    """Feature rows (48 BF16, 45 used), targets, one batch of row numbers and
    Adam's moments in the middle of a training."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.randn((c["rows"], KIN), generator=g, device=DEV)
    x[:, 45:] = 0.0
    t = 0.5 * torch.tanh(x[:, :NOUT] + 0.3 * x[:, 9:9 + NOUT] * x[:, 18:18 + NOUT])
    idx = torch.randint(0, c["rows"], (c["batch"],), generator=g, device=DEV, dtype=torch.int32)
    m = 1e-3 * torch.randn(7816, generator=g, device=DEV)
    v = 1e-5 * (0.5 + torch.rand(7816, generator=g, device=DEV))
    used = _unpadded()
    return x.to(torch.bfloat16), t.contiguous(), idx, m * used, v * used


def _unpadded():
    """1 at the parameters in use: inputs 45..47 and outputs 2..7 are padding."""
    u = torch.ones(7816, device=DEV)
    u[45 * HID:KIN * HID] = 0.0
    o = KIN * HID + HID + HID * HID + HID
    u[o:o + 8 * HID].view(HID, 8)[:, NOUT:] = 0.0
    u[o + 8 * HID + NOUT:] = 0.0
    return u


def _host_of(t):
    """Device field (levels, rows, columns) -> pinned Fortran-ordered array."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy().transpose(*reversed(range(t.dim())))


def _makers(b, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    shp = tuple(reversed(b.bounds.shape))

    def normal(s, lev=None, loc=0.0):
        return loc + s * torch.randn(shp if lev is None else (lev, *shp), generator=g, device=DEV, dtype=F64)

    def uniform(lo, hi, lev=None):
        return lo + (hi - lo) * torch.rand(shp if lev is None else (lev, *shp), generator=g, device=DEV, dtype=F64)

    return g, shp, normal, uniform


def _column_fields(b, nz, seed, depth=50.0):
    """The distributions of basins.column_fields, made on the device."""
    _, _, nrm, uni = _makers(b, seed)
    s = depth * float(np.median(b.metrics["dxt"]) * np.median(b.metrics["dyh"])) / TAU * 0.1
    f = {k: nrm(0.1, nz) for k in ("uu", "uup", "vv", "vvp")}
    f.update(ww=nrm(1e-3, nz + 1), nu=uni(1e-4, 1e-2, nz + 1))
    f.update({k: nrm(0.05 * s, nz) for k in ("rhsx", "rhsy", "rhsx_tran", "rhsy_tran")})
    f.update(pgrx=nrm(0.05 * s), pgry=nrm(0.05 * s), rdis=uni(0.0, 2e-5))
    f.update({k: nrm(1e-4) for k in ("tx_surf", "ty_surf", "tx_bot", "ty_bot")})
    f.update({k: uni(0.8 * depth, 1.2 * depth) for k in ("hhu", "hhup", "hhun", "hhv", "hhvp", "hhvn", "hhh")})
    f["wflux"] = nrm(1e-2)
    return f


def _tracer_fields(b, nz, seed, depth=50.0):
    """The distributions of basins.tracer_fields, made on the device."""
    g, shp, nrm, uni = _makers(b, seed)
    f = dict(ff=nrm(3.0, nz, 10.0), ffp=nrm(3.0, nz, 10.0), uu=nrm(0.1, nz), vv=nrm(0.1, nz), ww=nrm(1e-3, nz + 1),
             mu=uni(50.0, 500.0, nz), nu=uni(1e-5, 1e-3, nz + 1))
    f.update({k: nrm(1e-3, nz + 1) for k in ("slrx", "slry", "slzx", "slzy")})
    f.update(ff_top=nrm(2.0, None, 15.0), ff_bot=nrm(1.0, None, 4.0), swbal=uni(0.0, 1.0), src=nrm(1e-6, nz))
    f.update({k: torch.randint(1, 3, shp, generator=g, device=DEV, dtype=torch.int32) for k in ("ig_top", "ig_bot")})
    f.update({k: uni(0.8 * depth, 1.2 * depth) for k in ("hhu", "hhv", "hhqn", "hhqp")})
    f.update(factor_mu=1.0, factor_nu=1.0, az=0.3, ar=0.7, alpha_gm=1.0, src_factor=1.0)
    return f


# ------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "run":
        b = _basin(c["basin"], c["nx"], c["ny"], seed)
        return _exact_run(b, c["steps"], _scale(c, b.dt))
    if kind == "call":
        b = _basin(c["basin"], c["nx"], c["ny"], seed, varied=c["ksw4"] > 0)
        r = _Step(b)
        means = r.dynamics(c["nstep"] * b.dt, c["nstep"], c["ksw4"])
        if c["resident"]:
            return means
        return {"state": r.out(), "means": means, "scratch": {k: _np(r.scr[k]) for k in SCRATCH}}
    if kind == "ens":
        return [_exact_run(_basin("regional", nx, ny, seed * 64 + k), c["steps"], None)
                for k, (nx, ny) in enumerate(_sides(c))]
    if kind == "closure":
        b = _basin("closure", c["n"], c["n"], seed)
        return _exact_closure(b, MLP(seed=seed), c["steps"], c["every"])
    if kind == "train":
        return _exact_train(c, seed)
    b = _basin("regional", c["nx"], c["ny"], seed)
    dz, hzt = (v.tolist() for v in basins.vertical_grid(c["nz"], 0))
    if kind == "baroclinic":
        return _exact_baroclinic(b, dz, hzt, _column_fields(b, c["nz"], seed))
    return _exact_tracer(b, dz, hzt, _tracer_fields(b, c["nz"], seed))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a.T)).to(DEV, F64)


def _np(t):
    return t.cpu().numpy().transpose(*reversed(range(t.dim())))


def _e(a): return torch.roll(a, -1, -1)      # value at m + 1
def _w(a): return torch.roll(a, 1, -1)       # m - 1
def _n(a): return torch.roll(a, -1, -2)      # n + 1
def _s(a): return torch.roll(a, 1, -2)       # n - 1


class _Grid:
    def __init__(self, b):
        self.b = B = b.bounds
        self.__dict__.update({k: _dev(v) for k, v in b.metrics.items()})
        self.rlh, self.hr = _dev(b.rlh_s), _dev(b.hhq_rest)
        self.k = b.consts

        def box(lo, hi):
            z = torch.zeros(tuple(reversed(B.shape)), dtype=torch.bool, device=DEV)
            z[B.ny_start - lo - B.bnd_y1:B.ny_end + hi + 1 - B.bnd_y1, B.nx_start - lo - B.bnd_x1:B.nx_end + hi + 1 - B.bnd_x1] = True
            return z

        self.m = {k: _dev(v) for k, v in b.masks.items()}
        wet = {k: v > 0.5 for k, v in self.m.items()}
        self.inner = {k: v & box(0, 0) for k, v in wet.items()}
        self.ring = {k: v & box(1, 1) for k, v in wet.items()}
        self.low = {k: v & box(1, 0) for k, v in wet.items()}

    def wrap(self, a):
        B = self.b
        if B.periodicity_x:
            i0, i1 = B.mmm - B.bnd_x1, B.mm - B.bnd_x1
            l, r = a[..., i1].clone(), a[..., i0].clone()
            a[..., i0 - 1], a[..., i1 + 1] = l, r
        return a


class _Step(_Grid):
    """The leap-frog barotropic substep, loop by loop (Function/vel_ssh.f90:
    379-679), on whole arrays."""

    def __init__(self, b):
        super().__init__(b)
        self.st = {k: _dev(v) for k, v in b.state.items()}
        self.f = {k: _dev(b.forcing[k]) for k in FORCING}
        z = torch.zeros_like(self.hr)
        self.scr = {k: z.clone() for k in SCRATCH}
        self.un, self.vn, self.sn = z.clone(), z.clone(), z.clone()
        self.h = None

    def out(self):
        return {k: _np(v) for k, v in self.st.items()}

    def depths(self, hq, old=None):
        m, where = self.m, torch.where
        a = hq * self.dx * self.dy * m["lu"]
        u = (a + _e(a)) / (m["lu"] + _e(m["lu"])) / self.dxt / self.dyh
        v = (a + _n(a)) / (m["lu"] + _n(m["lu"])) / self.dxh / self.dyt
        s = a + _e(a) + _n(a) + _n(_e(a))
        c = m["lu"] + _e(m["lu"]) + _n(m["lu"]) + _n(_e(m["lu"]))
        h = s / c / self.dxb / self.dyb
        z = torch.zeros_like(hq)
        return [hq] + [self.wrap(where(self.low[k], x, z)) for k, x in (("llu", u), ("llv", v), ("luh", h))]

    def stress(self, u, v, t, s):
        a, b = u / self.dyh, v / self.dxh
        tn = self.dy / self.dx * (a - _w(a)) - self.dx / self.dy * (b - _s(b))
        a, b = u / self.dxt, v / self.dyt
        sn = self.dxb / self.dyb * (_n(a) - a) + self.dyb / self.dxb * (_e(b) - b)
        return self.wrap(torch.where(self.inner["lu"], tn, t)), self.wrap(torch.where(self.inner["luu"], sn, s))

    def diff(self, mu, t, s, hq, hh):
        a = self.dy * self.dy * mu * hq * t
        b = self.dx * self.dx * mu * hq * t
        muh = (mu + _e(mu) + _n(mu) + _n(_e(mu))) / 4.0
        p = self.dxb * self.dxb * muh * hh * s
        q = self.dyb * self.dyb * muh * hh * s
        return (_e(a) - a) / self.dyh + (p - _s(p)) / self.dxt, -(_n(b) - b) / self.dxh + (q - _w(q)) / self.dyt

    def substep(self, ti, nstep, ksw4, scale, means=None):
        where, I, R, st, f, g, scr = torch.where, self.inner, self.ring, self.st, self.f, self.k.free_fall_acc, self.scr
        u, up, v, vp, e, ep = (st[k] for k in STATE)
        (hq, hu, hv, hh), (_, hup, hvp, _) = self.h[0], self.h[1]
        U, V = u * hu * self.dyh, v * hv * self.dxh
        div = U - _w(U) + V - _s(V)
        self.sn = self.wrap(where(I["lu"], ep + 2.0 * ti * (f["wflux"] / self.k.ref_den - div / (self.dx * self.dy)), self.sn))
        new = self.depths(self.hr + self.sn)
        hun, hvn = new[1], new[2]
        t, s = self.stress(up, vp, scr["str_t2d"], scr["str_s2d"])
        a, b = v * self.dyt, u * self.dxt
        vort = (_e(a) - a) - (_n(b) - b) - ((_e(v) - v) * self.dyb - (_n(u) - u) * self.dxb)
        vort = self.wrap(where(I["luu"], vort, scr["vort"]))
        fx, fy = (U + _e(U)) / 2.0 * (u + _e(u)) / 2.0, (V + _e(V)) / 2.0 * (_n(u) + u) / 2.0 * self.m["luu"]
        w = vort * hh * (_e(v) + v)
        ax = -(fx - _w(fx) + fy - _s(fy)) + (w + _s(w)) / 4.0
        fy, fx = (V + _n(V)) / 2.0 * (v + _n(v)) / 2.0, (U + _n(U)) / 2.0 * (_e(v) + v) / 2.0
        w = vort * hh * (_n(u) + u)
        ay = -(fx - _w(fx) + fy - _s(fy)) - (w + _w(w)) / 4.0
        dx, dy = self.diff(f["mu"], t, s, hq, hh)
        if ksw4:
            px, py = self.diff(f["mu4"], t, s, hq, hh)
            z = torch.zeros_like(px)
            scr["fx"] = self.wrap(where(I["lcu"], -px / hu / self.dxt / self.dyh, z))
            scr["fy"] = self.wrap(where(I["lcv"], -py / hv / self.dxh / self.dyt, z))
            t, s = self.stress(scr["fx"], scr["fy"], t, s)
            px, py = self.diff(f["mu4"], t, s, hq, hh)
            dx, dy = dx + px, dy + py
        scr.update(vort=vort, str_t2d=t, str_s2d=s)
        for k, x, m in (("RHSx_adv", ax, "lcu"), ("RHSy_adv", ay, "lcv"), ("RHSx_dif", dx, "lcu"), ("RHSy_dif", dy, "lcv")):
            scr[k] = where(I[m], x, scr[k])
        k = self.rlh * hh * self.dxb * self.dyb
        sl, sln = -g * (_e(e) - e) * self.dyh * hu, -g * (_e(self.sn) - self.sn) * self.dyh * hun
        cx = k * (_e(v) + v)
        area = self.dxt * self.dyh
        gr = f["RHSx"] * scale + sl + dx + ax - (f["rdis"] + _e(f["rdis"])) / 2.0 * up * area * hu + (cx + _s(cx)) / 4.0
        un = (up * hup * area / 2.0 / ti + gr) / (hun * area / 2.0 / ti)
        self.un = where(I["lcu"], un, self.un)
        tl, tln = -g * (_n(e) - e) * self.dxh * hv, -g * (_n(self.sn) - self.sn) * self.dxh * hvn
        cy = k * (_n(u) + u)
        area = self.dyt * self.dxh
        gr = f["RHSy"] * scale + tl + dy + ay - (f["rdis"] + _n(f["rdis"])) / 2.0 * vp * area * hv - (cy + _w(cy)) / 4.0
        vn = (vp * hvp * area / 2.0 / ti + gr) / (hvn * area / 2.0 / ti)
        self.vn = where(I["lcv"], vn, self.vn)
        if means is not None:
            for n, x, m in (("ubrtr_i", u * hu + self.un * hun, "lcu"), ("vbrtr_i", v * hv + self.vn * hvn, "lcv"),
                            ("ssh4gradx", sl + sln, "lcu"), ("ssh4grady", tl + tln, "lcv")):
                means[n] = where(I[m], means[n] + x / (4.0 * nstep), means[n])
        self.un, self.vn = self.wrap(self.un.clone()), self.wrap(self.vn.clone())
        c = self.k.time_smooth / 2.0 / nstep
        for cur, prev, new_, m in (("ssh_e", "sshp_e", self.sn, "lu"), ("ubrtr_e", "ubrtrp_e", self.un, "lcu"),
                                   ("vbrtr_e", "vbrtrp_e", self.vn, "lcv")):
            x, y = st[cur], st[prev]
            st[prev] = where(R[m], x + c * (new_ - 2.0 * x + y), y)
            st[cur] = where(R[m], new_, x)
        out = []
        for i, m in enumerate(("lu", "llu", "llv", "luh")):
            x, y, z = self.h[0][i], self.h[1][i], new[i]
            out.append((where(R[m], z, x), where(R[m], x + c * (z - 2.0 * x + y), y)))
        self.h = [[o[0] for o in out], [o[1] for o in out]]

    def depths_of_state(self):
        self.h = [self.depths(self.hr + self.st["ssh_e"]), self.depths(self.hr + self.st["sshp_e"])]

    def dynamics(self, tau, nstep, ksw4):
        self.depths_of_state()
        means = {k: torch.zeros_like(self.hr) for k in MEANS}
        keep = None
        for k in range(1, 2 * nstep + 1):
            self.substep(tau / nstep, nstep, ksw4, 1.0, means)
            if k == nstep:
                keep = dict(self.st)
        self.st = keep
        self.wrap(means["ubrtr_i"])
        self.wrap(means["vbrtr_i"])
        return {k: _np(v) for k, v in means.items()}

    def steps(self, n, dt, scale):
        for k in range(n):
            self.depths_of_state()
            self.substep(dt, 1, 0, 1.0 if scale is None else float(scale[k]))


def _exact_run(b, steps, scale):
    r = _Step(b)
    r.steps(steps, b.dt, scale)
    return r.out()


def _layers(net_wb, prm):
    """Weights as the network holds them (BF16 copies, FP32 biases) in 64 bits."""
    w, p = net_wb.double(), prm.double()
    n1, n2 = KIN * HID, KIN * HID + HID * HID
    o = n1 + HID + HID * HID
    return (w[:n1].view(KIN, HID), p[n1:n1 + HID], w[n1:n2].view(HID, HID), p[o:o + HID], w[n2:].view(HID, 8),
            p[o + HID + 8 * HID:])


_C0 = math.sqrt(2.0 / math.pi)
_C1 = _C0 * 0.044715


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(z * (_C0 + _C1 * z * z)))


def _gelu_d(z):
    t = torch.tanh(z * (_C0 + _C1 * z * z))
    return 0.5 * (1.0 + t) + 0.5 * z * (1.0 - t * t) * (_C0 + 3.0 * _C1 * z * z)


def _exact_closure(b, net, steps, every):
    st = b.state
    norm = make_norm(b, st["ubrtr_e"], st["vbrtr_e"], st["ssh_e"], (1.0e-7, 1.0e-7))
    w1, b1, w2, b2, w3, b3 = _layers(net.wbf16, net.params)
    r = _Step(b)
    base = r.f["RHSx"], r.f["RHSy"]
    z = torch.zeros_like(r.hr)
    fac = [torch.where(r.inner["lcu"], 0.5 * (r.hr + _e(r.hr)) * r.dxt * r.dyh, z),
           torch.where(r.inner["lcv"], 0.5 * (r.hr + _n(r.hr)) * r.dyt * r.dxh, z)]
    for k in range(0, steps, every):
        x = []
        for i, a in enumerate((r.st["ubrtr_e"], r.st["vbrtr_e"], r.st["ssh_e"], r.hr, r.rlh)):
            a = (a - norm.mean[i]) * norm.inv_std[i]
            x += [torch.roll(a, (-dy, -dx), (0, 1)) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
        x = torch.stack(x, -1)
        y = _gelu(_gelu(x @ w1[:45] + b1) @ w2 + b2) @ w3 + b3
        r.f["RHSx"] = base[0] + y[..., 0] * norm.out_scale[0] * fac[0]
        r.f["RHSy"] = base[1] + y[..., 1] * norm.out_scale[1] * fac[1]
        r.steps(every, b.dt, None)
    return r.out()


def _exact_train(c, seed):
    x, t, idx, m, v = _batch(c, seed)
    net = MLP(seed=seed)
    w1, b1, w2, b2, w3, b3 = _layers(net.wbf16, net.params)
    x, t = x[idx.long()].double(), t[idx.long()].double()
    z1 = x @ w1 + b1
    a1 = _gelu(z1)
    z2 = a1 @ w2 + b2
    a2 = _gelu(z2)
    err = (a2 @ w3 + b3)[:, :NOUT] - t
    d3 = torch.zeros((x.shape[0], 8), dtype=F64, device=DEV)
    d3[:, :NOUT] = 2.0 * err / (x.shape[0] * NOUT)
    d2 = (d3 @ w3.T) * _gelu_d(z2)
    d1 = (d2 @ w2.T) * _gelu_d(z1)
    g = torch.cat([(x.T @ d1).reshape(-1), d1.sum(0), (a1.T @ d2).reshape(-1), d2.sum(0), (a2.T @ d3).reshape(-1),
                   d3.sum(0)])
    loss = (err * err).mean().reshape(1)
    used = _unpadded().double()
    m, v = m.double(), v.double()
    m = torch.where(used > 0, 0.9 * m + 0.1 * g, m)
    v = torch.where(used > 0, 0.999 * v + 0.001 * g * g, v)
    step = 1001
    upd = 1e-3 * (m / (1.0 - 0.9 ** step)) / (torch.sqrt(v / (1.0 - 0.999 ** step)) + 1e-8)
    return {"grad": torch.cat([g, loss]), "params": net.params.double() - upd * used, "m": m, "v": v}


def _thomas(A, D, C, E):
    x, y = [-C[0] / D[0]], [E[0] / D[0]]
    for j in range(1, len(A)):
        s = 1.0 / (A[j] * x[-1] + D[j])
        y.append((E[j] - A[j] * y[-1]) * s)
        x.append(-C[j] * s)
    r = [y[-1]]
    for j in range(len(A) - 2, -1, -1):
        r.append(x[j] * r[-1] + y[j])
    return torch.stack(r[::-1])


def _filtered(g, mask, cur, prev, new):
    """The Robert-Asselin filter on the interior and its ring; the new value
    is zero where no column was solved."""
    ts = g.k.time_smooth
    new = torch.where(g.inner[mask], new, torch.zeros_like(new))
    g.wrap(new)
    return (_np(torch.where(g.ring[mask], new, cur)),
            _np(torch.where(g.ring[mask], cur + ts * (new - 2.0 * cur + prev) / 2.0, prev)))


def _exact_baroclinic(b, dz, hzt, f):
    """Function/vel_ssh.f90:794-1027 in every water column at once."""
    g = _Grid(b)
    nz, out = len(dz), []
    for V in (False, True):
        far, partner = (_n, _w) if V else (_e, _s)
        x = (lambda a, b_: b_) if V else (lambda a, b_: a)
        cur, prev, other = x(f["uu"], f["vv"]), x(f["uup"], f["vvp"]), x(f["vv"], f["uu"])
        f1, f2 = x(g.dxt, g.dxh), x(g.dyh, g.dyt)
        hn = x(f["hhun"], f["hhvn"])
        bp, bp0 = hn * f1 * f2 / TAU / 2.0, x(f["hhup"], f["hhvp"]) * f1 * f2 / TAU / 2.0
        kc = g.rlh * f["hhh"] * g.dxb * g.dyb
        cor = kc * (far(other) + other)
        cor = (cor + partner(cor)) / 4.0
        drag = (f["rdis"] + far(f["rdis"])) / 2.0 * f1 * f2 * x(f["hhu"], f["hhv"])
        rhs = x(f["rhsx"], f["rhsy"]) + x(f["rhsx_tran"], f["rhsy_tran"]) + x(f["pgrx"], f["pgry"])
        A, D, C, E = [], [], [], []
        z = torch.zeros_like(bp)
        dp, fz = z, z
        for q in range(nz):
            dm, fm = dp, fz
            dp = fz = z
            if q < nz - 1:
                dp = (f["nu"][q + 1] + far(f["nu"][q + 1])) / 2.0 / hn / hzt[q + 1] * f1 * f2
                ww = f["ww"][q + 1] * g.dx * g.dy
                fz = (ww + far(ww)) / 2.0 * (cur[q] + cur[q + 1]) / 2.0
            eta = bp0 * prev[q] + rhs[q] - (fz - fm) / dz[q] + x(cor, -cor)[q] - drag * prev[q]
            if q == 0:
                eta = eta + x(f["tx_surf"], f["ty_surf"]) / dz[q] * f1 * f2
            if q == nz - 1:
                eta = eta + x(f["tx_bot"], f["ty_bot"]) / dz[q] * f1 * f2
            A.append(-dm / dz[q])
            C.append(-dp / dz[q])
            D.append(bp + (dp + dm) / dz[q])
            E.append(eta)
        out += _filtered(g, "lcv" if V else "lcu", cur, prev, _thomas(A, D, C, E))
    return out


def _exact_tracer(b, dz, hzt, f):
    """Function/tem_sal.f90:1-422 in every water column at once."""
    g = _Grid(b)
    nz, ff, ffp = len(dz), f["ff"], f["ffp"]
    z = torch.zeros_like(g.hr)
    F, FZ, CO, SG, FO = {}, {}, {}, {}, {}
    for d, far, mask, h, side, norm, vel in (("x", _e, "lcu", "hhu", g.dyh, g.dxt, "uu"), ("y", _n, "lcv", "hhv", g.dxh, g.dyt, "vv")):
        wet, hh = g.inner[mask], f[h]
        fd1, fz, co, sg = ([z] * (nz + 1) for _ in range(4))
        fd1, fz, co, sg = list(fd1), list(fz), list(co), list(sg)
        for k in range(1, nz):
            p, q = ffp[k], ffp[k - 1]
            dfdz = (p - q + far(p) - far(q)) / 2.0
            dfdh = (far(p) - p + far(q) - q) / 2.0
            mu = f["mu"][k] + f["mu"][k - 1]
            mu = (mu + far(mu)) / 4.0 * f["factor_mu"] * side / norm
            slr, slz = f["slr" + d][k], f["slz" + d][k]
            sl = f["ar"] * slr + f["az"] * slz
            fd1[k] = torch.where(wet, mu * (hh * dfdh * hzt[k] - sl * dfdz), z)
            fz[k] = torch.where(wet, mu * sl * dfdh, z)
            co[k] = torch.where(wet, mu * sl * sl / hh / hzt[k], z)
            sg[k] = torch.where(wet, mu * (slr - slz) * f["alpha_gm"], z)
        tot, F[d] = [z, z, z, z], []
        for q in range(nz):
            if q == 0:
                fd = fd1[1] / hzt[1]
            elif q < nz - 1:
                fd = (fd1[q] + fd1[q + 1]) / dz[q] / 2.0
            else:
                fd = fd1[q] / hzt[q]
            s2 = ff[q] + far(ff[q])
            fa = -(f[vel][q] * hh * side * s2 / 2.0)
            fg = -((sg[q + 1] - sg[q]) / dz[q] * s2 / 2.0)
            F[d].append(torch.where(wet, fa + fd + fg, z))
            tot = [t + dz[q] * v for t, v in zip(tot, (fa + fd + fg, fa, fd, fg))]
        FZ[d], CO[d], SG[d] = fz, co, sg
        FO[d] = _np(torch.stack([torch.where(wet, t, z) for t in tot]))
    hn, dxy = f["hhqn"], g.dx * g.dy
    bp, bp0 = hn * dxy / TAU / 2.0, f["hhqp"] * dxy / TAU / 2.0
    cu, cv = ((g.m[k] + s(g.m[k])).clamp_min(1e-10) for k, s in (("lcu", _w), ("lcv", _s)))
    A, D, C, E = [], [], [], []
    fz, dp = z, z
    for q in range(nz):
        k = q + 1
        fm = fz
        nu = f["nu"][k] * f["factor_nu"] * dxy / hn / hzt[k]
        dm = f["nu"][0] * f["factor_nu"] * dxy / hn / hzt[0] if q == 0 else dp
        if k < nz:
            sx, sy, dq = SG["x"][k], SG["y"][k], ffp[k] - ffp[q]
            vg = -(sx - _w(sx) + sy - _s(sy))
            cx, cy = CO["x"][k], CO["y"][k]
            fz = (-(FZ["x"][k] + _w(FZ["x"][k])) / cu - (FZ["y"][k] + _s(FZ["y"][k])) / cv
                  + (cx * _e(dq) + _w(cx) * _w(dq)) / cu / 2.0 + (cy * _n(dq) + _s(cy) * _s(dq)) / cv / 2.0
                  - (f["ww"][k] * dxy + vg) * (ff[q] + ff[k]) / 2.0)
            dp = (cx + _w(cx)) / cu / 2.0 + (cy + _s(cy)) / cv / 2.0 + nu
        else:
            fz, dp = z, nu
        eta = bp0 * ffp[q] + (F["x"][q] - _w(F["x"][q]) + F["y"][q] - _s(F["y"][q]) + (fz - fm) / dz[q]
                              + f["src"][q] * g.hr * f["swbal"] * f["src_factor"] * dxy)
        up, lo = dm / dz[q], dp / dz[q]
        if q == 0:
            one = f["ig_top"] == 1
            eta = eta + torch.where(one, dm * f["ff_top"] / dz[q], f["ff_top"] / dz[q] * dxy)
            D.append(bp + lo + torch.where(one, up, z))
        elif q == nz - 1:
            one = f["ig_bot"] == 1
            eta = eta + torch.where(one, dp * f["ff_bot"] / dz[q], f["ff_bot"] / dz[q] * dxy)
            D.append(bp + up + torch.where(one, lo, z))
        else:
            D.append(bp + lo + up)
        A.append(-up)
        C.append(-lo if q < nz - 1 else z)
        E.append(eta)
    return [*_filtered(g, "lu", ff, ffp, _thomas(A, D, C, E)), FO["x"], FO["y"]]
