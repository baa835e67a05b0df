"""The workloads this framework is timed on: discs advanced through the public
Python entry points (Disc, Batch), the allocation-free transport of the C ABI
and the learned closure's two directions.

A gas pass is what a run does between two outputs: the state is taken from the
host (a restart, or the next member of a parameter study in the same context),
a few DTs are advanced and the fields come back.  Particle and batch passes go
on from where the last one ended, as a run does.  Sizes come from the
repository's configurations (configs/*.par), its sweep (sweep.py) and its
tests, and odd ones between them; both builds of the library are used (the
parity build is Disc's default, the fast build is what bench.py times), with
the shipped table of launch shapes, which knows only the sweep's grids.
"""
import ctypes as C
import math
import os
import tempfile

import numpy as np
import torch

import dustyfargoadsg_b200 as fb
from dustyfargoadsg_b200 import _ffi, closure, sweep, tune

ISO, ADIABATIC, DUST = "iso_128x384.par", "adiabatic_sg_512x1536.par", "dust_256x768.par"
FIELDS = ("dens", "vrad", "vtheta", "energy")
# case keys that go into the parameters (fields of FbParams) as they are
OPTIONS = ("nrad", "nsec", "rmin", "rmax", "wkzrmin", "wkzrmax", "energy_equation", "self_gravity", "beta_cooling",
           "viscous_heating", "thermal_cooling", "radiative_diffusion", "corotating", "forced_circular",
           "wall_boundary", "non_reflecting", "nbpart")


def listed():
    return [
        # the smallest discs of the tests, one DT per restart: every call's
        # fixed costs and the latency of the substep's launches decide
        dict(name="iso_48x144", kind="gas", par=ISO, mode="parity", nrad=48, nsec=144, dts=1),
        # the plain isothermal disc that the reference can run on a CPU, with
        # the library build a user gets without asking
        dict(name="iso_128x384", kind="gas", par=ISO, mode="parity", nrad=128, nsec=384, dts=4),
        # the size and physics of the reference's own example files: energy
        # equation with radiative cooling, corotating frame, a free planet,
        # non-reflecting edges; a grid the tuning table does not know
        dict(name="cooling_200x400", kind="gas", par=ADIABATIC, mode="parity", nrad=200, nsec=400, dts=4,
             rmin=0.4, rmax=2.5, wkzrmin=0.5, wkzrmax=2.1, self_gravity=0, beta_cooling=0, thermal_cooling=1,
             corotating=1, forced_circular=0, wall_boundary=0, non_reflecting=1),
        # an odd grid, as a user picks one, adiabatic with beta cooling and
        # viscous heating
        dict(name="adiabatic_333x1001", kind="gas", par=ADIABATIC, mode="fast", nrad=333, nsec=1001, dts=4,
             self_gravity=0),
        # radiative diffusion by the implicit solver
        dict(name="diffusion_128x384", kind="gas", par=ADIABATIC, mode="parity", nrad=128, nsec=384, dts=1,
             self_gravity=0, radiative_diffusion=2),
        # the flagship: adiabatic, beta cooling and self-gravity
        dict(name="adiabatic_sg_512x1536", kind="gas", par=ADIABATIC, mode="fast", nrad=512, nsec=1536, dts=8),
        # the same physics with the default build on a smaller disc whose
        # radial transform is not a power of two
        dict(name="adiabatic_sg_192x576", kind="gas", par=ADIABATIC, mode="parity", nrad=192, nsec=576, dts=4),
        # the largest grid, beyond the L2 cache
        dict(name="iso_768x2304", kind="gas", par=ISO, mode="fast", nrad=768, nsec=2304, dts=8),
        # gas and 200,000 Lagrangian particles with turbulent kicks
        dict(name="dust_256x768", kind="dust", par=DUST, mode="fast", nrad=256, nsec=768, nbpart=200000, dts=2),
        # a parameter study: discs of five grid sizes in one graph launch
        dict(name="sweep_16", kind="batch", mode="fast", discs=16, sweep_seed=2, dts=1),
        # the transport alone on a caller's device arrays
        dict(name="transport_128x384", kind="transport", par=ISO, mode="parity", nrad=128, nsec=384),
        # training direction of the learned closure: loss and gradients of a
        # minibatch
        dict(name="closure_grad_128x384", kind="closure", mode="parity", nrad=128, nsec=384, batch=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gas"] * 6 + ["dust", "transport", "closure"])
    mode = rng.choice(["parity", "fast"])
    if kind == "transport":
        nrad = _log_int(rng, 24, 256)
        c = dict(kind=kind, par=rng.choice([ISO, ADIABATIC]), mode=mode, nrad=nrad,
                 nsec=min(rng.randint(2 * nrad, 4 * nrad), 131072 // (nrad + 1)))
        if c["par"] == ADIABATIC:
            c["self_gravity"] = 0
        return c
    if kind == "closure":
        return dict(kind=kind, mode=mode, nrad=_log_int(rng, 16, 128), nsec=64 * rng.randint(1, 6),
                    batch=rng.randint(1, 8))
    if kind == "dust":
        nrad = _log_int(rng, 32, 256)
        return dict(kind=kind, par=DUST, mode=mode, nrad=nrad, nsec=rng.randint(2 * nrad, 3 * nrad),
                    nbpart=_log_int(rng, 500, 200000), dts=1)
    nrad = _log_int(rng, 32, 700)
    c = dict(kind=kind, par=rng.choice([ISO, ADIABATIC]), mode=mode, nrad=nrad,
             nsec=min(2300, rng.randint(2 * nrad, int(3.3 * nrad))), dts=rng.choice([1, 1, 2]))
    if c["par"] == ADIABATIC:
        c["self_gravity"] = rng.choice([0, 1])
        if c["self_gravity"]:  # the log-polar transforms take lengths of small factors
            c["nrad"] = rng.choice([32, 48, 64, 96, 128, 160, 200, 256, 320, 384, 400, 512])
            c["nsec"] = c["nrad"] * rng.choice([2, 3])
        else:
            c["viscous_heating"] = rng.choice([1, 1, 0])
    return c


# ------------------------------------------------------------------ inputs
def _params(case):
    over = {k: case[k] for k in OPTIONS if k in case}
    return fb.read_par(os.path.join(fb.CONFIG_DIR, case["par"]), **over)


def _disc(case, seed):
    return fb.Disc(_params(case), noise=1e-4, seed=seed % 100003, dust_seed=seed % 100003 if "nbpart" in case else None,
                   tuning=tune.load_table(), mode=case["mode"])


def _saved(disc):
    """A disc's state as a host program keeps it for a restart."""
    s = disc.download()
    for name, key in (("SigmaMed", "sigma_med"), ("SigmaInf", "sigma_inf"), ("EnergyMed", "energy_med"),
                      ("VthetaMed", "vtheta_med"), ("VradMed", "vrad_med"), ("GLOBAL_SoundSpeed", "global_soundspeed")):
        s[name] = disc.prof[key].copy()
    return s


CHANNELS = [16, 32, 32, 32, 16]  # the closure network's layers


def _closure_inputs(case, seed):
    """Weights, biases, features, targets and initial density profiles."""
    g = np.random.default_rng(seed)
    nr, ns, nb = case["nrad"], case["nsec"], case["batch"]
    w = np.concatenate([(g.standard_normal(o * 9 * i) * math.sqrt(2.0 / (9 * i))) for i, o in
                        zip(CHANNELS, CHANNELS[1:])]).astype(np.float32)
    b = (0.05 * g.standard_normal(sum(CHANNELS[1:]))).astype(np.float32)
    x = np.zeros((nb, nr, ns, 16), dtype=np.float32)
    x[..., :7] = torch.from_numpy(0.5 * g.standard_normal((nb, nr, ns, 7), dtype=np.float32)).bfloat16().float().numpy()
    sig = np.tile((6.3e-4 * np.linspace(1.5, 0.6, nr)).astype(np.float32), (nb, 1))
    y = np.zeros((nb, 3, nr, ns), dtype=np.float32)
    y[:, 0] = 1e-2 * sig[:, :, None] * g.standard_normal((nb, nr, ns), dtype=np.float32)
    scale, wq = np.array([1e-6, 1.0, 1.0]), np.array([1.0 / float(np.mean(y[:, 0].astype(np.float64) ** 2)), 1.0, 1.0])
    return dict(w=w, b=b, x=x, y=y, sig=sig, scale=scale, wq=wq)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gas":
        disc = _disc(case, seed)
        return dict(case=case, disc=disc, start=_saved(disc))
    if kind == "dust":
        return dict(case=case, disc=_disc(case, seed))
    if kind == "batch":
        discs = []
        with tempfile.TemporaryDirectory() as wd:
            for n, d in enumerate(sweep.draw_discs(case["discs"], case["sweep_seed"])):
                par = sweep.write_disc_files(d, wd, "disc%03d" % n)
                discs.append(fb.Disc(fb.read_par(par), noise=1e-4, seed=(seed + n) % 100003,
                                     tuning=tune.load_table(), mode=case["mode"]))
        return dict(case=case, discs=discs, batch=fb.Batch(discs))
    if kind == "transport":
        p = _params(case)
        with fb.Disc(p, noise=1e-2, seed=seed % 100003, mode=case["mode"]) as disc:
            s = disc.download()
        g = np.random.default_rng(seed)
        s["vrad"] = s["vrad"] + 1e-3 * g.standard_normal(s["vrad"].shape)
        s["vrad"][:case["nsec"]] = 0.0
        t0 = torch.tensor(np.stack([s[k] for k in FIELDS]), device="cuda")
        return dict(case=case, p=p, lib=fb.load(case["mode"]), t0=t0, t=torch.empty_like(t0), lost=C.c_double(),
                    dt=_transport_dt(p))
    d = _closure_inputs(case, seed)
    disc = fb.Disc(fb.read_par(os.path.join(fb.CONFIG_DIR, ISO), nrad=case["nrad"], nsec=case["nsec"]),
                   mode=case["mode"])
    net = closure.Closure(disc, capacity=case["batch"], batch=case["batch"], seed=1)
    net.set_params({"w": d["w"], "b": d["b"], "scale": d["scale"], "wq": d["wq"]})
    fp = C.POINTER(C.c_float)
    for n in range(case["batch"]):
        x, y, sig = (np.ascontiguousarray(d[k][n]) for k in ("x", "y", "sig"))
        _ffi.check(net.lib.fb_closure_set_sample(net.c, n, x.ctypes.data_as(fp), y.ctypes.data_as(fp),
                                                 sig.ctypes.data_as(fp)), "fb_closure_set_sample")
    return dict(case=case, disc=disc, net=net, gw=np.zeros(net.nw, np.float32), gb=np.zeros(net.nb, np.float32),
                out=np.zeros((case["nrad"], case["nsec"], 16), np.float32))


def _transport_dt(p):
    """A time step the CFL condition of this grid would give."""
    return 0.25 * math.log(p.rmax / p.rmin) / p.nrad / p.aspectratio * p.rmin ** 1.5


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "gas":
        disc = state["disc"]
        disc.set_state(state["start"])
        sub = [disc.step().substeps for _ in range(case["dts"])]
        out = disc.download()
        return [sum(sub)] + [out[k] for k in FIELDS] + [out["LostMass"], out["pl_x"], out["pl_y"]]
    if kind == "dust":
        disc = state["disc"]
        sub = [disc.step().substeps for _ in range(case["dts"])]
        out, parts = disc.download(), disc.dust()
        return [sum(sub)] + [out[k] for k in FIELDS[:3]] + [parts["pc_" + k] for k in disc.DUST_ARRAYS] + [parts["pc_kicks"]]
    if kind == "batch":
        sub = [r.substeps for _ in range(case["dts"]) for r in state["batch"].step()]
        outs = [d.download() for d in state["discs"]]
        return [sum(sub)] + [o[k] for o in outs for k in FIELDS[:3]]
    if kind == "transport":
        t, lib = state["t"], state["lib"]
        t.copy_(state["t0"])
        ptr = [C.c_void_p(t[q].data_ptr()) for q in range(4)]
        _ffi.check(lib.fb_transport_noalloc(C.byref(state["p"]), *ptr, state["dt"], None, C.byref(state["lost"])),
                   "fb_transport_noalloc")
        return [t[0], t[1], t[2], t[3], state["lost"].value]
    net, fp = state["net"], C.POINTER(C.c_float)
    loss = C.c_double()
    _ffi.check(net.lib.fb_closure_loss_grad(net.c, 0, case["batch"], C.byref(loss), state["gw"].ctypes.data_as(fp),
                                            state["gb"].ctypes.data_as(fp)), "fb_closure_loss_grad")
    # the forward direction: the network's face fluxes of one sample
    _ffi.check(net.lib.fb_closure_infer(net.c, None, 0, state["out"].ctypes.data_as(fp)), "fb_closure_infer")
    return [loss.value, state["gw"], state["gb"], state["out"]]


# -------------------------------------------------------------------- work
def _substeps(p):
    """Substeps of one DT from the sound and viscous limits at the inner edge
    alone (the flow's own velocities add to them)."""
    dx = min(math.log(p.rmax / p.rmin) / p.nrad, 2.0 * math.pi / p.nsec)
    cs = p.aspectratio * p.rmin ** -1.5
    return max(1.0, p.dt * 2.0 * math.hypot(cs / dx, 4.0 * p.alphaviscosity * p.aspectratio * cs / dx ** 2))


def _gas_work(p, dts):
    # state in and out once; about 450 (600) FP64 operations per cell and
    # substep isothermal (with the energy equation), counting a quotient or a
    # root as one: sources 90 (150), two van Leer passes in azimuth and one in
    # radius of 5 (6) quantities, the time step's limits; the transforms of
    # self-gravity 5 N log2 N each
    cells, e = p.nrad * p.nsec, p.energy_equation
    flops = (600.0 if e else 450.0) * cells
    if p.self_gravity:
        flops += 2 * 5.0 * cells * math.log2(p.nsec) + 2 * 2 * 5.0 * cells * math.log2(2 * p.nrad)
    return dict(bytes=2.0 * 8 * (4 if e else 3) * cells, flops=flops * _substeps(p) * dts)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = []
        for d in sweep.draw_discs(case["discs"], case["sweep_seed"]):
            p = fb.read_par(os.path.join(fb.CONFIG_DIR, ISO), nrad=d["Nrad"], nsec=d["Nsec"],
                            aspectratio=d["AspectRatio"], alphaviscosity=d["AlphaViscosity"])
            parts.append(_gas_work(p, case["dts"]))
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    cells = case["nrad"] * case["nsec"]
    if kind == "transport":
        nf = 4 if case["par"] == ADIABATIC else 3
        return dict(bytes=2.0 * 8 * nf * cells, flops=320.0 * cells)
    if kind == "closure":
        macs = sum(9 * i * o for i, o in zip(CHANNELS, CHANNELS[1:]))
        nb = case["batch"]
        # forward, gradients of the weights and (but for the first layer) of
        # the layer inputs, and one sample's forward pass
        flops = 2.0 * cells * (nb * (3 * macs - 9 * 16 * 32) + macs)
        return dict(bytes=cells * (nb * (2.0 * 16 + 4 * 3) + 2 * 16 + 4 * 16), flops=flops)
    w = _gas_work(_params(case), case["dts"])
    if kind == "dust":
        w["bytes"] += 2.0 * 8 * 7 * case["nbpart"]
        w["flops"] += 300.0 * case["nbpart"] * _substeps(_params(case)) * case["dts"]
    return w


# ------------------------------------------------------------------- exact
# The same step in plain numpy, for the discs it covers: log grid, fixed
# frame, one planet on a circular orbit, walls and Stockholm damping,
# isothermal or adiabatic with beta cooling.
class _Grid:
    def __init__(self, p):
        nr, ns = p.nrad, p.nsec
        radii = p.rmin * np.exp(np.arange(nr + 1) / nr * math.log(p.rmax / p.rmin))
        self.nr, self.ns, self.rinf, self.rsup = nr, ns, radii[:-1], radii[1:]
        self.rmed = 2.0 / 3.0 * (self.rsup ** 3 - self.rinf ** 3) / (self.rsup ** 2 - self.rinf ** 2)
        self.surf = 0.5 * (p.pmax - p.pmin) * (self.rsup ** 2 - self.rinf ** 2) / ns
        self.dphi = (p.pmax - p.pmin) / ns
        az = p.pmin + self.dphi * np.arange(ns)
        self.x, self.y = self.rmed[:, None] * np.cos(az), self.rmed[:, None] * np.sin(az)
        self.dxt = self.dphi * self.rmed
        self.idrm = np.concatenate([[0.0], 1.0 / np.diff(self.rmed)])


def _c(a):
    return np.asarray(a)[:, None]


def _van_leer(dm, dp):
    prod, tot = dm * dp, dm + dp
    with np.errstate(divide="ignore", invalid="ignore"):
        return np.where(prod > 0.0, prod / np.where(prod > 0.0, tot, 1.0), 0.0)


def _theta_pass(q, v, dt, g):
    """One azimuthal van Leer pass of all quantities (the density last) at the
    face velocities v."""
    dxt, invdx = _c(g.dxt), 1.0 / _c(g.dxt)

    def star(a):
        d = _van_leer(a - np.roll(a, 1, 1), np.roll(a, -1, 1) - a) * invdx
        return np.where(v * dt > 0.0, np.roll(a, 1, 1) + (dxt - v * dt) * np.roll(d, 1, 1), a - (dxt + v * dt) * d)

    rho = q[-1]
    rs = star(rho)
    out = []
    for a in q:
        f = _c(g.rsup - g.rinf) * dt * star(a / (rho + 1e-20)) * rs * v
        out.append(a + (f - np.roll(f, -1, 1)) / _c(g.surf))
    return out


def _transport(f, dt, g, energy):
    """Radial and azimuthal transport of the fields (nr + 1 rings); returns
    the new ones before floors and boundaries, and the ring-0 outflow."""
    nr, ns = g.nr, g.ns
    rho, vr, vt = f["dens"][:nr], f["vrad"], f["vtheta"][:nr]
    rm = _c(g.rmed)
    q = [rho * vr[1:], rho * vr[:nr], rho * np.roll(vt, -1, 1) * rm, rho * vt * rm]
    q += ([f["energy"][:nr]] if energy else []) + [rho]
    v = vr[1:nr]  # faces 1 .. nr-1

    def star(a):
        dq = np.zeros_like(a)
        d = np.diff(a, axis=0) * _c(g.idrm[1:])
        dq[1:-1] = 2.0 * _van_leer(d[:-1], d[1:])
        lo = _c(np.diff(g.rmed))  # the reference takes the gap above the face's upper ring when the flow goes inwards
        hi = np.concatenate([lo[1:], lo[:1]])  # no slope on the last ring
        return np.where(v > 0.0, a[:-1] + (lo - v * dt) * 0.5 * dq[:-1], a[1:] - (hi + v * dt) * 0.5 * dq[1:])

    rs = star(rho)
    new = []
    for a in q:
        flux = np.zeros((nr + 1, ns))
        flux[1:nr] = dt * g.dphi * _c(g.rinf[1:]) * star(a / (rho + 1e-20)) * rs * v
        new.append(a + (flux[:-1] - flux[1:]) / _c(g.surf))
        lost = float(np.sum(flux[0] - flux[1]))
    vmed = _c(vt.mean(axis=1))
    nt = vmed / rm * dt / g.dphi
    nround = np.floor(nt + 0.5)
    q = _theta_pass(new, vt - vmed, dt, g)
    q = _theta_pass(q, np.broadcast_to((nt - nround) * rm / dt * g.dphi, vt.shape), dt, g)
    cols = (np.arange(ns)[None, :] - nround.astype(np.int64)) % ns
    q = [np.take_along_axis(a, cols, axis=1) for a in q]
    out = {k: a.copy() for k, a in f.items()}
    r = q[-1]
    out["dens"][:nr] = r
    out["vtheta"][:nr] = (np.roll(q[2], 1, 1) + q[3]) / (r + np.roll(r, 1, 1) + 1e-20) / rm
    out["vrad"][0] = 0.0
    out["vrad"][1:nr] = (q[0][:-1] + q[1][1:]) / (r[1:] + r[:-1] + 1e-20)
    if energy:
        out["energy"][:nr] = q[4]
    return out, lost


def _stress(vr, vt, rho, nu, g):
    """Divergence and stress tensor of rings 0 .. nr-1 (the shear on ring 0 is
    zero); vr has nr + 1 rings."""
    nr = g.nr
    v, vtp = vr[:nr], np.roll(vt, -1, 1)
    irm, isup = 1.0 / _c(g.rmed), 1.0 / _c(g.rsup - g.rinf)
    div = (vr[1:] * _c(g.rsup) - v * _c(g.rinf)) * isup * irm + (vtp - vt) / g.dphi * irm
    drr = (vr[1:] - v) * isup
    dpp = (vtp - vt) / g.dphi * irm + 0.5 * (vr[1:] + v) * irm
    trr, tpp = 2.0 * rho * nu * (drr - div / 3.0), 2.0 * rho * nu * (dpp - div / 3.0)
    trp = np.zeros_like(rho)
    om = vt * irm
    drp = 0.5 * (_c(g.rinf[1:]) * (om[1:] - om[:-1]) * _c(g.idrm[1:]) +
                 (v - np.roll(v, 1, 1))[1:] / g.dphi / _c(g.rinf[1:]))
    mean = 0.25 * (rho[1:] + rho[:-1] + np.roll(rho, 1, 1)[1:] + np.roll(rho, 1, 1)[:-1])
    trp[1:] = 2.0 * mean * nu[1:] * drp
    return div, trr, tpp, trp


def _gas_dt(p, g, prof, st, cs):
    """One DT of the state dict st in place; returns the substeps."""
    nr, ns, energy = g.nr, g.ns, bool(p.energy_equation)
    gam, cvnr2 = p.adiabaticindex, 1.41 ** 2
    rm, isup = _c(g.rmed), 1.0 / _c(g.rsup - g.rinf)
    dxr, dxt = _c(g.rsup - g.rinf), _c(g.dxt)
    dxm, idrm1 = np.minimum(dxr, dxt), _c(g.idrm[1:])
    f = {k: st[k].reshape(nr + 1, ns).copy() for k in FIELDS}
    if energy:
        cs[:] = np.sqrt(gam * (gam - 1.0) * f["energy"][:nr] / f["dens"][:nr])
    done, count = 0.0, 0
    while count == 0 or done < 0.999999999 * p.dt:
        rho, vr, vt = f["dens"][:nr], f["vrad"], f["vtheta"][:nr]
        gcs = st["gcs"]
        nu = p.alphaviscosity * gcs ** 2 * g.rmed ** 1.5
        # time step
        vmoy = vt.mean(axis=1)
        dvr, dvt = vr[1:] - vr[:nr], np.roll(vt, -1, 1) - vt
        dvr, dvt = np.where(dvr >= 0.0, 1e-10, -dvr), np.where(dvt >= 0.0, 1e-10, -dvt)
        s = (cs / dxm) ** 2 + (vr[:nr] / dxr) ** 2 + ((vt - _c(vmoy)) / dxt) ** 2
        s = s + (4.0 * cvnr2 * np.maximum(dvr / dxr, dvt / dxt)) ** 2 + _c((4.0 * nu / dxm[:, 0] ** 2) ** 2) + 1e-20
        new = min(float((0.5 / np.sqrt(s[1:])).min()),
                  float((2.0 * math.pi * 0.5 / ns / np.abs(np.diff(vmoy / g.rmed))).min()), p.dt - done)
        dt = (p.dt - done) / math.ceil((p.dt - done) / new)
        done += dt
        count += 1
        # potential: star, planet, indirect terms
        mass = _c(g.surf) * rho
        ax, ay = float((mass * g.x / rm ** 3).sum()), float((mass * g.y / rm ** 3).sum())
        m, px, py = st["pl_mass"], st["pl_x"], st["pl_y"]
        d = math.hypot(px, py)
        eps = p.thicknesssmoothing * p.aspectratio * d ** (1.0 + p.flaringindex)
        pot = (-m / np.sqrt((g.x - px) ** 2 + (g.y - py) ** 2 + eps * eps) + m / d ** 3 * (g.x * px + g.y * py)
               - 1.0 / rm + ax * g.x + ay * g.y)
        th, om = math.atan2(py, px), (px * st["pl_vy"] - py * st["pl_vx"]) / d / d
        sp = math.hypot(st["pl_vx"], st["pl_vy"])
        th += om * dt
        st["pl_x"], st["pl_y"], st["pl_vx"], st["pl_vy"] = (d * math.cos(th), d * math.sin(th), -sp * math.sin(th),
                                                            sp * math.cos(th))
        if energy:
            cs[:] = np.sqrt(gam * (gam - 1.0) * f["energy"][:nr] / rho)
            st["gcs"] = gcs = cs.mean(axis=1)
            pres = (gam - 1.0) * f["energy"][:nr]
        else:
            pres = rho * cs * cs
        nu = _c(p.alphaviscosity * gcs ** 2 * g.rmed ** 1.5)
        # pressure, potential and curvature
        rhom, rr = np.roll(rho, 1, 1), rho[1:] + rho[:-1]
        vri = np.zeros((nr + 1, ns))
        vt4 = (vt + np.roll(vt, -1, 1))
        vt4 = 0.25 * (vt4[1:] + vt4[:-1])
        vri[1:nr] = vr[1:nr] + dt * (-(np.diff(pres, axis=0) * 2.0 / rr + np.diff(pot, axis=0)) * idrm1 +
                                     vt4 ** 2 / _c(g.rinf[1:]))
        vti = vt - dt * ((pres - np.roll(pres, 1, 1)) * 2.0 / (rho + rhom) + pot - np.roll(pot, 1, 1)) / dxt
        # viscosity
        div, trr, tpp, trp = _stress(vri, vti, rho, nu, g)
        trp1 = np.concatenate([trp[1:], np.zeros((1, ns))])
        dvt_ = dt / rm * ((_c(g.rsup) * trp1 - _c(g.rinf) * trp) * isup + (tpp - np.roll(tpp, 1, 1)) / g.dphi +
                          0.5 * (trp + trp1)) / (0.5 * (rho + rhom))
        dvr_ = dt / _c(g.rinf[1:]) * (np.diff(rm * trr, axis=0) * idrm1 + (np.roll(trp, -1, 1) - trp)[1:] / g.dphi -
                                      0.5 * (tpp[1:] + tpp[:-1])) / (0.5 * rr)
        vti[1:nr - 1] += dvt_[1:nr - 1]
        vri[1:nr] += dvr_
        # artificial viscosity
        dv, dw = np.diff(vri, axis=0), np.roll(vti, -1, 1) - vti
        qr, qt = np.where(dv < 0.0, cvnr2 * rho * dv * dv, 0.0), np.where(dw < 0.0, cvnr2 * rho * dw * dw, 0.0)
        f["vrad"][:] = 0.0
        f["vrad"][1:nr] = vri[1:nr] - dt * 2.0 / rr * np.diff(qr, axis=0) * idrm1
        f["vtheta"][:nr] = vti - dt * 2.0 / (rho + rhom) * (qt - np.roll(qt, 1, 1)) / dxt
        f["vtheta"][nr] = 0.0
        if energy:
            en = f["energy"][:nr] - dt * qr * dv * isup - dt * qt * dw / dxt
            div, trr, tpp, trp = _stress(f["vrad"], f["vtheta"][:nr], rho, nu, g)
            heat = 0.0
            if p.viscous_heating:
                heat = 0.5 / nu / rho * (trr ** 2 + 2.0 * trp ** 2 + tpp ** 2) + 2.0 / 9.0 * nu * rho * div ** 2
                heat[0] = heat[1] * np.exp(np.log(heat[1] / heat[2]) * math.log(g.rmed[0] / g.rmed[1]) /
                                           math.log(g.rmed[1] / g.rmed[2]))
            en = (en + heat * dt) / (1.0 + (gam - 1.0) * dt * div)
            if p.beta_cooling:
                omega = f["vtheta"][:nr].mean(axis=1) / g.rmed
                en = en / (1.0 + dt * _c(omega) / p.betacoolingtime * _c(g.rmed ** p.betacoolingslope))
            f["energy"][:nr] = en
            f["energy"][nr] = 0.0
        # transport, floors, walls, damping zones
        f, lost = _transport(f, dt, g, energy)
        st["LostMass"] += lost
        f["vtheta"][[0, nr - 1]] = prof["VthetaMed"][[0, nr - 1], None]
        if energy:
            f["energy"][:nr] = np.maximum(f["energy"][:nr], 1e-3 * _c(prof["EnergyMed"]))
        v, r = f["vrad"], f["dens"]
        r[:nr] = np.maximum(r[:nr], p.densityfloor)
        v[0], v[nr], v[1], v[nr - 1] = -v[2], -v[nr - 2], 0.0, 0.0
        edge = [0, 1, nr - 2, nr - 1]
        r[edge] = prof["SigmaMed"][edge, None]
        for i in range(nr):
            lo, hi = g.rmed[i] < p.wkzrmin, g.rmed[i] > p.wkzrmax
            if lo or hi:
                ref, end = (p.wkzrmin, g.rmed[0]) if lo else (p.wkzrmax, g.rmed[nr - 1])
                lam = ((g.rmed[i] - ref) / (end - ref)) ** 2 * dt / (p.dampingtodynamicaltimeratio * g.rmed[i] ** 1.5)
                for k in FIELDS[:4 if energy else 3]:
                    f[k][i] = (f[k][i] + lam * f[k][i].mean()) / (1.0 + lam)
    for k in FIELDS:
        st[k] = f[k].ravel()
    return count


def _exact_gas(case, seed):
    p = _params(case)
    if (p.self_gravity or p.thermal_cooling or p.radiative_diffusion or p.corotating or not p.forced_circular or
            not p.wall_boundary):
        return None
    if p.nrad * p.nsec * _substeps(p) * case["dts"] > 3e6:  # over 20 s in numpy
        return None
    with _disc(case, seed) as disc:
        st = _saved(disc)
    prof = {k: st[k] for k in ("VthetaMed", "EnergyMed", "SigmaMed")}
    st.update({k: float(st[k][0]) for k in ("pl_mass", "pl_x", "pl_y", "pl_vx", "pl_vy")}, gcs=st["GLOBAL_SoundSpeed"])
    g = _Grid(p)
    cs = np.repeat(_c(p.aspectratio * g.rmed ** (p.flaringindex - 0.5)), p.nsec, axis=1)
    for _ in range(case["dts"]):
        _gas_dt(p, g, prof, st, cs)
    return [None] + [st[k] for k in FIELDS] + [st["LostMass"], np.array([st["pl_x"]]), np.array([st["pl_y"]])]


def _exact_transport(case, seed):
    s = prepare(case, seed)
    p, nr = s["p"], case["nrad"]
    f = {k: s["t0"][q].cpu().numpy().reshape(nr + 1, -1) for q, k in enumerate(FIELDS)}
    out, lost = _transport(f, s["dt"], _Grid(p), bool(p.energy_equation))
    return [out[k].ravel() for k in FIELDS] + [lost]


def _exact_closure(case, seed):
    d = _closure_inputs(case, seed)
    nr, nb = case["nrad"], case["batch"]
    ws, bs, ow, ob = [], [], 0, 0
    for i, o in zip(CHANNELS, CHANNELS[1:]):
        w = torch.from_numpy(d["w"][ow:ow + o * 9 * i]).double().reshape(o, 3, 3, i)
        ws.append(w.requires_grad_())
        bs.append(torch.from_numpy(d["b"][ob:ob + o]).double().requires_grad_())
        ow, ob = ow + o * 9 * i, ob + o
    pad, conv, gelu = torch.nn.functional.pad, torch.nn.functional.conv2d, torch.nn.functional.gelu
    h = torch.from_numpy(d["x"]).double().permute(0, 3, 1, 2)
    for n, (w, b) in enumerate(zip(ws, bs)):
        h = conv(pad(pad(h, (1, 1, 0, 0), mode="circular"), (0, 0, 1, 1)), w.permute(0, 3, 1, 2), b)
        h = gelu(h) if n < 3 else h
    p = fb.read_par(os.path.join(fb.CONFIG_DIR, ISO), nrad=nr, nsec=case["nsec"])
    sig = torch.from_numpy(d["sig"]).double()
    face = torch.zeros(nb, nr + 1, dtype=torch.float64)
    face[:, 1:nr] = torch.sqrt(sig[:, :-1] * sig[:, 1:])
    fr = torch.cat([h[:, 0], torch.zeros_like(h[:, 0, :1])], dim=1) * face[:, :, None]
    ft = h[:, 1] * sig[:, :, None]
    ds = d["scale"][0] * (fr[:, :-1] - fr[:, 1:] + ft - torch.roll(ft, -1, 2))
    ds = ds / torch.from_numpy(_Grid(p).surf)[None, :, None]
    loss = d["wq"][0] * ((ds - torch.from_numpy(d["y"][:, 0]).double()) ** 2).mean()
    loss.backward()
    grads = [torch.cat([t.grad.reshape(-1) for t in ts]).numpy() for ts in (ws, bs)]
    return [float(loss.detach())] + grads + [h[0].detach().permute(1, 2, 0).contiguous().numpy()]


def exact(case, seed):
    """What run returns, in 64 bits; None for what numpy does not reach in
    time (large grids, batches, the implicit solver) or at all (particles,
    whose kicks follow the library's random stream)."""
    if case["kind"] == "gas":
        return _exact_gas(case, seed)
    if case["kind"] == "transport":
        return _exact_transport(case, seed)
    if case["kind"] == "closure":
        return _exact_closure(case, seed)
    return None
