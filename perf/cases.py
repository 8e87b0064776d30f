"""The framework's work as its users have it done, for measuring speed and accuracy.

A case is one stretch of a disk's run between two outputs, driven the way a run loop
drives it: per step the CFL time step is read back, the bodies are moved and handed in,
the gas step runs and the disk's force on every body is read back; at the end the evolved
fields are snapshotted into page-locked buffers.  The batch cases advance a parameter
study of independent disks.

* ``listed()``   the cases; ``draw(rng)`` one more of the same ranges;
* ``prepare``    a disk (or batch) in mid-run: seeded fields with a spiral, noise and
  subsonic motions, uploaded to an engine, with its CFL step, bodies and snapshot buffers;
* ``run``        one such stretch; it returns the snapshotted fields, the forces of the
  last step and the time reached.  Calling it again goes on from there;
* ``work``       the bytes and operations one stretch cannot do without;
* ``exact``      the same stretch in 64-bit torch, from the scheme's formulas.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fargocpt_gb300 import setups
from fargocpt_gb300.abi import params_from_dict
from fargocpt_gb300.batch import Batch
from fargocpt_gb300.engine import Engine
from fargocpt_gb300.output import Snapshotter
from fargocpt_gb300.simulation import step_leapfrog

PLANETS = [(1e-3, 1.0, 0.0), (3e-4, 1.6, 2.1), (1e-4, 2.5, 4.2)]
FP64, FP32 = "fp64", "fp32"


def _case(name, nr, nz, *, form=FP64, adiabatic=True, planets=1, steps=8, integrator="euler",
          art_visc="sn", limiter="vanleer", fargo=True):
    return dict(name=name, kind="disk", nr=nr, nz=nz, form=form, adiabatic=adiabatic,
                planets=planets, steps=steps, integrator=integrator, art_visc=art_visc,
                limiter=limiter, fargo=fargo)


def _batch(name, disks, seed, *, steps, clock):
    return dict(name=name, kind="batch", disks=disks, sweep=seed, steps=steps, clock=clock)


def listed():
    return [
        # the drop-in FP64 form.  The smallest disk in use: a quick look or a test run,
        # where launches and read-backs count
        _case("fp64_iso_128x384", 128, 384, adiabatic=False, steps=24),
        # the usual production disk with an energy equation
        _case("fp64_adi_512x1536", 512, 1536, steps=12),
        # a high-resolution locally isothermal disk
        _case("fp64_iso_1024x3072", 1024, 3072, adiabatic=False, steps=8),
        # the largest single-GPU disk: three planets, energy equation
        _case("fp64_adi_2048x6144", 2048, 6144, planets=3, steps=8),
        # a grid chosen for its cell aspect, no round numbers, LeapFrog
        _case("fp64_leapfrog_395x1187", 395, 1187, planets=2, steps=8, integrator="leapfrog"),
        # other options of the scheme on an odd ring: TW viscosity, MC limiter
        _case("fp64_tw_mc_301x1001", 301, 1001, art_visc="tw", limiter="mc", steps=12),
        # the FP32-mixed form: small, ragged and large
        _case("fp32_iso_192x576", 192, 576, form=FP32, adiabatic=False, steps=24),
        _case("fp32_adi_777x2345", 777, 2345, form=FP32, planets=2, steps=8),
        _case("fp32_adi_2048x6144", 2048, 6144, form=FP32, planets=3, steps=8),
        # a parameter study: disks of several sizes stepped together, by the device's
        # clock and by the host's
        _batch("batch_device_clock_16", 16, 4, steps=16, clock="device"),
        _batch("batch_host_clock_12", 12, 9, steps=12, clock="host"),
    ]


def draw(rng):
    if rng.random() < 0.2:
        return dict(kind="batch", disks=rng.randint(3, 16), sweep=rng.randint(0, 10 ** 6),
                    steps=rng.randint(4, 16), clock=rng.choice(["device", "host"]))
    nr = int(round(math.exp(rng.uniform(math.log(96), math.log(1800)))))
    nz = max(64, min(6144, int(round(nr * rng.uniform(2.0, 4.0)))))
    steps = max(4, min(24, int(2048 * 6144 * 4 / (nr * nz))))
    c = _case(None, nr, nz, form=rng.choice([FP64, FP64, FP32]), adiabatic=rng.random() < 0.6,
              planets=rng.randint(1, 3), steps=steps,
              integrator=rng.choice(["euler", "euler", "euler", "leapfrog"]),
              art_visc=rng.choice(["sn", "sn", "sn", "tw"]),
              limiter=rng.choice(["vanleer", "vanleer", "vanleer", "mc"]),
              fargo=rng.random() < 0.9)
    del c["name"]
    return c


# -- inputs ---------------------------------------------------------------------------
def _params(case):
    d = setups.base_params(case["nr"], case["nz"], 0.3, 5.0 if case["planets"] > 1 else 3.0,
                           adiabatic=case["adiabatic"],
                           flaring=0.25 if case["adiabatic"] else 0.0)
    d.update(precision=1 if case["form"] == FP32 else 0,
             integrator=1 if case["integrator"] == "leapfrog" else 0,
             art_visc={"sn": 1, "tw": 2}[case["art_visc"]],
             flux_limiter=1 if case["limiter"] == "mc" else 0,
             fast_transport=1 if case["fargo"] else 0)
    return d


def _radii(d):
    q = math.pow(d["rmax"] / d["rmin"], 1.0 / (d["nrad"] - 2.0))
    return np.array([d["rmin"] * math.pow(q, n - 1.0) for n in range(d["nrad"] + 2)])


def _fields(d, radii, slope, seed):
    """A disk in mid-run: the power-law profiles with a two-armed spiral (5 %), noise
    (0.1 %) and motions of a few per cent of the sound speed."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    nr, nz = d["nrad"], d["naz"]

    def noise(rows):
        return 2.0 * torch.rand((rows, nz), generator=g, device=dev, dtype=torch.float64) - 1.0

    r0 = torch.tensor(radii[:nr], device=dev)
    r1 = torch.tensor(radii[1:nr + 1], device=dev)
    rm = (2.0 / 3.0 * (r1 ** 3 - r0 ** 3) / (r1 ** 2 - r0 ** 2))[:, None]
    ri = torch.tensor(radii[:nr + 1], device=dev)[:, None]
    phi = torch.arange(nz, device=dev, dtype=torch.float64)[None, :] * (2.0 * math.pi / nz)
    turn = 2.0 * math.pi * torch.rand(3, generator=g, device=dev, dtype=torch.float64)
    vk = torch.sqrt(d["G"] * d["hydro_center_mass"] / rm)
    h = d["aspect_ratio"] * rm ** d["flaring_index"]
    arm = torch.cos(2.0 * phi + 8.0 * torch.log(rm) + turn[0])
    sigma = d["sigma0"] * rm ** -slope * (1.0 + 0.05 * arm + 1e-3 * noise(nr))
    cs = h * vk
    vaz = vk * torch.sqrt(1.0 + h * h * (2.0 * d["flaring_index"] - 1.0 - slope)) + \
        cs * (0.02 * torch.sin(2.0 * phi + 8.0 * torch.log(rm) + turn[1]) + 1e-3 * noise(nr))
    csi = d["aspect_ratio"] * ri ** (d["flaring_index"] - 0.5)
    vr = csi * (0.03 * torch.sin(2.0 * phi + 8.0 * torch.log(ri) + turn[2]) +
                1e-3 * noise(nr + 1))
    out = dict(SIGMA=sigma, V_RADIAL=vr, V_AZIMUTHAL=vaz)
    if d["eos"] == 1:
        out["ENERGY"] = sigma * cs ** 2 / (d["gamma"] - 1.0) * (1.0 + 1e-3 * noise(nr))
    return out


def _disk_inputs(case, seed):
    d = _params(case)
    radii = _radii(d)
    return d, radii, _fields(d, radii, 1.0, seed), setups.CircularPlanets(PLANETS[:case["planets"]])


def _batch_inputs(case, seed):
    """The study's disks (sizes, viscosity, planet mass, aspect ratio from the study's own
    seed) with fields from the run's seed."""
    rng = np.random.default_rng(case["sweep"])
    out = []
    for k in range(case["disks"]):
        nr = int(rng.choice(setups.SWEEP_NR))
        alpha, q = 10.0 ** rng.uniform(-4.0, -2.0), 10.0 ** rng.uniform(-5.0, -2.5)
        h, slope = rng.uniform(0.03, 0.07), rng.uniform(0.5, 1.5)
        d = setups.base_params(nr, 3 * nr, 0.4, 2.5, adiabatic=False, alpha=alpha, h=h)
        d["precision"] = 1
        radii = _radii(d)
        out.append((d, radii, _fields(d, radii, slope, seed * 1000 + k),
                    setups.CircularPlanets([(q, 1.0, 0.0)])))
    return out


def _load(engine, fields, nbody):
    for name, a in fields.items():
        a = a.cpu().numpy()
        engine.set_field(name, a)
        engine.set_field(name + "0", a)
    b = nbody.bodies(0.0)
    engine.set_bodies(b, *nbody.indirect(b))
    engine.init_euler(0.0)
    engine.apply_boundary_condition(0.0, 0.0, False)
    return engine.condition_cfl()


# -- the runs -------------------------------------------------------------------------
class _Pages:
    """A snapshot buffer as an array that keeps the snapshot (and its engine) alive."""

    def __init__(self, snap, a):
        self.snap, self.__array_interface__ = snap, a.__array_interface__


def _snapshot(engine, fields):
    snap = Snapshotter(engine, list(fields))
    return snap, {k: np.asarray(_Pages(snap, a)) for k, a in snap.arrays.items()}


def prepare(case, seed):
    s = dict(case=case, t=0.0)
    if case["kind"] == "disk":
        d, radii, fields, nbody = _disk_inputs(case, seed)
        e = Engine(params_from_dict(d), radii)
        s.update(engine=e, nbody=nbody, last_dt=_load(e, fields, nbody),
                 max_var=d["cfl_max_var"], snap=[_snapshot(e, fields)])
        return s
    disks = _batch_inputs(case, seed)
    b = Batch([params_from_dict(d) for d, *_ in disks], [r for _, r, *_ in disks])
    dts = [_load(e, f, n) for e, (_, _, f, n) in zip(b.disks, disks)]
    for k, (d, _, _, n) in enumerate(disks):
        b.set_clock(k, time=0.0, last_dt=dts[k], t_end=1e6, monitor_dt=1e6,
                    cfl_max_var=d["cfl_max_var"], star_mass=n.mstar,
                    planets=[(q * n.mstar, a, p) for q, a, p in n.planets])
    s.update(batch=b, nbody=[n for *_, n in disks], last_dt=dts, times=[0.0] * b.n,
             max_var=[d["cfl_max_var"] for d, *_ in disks],
             snap=[_snapshot(e, f) for e, (_, _, f, _) in zip(b.disks, disks)])
    return s


def _run_disk(s):
    e, nbody = s["engine"], s["nbody"]
    force = []
    for _ in range(s["case"]["steps"]):
        t = s["t"]
        dt = min(s["max_var"] * s["last_dt"], e.condition_cfl())
        if s["case"]["integrator"] == "leapfrog":
            b = nbody.bodies(t + dt / 2)
            first = (b, *nbody.indirect(b))
            step_leapfrog(e, dt, t, first, first)
        else:
            b = nbody.bodies(t)
            e.set_bodies(b, *nbody.indirect(b), 0.0)
            e.step_euler(dt, t)
        force = e.disk_on_nbody_accel(len(b))
        s["t"], s["last_dt"] = t + dt, dt
    return {"force": np.array(force), "time": s["t"]}


def _run_batch(s):
    b = s["batch"]
    if s["case"]["clock"] == "device":
        b.run(s["case"]["steps"], steps_per_graph=s["case"]["steps"])
        return {"time": np.array([b.clock(k)["time"] for k in range(b.n)])}
    for _ in range(s["case"]["steps"]):
        dts = []
        for k, (e, nbody) in enumerate(zip(b.disks, s["nbody"])):
            dts.append(min(s["max_var"][k] * s["last_dt"][k], e.condition_cfl()))
            bodies = nbody.bodies(s["times"][k])
            e.set_bodies(bodies, *nbody.indirect(bodies))
        b.step(dts, s["times"])
        s["times"] = [t + dt for t, dt in zip(s["times"], dts)]
        s["last_dt"] = dts
    return {"time": np.array(s["times"])}


def run(state):
    out = _run_disk(state) if state["case"]["kind"] == "disk" else _run_batch(state)
    for snap, _ in state["snap"]:
        snap.begin()
    for snap, _ in state["snap"]:
        snap.wait()
    out["disks"] = [dict(views) for _, views in state["snap"]]
    return out


def work(case):
    """Per step the evolved state read once and written once in its type, and the scheme's
    additions, multiplications, divisions and roots per cell; the snapshot written once."""
    def one(cells, fields, planets, size):
        flops = {3: 560, 4: 730}[fields] + 45 * (planets + 1)
        return (case["steps"] * 2 * size * fields + 8 * fields) * cells, \
            case["steps"] * flops * cells

    if case["kind"] == "disk":
        b, f = one(case["nr"] * case["nz"], 4 if case["adiabatic"] else 3, case["planets"],
                   8 if case["form"] == FP64 else 4)
        return {"bytes": b, "flops": f}
    rng = np.random.default_rng(case["sweep"])
    cells = 0
    for _ in range(case["disks"]):
        nr = int(rng.choice(setups.SWEEP_NR))
        rng.uniform(size=4)
        cells += nr * 3 * nr
    b, f = one(cells, 3, 1, 4)
    return {"bytes": b, "flops": f}


# -- the scheme in 64-bit torch -------------------------------------------------------
class _Exact:
    """The step's formulas on whole (rings x azimuth) tensors: a staggered polar grid,
    v_r at inner faces (one row more), v_phi at left faces."""

    def __init__(self, d, radii, fields):
        self.d, self.nr, self.nz = d, d["nrad"], d["naz"]
        nr, dev = self.nr, fields["SIGMA"].device
        ra = torch.tensor(radii, device=dev)
        self.ri, self.rs = ra[:nr + 1, None], ra[1:nr + 2, None]
        self.rm = 2.0 / 3.0 * (self.rs ** 3 - self.ri ** 3) / (self.rs ** 2 - self.ri ** 2)
        self.dphi = 2.0 * math.pi / self.nz
        phi = torch.arange(self.nz, device=dev, dtype=torch.float64)[None] * self.dphi
        self.x, self.y = self.rm[:nr] * torch.cos(phi), self.rm[:nr] * torch.sin(phi)
        self.surf = math.pi * (self.rs ** 2 - self.ri ** 2)[:nr] / self.nz
        self.drm = self.rm[1:nr] - self.rm[:nr - 1]
        self.drs = (self.rs - self.ri)[:nr]
        self.S, self.vr, self.va = (fields[k].clone() for k in
                                    ("SIGMA", "V_RADIAL", "V_AZIMUTHAL"))
        self.adi = d["eos"] == 1
        self.E = fields["ENERGY"].clone() if self.adi else None
        self.ref = {k: v.clone() for k, v in fields.items()}
        gm = d["G"] * d["hydro_center_mass"]
        self.omk = torch.sqrt(gm / self.rm[:nr] ** 3)
        self.cs_iso = d["aspect_ratio"] * self.rm[:nr] ** d["flaring_index"] * \
            torch.sqrt(gm / self.rm[:nr])
        self.derived()
        self.qp = self.qm = torch.zeros_like(self.S)
        if self.adi:
            self.stress()
            self.heating()
        self.ghosts()

    def derived(self):
        d = self.d
        if self.adi:
            self.cs = torch.sqrt(d["gamma"] * (d["gamma"] - 1.0) * self.E / self.S)
            self.H = self.cs / math.sqrt(d["gamma"]) / self.omk
        else:
            self.cs = self.cs_iso.expand_as(self.S)
            self.H = self.cs / self.omk
        self.pressure()
        self.nu = d["viscous_alpha"] * self.H * self.cs

    def pressure(self):
        self.P = (self.d["gamma"] - 1.0) * self.E if self.adi else self.S * self.cs ** 2

    def floor_e(self):
        d = self.d
        k = self.S / d["mu"] * d["R_gas"] / (d["gamma"] - 1.0)
        lo = d["minimum_temperature"] * k
        self.E = torch.where(self.E > lo, self.E, lo)  # the upper bound (1e300 K) is never met

    def kick(self, dt, bodies, ix, iy):
        d, nr, act, vact = self.d, self.nr, slice(1, self.nr - 1), slice(2, self.nr - 1)
        below = slice(1, self.nr - 2)
        left = lambda a: torch.roll(a, 1, 1)   # noqa: E731  the value at j - 1
        right = lambda a: torch.roll(a, -1, 1)  # noqa: E731  and at j + 1
        s2 = (d["thickness_smoothing"] * self.H) ** 2
        pot = -ix * self.x - iy * self.y
        for bx, by, m, *_ in bodies:
            pot = pot - d["G"] * m / torch.sqrt((self.x - bx) ** 2 + (self.y - by) ** 2 + s2)
        # pressure, gravity, centrifugal force
        S, P, vr, va = self.S, self.P, self.vr.clone(), self.va
        idr = 1.0 / self.drm[1:nr - 2]
        vt = 0.25 * (va[vact] + right(va)[vact] + va[below] + right(va)[below])
        vr[vact] += dt * (-2.0 / (S[vact] + S[below]) * (P[vact] - P[below]) * idr
                          - (pot[vact] - pot[below]) * idr + vt ** 2 / self.ri[vact])
        idx = 2.0 / (self.dphi * (self.rs[act] + self.ri[act]))
        va = va.clone()
        va[act] -= dt * (2.0 / (S + left(S)) * (P - left(P)) + (pot - left(pot)))[act] * idx
        self.vr, self.va = vr, va
        # compression heating, artificial viscosity
        dvr, dva = vr[1:] - vr[:-1], right(va) - va
        rmn = self.rm[:nr]
        if self.adi:
            div = ((vr[1:] * self.ri[1:] - vr[:-1] * self.ri[:-1]) / (self.drs * rmn)
                   + dva / (self.dphi * rmn))
            e = self.E * torch.exp(-(d["gamma"] - 1.0) * dt * div)
            e[nr - 1] = self.E[nr - 1]
            self.E = e
        C2 = d["art_visc_factor"] ** 2
        vr, va = vr.clone(), va.clone()
        if d["art_visc"] == 1:
            qr = torch.where(dvr < 0, C2 * S * dvr ** 2, 0.0)
            qf = torch.where(dva < 0, C2 * S * dva ** 2, 0.0)
            if self.adi:
                self.E[act] -= dt * (qr * dvr / self.drs + qf * dva / (self.dphi * rmn))[act]
            vr[vact] -= dt * 2.0 / (S[vact] + S[below]) * (qr[vact] - qr[below]) * idr
            va[act] -= (dt * 2.0 / (S + left(S)) * (qf - left(qf)) / (self.dphi * rmn))[act]
        else:
            err = dvr / self.drs
            epp = (dva / self.dphi + 0.5 * (vr[1:] + vr[:-1])) / rmn
            div = torch.clamp(err + epp, max=0.0)
            l2 = C2 * torch.maximum(self.drs, rmn * self.dphi) ** 2
            qr, qf = (-l2 * S * div * (x - div / 3.0) for x in (err, epp))
            if self.adi:
                self.E[act] += dt * (-l2 * div * S / 3.0
                                     * (err ** 2 + epp ** 2 + (err - epp) ** 2))[act]
            va[act] += (2.0 * dt / ((self.rs[:nr] + self.ri[:nr]) * 0.5 * (S + left(S)))
                        * (qf - left(qf)) / self.dphi)[act]
            vr[vact] += dt / (0.5 * (S[vact] + S[below])) * 2.0 / \
                (rmn[vact] ** 2 - rmn[below] ** 2) * (
                    (qr[vact] * rmn[vact] - qr[below] * rmn[below])
                    - 0.5 * (qf[vact] + qf[below]) * (rmn[vact] - rmn[below]))
        self.vr, self.va = vr, va
        if self.adi:
            self.floor_e()
            P = self.P
            self.derived()
            self.P = P
        # viscosity
        self.stress()
        trr, tpp, trp = self.trr, self.tpp, self.trp
        r2 = self.ri ** 2
        self.va[act] += (dt / rmn / (0.5 * (S + left(S)))
                         * (2.0 / (r2[1:] - r2[:-1]) * (r2[1:] * trp[1:] - r2[:-1] * trp[:-1])
                            + (tpp - left(tpp)) / self.dphi))[act]
        self.vr[vact] += dt / (0.5 * (S[vact] + S[below])) * 2.0 / (rmn[vact] + rmn[below]) * (
            (rmn[vact] * trr[vact] - rmn[below] * trr[below]) * idr
            + (right(trp)[vact] - trp[vact]) / self.dphi - 0.5 * (tpp[vact] + tpp[below]))
        if self.adi:
            self.heating()
            self.E[act] += dt * (self.qp - self.qm)[act]
            self.floor_e()

    def stress(self):
        nr, vr, va, S, nu = self.nr, self.vr, self.va, self.S, self.nu
        left, rmn = (lambda a: torch.roll(a, 1, 1)), self.rm[:nr]
        dva = (torch.roll(va, -1, 1) - va) / (self.dphi * rmn)
        self.div = (vr[1:] * self.ri[1:] - vr[:-1] * self.ri[:-1]) / (self.drs * rmn) + dva
        ns = 2.0 * nu * S
        self.trr = ns * ((vr[1:] - vr[:-1]) / self.drs - self.div / 3.0)
        self.tpp = ns * (dva + 0.5 * (vr[1:] + vr[:-1]) / rmn - self.div / 3.0)
        om = va / rmn
        ri = self.ri[1:nr]
        drp = ri * (om[1:] - om[:-1]) / self.drm + (vr - left(vr))[1:nr] / (self.dphi * ri)
        avg = lambda a: 0.25 * (a[1:] + a[:-1] + left(a)[1:] + left(a)[:-1])  # noqa: E731
        self.trp = torch.zeros_like(vr)
        self.trp[1:nr] = avg(nu) * avg(S) * drp

    def heating(self):
        d, nr, S, E = self.d, self.nr, self.S, self.E
        trp = self.trp + torch.roll(self.trp, -1, 1)
        trp = 0.25 * (trp[1:] + trp[:-1])
        ns = self.nu * S
        qp = (self.trr ** 2 + 2.0 * trp ** 2 + self.tpp ** 2) / (2.0 * ns) \
            + 2.0 / 9.0 * ns * self.div ** 2
        qm = E * self.omk / d["cooling_beta_value"]
        a = 1.0 + 8.0 * self.H * d["sigma_sb"] / d["c_light"] * \
            (d["mu"] * (d["gamma"] - 1.0) / (d["R_gas"] * S)) ** 4 * E ** 3
        self.qp, self.qm = qp / a, qm / a
        for q in (self.qp, self.qm):
            q[0] = q[nr - 1] = 0.0

    def ghosts(self):
        n = self.nr
        for q in (self.S, self.E):
            if q is not None:
                q[0], q[n - 1] = q[1].clone(), q[n - 2].clone()
        inner = torch.where(self.vr[2] > 0, 0.0, self.vr[2])
        outer = torch.where(self.vr[n - 2] < 0, 0.0, self.vr[n - 2])
        self.vr[0] = self.vr[1] = inner
        self.vr[n] = self.vr[n - 1] = outer
        for i in (0, n - 1):
            self.va[i] = math.sqrt(self.d["G"] * self.d["hydro_center_mass"] / float(self.rm[i, 0]))

    def limit(self, a, b):
        if self.d["flux_limiter"] == 1:
            m = 2.0 * torch.where(a.abs() < b.abs(), a, b)
            c = 0.5 * (a + b)
            return torch.where(a * b > 0, torch.where(c.abs() < m.abs(), c, m), 0.0)
        s = a + b
        return torch.where(a * b > 0, 2.0 * a * b / torch.where(s == 0, 1.0, s), 0.0)

    def star_r(self, Q, dt):
        nr, v = self.nr, self.vr[1:self.nr]
        g = (Q[1:] - Q[:-1]) / self.drm
        dq = torch.zeros_like(Q)
        dq[1:nr - 1] = self.limit(g[1:], g[:-1])
        up = self.rm[2:nr + 1] - self.rm[1:nr]
        return torch.where(v > 0, Q[:-1] + (self.drm - v * dt) * 0.5 * dq[:-1],
                           Q[1:] - (up + v * dt) * 0.5 * dq[1:])

    def star_phi(self, Q, v, dt):
        dx = self.dphi * self.rm[:self.nr]
        m = torch.roll(Q, 1, 1)
        dq = 0.5 * self.limit(torch.roll(Q, -1, 1) - Q, Q - m) / dx
        ksi = v * dt
        return torch.where(ksi > 0, m + (dx - ksi) * torch.roll(dq, 1, 1), Q - (dx + ksi) * dq)

    def transport(self, dt):
        nr, rmn, S, vr, va = self.nr, self.rm[:self.nr], self.S, self.vr, self.va
        q = [S * vr[1:], S * vr[:-1], S * torch.roll(va, -1, 1) * rmn, S * va * rmn]
        if self.adi:
            q.append(self.E)
        face = torch.zeros_like(vr)
        face[1:nr] = dt * self.dphi * self.ri[1:nr] * vr[1:nr] * self.star_r(S, dt)

        def radial(Q, star):
            f = face.clone()
            if star is not None:
                f[1:nr] *= star
            return Q + (f[:-1] - f[1:]) / self.surf

        q = [radial(Q, self.star_r(Q / S, dt)) for Q in q]
        S = radial(S, None)
        mean = va.mean(1, keepdim=True)
        N = mean / rmn * dt / self.dphi
        whole = torch.floor(N + 0.5)
        uni = (N - whole) * rmn / dt * self.dphi
        res = va - mean
        passes = [res, uni.expand_as(va)] if self.d["fast_transport"] else [uni + res]
        for v in passes:
            f0 = self.drs * dt * v * self.star_phi(S, v, dt) / self.surf

            def azimuthal(Q, f):
                return Q + f - torch.roll(f, -1, 1)

            q = [azimuthal(Q, f0 * self.star_phi(Q / S, v, dt)) for Q in q]
            S = azimuthal(S, f0)
        j = torch.arange(self.nz, device=S.device)[None, :]
        j = torch.remainder(j - whole.to(torch.int64), self.nz)
        S, *q = (torch.gather(a, 1, j) for a in (S, *q))
        vr = self.vr.clone()
        vr[0] = 0.0
        vr[1:nr] = (q[0][:-1] + q[1][1:]) / (S[:-1] + S[1:])
        left = lambda a: torch.roll(a, 1, 1)  # noqa: E731
        self.vr, self.va = vr, (left(q[2]) + q[3]) / (left(S) + S) / rmn
        self.S = torch.clamp(S, min=self.d["sigma_floor"] * self.d["sigma0"])
        if self.adi:
            self.E = q[4]
            self.floor_e()

    def damp(self, dt):
        d, nr = self.d, self.nr
        g = math.pow(d["rmax"] / d["rmin"], 1.0 / (nr - 2.0))
        oc = 1.5 / d["rmin"] * (1 - g ** 2) / (1 - g ** 3)
        for name, attr in (("V_RADIAL", "vr"), ("V_AZIMUTHAL", "va"), ("SIGMA", "S"),
                           ("ENERGY", "E")):
            x = getattr(self, attr)
            if x is None:
                continue
            vec = attr == "vr"
            radius = self.ri if vec else self.rm[:nr]
            top = nr if vec else nr - 1
            for edge, lim, rt in ((d["rmin"], d["damping_inner_limit"], d["rmin"]),
                                  (d["rmax"], d["damping_outer_limit"],
                                   d["damping_time_radius_outer"])):
                r = edge * lim
                k = int(math.floor(math.log(r / d["rmin"] if vec else r * oc) / math.log(g))) + 1
                k = max(0, min(k, nr - 1))
                rows = slice(0, min(k, top) + 1) if lim > 1 else slice(min(k + 1, top), None)
                tau = d["damping_time_factor"] * 2.0 * math.pi / \
                    math.sqrt(d["G"] * d["hydro_center_mass"] / rt ** 3)
                x0 = self.ref[name][rows]
                x[rows] = (x[rows] - x0) * torch.exp(
                    -dt * ((radius[rows] - r) / (edge - r)) ** 2 / tau) + x0

    def cfl(self):
        d, nr, act = self.d, self.nr, slice(1, self.nr - 1)
        rmn, vr, va = self.rm[:nr], self.vr, self.va
        mean = va.mean(1, keepdim=True)
        om = mean / rmn
        shear = d["cfl"] * self.dphi / ((om[:-1] - om[1:]).abs() + 1e-100)
        dxa = rmn * self.dphi
        cell = torch.minimum(self.drs, dxa)
        lf = 0.6 if d.get("integrator") == 1 else 1.0
        dvr, dva = vr[1:] - vr[:-1], torch.roll(va, -1, 1) - va
        if d["art_visc"] == 1:
            q = torch.maximum(torch.clamp(-dvr, min=0.0) / self.drs,
                              torch.clamp(-dva, min=0.0) / dxa)
        else:
            q = torch.clamp(-(dvr / self.drs + (dva / self.dphi + 0.5 * (vr[1:] + vr[:-1])) / rmn),
                            min=0.0)
        total = (self.cs / cell) ** 2 + (vr[:-1] / self.drs) ** 2
        total = total + ((va - mean if d["fast_transport"] else va) / dxa) ** 2
        total = total + (4.0 * d["art_visc_factor"] ** 2 * q * lf) ** 2
        total = total + (4.0 * self.nu / cell ** 2 * lf) ** 2
        if self.adi:
            total = total + (((self.qp - self.qm) / self.E) / d["heating_cooling_cfl_limit"] * lf) ** 2
        return min(float(shear[:nr - 1].min()), float((d["cfl"] / torch.sqrt(total[act])).min()))

    def force(self, bodies):
        act = slice(1, self.nr - 1)
        mass = (self.surf * (self.S - self.S.mean(1, keepdim=True)))[act]
        s2 = (self.d["thickness_smoothing"] * self.H[act]) ** 2
        out = []
        for bx, by, *_ in bodies:
            dx, dy = self.x[act] - bx, self.y[act] - by
            w = self.d["G"] * mass * (dx ** 2 + dy ** 2 + s2) ** -1.5
            out.append([float((w * dx).sum()), float((w * dy).sum())])
        return torch.tensor(out, dtype=torch.float64)

    def step(self, dt, t, nbody, leapfrog):
        b = nbody.bodies(t + dt / 2 if leapfrog else t)
        ind = nbody.indirect(b)
        self.kick(dt / 2 if leapfrog else dt, b, *ind)
        self.ghosts()
        self.transport(dt)
        if leapfrog:
            self.pressure()
            self.kick(dt / 2, b, *ind)
        self.damp(dt)
        self.ghosts()
        self.derived()
        return b

    def outputs(self):
        out = dict(SIGMA=self.S, V_RADIAL=self.vr, V_AZIMUTHAL=self.va)
        if self.adi:
            out["ENERGY"] = self.E
        return out


def _exact_disk(d, radii, fields, nbody, steps):
    x = _Exact(d, radii, fields)
    t, last, b = 0.0, x.cfl(), []
    for _ in range(steps):
        dt = min(d["cfl_max_var"] * last, x.cfl())
        b = x.step(dt, t, nbody, d.get("integrator") == 1)
        t, last = t + dt, dt
    return x, t, b


def exact(case, seed):
    if case["kind"] == "disk":
        d, radii, fields, nbody = _disk_inputs(case, seed)
        x, t, b = _exact_disk(d, radii, fields, nbody, case["steps"])
        return {"force": x.force(b), "time": t, "disks": [x.outputs()]}
    times, disks = [], []
    for d, radii, fields, nbody in _batch_inputs(case, seed):
        x, t, _ = _exact_disk(d, radii, fields, nbody, case["steps"])
        times.append(t)
        disks.append(x.outputs())
    return {"time": np.array(times), "disks": disks}
