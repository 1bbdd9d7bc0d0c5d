"""Timed workloads of the library: what a simulation host has it do, from a
2D column of a few thousand particles to a box of eight million.

A case names a workload (`kind`), its size (`dx` or `n`), the precision form
and the number of whole steps of one pass.  A pass starts from a state that
the program holds (on the device, or in page-locked host memory), so every
pass does the same work: it hands the state over (sph_upload, the IC part of
the time loop), advances it and takes the new state back.
"""
import ctypes as C
import math

import numpy as np
import torch

import sphera_b200
from sphera_b200 import Batch, Simulation, abi, cases
from sphera_b200.slab import DeviceState

FORMS = {"fp64": abi.SPH_PREC_FP64, "fp32c": abi.SPH_PREC_FP32C}

# the most particle-steps of a drawn case
MOST_PARTICLE_STEPS = 16.0e6


def listed():
    return [
        # the smallest job: the 5,000-particle 2D column between two output
        # frames; launches and latency are all of it
        dict(name="column_2d_fp64", kind="column", dx=0.02, form="fp64", steps=40),
        # a 2D column at an odd resolution, read back to the host every frame
        dict(name="column_2d_fp32c", kind="column", dx=0.0113, form="fp32c", steps=40, to_host=True),
        # a coarse 3D run (13,500 particles), as parameter studies use
        dict(name="dam_3d_small", kind="dam", dx=0.02, form="fp32c", steps=20),
        # the headline workload: 864,000 particles, tuned once before a long run
        dict(name="dam_3d_fp32c", kind="dam", dx=0.005, form="fp32c", steps=10, tuned=True),
        # the reference's own arithmetic at an ordinary size
        dict(name="dam_3d_fp64", kind="dam", dx=0.0075, form="fp64", steps=10),
        # a forced sloshing tank with partial smoothing of velocity and pressure
        dict(name="slosh_3d_smoothed", kind="slosh", dx=0.0095, form="fp32c", steps=10, teta=0.2),
        # first-order consistency (renormalised gradients) as its tutorials set it
        dict(name="dam_3d_c1", kind="dam", dx=0.0105, form="fp64", steps=5, c1=0.614),
        # an ensemble study: 64 members of 2.5k-50k particles in one batch
        dict(name="ensemble_2d", kind="ensemble", members=64, dx=0.01, form="fp32c", steps=10, tuned=True),
        # the random-box microbenchmark, small, in FP64
        dict(name="box_3d_fp64", kind="box", n=400009, form="fp64", steps=1),
        # and large, in the compensated FP32 form
        dict(name="box_3d_fp32c", kind="box", n=8000003, form="fp32c", steps=2),
        # a host that keeps the particles in its own (page-locked) memory and
        # hands them over at every step
        dict(name="coupled_3d_fp32c", kind="coupled", dx=0.006, form="fp32c", steps=1),
        # a host loop that replaces the reference's subroutines one by one
        dict(name="calls_3d_fp64", kind="calls", dx=0.012, form="fp64", steps=4),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    form = rng.choice(["fp64", "fp32c"])
    kind = rng.choice(["column", "dam", "dam", "slosh", "ensemble", "box", "coupled", "calls", "order"])
    if kind == "column":
        c = dict(kind=kind, dx=log(0.0065, 0.028), form=form, steps=rng.choice([20, 40]),
                 to_host=rng.random() < 0.5)
    elif kind in ("dam", "slosh"):
        option = rng.choice(["plain", "plain", "teta", "c1", "tuned"])
        c = dict(kind=kind, dx=log(0.0075, 0.025), form=form, steps=rng.choice([5, 10]))
        if option == "teta":
            c["teta"] = round(rng.uniform(0.05, 0.3), 3)
        elif option == "c1":
            c["c1"] = 0.614
        elif option == "tuned":
            c["tuned"] = True
    elif kind == "ensemble":
        c = dict(kind=kind, members=rng.randint(3, 40), dx=0.01, form=form, steps=rng.choice([5, 10]),
                 tuned=rng.random() < 0.5)
    elif kind == "box":
        c = dict(kind=kind, n=int(log(50e3, 4e6)) | 1, form=form, steps=1)
    elif kind == "coupled":
        c = dict(kind=kind, dx=log(0.006, 0.025), form=form, steps=rng.choice([1, 2]))
    elif kind == "calls":
        c = dict(kind=kind, dx=log(0.009, 0.025), form=form, steps=rng.choice([2, 4]))
    else:
        c = dict(kind=kind, n=int(log(1e3, 1e6)) | 1, dim=rng.choice([2, 3]), steps=1)
    if c["kind"] != "order" and _count(c) * c["steps"] > MOST_PARTICLE_STEPS:
        c["steps"] = max(1, int(MOST_PARTICLE_STEPS / _count(c)))
    return c


# ----------------------------------------------------------------- workloads
def _count(case):
    """Particles of a case."""
    kind = case["kind"]
    if kind in ("box", "order"):
        return case["n"]
    dx = case["dx"]
    if kind == "column":
        return round(1.0 / dx) * round(2.0 / dx)
    if kind == "slosh":
        return round(1.0 / dx) * round(0.5 / dx) * round(0.25 / dx)
    if kind == "ensemble":
        return int(case["members"] * 1.25 * 1.5 / dx ** 2)   # mean width and height
    return round(0.6 / dx) * round(0.3 / dx) * round(0.6 / dx)


def _collapse(case, dims, seed):
    """The velocities of a column in collapse: the stagnation flow that
    spreads it along x as it falls, and a disturbance of 2 cm/s."""
    rng = np.random.Generator(np.random.PCG64([seed, 0x5EED]))
    st = case.state
    lx, lz = dims
    st.v[:, 0] = 0.8 * st.x[:, 0] / lx
    st.v[:, 2] = -0.8 * (lz / lx) * st.x[:, 2] / lz
    axes = [0, 2] if case.params.dim == 2 else [0, 1, 2]
    for d in axes:
        st.v[:, d] += rng.uniform(-0.02, 0.02, size=st.n)
    return case


def _build(case, seed):
    """The workload as the library's generators make it, on a jittered
    lattice (a tenth of the spacing: a flow has lost its lattice)."""
    kind, precision = case["kind"], FORMS[case.get("form", "fp64")]
    if kind == "column":
        c = _collapse(cases.dam_break_2d(dx=case["dx"], jitter=0.1, seed=seed, precision=precision), (1.0, 2.0), seed)
    elif kind == "box":
        c = cases.random_box(n=case["n"], seed=seed, precision=precision)
    elif kind == "slosh":
        c = cases.sloshing_3d(dx=case["dx"], jitter=0.1, seed=seed, precision=precision)
    else:
        c = _collapse(cases.dam_break_3d(dx=case["dx"], jitter=0.1, seed=seed, precision=precision), (0.6, 0.6), seed)
    if case.get("teta"):
        c.params.teta_p = c.params.teta_v = case["teta"]
    if case.get("c1"):
        c.params.c1_be = c.params.c1_divu = 1
        c.params.invb_det_thresh = case["c1"]
    return c


def _ensemble(case, seed):
    """The columns of an ensemble study, as cases.ensemble_2d sizes them
    (width U[0.5, 2.0] m, height U[0.5, 2.5] m); the seed disturbs them."""
    rng, dx = np.random.Generator(np.random.PCG64(0xC3)), case["dx"]
    out = []
    for i in range(case["members"]):
        size = tuple(round(rng.uniform(0.5, hi) / dx) * dx for hi in (2.0, 2.5))
        c = cases.dam_break_2d(dx=dx, column=size, jitter=0.1, seed=[seed, i], precision=FORMS[case["form"]])
        out.append(_collapse(c, size, seed + i))
    return out


def _on_device(st):
    return DeviceState(*(torch.from_numpy(getattr(st, f)).cuda() for f in ("x", "v", "rho", "p", "m")))


def _blank_device(n):
    return DeviceState(*(torch.empty(s, dtype=torch.float64, device="cuda") for s in ((n, 3), (n, 3), (n,), (n,), (n,))))


def _pinned(n, like=None):
    bufs = [torch.empty(s, dtype=torch.float64, pin_memory=True) for s in ((n, 3), (n, 3), (n,), (n,), (n,))]
    st = abi.State(*(b.numpy() for b in bufs))
    if like is not None:
        for f in ("x", "v", "rho", "p", "m"):
            getattr(st, f)[...] = getattr(like, f)
    st.pins = bufs
    return st


def _fields(st, n):
    return {f: getattr(st, f)[:n] for f in ("x", "v", "rho", "p", "m")}


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "order":
        return _prepare_order(case, seed)
    s = dict(kind=kind, steps=case["steps"])
    if kind == "ensemble":
        cs = _ensemble(case, seed)
        s["sim"] = Batch(cs)
        s["states"] = [_on_device(c.state) for c in cs]
        n = sum(c.n for c in cs)
        s["all"] = _blank_device(n)
        at, s["outs"] = 0, []
        for c in cs:   # the members' rows of one set of arrays
            s["outs"].append(DeviceState(*(getattr(s["all"], f)[at:at + c.n] for f in ("x", "v", "rho", "p", "m"))))
            at += c.n
    else:
        c = _build(case, seed)
        s["sim"] = Simulation(c)
        if kind == "coupled":
            s["state"], s["out"] = _pinned(c.n, c.state), _pinned(c.n)
        elif kind == "calls" or case.get("to_host"):
            s["state"] = c.state
        else:
            s["state"], s["out"] = _on_device(c.state), _blank_device(c.n)
    torch.cuda.synchronize()
    if case.get("tuned"):
        s["sim"].upload(s["states"] if kind == "ensemble" else s["state"])
        s["sim"].autotune(reps=2)
    return s


def _prepare_order(case, seed):
    """Positions for OrdGrid1 alone, on a caller's stream and buffers: a
    filled box at 18 (3D) or 7 (2D) particles per cell, in caller order."""
    n, dim = case["n"], case["dim"]
    rng = np.random.Generator(np.random.PCG64(seed))
    dx = 0.01
    side = dx * n ** (1.0 / dim)
    x = rng.uniform(0.0, side, size=(n, 3))
    if dim == 2:
        x[:, 1] = 0.0
    p = abi.make_params(dim=dim, precision=abi.SPH_PREC_FP64, dx=dx, trunc=1.3, domain_lo=(0.0, 0.0, 0.0),
                        domain_hi=(side, side if dim == 3 else 0.0, side))
    ncd, _, _ = _grid(p)
    i32 = dict(dtype=torch.int32, device="cuda")
    s = dict(kind="order", params=p, n=n, x=torch.from_numpy(x).cuda(), cella=torch.empty(n, **i32),
             icont=torch.empty(ncd[0] * ncd[1] * ncd[2] + 1, **i32), order=torch.empty(n, **i32))
    f = sphera_b200.lib().sph_ord_grid_static
    f.argtypes = [C.POINTER(abi.SphParams), C.c_int32] + [C.c_void_p] * 5
    f.restype = C.c_int
    s["call"] = f
    return s


# ----------------------------------------------------------------------- run
def _ok(code):
    if code != abi.SPH_OK:
        raise sphera_b200.SphError(code, "sphera_b200")


def run(s):
    kind = s["kind"]
    if kind == "order":
        _ok(s["call"](C.byref(s["params"]), s["n"], s["x"].data_ptr(), s["cella"].data_ptr(), s["icont"].data_ptr(),
                      s["order"].data_ptr(), torch.cuda.current_stream().cuda_stream))
        return {"cella": s["cella"], "icont": s["icont"], "order": s["order"]}
    sim, lib = s["sim"], sphera_b200.lib()
    if kind == "ensemble":
        sim.upload(s["states"])
        sim.step(s["steps"])
        for i, out in enumerate(s["outs"]):
            _ok(lib.sph_batch_download(sim._h, i, C.byref(out.struct)))
        return _fields(s["all"], s["all"].n)
    sim.upload(s["state"])
    if kind == "coupled":
        out = s["out"]
        out.struct.n = out.n
        _ok(lib.sph_step_download(sim._h, s["steps"], C.byref(out.struct)))
        return _fields(out, out.struct.n)
    if kind == "calls":
        for _ in range(s["steps"]):
            sim.time_step_duration()
            sim.rhs_momentum(want=False)
            sim.leapfrog_momentum()
            sim.leapfrog_trajectories()
            sim.ord_grid()
            sim.boundary_data_tab()
            sim.continuity(want=False)
            sim.leapfrog_continuity()
            sim.eos()
        st = sim.download()
        return _fields(st, st.n)
    sim.step(s["steps"])
    if "out" not in s:
        st = sim.download()
        return _fields(st, st.n)
    return _fields(s["out"], sim.download_into(s["out"]))


# ---------------------------------------------------------------------- work
def work(case):
    """The 72-byte state of a particle read once and written once, and for
    every step and accepted pair 9 flops of distance, 107 of the momentum
    terms and 34 of the continuity terms (30 more with partial smoothing,
    230 more with C1)."""
    n, steps = _count(case), case["steps"]
    if case["kind"] == "order":
        cells = n / (2.6 ** case["dim"])
        return {"bytes": 24.0 * n + 8.0 * n + 4.0 * cells, "flops": 0.0}
    two_d = case["kind"] in ("column", "ensemble")
    pairs = math.pi * 2.6 ** 2 if two_d else 4.0 / 3.0 * math.pi * 2.6 ** 3
    flops = 150.0 + (30.0 if case.get("teta") else 0.0) + (230.0 if case.get("c1") else 0.0)
    return {"bytes": 144.0 * n, "flops": flops * pairs * n * steps}


# --------------------------------------------------------------------- exact
def exact(case, seed):
    """The pass in 64 bits without the library, for the workloads without
    walls (the wall terms are defined by the method's own tabulated
    quadrature, which has no plain form to hold them against) and for the
    cell order."""
    if case["kind"] == "order":
        return _exact_order(case, seed)
    if case["kind"] != "box":
        return None
    c = _build(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, v, rho, p, m = (torch.from_numpy(getattr(c.state, f)).to(dev) for f in ("x", "v", "rho", "p", "m"))
    s = c.params
    h, cs = s.dx * s.trunc, math.sqrt(s.eps / s.den0)

    def step_length(vel):
        return min(s.cfl * 2.0 * h / (cs + float(vel.norm(dim=1).max())), s.vsc_coeff * h * h / (0.5 * s.kin_visc))

    dt = dt_prev = step_length(v)
    nb = _Neighbours(s, x)
    grav = torch.tensor(list(s.grav), dtype=torch.float64, device=dev)
    for _ in range(case["steps"]):
        v = v + 0.5 * (dt + dt_prev) * (nb.momentum(v, rho, p, m) + grav)
        x = x + dt * v
        nb = _Neighbours(s, x)
        rho = rho - dt * nb.continuity(v, rho, m)
        p = s.eps / s.den0 * (rho - s.den0) + s.p_ref
        dt, dt_prev = step_length(v), dt
    return {"x": x, "v": v, "rho": rho, "p": p, "m": m}


def _grid(s):
    """CreaGrid.f90:51-74: cells per axis, origin and cell size."""
    doubleh, epsi = 2.0 * s.dx * s.trunc, 0.01 * s.dx
    ncd, lo, dcd = [], [], []
    for d in range(3):
        a, b = s.domain_lo[d] - doubleh - epsi, s.domain_hi[d] + doubleh + epsi
        k = int(math.floor((b - a) / doubleh + 0.5))
        ncd.append(k if d != 1 or s.dim == 3 else 1)
        lo.append(a)
        dcd.append((b - a) / k)
    return ncd, lo, dcd


def _exact_order(case, seed):
    s = _prepare_order(case, seed)
    ncd, lo, dcd = _grid(s["params"])
    x = s["x"]
    i, j, k = (torch.ceil((x[:, d] - lo[d]) / dcd[d]).to(torch.int64) for d in range(3))
    if case["dim"] == 2:
        j = torch.ones_like(j)
    cella = ((k - 1) * ncd[1] + (j - 1)) * ncd[0] + i
    order = torch.sort(cella, stable=True).indices + 1
    count = torch.bincount(cella - 1, minlength=ncd[0] * ncd[1] * ncd[2])
    icont = torch.cat([count.new_ones(1), 1 + torch.cumsum(count, 0)])
    return {"cella": cella.to(torch.int32), "icont": icont.to(torch.int32), "order": order.to(torch.int32)}


class _Neighbours:
    """Pair sums over the particles of the 27 cells around each one, the
    m-th particle of a neighbouring cell for all particles at a time."""

    def __init__(self, s, x):
        self.s, self.x = s, x
        self.h = s.dx * s.trunc
        ncd, lo, dcd = _grid(s)
        c = [torch.ceil((x[:, d] - lo[d]) / dcd[d]).to(torch.int64) - 1 for d in range(3)]
        cells = ncd[0] * ncd[1] * ncd[2]
        key = (c[1] * ncd[0] + c[0]) * ncd[2] + c[2]
        self.order = torch.sort(key).indices
        self.count = torch.bincount(key, minlength=cells)
        self.start = torch.cumsum(self.count, 0) - self.count
        self.cell, self.ncd = [t[self.order] for t in c], ncd

    def pairs(self):
        """(rows i, rows j) in sorted order, pair by pair of cell offsets."""
        n = len(self.order)
        rows = torch.arange(n, device=self.x.device)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    at = [self.cell[0] + dx, self.cell[1] + dy, self.cell[2] + dz]
                    inside = torch.ones(n, dtype=torch.bool, device=self.x.device)
                    for a, k in zip(at, self.ncd):
                        inside &= (a >= 0) & (a < k)
                    key = torch.where(inside, (at[1] * self.ncd[0] + at[0]) * self.ncd[2] + at[2], 0)
                    first, left = self.start[key], torch.where(inside, self.count[key], 0)
                    for m in range(int(left.max())):
                        i = rows[left > m]
                        yield i, first[i] + m

    def kernel(self, rr):
        s, h = self.s, self.h
        r = rr.sqrt()
        q, q2, eta, eta2 = r / h, rr / (h * h), 1.0e-3 * h, 1.0e-2 * h * h
        ke, kacl = 0.477464 / h ** 4, 0.074603 / h ** 4
        g = torch.where(q < 1.0, 1.5 * q2 - 2.0 * q, 2.0 * q - 0.5 * q2 - 2.0) * ke
        pk1 = g / (r + eta)
        return pk1, pk1 / (rr + eta2), (12.0 * q - 3.0 * q2 - 12.0) * kacl / (r + eta)

    def accepted(self):
        x = self.x[self.order]
        for i, j in self.pairs():
            d = x[i] - x[j]
            rr = (d * d).sum(1)
            keep = (rr <= 4.0 * self.h * self.h) & (i != j)
            i, j, d, rr = i[keep], j[keep], d[keep], rr[keep]
            yield i, j, d, rr, self.kernel(rr)

    def back(self, t):
        out = torch.empty_like(t)
        out[self.order] = t
        return out

    def momentum(self, v, rho, p, m):
        s, h, nu = self.s, self.h, self.s.kin_visc
        cs = math.sqrt(s.eps / s.den0)
        v, rho, p, m = (t[self.order] for t in (v, rho, p, m))
        acc = torch.zeros_like(v)
        for i, j, d, rr, (_, pk2, pk3) in self.accepted():
            dv, rs = v[j] - v[i], rho[i] + rho[j]
            f = -m[j] * (p[i] / rho[i] ** 2 + p[j] / rho[j] ** 2) * pk3
            f = f - m[j] * (s.alfa_mon * 2.0 * cs * h / rs) * (dv * d).sum(1) * pk2
            w = -m[j] * 4.0 * nu * nu / (nu * rs + 1.0e-3) * pk2 * rr
            acc[i] += f[:, None] * d + w[:, None] * dv   # each i at most once
        return self.back(acc)

    def continuity(self, v, rho, m):
        """Minus the density rate: sum of rho_i (m_j / rho_j) PK1 (v_j - v_i) . (x_i - x_j)."""
        v, rho, m = (t[self.order] for t in (v, rho, m))
        out = torch.zeros_like(rho)
        for i, j, d, _, (pk1, _, _) in self.accepted():
            out[i] += rho[i] * (m[j] / rho[j]) * pk1 * ((v[j] - v[i]) * d).sum(1)
        return self.back(out)
