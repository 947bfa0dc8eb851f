"""The work that a user of tcad_b200 has it do, as timed cases.

Each case is one use of a public entry point (Device2D / Device3D,
DeviceBatch, solve_transient, solve_linear, the pack's assembly) on a device
of workloads.py's kinds, from a converged starting point where the call
needs one.  listed() names the cases, draw(rng) gives more of the same
ranges, prepare / run / work / exact serve one case.

The state that a pass starts from is put back at the start of the pass, the
way a program that explores several biases from one converged point does it.
"""
import math
import warnings

import numpy as np
import torch

import tcad_b200 as tb
from tcad_b200 import _lib
from tcad_b200 import workloads as W
from tcad_b200.batch import DeviceBatch
from tcad_b200.linsolve import solve_linear
from tcad_b200.physics import Mesh2D, Semiconductor
from tcad_b200.transient import RampWaveform, solve_transient


def listed():
    return [
        # reading the terminal currents of a converged small 2D device: the
        # smallest call, after every bias point of a sweep
        dict(name="currents_diode_201x101", kind="currents", device="diode", nx=201, ny=101),
        # the coupled residual and Jacobian alone, for a program with its own
        # Newton loop: a 2D MOSFET and the full-size 3D tri-gate
        dict(name="assemble_mosfet_256x128", kind="assemble", device="mosfet", nx=256, ny=128),
        dict(name="assemble_trigate_160x96x64", kind="assemble", device="trigate", nx=160,
             ny=96, nz=64),
        # the first solve of every device: 2D and 3D equilibrium
        dict(name="equilibrium_mosfet_240x120", kind="equilibrium", device="mosfet", nx=240,
             ny=120),
        dict(name="equilibrium_trigate_96x56x40", kind="equilibrium", device="trigate", nx=96,
             ny=56, nz=40),
        # a bias sweep of one small device (interactive use): the plain-method
        # p-n diode and a coarse tri-gate
        dict(name="sweep_diode_201x101", kind="sweep", device="diode", nx=201, ny=101, points=3),
        dict(name="sweep_trigate_40x24x16", kind="sweep", device="trigate", nx=40, ny=24, nz=16,
             points=3),
        # one bias point of a large 3D device: the Id-Vg tri-gate at its full
        # mesh, and a million-node p-i-n
        dict(name="point_trigate_160x96x64", kind="sweep", device="trigate", nx=160, ny=96,
             nz=64, points=1),
        dict(name="point_pin_128x128x64", kind="sweep", device="pin", nx=128, ny=128, nz=64,
             points=1),
        # device variants of uneven size through equilibrium and the first
        # ramp step as one batch (design-of-experiments use)
        dict(name="batch_mosfet_16", kind="batch", count=16, nx_lo=40, nx_hi=120, ny_lo=20,
             ny_hi=60, precision="fp64"),
        # switching transient of a small diode, backward Euler
        dict(name="transient_diode_81x41", kind="transient", device="diode", nx=81, ny=41,
             steps=6, theta=1.0),
        # the general sparse drop-in: one implicit time step's Jacobian of a
        # MOSFET as CSR, GMRES with node-block Jacobi
        dict(name="linear_gmres_mosfet_96x48", kind="linear", device="mosfet", nx=96, ny=48,
             method="gmres"),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh3(rng, lo, hi):
    """An nx >= ny >= nz mesh of about lo .. hi nodes, proportions near the
    listed ones."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    c = (n / (10 * 6 * 4)) ** (1 / 3)
    return dict(nx=max(12, int(10 * c * rng.uniform(0.9, 1.1))),
                ny=max(8, int(6 * c * rng.uniform(0.9, 1.1))),
                nz=max(6, int(4 * c * rng.uniform(0.9, 1.1))))


def _mesh2(rng, lo, hi):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = rng.uniform(1.4, 2.4)
    return dict(nx=max(20, int(math.sqrt(n * a))), ny=max(10, int(math.sqrt(n / a))))


def draw(rng):
    kind = rng.choice(["currents", "assemble", "assemble", "equilibrium", "equilibrium", "sweep",
                       "sweep", "sweep", "point", "batch", "transient", "linear"])
    if kind == "currents":
        return dict(kind=kind, device="diode", **_mesh2(rng, 2e3, 1e5))
    if kind == "assemble":
        if rng.random() < 0.5:
            return dict(kind=kind, device="mosfet", **_mesh2(rng, 2e3, 3e5))
        return dict(kind=kind, device=rng.choice(["trigate", "pin"]), **_mesh3(rng, 6e3, 9e5))
    if kind == "equilibrium":
        if rng.random() < 0.6:
            return dict(kind=kind, device=rng.choice(["mosfet", "diode"]),
                        **_mesh2(rng, 1e3, 3e4))
        return dict(kind=kind, device=rng.choice(["trigate", "pin"]), **_mesh3(rng, 5e3, 3e5))
    if kind == "sweep":
        if rng.random() < 0.5:
            return dict(kind=kind, device="diode", points=rng.randint(1, 3),
                        **_mesh2(rng, 1e3, 4e4))
        return dict(kind=kind, device=rng.choice(["trigate", "pin"]), points=rng.randint(1, 2),
                    **_mesh3(rng, 5e3, 6e4))
    if kind == "point":
        return dict(kind="sweep", device=rng.choice(["trigate", "pin"]), points=1,
                    **_mesh3(rng, 8e4, 6e5))
    if kind == "batch":
        nx, ny = rng.randint(30, 60), rng.randint(14, 30)
        return dict(kind=kind, count=_loguniform(rng, 2, 24), nx_lo=nx, nx_hi=2 * nx, ny_lo=ny,
                    ny_hi=2 * ny, precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "transient":
        return dict(kind=kind, device="diode", steps=rng.randint(3, 6),
                    theta=rng.choice([1.0, 1.0, 0.5]), **_mesh2(rng, 1e3, 6e3))
    return dict(kind=kind, device="mosfet", method=rng.choice(["gmres", "bicgstab"]),
                **_mesh2(rng, 1e3, 9e3))


# ---- devices ---------------------------------------------------------------
def _diode(rng, nx, ny):
    """workloads.diode2d's structure with seeded doping levels (for even nx
    the junction falls between two nodes)."""
    L = 2.0e-4
    x = W.diode_x(nx) if nx % 2 else np.linspace(0.0, L, nx)
    y = np.linspace(0.0, 1.0e-4, ny)
    na, nd = 1e17 * rng.uniform(0.7, 1.4), 1e18 * rng.uniform(0.7, 1.4)
    dop = np.where(np.meshgrid(x, y)[0] < 0.5 * L, -na, nd)
    mat = Semiconductor(tau_n0=1e-7, tau_p0=1e-7, tau_Nref=1e300)
    dev = tb.Device2D(Mesh2D(x, y), dop, material=mat,
                      models=tb.Models(doping_mobility=False, srh=True, auger=False, bgn=False))
    dev.add_contact("anode", np.zeros(ny, int), np.arange(ny))
    dev.add_contact("cathode", np.full(ny, nx - 1), np.arange(ny))
    return dev


def _device(case, seed):
    """(device, the bias points of its sweep)."""
    rng = np.random.default_rng([seed, 7])
    kind = case["device"]
    points = int(case.get("points", 1))
    if kind == "diode":
        dev = _diode(rng, case["nx"], case["ny"])
        top = 0.55 + 0.05 * rng.random()
        volts = [{"anode": top * (k + 1) / points} for k in range(points)]
    elif kind == "mosfet":
        dev = W.mosfet2d(tb.Device2D, case["nx"], case["ny"], Lg=100e-7 * rng.uniform(0.8, 1.2),
                         Na=1e17 * rng.uniform(0.6, 1.6), Nsd_peak=1e20 * rng.uniform(0.5, 1.0))
        volts = [{"gate": 0.3, "drain": 0.05}]
    elif kind == "trigate":
        dev = W.trigate3d(tb.Device3D, case["nx"], case["ny"], case["nz"],
                          Na=1e18 * rng.uniform(0.8, 1.25),
                          Nsd_peak=1e20 * rng.uniform(0.6, 1.0))
        vg = 0.2 + 0.05 * rng.random()
        volts = [W.trigate_bias(0.05, vg + 0.1 * k) for k in range(points)]
    else:
        dev = W.pin3d(tb.Device3D, case["nx"], case["ny"], case["nz"],
                      NA=1e19 * rng.uniform(0.7, 1.4), ND=1e19 * rng.uniform(0.7, 1.4))
        top = 0.6 + 0.05 * rng.random()
        volts = [{"anode": top * (k + 1) / points} for k in range(points)]
    return dev, volts


def _biased_state(dev, seed):
    """A smooth non-equilibrium state near the neutral bulk, on the host:
    what a Newton loop's iterate looks like, from the seed alone."""
    rng = np.random.default_rng([seed, 11])
    s = dev.setup
    r = [c / c[-1] for c in s.coords]
    g = np.meshgrid(*reversed(r), indexing="ij")
    wave = sum(np.sin((2 + k) * np.pi * q + rng.uniform(0, 6.28)) for k, q in enumerate(g))
    psi = s.bulk_guess() + 0.3 * wave
    fn, fp = (2.0 * (a * g[-1] + b * g[0]) for a, b in rng.uniform(0.5, 1.0, (2, 2)))
    return psi, s.nie_s * np.exp(psi - fn), s.nie_s * np.exp(fp - psi)


def _batch_devices(case, seed):
    q = W.mosfet_batch_params(count=case["count"], seed=1000,
                              nx=(case["nx_lo"], case["nx_hi"]),
                              ny=(case["ny_lo"], case["ny_hi"]), Lg=(60e-7, 150e-7),
                              Na=(5e16, 5e17), Npk=(2e19, 1e20), V=(0.2, 0.6))
    f = np.random.default_rng([seed, 17]).uniform(0.8, 1.25, (len(q), 2))
    devs = [W.mosfet2d(tb.Device2D, p["nx"], p["ny"], Lg=p["Lg"] * a, Na=p["Na"] * b,
                       Nsd_peak=p["Nsd_peak"]) for p, (a, b) in zip(q, f)]
    return devs, [{"gate": 0.5 * p["Vg"], "drain": 0.25 * p["Vd"]} for p in q]


def _linear_system(dev, seed):
    """One implicit time step's Jacobian of the device as CSR with its rows
    scaled to unit diagonal, the right-hand side of a known solution, and
    that solution."""
    rng = np.random.default_rng([seed, 13])
    psi, n, p = _biased_state(dev, seed)
    A = dev._residual_jacobian(psi, n, p, {})[1].tocsr()
    A.sum_duplicates()
    dV = np.outer(dev.setup.dv[1], dev.setup.dv[0]).ravel()
    shift = np.zeros(3 * dev.N)
    shift[1::3], shift[2::3] = -dV / 1e-3, dV / 1e-3
    shift[dev._dirichlet_rows] = 0.0
    A.setdiag(A.diagonal() + shift)
    A.data /= np.repeat(A.diagonal(), np.diff(A.indptr))
    gy, gx = np.meshgrid(*(np.linspace(0.0, np.pi, m) for m in dev.setup.shape), indexing="ij")
    x = np.stack([np.sin(k * gx + a) * np.cos(k * gy + b) for k, (a, b) in
                  enumerate(rng.uniform(0, 6.28, (3, 2)), 1)], -1).ravel()
    return A, A @ x, x


# ---- one case --------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        devs, volts = _batch_devices(case, seed)
        return dict(kind=kind, batch=DeviceBatch(devs), volts=volts,
                    opts=tb.NewtonOptions(precision=case["precision"]))
    dev, volts = _device(case, seed)
    st = dict(kind=kind, dev=dev, volts=volts)
    if kind in ("currents", "assemble"):
        for name, a in zip(("psi", "n", "p"), _biased_state(dev, seed)):
            setattr(dev, name, a)
        dev.pack.set_bias()
    elif kind == "equilibrium":
        dev.pack
    elif kind in ("sweep", "transient"):
        dev.solve_equilibrium()
        st["start"] = dev.save_state()
    elif kind == "linear":
        st["A"], st["b"], _ = _linear_system(dev, seed)
        st["method"] = case["method"]
    if kind == "transient":
        st["steps"], st["theta"] = case["steps"], case["theta"]
    return st


def run(st):
    kind = st["kind"]
    if kind == "batch":
        b = st["batch"]
        b.solve_equilibrium(st["opts"])
        b.solve_bias(st["volts"], st["opts"])
        return dict(psi=b.pack.psi, n=b.pack.n, p=b.pack.p)
    dev = st["dev"]
    if kind == "currents":
        return [dev.terminal_current(c) for c in dev.bcs]
    if kind == "assemble":
        dev.pack.assemble(_lib.MODE_ELIMINATE)
        return dict(F=dev.pack.F, J=dev.pack.J)
    if kind == "linear":
        x, _ = solve_linear(st["A"], st["b"], method=st["method"], rtol=1e-14, maxiter=4000,
                            restart=100, block_size=3)
        return x
    if kind == "equilibrium":
        dev.solve_equilibrium()
    elif kind == "sweep":
        dev.restore_state(st["start"])
        for v in st["volts"]:
            dev.solve_bias(v)
    else:
        dev.restore_state(st["start"])
        dev.bcs["anode"].V = 0.0
        dt = 2e-11
        res = solve_transient(dev, {"anode": RampWaveform(0.0, 0.5, 0.0, st["steps"] * dt)},
                              st["steps"] * dt, dt, theta=st["theta"], dt_max=dt)
        return dict(psi=dev.psi_gpu, n=dev.n_gpu, p=dev.p_gpu, times=res.times,
                    I=res.terminal_current["anode"])
    return dict(psi=dev.psi_gpu, n=dev.n_gpu, p=dev.p_gpu)


def work(case):
    """Bytes and flops of one pass that no method avoids: its inputs (state
    and coefficients: 16 doubles and a flag per node in 3D, 13 in 2D) read
    once and its outputs written once; a Newton solve's least is one
    linearisation written and read (its block system has 39 / 29 entries a
    node) and three state arrays."""
    if case["kind"] == "batch":
        rng = W.mosfet_batch_params(count=case["count"], seed=1000,
                                    nx=(case["nx_lo"], case["nx_hi"]),
                                    ny=(case["ny_lo"], case["ny_hi"]))
        n, d3 = sum(q["nx"] * q["ny"] for q in rng), False
    else:
        d3 = "nz" in case
        n = case["nx"] * case["ny"] * (case["nz"] if d3 else 1)
    ne, coef = (39, 16) if d3 else (29, 13)
    if case["kind"] == "currents":   # the edges at the contact nodes
        return {"bytes": 8.0 * 2 * case["ny"] * 24, "flops": 2.0 * case["ny"] * 300}
    if case["kind"] == "assemble":
        return {"bytes": n * (8.0 * (coef + 3 + ne) + 1), "flops": n * (300.0 if d3 else 200.0)}
    if case["kind"] == "equilibrium":
        return {"bytes": n * 8.0 * (coef + 2 * (7 if d3 else 5)), "flops": n * 100.0}
    if case["kind"] == "linear":
        return {"bytes": n * 12.0 * ne, "flops": 2.0 * n * ne}
    solves = case.get("points", case.get("steps", 2))
    return {"bytes": solves * n * 8.0 * (coef + 3 + 2 * ne), "flops": solves * n * 4.0 * ne}


# ---- the same in plain numpy, 64 bits -----------------------------------------
def _bern(x):
    """B(x) = x / (e^x - 1) and B'(x)."""
    x = np.clip(x, -700.0, 700.0)
    small = np.abs(x) < 1e-4
    xs = np.where(small, 1.0, x)
    b = np.where(small, 1 - x / 2 + x * x / 12, xs / np.expm1(xs))
    db = np.where(small, -0.5 + x / 6 - x ** 3 / 180, b * (1 / xs + 1 / np.expm1(-xs)))
    return b, db


def _on(s, name):
    mask = np.zeros(s.N, dtype=bool)
    for b in s.bcs.values():
        if b.kind == name:
            mask[b.nodes] = True
    return mask


def _contact_targets(s):
    """psi, n, p that the contacts hold (charge neutrality and mass action
    at the contact's bias)."""
    t = np.zeros((3, s.N))
    C, ns = s.C.ravel(), s.nie_s.ravel()
    for b in s.bcs.values():
        if b.kind != "contact":
            continue
        k = b.nodes
        root = np.sqrt(C[k] ** 2 + 4 * ns[k] ** 2)
        maj = 0.5 * (np.abs(C[k]) + root)
        mino = ns[k] ** 2 / maj
        t[1, k], t[2, k] = np.where(C[k] >= 0, maj, mino), np.where(C[k] >= 0, mino, maj)
        t[0, k] = b.V / s.VT + np.log(t[1, k] / ns[k])
    return t


def _gate_terms(s):
    """Robin coefficient and right-hand potential of every gate node."""
    gk, gr = np.zeros(s.N), np.zeros(s.N)
    bulk = s.bulk_guess().ravel()
    for b in s.bcs.values():
        if b.kind == "gate":
            kw = b.kappa * b.w
            np.add.at(gk, b.nodes, kw)
            np.add.at(gr, b.nodes, kw * ((b.Vg - b.Vfb) / s.VT + bulk[b.nodes]))
    return gk, gr


def _coupled(s, psi, n, p):
    """Coupled Scharfetter-Gummel residual [3][N] and Jacobian in the
    node-block layout [9 + 5 x 2 dim][N], contact rows and columns
    eliminated."""
    dim, shp = s.dim, s.shape
    psi, n, p = (np.asarray(a, float).reshape(shp) for a in (psi, n, p))
    dvs = [s.bcast(s.dv[a], a) * np.ones(shp) for a in range(dim)]
    dV = np.prod(dvs, axis=0)
    F = np.zeros((3,) + shp)
    J = np.zeros((9 + 10 * dim,) + shp)
    for a in range(dim):
        lo, hi = s.lo(a), s.hi(a)
        face = (dV / dvs[a])[lo]
        h = s.bcast(s.h[a], a)
        an, ap, dl = s.an[a][lo], s.ap[a][lo], s.dl[a][lo]
        d = psi[hi] - psi[lo]
        Bp, dBp = _bern(d + dl)
        Bm, dBm = _bern(-(d + dl))
        Hp, dHp = _bern(d - dl)
        Hm, dHm = _bern(-(d - dl))
        f = face * d / h
        Jn = face * an * (n[hi] * Bp - n[lo] * Bm)
        Jp = -face * ap * (p[hi] * Hm - p[lo] * Hp)
        g = face / h
        npsi = face * an * (n[hi] * dBp + n[lo] * dBm)
        ppsi = face * ap * (p[hi] * dHm + p[lo] * dHp)
        nlo, nhi = -face * an * Bm, face * an * Bp
        plo, phi = face * ap * Hp, -face * ap * Hm
        for r, q in enumerate((f, Jn, Jp)):
            F[r][lo] += q
            F[r][hi] -= q
        for end, sg, kn, kp, d0 in ((lo, 1.0, nlo, plo, 2 * a + 1), (hi, -1.0, nhi, phi, 2 * a)):
            J[0][end] -= g
            J[3][end] -= npsi
            J[6][end] -= ppsi
            J[4][end] += sg * kn
            J[8][end] += sg * kp
            e = 9 + 5 * d0
            J[e][end], J[e + 1][end], J[e + 3][end] = g, npsi, ppsi
            J[e + 2][end] = nhi if sg > 0 else -nlo
            J[e + 4][end] = phi if sg > 0 else -plo
    R, dRn, dRp = np.zeros(shp), np.zeros(shp), np.zeros(shp)
    if s.models.srh:
        nn, pp = n * s.Ns, p * s.Ns
        ex = nn * pp - s.nie ** 2
        den = s.tau_p * (nn + s.nie) + s.tau_n * (pp + s.nie)
        R = ex / den
        dRn = (pp * den - ex * s.tau_p) / den ** 2
        dRp = (nn * den - ex * s.tau_n) / den ** 2
        if s.models.auger:
            cc = s.mat.Cn_auger * nn + s.mat.Cp_auger * pp
            R = R + cc * ex
            dRn = dRn + s.mat.Cn_auger * ex + cc * pp
            dRp = dRp + s.mat.Cp_auger * ex + cc * nn
        R, dRn, dRp = R / s.R0, dRn * s.Ns / s.R0, dRp * s.Ns / s.R0
    gk, gr = (a.reshape(shp) for a in _gate_terms(s))
    F[0] += -dV * (n - p - s.C) + gr - gk * psi
    F[1] -= R * dV
    F[2] += R * dV
    J[0] -= gk
    J[1], J[2] = -dV, dV
    J[4] -= dRn * dV
    J[5] = -dRp * dV
    J[7] = dRn * dV
    J[8] += dRp * dV
    on = _on(s, "contact").reshape(shp)
    tgt = _contact_targets(s).reshape((3,) + shp)
    off = np.where(on, np.stack([psi, n, p]) - tgt, 0.0)
    for a in range(dim):
        for end, nbr, d0 in ((s.lo(a), s.hi(a), 2 * a + 1), (s.hi(a), s.lo(a), 2 * a)):
            e = 9 + 5 * d0
            F[0][end] -= J[e][end] * off[0][nbr]
            F[1][end] -= J[e + 1][end] * off[0][nbr] + J[e + 2][end] * off[1][nbr]
            F[2][end] -= J[e + 3][end] * off[0][nbr] + J[e + 4][end] * off[2][nbr]
            keep = ~on[nbr]
            for m in range(5):
                J[e + m][end] *= keep
    F[:, on] = off[:, on]
    J[:, on] = 0.0
    for e in (0, 4, 8):
        J[e][on] = 1.0
    return F.reshape(3, -1), J.reshape(9 + 10 * dim, -1)


_PAIRS = ((0, 0), (1, 0), (1, 1), (2, 0), (2, 2))


def _lines(s, a):
    """Node values [..][N] as [..][lines][nodes], the lines along the shorter
    side (the size of the direct solves' blocks)."""
    ny, nx = s.shape
    a = torch.from_numpy(np.ascontiguousarray(a).reshape(a.shape[:-1] + (ny, nx)))
    return a if nx <= ny else a.transpose(-1, -2).contiguous()


def _nodes(s, a):
    """The inverse of _lines."""
    ny, nx = s.shape
    return (a if nx <= ny else a.transpose(-1, -2)).reshape(a.shape[:-2] + (ny * nx,)).numpy()


def _line_blocks(s, J):
    """The 2D block system as block-tridiagonal over the lines: diagonal and
    the two coupling blocks of each line, unknowns 3 i + c along it."""
    J = _lines(s, J)
    if s.shape[1] > s.shape[0]:          # along a line is y: W, E <-> S, N
        J = torch.cat([J[:9], J[19:29], J[9:19]])
    m, q = J.shape[1:]
    i = torch.arange(q)
    D = torch.zeros(m, 3 * q, 3 * q, dtype=torch.float64)
    lo, up = torch.zeros_like(D), torch.zeros_like(D)
    for r in range(3):
        for c in range(3):
            D[:, 3 * i + r, 3 * i + c] = J[3 * r + c]
    for k, (r, c) in enumerate(_PAIRS):
        D[:, 3 * i[1:] + r, 3 * i[1:] - 3 + c] = J[9 + k][:, 1:]
        D[:, 3 * i[:-1] + r, 3 * i[:-1] + 3 + c] = J[14 + k][:, :-1]
        lo[:, 3 * i + r, 3 * i + c] = J[19 + k]
        up[:, 3 * i + r, 3 * i + c] = J[24 + k]
    return D, lo, up


def _line_solve(D, lo, up, b):
    """Block-tridiagonal LU (torch.linalg.solve per row), b [rows][m]."""
    m = len(b)
    G, y = [], []
    for j in range(m):
        Dj, bj = D[j], b[j]
        if j:
            Dj = Dj - lo[j] @ G[-1]
            bj = bj - lo[j] @ y[-1]
        sol = torch.linalg.solve(Dj, torch.cat([up[j], bj[:, None]], 1))
        G.append(sol[:, :-1])
        y.append(sol[:, -1])
    x = [y[-1]]
    for j in range(m - 2, -1, -1):
        x.append(y[j] - G[j] @ x[-1])
    return torch.stack(x[::-1])


def _exact_equilibrium(s):
    """2D equilibrium potential by Newton with direct solves."""
    saved = {n: (b.V if b.kind == "contact" else b.Vg) for n, b in s.bcs.items()}
    for b in s.bcs.values():
        if b.kind == "contact":
            b.V = 0.0
        else:
            b.Vg = 0.0
    tgt = _contact_targets(s)[0].reshape(s.shape)
    gk, gr = (a.reshape(s.shape) for a in _gate_terms(s))
    for n, b in s.bcs.items():
        if b.kind == "contact":
            b.V = saved[n]
        else:
            b.Vg = saved[n]
    on = _on(s, "contact").reshape(s.shape)
    dvx, dvy = s.dv[0][None, :], s.dv[1][:, None]
    dV = dvy * dvx
    gx, gy = dvy / s.h[0][None, :], dvx / s.h[1][:, None]
    psi = np.where(on, tgt, s.bulk_guess())
    for _ in range(60):
        n, p = s.nie_s * np.exp(psi), s.nie_s * np.exp(-psi)
        F = -dV * (n - p - s.C) + gr - gk * psi
        fx, fy = gx * np.diff(psi, axis=1), gy * np.diff(psi, axis=0)
        F[:, :-1] += fx
        F[:, 1:] -= fx
        F[:-1] += fy
        F[1:] -= fy
        dg = -dV * (n + p) - gk
        dg[:, :-1] -= gx
        dg[:, 1:] -= gx
        dg[:-1] -= gy
        dg[1:] -= gy
        F[on], dg[on] = 0.0, 1.0
        cx, cy = np.zeros(s.shape), np.zeros(s.shape)     # couplings to +x and +y
        cx[:, :-1] = gx * ~(on[:, 1:] | on[:, :-1])
        cy[:-1] = gy * ~(on[1:] | on[:-1])
        dl, along, across = _lines(s, np.stack([dg, cx, cy]).reshape(3, -1))
        if s.shape[1] > s.shape[0]:
            along, across = across, along
        D = torch.diag_embed(dl) + torch.diag_embed(along[:, :-1], 1) \
            + torch.diag_embed(along[:, :-1], -1)
        up = torch.diag_embed(across)
        d = _line_solve(D, torch.cat([up[-1:], up[:-1]]), up, _lines(s, -F.ravel()))
        d = _nodes(s, d).reshape(s.shape)
        d = np.clip(d, -5.0, 5.0)
        psi = psi + d
        if np.abs(d).max() < 1e-12:
            break
    return psi, s.nie_s * np.exp(psi), s.nie_s * np.exp(-psi)


def _exact_points(s, state, volts):
    """The sweep's last state by Newton with direct solves (2D)."""
    psi, n, p = (np.array(a, float).ravel() for a in state)
    on = _on(s, "contact")
    for v in volts:
        for name, val in v.items():
            s.bcs[name].V = float(val)
        tgt = _contact_targets(s)
        psi[on], n[on], p[on] = tgt[0][on], tgt[1][on], tgt[2][on]
        left = 3
        for _ in range(60):
            F, J = _coupled(s, psi, n, p)
            sc = np.stack([np.ones_like(n), n, p])          # unknowns: dpsi, dn/n, dp/p
            D, lo, up = _line_blocks(s, J)
            r, b = (_lines(s, a).permute(1, 2, 0).flatten(1) for a in (sc, -F))
            D, lo[1:], up[:-1] = D * r[:, None, :], lo[1:] * r[:-1, None, :], \
                up[:-1] * r[1:, None, :]
            w = 1.0 / D.abs().amax(2)                        # row scaling
            u = _line_solve(D * w[..., None], lo * w[..., None], up * w[..., None], b * w)
            u = _nodes(s, u.unflatten(1, (-1, 3)).permute(2, 0, 1)) * sc
            psi = psi + np.clip(u[0], -5.0, 5.0)
            n1 = np.clip(n + u[1], 0.1 * n, 10.0 * n)
            p1 = np.clip(p + u[2], 0.1 * p, 10.0 * p)
            err = max(np.abs(u[0]).max(), np.abs(n1 / n - 1).max(), np.abs(p1 / p - 1).max())
            n, p = n1, p1
            if err < 1e-6:
                left -= 1
                if left == 0:
                    break
    return psi, n, p


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch" or kind == "transient":
        return None                 # many devices, or many steps: over 20 s
    dev, volts = _device(case, seed)
    s = dev.setup
    nx, ny = s.nax[:2]
    if kind == "linear":
        return _linear_system(dev, seed)[2]
    if kind == "currents":
        psi, n, p = _biased_state(dev, seed)
        # the continuity residuals of the contact rows, as if they were free
        bcs, s.bcs = dict(s.bcs), {}
        F, _ = _coupled(s, psi, n, p)
        s.bcs = bcs
        f = F[1] + F[2]
        return [float(f[np.unique(b.nodes)].sum() * s.J0 * s.LD) for b in bcs.values()]
    if kind == "assemble":
        F, J = _coupled(s, *_biased_state(dev, seed))
        return dict(F=F.ravel(), J=J.ravel())
    if s.dim == 3 or kind == "sweep" and max(nx, ny) * min(nx, ny) ** 3 > 2.2e8:
        return None                 # a direct solve of it takes over 20 s
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        st = _exact_equilibrium(s)
        if kind == "sweep":
            st = _exact_points(s, st, volts)
    return dict(zip(("psi", "n", "p"), (np.asarray(a).ravel() for a in st)))
