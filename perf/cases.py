"""Performance cases of the WCNS path, through the public Python mirror of the
C ABI (wcns_b200.solver.Wcns).

Kinds of work, each what a program that drives the library does:

  steps     advance a state that is on the device by a few whole time steps
            (wcns_step, the CUDA-graph path) and hand the new state on.  Every
            pass starts from the same saved state, which the program copies
            into the context's fields on the device, as a coupled or a
            parametric run does.
  restart   the flow-file way: the interior state comes from pinned host
            memory (wcns_set_interior), steps, and goes back
            (wcns_get_interior) with the residual norms of every block.
  phases    one step driven phase by phase under the reference's subroutine
            names, as a Fortran time loop bound to the C ABI runs it.
  residual  the inviscid residual alone (initial_q_dq_c_t, r_h_s_invis), as a
            solver with its own time integration uses it, FP64 or mixed.
  adjoint   the linear operators of the discrete adjoint at a state: tangent,
            adjoint, and the LU-SGS pair both ways, on device vectors.

Workloads are the seeded generators of wcns_b200.cases: the isentropic vortex,
the laminar flat plate, the SA channel with a wall bump, and the batch of
independent bump cases.  The grids depend on the case alone; the flow states
(a smooth disturbance plus short waves) on the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from wcns_b200 import cases as workloads
from wcns_b200.solver import Wcns

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest call: one step of a small vortex block, as an
        # interactive or unit-sized run makes it; launches and host work count
        dict(name="vortex_one_step", kind="steps", flow="vortex", ni=33, nj=17, nk=9, nscheme=42, nflux=2, steps=1,
             bits=64, tune=False),
        # a small multi-block laminar case, stepped and monitored: residual
        # norms of every block and the wall forces after the step
        dict(name="plate_monitor", kind="steps", flow="plate", a=9, e=7, h1=11, h2=7, hc=7, nk=7, nscheme=41, nflux=3,
             steps=1, bits=64, tune=False, monitor=True),
        # the vortex configuration of the benchmark set, ten steps per call
        dict(name="vortex_ten_steps", kind="steps", flow="vortex", ni=65, nj=33, nk=17, nscheme=4, nflux=1, steps=10,
             bits=64, tune=False),
        # the laminar plate configuration (8 blocks, 228,888 points)
        dict(name="plate_steps", kind="steps", flow="plate", a=65, e=33, h1=65, h2=33, hc=49, nk=9, nscheme=41,
             nflux=3, steps=5, bits=64, tune=False),
        # the SA channel configuration (24 blocks, 4.16 M points), the flagship
        dict(name="channel_steps", kind="steps", flow="channel", ni=385, nj=129, nk=81, bx=6, by=2, bz=2, nscheme=41,
             nflux=3, steps=2, bits=64, tune=False),
        # the channel at a middle, ragged size in mixed precision, tuned
        dict(name="channel_mixed", kind="steps", flow="channel", ni=211, nj=103, nk=59, bx=5, by=2, bz=2, nscheme=41,
             nflux=3, steps=3, bits=32, tune=True),
        # the 64-case batch (one block each, SA), FP64, tuned
        dict(name="batch64_steps", kind="steps", flow="batch", ncases=64, grid_seed=0, steps=3, bits=64, tune=True),
        # restart from host memory, one step, state and residual back
        dict(name="channel_restart", kind="restart", flow="channel", ni=150, nj=87, nk=45, bx=3, by=2, bz=1,
             nscheme=41, nflux=3, steps=1, bits=64, tune=False),
        # the phases called one by one on a plate of odd sizes
        dict(name="plate_phases", kind="phases", flow="plate", a=41, e=23, h1=47, h2=27, hc=31, nk=13, nscheme=41,
             nflux=2, steps=1, bits=64, tune=False),
        # the inviscid residual alone, ragged block, Roe
        dict(name="residual_fp64", kind="residual", flow="vortex", ni=121, nj=75, nk=51, nscheme=4, nflux=3, bits=64),
        # the same kernel family in mixed precision
        dict(name="residual_mixed", kind="residual", flow="vortex", ni=121, nj=75, nk=51, nscheme=4, nflux=1, bits=32),
        # the adjoint's operators on the vortex configuration
        dict(name="adjoint_operators", kind="adjoint", flow="vortex", ni=65, nj=33, nk=17, nscheme=4, nflux=3,
             bits=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 5 + ["restart", "phases", "residual", "residual", "adjoint"])
    bits = 32 if kind != "adjoint" and rng.random() < 0.3 else 64
    scheme = dict(nscheme=rng.choice([4, 41, 42]), nflux=rng.choice([1, 2, 3]), bits=bits)
    if kind in ("residual", "adjoint"):
        top = 129 if kind == "residual" else 81
        return dict(scheme, kind=kind, flow="vortex", ni=_log(rng, 17, top), nj=_log(rng, 11, top * 2 // 3),
                    nk=_log(rng, 9, top // 2), nscheme=4, nflux=rng.choice([1, 3]))
    scheme.update(kind=kind, steps=1 if kind != "steps" else rng.choice([1, 2, 4]), tune=rng.random() < 0.4)
    flow = rng.choice(["vortex", "plate", "channel", "channel", "batch"] if kind == "steps" else
                      ["vortex", "plate", "channel"])
    if flow == "vortex":
        return dict(scheme, flow=flow, ni=_log(rng, 17, 161), nj=_log(rng, 13, 97), nk=_log(rng, 9, 65))
    if flow == "plate":
        return dict(scheme, flow=flow, a=_log(rng, 9, 73), e=_log(rng, 7, 41), h1=_log(rng, 11, 73),
                    h2=_log(rng, 7, 41), hc=_log(rng, 7, 53), nk=_log(rng, 7, 17), monitor=rng.random() < 0.5)
    if flow == "batch":
        return dict(kind=kind, flow=flow, ncases=_log(rng, 4, 64), grid_seed=rng.randrange(1000),
                    steps=scheme["steps"], bits=bits, tune=scheme["tune"])
    bx, by, bz = rng.choice([(2, 2, 1), (3, 2, 1), (4, 2, 2), (5, 2, 2)])
    if kind == "restart":
        bx, by, bz = rng.choice([(2, 2, 1), (3, 2, 1)])
    return dict(scheme, flow=flow, ni=_log(rng, 12 * bx, 230), nj=_log(rng, 12 * by, 115), nk=_log(rng, 12 * bz, 75),
                bx=bx, by=by, bz=bz)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _workload(case):
    f = case["flow"]
    if f == "vortex":
        return workloads.vortex_case(ni=case["ni"], nj=case["nj"], nk=case["nk"], nscheme=case["nscheme"],
                                     nflux=case["nflux"], noise=0.0)
    if f == "plate":
        keys = ("a", "e", "h1", "h2", "hc", "nk", "nscheme", "nflux")
        first = 1.0e-5 if case["h1"] >= 33 else 1.0e-3
        return workloads.plate_case(first=first, **{k: case[k] for k in keys})
    if f == "channel":
        keys = ("ni", "nj", "nk", "bx", "by", "bz", "nscheme", "nflux")
        first = 2.0e-6 if case["nj"] >= 97 else 1.0e-4 if case["nj"] >= 49 else 1.0e-3
        return workloads.channel_case(first=first, **{k: case[k] for k in keys})
    return workloads.batch_case(ncases=case["ncases"], seed=case["grid_seed"])


def _disturb(w, seed):
    """A smooth density and pressure disturbance and a little short-wave noise
    on every block's interior, in place, from the seed.  Both are functions of
    the coordinates, so that the copies of an interface point agree, as they
    do in any state that the solver has stepped."""
    rng = np.random.default_rng(seed)
    ax, ay, az = rng.uniform(1.0, 3.0, 3)
    px, py, pz = rng.uniform(0.0, 2.0 * math.pi, 3)
    amp = rng.uniform(0.01, 0.03)
    bx, by, bz = rng.uniform(50.0, 500.0, 3)
    for (ni, nj, nk), (x, y, z), prim in zip(w.dims, w.xyz, w.prim):
        s = amp * np.sin(ax * x + px) * np.cos(ay * y + py) * np.cos(az * z + pz)
        s += 1.0e-6 * np.sin(bx * x + by * y + bz * z)
        for a, c in ((prim[0], 1.0), (prim[4], 1.4)):
            a[3:3 + nk, 3:3 + nj, 3:3 + ni] *= 1.0 + c * s


def _field(g, name):
    return [torch.as_tensor(g.device_view(name, nb), device="cuda") for nb in range(1, len(g.dims) + 1)]


def _state_names(w):
    return ["r", "u", "v", "w", "p"] + (["t"] if w.params.nvis else []) + (["qke", "vist"] if w.sa else [])


def prepare(case, seed):
    if case["kind"] in ("residual", "adjoint"):
        return _prepare_block(case, seed)
    w = _workload(case)
    _disturb(w, seed)
    g = Wcns(w)
    if w.sa:
        g.sa_setup(w.sa["timedt_turb"], w.sa["kmaxlim"])
    if case["bits"] == 32:
        g.set_precision(32)
    names = _state_names(w)
    views = [v for n in names for v in _field(g, n)]
    g.sync()
    saved = [v.clone() for v in views]
    s = dict(case=case, g=g, names=names, views=views, saved=saved)
    if case["tune"]:
        # on a stepped state, as the tuner times the phases on live fields
        g.step(1)
        g.autotune(3)
        torch._foreach_copy_(views, saved)
        torch.cuda.current_stream().synchronize()
    if case["kind"] == "restart":
        pin = [[torch.empty((nk, nj, ni), dtype=torch.float64, pin_memory=True).numpy() for _ in names]
               for ni, nj, nk in g.dims]
        out = [[torch.empty((nk, nj, ni), dtype=torch.float64, pin_memory=True).numpy() for _ in names]
               for ni, nj, nk in g.dims]
        g.get_interior(names, pin)
        s.update(host_in=pin, host_out=out)
    return s


def _prepare_block(case, seed):
    """One Cartesian block whose ghosted state is smooth everywhere, and for
    the adjoint a direction and a weight vector."""
    w = _workload(case)
    ni, nj, nk = w.dims[0]
    rng = np.random.default_rng(seed)
    w.prim = [tuple(_smooth_state(case, rng)) + (np.ones((nk + 6, nj + 6, ni + 6)),)]
    g = Wcns(w)
    if case["bits"] == 32:
        g.set_precision(32)
    s = dict(case=case, g=g, views=[_field(g, f"dq{m}")[0] for m in range(1, 6)])
    if case["kind"] == "adjoint":
        g.timestep_tgh()
        for slot in ("v", "lam", "b"):
            g.adj_set(slot, 1, _vector(case, rng))
    return s


def _smooth_state(case, rng):
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    z, y, x = np.meshgrid(np.arange(-2, nk + 4) / nk, np.arange(-2, nj + 4) / nj, np.arange(-2, ni + 4) / ni,
                          indexing="ij")
    p0 = 1.0 / (1.4 * 0.25)
    out = []
    for mean, amp in ((1.0, 0.2), (1.0, 0.3), (0.0, 0.3), (0.0, 0.2), (p0, 0.2 * p0)):
        a, b, c = rng.integers(1, 4, 3)
        f, h, e = rng.uniform(0.0, 2.0 * math.pi, 3)
        out.append(mean + amp * np.sin(2 * math.pi * a * x + f) * np.cos(2 * math.pi * b * y + h) *
                   np.cos(2 * math.pi * c * z + e) + rng.uniform(-1e-3, 1e-3, x.shape) * amp)
    return out


def _vector(case, rng):
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    out = []
    for _ in range(5):
        a = np.zeros((nk + 6, nj + 6, ni + 6))
        a[3:-3, 3:-3, 3:-3] = rng.standard_normal((nk, nj, ni))
        out.append(a)
    return out


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _taken(names, views, nb):
    """The program's own copy of fields, one tensor each over the blocks, the
    form in which a coupled program takes them: the views alias the context's
    memory, which the next call overwrites, so the copies are complete before
    anything else is asked of the context."""
    out = {n: torch.cat([a.view(-1) for a in views[q * nb:(q + 1) * nb]]) for q, n in enumerate(names)}
    torch.cuda.current_stream().synchronize()
    return out


def _new_state(s):
    return _taken(s["names"], s["views"], len(s["g"].dims))


def run(s):
    case, g = s["case"], s["g"]
    kind = case["kind"]
    if kind == "residual":
        g.initial_q_dq_c_t()
        g.r_h_s_invis()
        return _taken([f"dq{m}" for m in range(1, 6)], s["views"], 1)
    if kind == "adjoint":
        g.rhs_invis_tangent()
        g.rhs_invis_adjoint(fold=True)
        g.lusgs_operator(transpose=False)
        x = g.adj_get("x", 1)
        g.lusgs_operator(transpose=True)
        return dict(rdot=g.adj_get("rdot", 1), qbar=g.adj_get("qbar", 1), x=x, xt=g.adj_get("x", 1))
    if kind == "restart":
        g.set_interior(s["names"], s["host_in"])
        g.step(case["steps"], history=False)
        g.get_interior(s["names"], s["host_out"])
        res, rmax, rms = g.residual_curve()
        return dict(state=s["host_out"], res=res, rmax=rmax, rms=rms)
    torch._foreach_copy_(s["views"], s["saved"])
    torch.cuda.current_stream().synchronize()
    if kind == "steps":
        hist = g.step(case["steps"])
        out = dict(state=_new_state(s), history=hist)
        if case.get("monitor"):
            res, rmax, rms = g.residual_curve()
            out.update(res=res, rmax=rmax, rms=rms, forces=np.array([v for k, v in g.force().items() if k != "xcp"]))
        return out
    for _ in range(case["steps"]):
        g.boundary_all()
        g.initial_q_dq_c_t()
        g.timestep_tgh()
        if g.case.params.nvis:
            g.r_h_s_vis()
            g.communicate_dq_npp()
        g.r_h_s_invis()
        g.communicate_dq_npp()
        g.l_h_s_tgh()
        g.communicate_pv_npp()
    res, rmax, rms = g.residual_curve()
    return dict(state=_new_state(s), res=res, rmax=rmax, rms=rms)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _points(case):
    f = case["flow"]
    if f == "batch":
        rng = np.random.default_rng(case["grid_seed"])  # the draws of batch_case
        n = 0
        for _ in range(case["ncases"]):
            ni, nj = int(rng.integers(17, 50)), int(rng.integers(17, 34))
            rng.uniform(0.3, 0.8), rng.uniform(0.02, 0.08)
            n += ni * nj * 17
        return n
    if f == "plate":
        na, nb = 2 * case["a"] - 1, 3 * case["e"] - 2
        return case["nk"] * ((na + nb) * case["h1"] + case["a"] * case["hc"] + 2 * case["a"] * case["h2"] +
                             3 * case["e"] * case["h2"])
    if f == "channel":  # interface points are on both blocks
        return math.prod(case[n] + case[b] - 1 for n, b in (("ni", "bx"), ("nj", "by"), ("nk", "bz")))
    return case["ni"] * case["nj"] * case["nk"]


def work(case):
    """Per point and step: the state read and written (5 words, T for viscous
    flow, qke and vist with the SA model), the nine metrics and the volume,
    the wall distance; operations counted from the scheme's formulas with the
    weights at one division per side (inviscid 700 per direction, viscous 330,
    a sweep 150, the SA model 400, the rest 250)."""
    n = _points(case)
    if case["kind"] == "residual":
        return {"bytes": 8.0 * n * (5 + 9 + 5), "flops": 2100.0 * n}
    if case["kind"] == "adjoint":
        # tangent and adjoint: state, metrics, one vector in and one out each;
        # the LU-SGS operator and its transpose: state, metrics, radii and
        # time step, a vector in and one out each
        return {"bytes": 8.0 * n * (2 * (5 + 9 + 10) + 2 * (5 + 9 + 4 + 10)), "flops": n * (2 * 4200.0 + 4 * 150.0)}
    visc = case["flow"] != "vortex"
    sa = case["flow"] in ("channel", "batch")
    state = 5 + (1 if visc else 0) + (2 if sa else 0)
    words = 2 * state + 10 + (1 if sa else 0)
    flops = 2100.0 + 600.0 + 250.0 + (990.0 if visc else 0.0) + (400.0 if sa else 0.0)
    return {"bytes": 8.0 * n * words * case["steps"], "flops": flops * n * case["steps"]}


# ---------------------------------------------------------------------------
# 64-bit values of the block kinds (uniform Cartesian metrics, nscheme 4, all
# ghosts valid: every line runs the interior scheme), from the formulas
# ---------------------------------------------------------------------------

_G = 1.4


def _exact_flux(nflux, ql, qr, k, efix=0.1):
    nx = [torch.as_tensor(v, dtype=torch.float64) for v in k]
    kk = math.sqrt(sum(v * v for v in k))

    def euler(q):
        r, u, v, w, p = q
        c = nx[0] * u + nx[1] * v + nx[2] * w
        e = p / (_G - 1.0) + 0.5 * r * (u * u + v * v + w * w)
        return [r * c, r * c * u + nx[0] * p, r * c * v + nx[1] * p, r * c * w + nx[2] * p, (e + p) * c]

    def split(q, sign):  # Steger-Warming
        r, u, v, w, p = q
        c = torch.sqrt(_G * p / r)
        th = nx[0] * u + nx[1] * v + nx[2] * w
        lam = [th, th + c * kk, th - c * kk]
        l1, l4, l5 = (0.5 * (x + sign * torch.sqrt(x * x + (efix * kk) ** 2)) for x in lam)
        x1 = (2.0 * l1 - l4 - l5) / (2.0 * _G)
        x2 = c * (l4 - l5) / (2.0 * _G)
        n = [v / kk for v in nx]
        em = p / ((_G - 1.0) * r) + 0.5 * (u * u + v * v + w * w)
        hm = em + p / r
        return [r * (l1 - x1), r * (l1 * u - x1 * u + n[0] * x2), r * (l1 * v - x1 * v + n[1] * x2),
                r * (l1 * w - x1 * w + n[2] * x2), r * (l1 * em - x1 * hm + th / kk * x2)]

    if nflux == 1:
        return [a + b for a, b in zip(split(ql, 1.0), split(qr, -1.0))]
    fl, fr = euler(ql), euler(qr)
    d = [b - a for a, b in zip(ql, qr)]

    def enthalpy(q):
        return _G / (_G - 1.0) * q[4] / q[0] + 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)

    rho = torch.sqrt(ql[0] * qr[0])
    s = torch.sqrt(qr[0] / ql[0])
    u, v, w = ((ql[m] + qr[m] * s) / (1.0 + s) for m in (1, 2, 3))
    h = (enthalpy(ql) + enthalpy(qr) * s) / (1.0 + s)
    c2 = (h - 0.5 * (u * u + v * v + w * w)) * (_G - 1.0)
    c = torch.sqrt(c2)
    th = u * nx[0] + v * nx[1] + w * nx[2]
    l1, l4, l5 = (torch.sqrt(x * x + (efix * kk) ** 2) for x in (th - c * kk, th, th + c * kk))
    n = [x / kk for x in nx]
    dth = rho * (d[1] * n[0] + d[2] * n[1] + d[3] * n[2])
    a1 = l4 * (d[0] - d[4] / c2)
    a2 = 0.5 * l5 * (d[4] / c2 + dth / c)
    a3 = 0.5 * l1 * (d[4] / c2 - dth / c)
    a4, a5 = a1 + a2 + a3, c * (a2 - a3)
    a6, a7, a8 = (l4 * (rho * d[m + 1] - n[m] * dth) for m in range(3))
    df = [a4, u * a4 + n[0] * a5 + a6, v * a4 + n[1] * a5 + a7, w * a4 + n[2] * a5 + a8,
          h * a4 + th / kk * a5 + u * a6 + v * a7 + w * a8 - c2 * a1 / (_G - 1.0)]
    return [0.5 * (a + b - x) for a, b, x in zip(fl, fr, df)]


def _exact_line(q, nflux, k):
    """The flux difference along the last axis (ghosts included: n + 6)."""
    n = q[0].shape[-1] - 6

    def sl(a, first, count):  # points first .. first+count-1 (1-based, ghosts from -2)
        return a[..., first + 2:first + 2 + count]

    ql, qr = [], []
    for a in q:
        m2, m1, c0, p1, p2 = (sl(a, o, n + 2) for o in (-2, -1, 0, 1, 2))  # centres i = 0 .. n+1
        g = (0.5 * (m2 - 4.0 * m1 + 3.0 * c0), 0.5 * (p1 - m1), 0.5 * (-3.0 * c0 + 4.0 * p1 - p2))
        s = (m2 - 2.0 * m1 + c0, m1 - 2.0 * c0 + p1, c0 - 2.0 * p1 + p2)
        e = [(1.0e-6 + gg * gg + ss * ss) ** 2 for gg, ss in zip(g, s)]
        side = []
        for cs, sign in (((1.0, 10.0, 5.0), 1.0), ((5.0, 10.0, 1.0), -1.0)):
            b = [ck / ek for ck, ek in zip(cs, e)]
            t = b[0] + b[1] + b[2]
            side.append(c0 + 0.125 * sum(bk / t * (ss + sign * 4.0 * gg) for bk, gg, ss in zip(b, g, s)))
        ql.append(side[0][..., :-1])  # half nodes 0 .. n
        qr.append(side[1][..., 1:])
    out = []
    for f in _exact_flux(nflux, ql, qr, k):
        inner = (2250.0 * (f[..., 3:n - 1] - f[..., 2:n - 2]) - 125.0 * (f[..., 4:n] - f[..., 1:n - 3]) +
                 9.0 * (f[..., 5:n + 1] - f[..., 0:n - 4])) / 1920.0
        d1 = (-23.0 * f[..., 0:1] + 21.0 * f[..., 1:2] + 3.0 * f[..., 2:3] - f[..., 3:4]) / 24.0
        d2 = (f[..., 0:1] - 27.0 * f[..., 1:2] + 27.0 * f[..., 2:3] - f[..., 3:4]) / 24.0
        e1 = -(-23.0 * f[..., n:n + 1] + 21.0 * f[..., n - 1:n] + 3.0 * f[..., n - 2:n - 1] - f[..., n - 3:n - 2]) / 24.0
        e2 = -(f[..., n:n + 1] - 27.0 * f[..., n - 1:n] + 27.0 * f[..., n - 2:n - 1] - f[..., n - 3:n - 2]) / 24.0
        out.append(torch.cat([d1, d2, inner, e2, e1], dim=-1))
    return out


def _exact_residual(case, q):
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    dx, dy, dz = 10.0 / (ni - 1), 5.0 / (nj - 1), 2.5 / (nk - 1)
    inside = slice(3, -3)
    total = None
    for axis, k in ((2, (dy * dz, 0.0, 0.0)), (1, (0.0, dx * dz, 0.0)), (0, (0.0, 0.0, dx * dy))):
        cut = tuple(slice(None) if a == axis else inside for a in range(3))
        d = [f.movedim(-1, axis) for f in _exact_line([a[cut].movedim(axis, -1) for a in q], case["nflux"], k)]
        total = d if total is None else [a + b for a, b in zip(total, d)]
    return [torch.nn.functional.pad(a, (3,) * 6) for a in total]


def exact(case, seed):
    if case["kind"] not in ("residual", "adjoint"):
        return None
    rng = np.random.default_rng(seed)
    q = [torch.from_numpy(a).cuda() for a in _smooth_state(case, rng)]
    if case["kind"] == "residual":
        return {f"dq{m + 1}": a.reshape(-1) for m, a in enumerate(_exact_residual(case, q))}
    v, lam = ([torch.from_numpy(a).cuda() for a in _vector(case, rng)] for _ in range(2))
    rdot = torch.func.jvp(lambda *a: tuple(_exact_residual(case, list(a))), tuple(q), tuple(v))[1]
    for a in q:
        a.requires_grad_(True)
    res = _exact_residual(case, q)
    bar = list(torch.autograd.grad(res, q, lam))
    # interface ghosts of the periodic directions (i and k) are copies of the
    # points on the other side: their adjoint moves there.  A ghost is filled
    # over a whole face, edges excluded
    out = []
    ins = slice(3, -3)
    for b in bar:
        b = b.detach().clone()
        for axis in (2, 0):
            n = b.shape[axis] - 6
            for layer in (1, 2, 3):
                for ghost, point in ((1 - layer, n - layer), (n + layer, 1 + layer)):
                    g = tuple(ghost + 2 if a == axis else ins for a in range(3))
                    p = tuple(point + 2 if a == axis else ins for a in range(3))
                    b[p] += b[g]
                    b[g] = 0.0
        out.append(b)
    five = [None] * 5
    return dict(rdot=[a.cpu() for a in rdot], qbar=[a.cpu() for a in out], x=five, xt=five)
