"""The LU-SGS operator and its transpose at the edges of their forms: columns that
fill a cluster exactly and one row more (which goes plane by plane), a block of one
warp, blocks short in one direction.

P b is compared with a restatement plane by plane: sums of three products of O(1)
matrices along at most i+j+k planes, whose coefficients damp a disturbance, so the
round-off stays a few hundred roundings of 1e-16 of the field's maximum (bar 1e-12);
P^T y through <y, P b> = <P^T y, b> at the same bar."""
import numpy as np
import pytest

from tests.helpers import interior
from wcns_b200 import cases

pytestmark = pytest.mark.gpu


def _term(prim, nvec, rad, npn, dq):
    """mxdq_std (LHS.f90:756-828) for arrays of points."""
    rm, um, vm, wm, pm = prim
    g = 1.4
    c2 = g * pm / rm
    cm, v2 = np.sqrt(c2), um * um + vm * vm + wm * wm
    hm = g / (g - 1.0) * pm / rm + 0.5 * v2
    ct = nvec[0] * um + nvec[1] * vm + nvec[2] * wm
    cgm = np.maximum(np.sqrt(nvec[0] ** 2 + nvec[1] ** 2 + nvec[2] ** 2), 1e-30)
    l1, l4, l5 = 0.5 * (ct + npn * rad), 0.5 * (ct + cm * cgm + npn * rad), 0.5 * (ct - cm * cgm + npn * rad)
    x1, x2 = (2.0 * l1 - l4 - l5) / (2.0 * c2), (l4 - l5) / (2.0 * cm)
    nx, ny, nz, ct = nvec[0] / cgm, nvec[1] / cgm, nvec[2] / cgm, ct / cgm
    ae = g - 1.0
    dc = ct * dq[0] - nx * dq[1] - ny * dq[2] - nz * dq[3]
    dh = 0.5 * ae * v2 * dq[0] - ae * (um * dq[1] + vm * dq[2] + wm * dq[3] - dq[4])
    a, b = c2 * dc * x1 + dh * x2, dh * x1 + dc * x2
    return np.stack([l1 * dq[0] - b, l1 * dq[1] + nx * a - um * b, l1 * dq[2] + ny * a - vm * b,
                     l1 * dq[3] + nz * a - wm * b, l1 * dq[4] + ct * a - hm * b])


def _operator(g, dims, b):
    I = lambda f: interior(g.get(f, 1), dims)  # noqa: E731
    prim = np.stack([I(f) for f in ("r", "u", "v", "w", "p")])
    met = [np.stack([I(f) for f in n]) for n in (("kcx", "kcy", "kcz"), ("etx", "ety", "etz"), ("ctx", "cty", "ctz"))]
    rad = [I(f) for f in ("sra", "srb", "src")]
    coed = 1.0 / (1.0 / I("dtdt") + rad[0] + rad[1] + rad[2])
    ni, nj, nk = dims
    k, j, i = np.meshgrid(np.arange(nk), np.arange(nj), np.arange(ni), indexing="ij")
    planes = [np.nonzero(i + j + k == p) for p in range(ni + nj + nk - 2)]
    x = np.zeros_like(b)
    for lower in (True, False):
        for pk, pj, pi in planes if lower else planes[::-1]:
            acc = np.zeros((5, pk.size))
            for d in range(3):
                q = [pk.copy(), pj.copy(), pi.copy()]
                q[2 - d] += -1 if lower else 1
                ok = q[2 - d] >= 0 if lower else q[2 - d] < (nk, nj, ni)[2 - d]
                at = tuple(v[ok] for v in q)
                sel = (slice(None),) + at
                acc[:, ok] += _term(prim[sel], met[d][sel], rad[d][at], 1.0 if lower else -1.0, x[sel])
            at = (slice(None), pk, pj, pi)
            x[at] = (-b[at] + acc) * coed[pk, pj, pi] if lower else x[at] - acc * coed[pk, pj, pi]
    return x


@pytest.mark.parametrize("dims", [(9, 5, 6), (6, 33, 8), (7, 5, 129), (40, 16, 17), (6, 64, 64), (5, 65, 64)], ids=lambda d: "x".join(map(str, d)))
def test_operator_and_transpose(dims):
    from wcns_b200.solver import Wcns
    ni, nj, nk = dims
    g = Wcns(cases.vortex_case(ni=ni, nj=nj, nk=nk, nscheme=4, nflux=1, nsteps=1))
    g.boundary_all()
    g.initial_q_dq_c_t()
    g.timestep_tgh()
    rng = np.random.default_rng(ni + nj)
    vec = []
    for _ in range(2):
        v = np.zeros((5, nk + 6, nj + 6, ni + 6))
        v[:, 3:-3, 3:-3, 3:-3] = rng.uniform(-1.0, 1.0, (5, nk, nj, ni))
        vec.append(v)
    out = []
    for t in range(2):
        g.adj_set("b", 1, list(vec[t]))
        g.lusgs_operator(transpose=bool(t))
        out.append(np.stack([interior(a, dims) for a in g.adj_get("x", 1)]))
    b, y = (v[:, 3:-3, 3:-3, 3:-3] for v in vec)
    x = _operator(g, dims, b)
    assert np.max(np.abs(out[0] - x)) <= 1e-12 * np.max(np.abs(x))
    assert abs(np.vdot(y, out[0]) - np.vdot(out[1], b)) <= 1e-12 * np.linalg.norm(y) * np.linalg.norm(out[0])
