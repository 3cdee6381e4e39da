"""The residual's line kernels at the edges of their splits: the shortest lines
a direction takes (both ends' closures or boundary sections overlap), lines one
point longer or shorter than a warp or a thread block's pass, groups of lines
that fill a block partly, ends with and without boundary sections.

A state of order one with 20 % disturbances gives every component a residual of
the size of the flux differences, whose round-off is some ten roundings of
1e-16 of a flux; the bar is the one of the phases, 1e-12 of a field's maximum."""
import numpy as np
import pytest

from tests.helpers import compare_fields, supersonic_box_case
from wcns_b200 import cases

pytestmark = pytest.mark.gpu

DQ = ["dq1", "dq2", "dq3", "dq4", "dq5"]
DIMS = [(5, 6, 7), (7, 5, 8), (8, 9, 10), (12, 11, 5), (31, 8, 33), (10, 64, 6), (6, 13, 65), (71, 9, 11), (130, 7, 6), (9, 6, 257)]
# enough lines for the shortest chunks: lengths whose first chunk takes every remainder
LARGE = [(90 + q % 5, 96 + q, 92 + q % 3) for q in range(8)]
INVISCID = [(d, s, f) for d in DIMS for s in (4, 41, 42) for f in (1, 2, 3)] + \
    [(d, (4, 41, 42)[q % 3], (3, 2, 1)[q % 3 if q < 3 else 0]) for q, d in enumerate(LARGE)] + [(d, 41, 3) for d in LARGE]


def _case(dims, nscheme, nflux):
    """Box with far field (boundary sections) at both j faces, none at the
    others, and a disturbance without symmetry in all five variables."""
    case = supersonic_box_case(*dims, nscheme=nscheme, nflux=nflux)
    r, u, v, w, p, t = case.prim[0]
    rng = np.random.default_rng(dims[0] * 1000 + dims[1] * 10 + dims[2])
    k, j, i = np.meshgrid(*(np.linspace(0.0, 1.0, d) for d in dims[::-1]), indexing="ij")
    for f, amp in ((r, 0.2), (u, 0.2), (v, 0.3), (w, 0.3), (p, 0.1)):
        a, b, c = rng.uniform(2.0, 5.0, 3)
        x = cases.interior(f, dims)
        x[...] = x + amp * (np.sin(a * i + b * j + c * k) * (1.0 if f is not p else x))
    return case


@pytest.mark.parametrize("dims,nscheme,nflux", INVISCID, ids=str)
def test_inviscid_lines(dims, nscheme, nflux):
    from oracle.pyoracle import Oracle
    from wcns_b200.solver import Wcns
    case = _case(dims, nscheme, nflux)
    g, o = Wcns(case), Oracle(case)
    g.boundary_all(); o.phase("boundary_all")
    g.initial_q_dq_c_t(); o.phase("initial_q_dq_c_t")
    g.r_h_s_invis(); o.phase("rhs_invis")
    errs = compare_fields(g, o, DQ)
    assert max(errs.values()) <= 1e-12, errs


@pytest.mark.parametrize("dims", DIMS + LARGE + [(4, 6, 7), (9, 5, 3), (6, 4, 5)], ids=lambda d: "x".join(map(str, d)))
def test_viscous_lines(dims):
    from oracle.pyoracle import Oracle
    from wcns_b200.solver import Wcns
    case = _case(dims, 4, 1)
    case.params.nvis = 1
    g, o = Wcns(case), Oracle(case)
    g.boundary_all(); o.phase("boundary_all")
    g.initial_q_dq_c_t(); o.phase("initial_q_dq_c_t")
    g.r_h_s_vis(); o.phase("rhs_vis")
    errs = compare_fields(g, o, DQ)
    assert max(errs.values()) <= 1e-12, errs
