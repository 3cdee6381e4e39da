"""The viscous residual with every mixture of line ends: a line's end has a boundary
when its third ghost point has a negative density or, where that is positive, a
negative temperature, so the two ends of a line, and neighbouring lines, reach their
flag by different tests.  The flags are each thread's own reads: an exchange among the
lanes that happen to run together would be undefined after them.  The bar is the one of the phases: 1e-12 of a field's maximum
(a disturbed state whose residual has the size of the flux differences)."""
import os

import numpy as np
import pytest

from tests.helpers import compare_fields
from tests.test_residual_lines import DQ, _case


def test_no_exchange_among_whichever_lanes_run_together():
    from wcns_b200.build import CSRC
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            assert "__activemask" not in f.read(), name


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(12, 26, 9), (7, 33, 25), (65, 9, 17), (9, 64, 6)], ids=lambda d: "x".join(map(str, d)))
def test_mixed_ends(dims):
    from oracle.pyoracle import Oracle
    from wcns_b200.solver import Wcns
    case = _case(dims, 4, 1)
    case.params.nvis = 1
    g, o = Wcns(case), Oracle(case)
    g.boundary_all(); o.phase("boundary_all")
    g.initial_q_dq_c_t(); o.phase("initial_q_dq_c_t")
    r, t = (np.abs(o.get(f, 1)) for f in ("r", "t"))
    t = np.where(t > 0.0, t, 1.0)
    rng = np.random.default_rng(sum(dims))
    for axis in range(3):
        for end in (0, -1):  # the third ghost points of the two ends
            for f in (r, t):
                a = np.moveaxis(f, axis, 0)
                a[end] = a[end] * rng.choice([1.0, 1.0, -1.0], a[end].shape)
    for h in (g, o):
        h.set("r", 1, r)
        h.set("t", 1, t)
    g.r_h_s_vis(); o.phase("rhs_vis")
    errs = compare_fields(g, o, DQ)
    assert max(errs.values()) <= 1e-12, errs
