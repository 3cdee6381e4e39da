"""Residuals of states with a value that is not finite, not physical or far out of
scale at one point.  Such a value has to reach the residual, as it does in the
reference: the points that become infinite or undefined are the oracle's, and no point
beside them turns into a number (a Van Leer flux is zero where its Mach number is
undefined, so a state that loses an infinity hides it)."""
import numpy as np
import pytest

from tests.helpers import interior
from tests.test_residual_lines import DQ, _case

pytestmark = pytest.mark.gpu

DIMS = (20, 12, 11)
POINTS = [(8, 8, 11), (3, 8, 5), (8, 3, 11), (8, 5, 3), (8, 2, 9)]  # k, j, i of the ghosted arrays
INF = float("inf")


def _pair(nscheme, nflux, nvis):
    from oracle.pyoracle import Oracle
    from wcns_b200.solver import Wcns
    case = _case(DIMS, nscheme, nflux)
    case.params.nvis = nvis
    g, o = Wcns(case), Oracle(case)
    g.boundary_all(); o.phase("boundary_all")
    g.initial_q_dq_c_t(); o.phase("initial_q_dq_c_t")
    return g, o


def _kinds(a):
    return np.where(np.isnan(a), 3, np.where(np.isposinf(a), 1, np.where(np.isneginf(a), 2, 0)))


def _compare(field, values, points, nscheme, nflux, nvis):
    g, o = _pair(nscheme, nflux, nvis)
    clean = {f: o.get(f, 1) for f in DQ}
    good = o.get(field, 1)
    for value in values:
        for point in points:
            a = good.copy()
            a[point] = value
            for h, get in ((g, g.get), (o, o.get)):
                h.set(field, 1, a)
                for f in DQ:
                    h.set(f, 1, clean[f])
            try:
                g.r_h_s_vis() if nvis else g.r_h_s_invis()
            except Exception as e:  # c^2 <= 0 is reported by both
                assert "c^2" in str(e) or "sound" in str(e) or "Roe" in str(e), e
                with pytest.raises(RuntimeError):
                    o.phase("rhs_invis")
                continue
            o.phase("rhs_vis" if nvis else "rhs_invis")
            for f in DQ:
                x, y = interior(g.get(f, 1), DIMS), interior(o.get(f, 1), DIMS)
                np.testing.assert_array_equal(_kinds(x), _kinds(y), err_msg=f"{f} {field} {value} {point}")
                ok = np.isfinite(y)
                assert np.max(np.abs(x[ok] - y[ok]), initial=0.0) <= 1e-10 * np.max(np.abs(y[ok]), initial=0.0), (f, field, value, point)


@pytest.mark.parametrize("field", ["u", "w"])
def test_viscous(field):
    _compare(field, (INF, -INF, float("nan"), 1e60), POINTS, 4, 1, 1)


@pytest.mark.parametrize("nflux", [1, 2, 3])
@pytest.mark.parametrize("nscheme", [4, 41, 42])
@pytest.mark.parametrize("field", ["r", "u", "p"])
def test_inviscid(field, nscheme, nflux):
    _compare(field, (INF, float("nan"), 1e30, 1e60), POINTS, nscheme, nflux, 0)


@pytest.mark.parametrize("form", ["clustered", "wide", "plane"])
@pytest.mark.parametrize("field,value", [("p", -1.0), ("p", 0.0), ("p", INF), ("p", float("nan")), ("r", -1.0), ("r", 0.0), ("r", INF), ("r", float("nan")),
                                         ("u", INF), ("u", float("nan")), ("dq1", INF), ("dq5", float("nan")), ("sra", INF)], ids=str)
def test_sweeps(field, value, form, monkeypatch):
    """A state that turned bad between the time step and the sweeps: what the sweeps
    hand on from there is undefined, whatever form they take."""
    from oracle.pyoracle import Oracle
    from tests.helpers import perturbed
    from wcns_b200 import cases
    from wcns_b200.solver import FLAG_SWEEP_BY_PLANE, FLAG_SWEEP_WIDE, Wcns, WcnsError
    if form == "clustered":
        monkeypatch.setenv("WCNS_SWEEP_CLUSTER", "4")
    dims = (13, 9, 8)
    for point in ((6, 6, 7), (4, 5, 5)):
        case = perturbed(cases.vortex_case(ni=13, nj=9, nk=8, nscheme=4, nflux=1))
        g, o = Wcns(case, flags={"clustered": 0, "wide": FLAG_SWEEP_WIDE, "plane": FLAG_SWEEP_BY_PLANE}[form]), Oracle(case)
        assert g.sweep_mode() == form
        for gp, op in [("boundary_all", "boundary_all"), ("initial_q_dq_c_t", "initial_q_dq_c_t"), ("timestep_tgh", "timestep"),
                       ("r_h_s_invis", "rhs_invis"), ("communicate_dq_npp", "communicate_dq")]:
            getattr(g, gp)()
            o.phase(op)
        a = o.get(field, 1)
        a[point] = value
        g.set(field, 1, a)
        o.set(field, 1, a)
        try:
            g.l_h_s_tgh()
        except WcnsError:
            with pytest.raises(RuntimeError):
                o.phase("lhs")
            continue
        o.phase("lhs")
        for f in DQ + ["r", "u", "v", "w", "p"]:
            x, y = interior(g.get(f, 1), dims), interior(o.get(f, 1), dims)
            np.testing.assert_array_equal(_kinds(x), _kinds(y), err_msg=f"{f} {point}")
            ok = np.isfinite(y)
            assert np.max(np.abs(x[ok] - y[ok]), initial=0.0) <= 1e-10 * np.max(np.abs(y[ok]), initial=0.0), (f, point)
