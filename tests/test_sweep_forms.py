"""The wide sweeps at the edges of their splits: chunk widths that fill a warp
exactly or by one column more, chunks of one row (every j term crosses a
ring), several chunks per CTA (folding), fewer and more staged planes, and rows
longer than the usual CTA.

Every form and split evaluates a cell with the same operations in the same
order (csrc/wcns_sweep.cuh), so the states agree bit for bit with the
clustered sweeps wherever those can run; rows too long for them are compared
with the oracle at the parity bar of the phases (1e-12 of a field's maximum:
a sweep's terms are sums of a few products whose round-off is 1e-15 of their
size, and the disturbed state gives every component a dq of its own)."""
import numpy as np
import pytest

from tests.helpers import compare_fields, perturbed
from wcns_b200 import cases

pytestmark = pytest.mark.gpu

STATE = ("r", "u", "v", "w", "p")


def _states(g, case):
    return [g.get(f, nb) for nb in range(1, case.nblocks + 1) for f in STATE]


def _workload(name):
    if name == "vortex":  # one block, rows of 9: 4 rows are 36 columns, 32 and 33 columns come from nk 8 and 11
        return perturbed(cases.vortex_case(ni=29, nj=17, nk=9))
    if name == "vortex_nk8":
        return perturbed(cases.vortex_case(ni=12, nj=13, nk=8, nscheme=41, nflux=3))
    if name == "vortex_rows_j":  # k longer than j
        return perturbed(cases.vortex_case(ni=14, nj=7, nk=19, nscheme=41, nflux=3))
    if name == "vortex_nk11":
        return perturbed(cases.vortex_case(ni=9, nj=21, nk=11, nscheme=41, nflux=3))
    return perturbed(cases.small_plate_case())


@pytest.mark.parametrize("env", [
    {"WCNS_WIDE_MIN_COLS": "1", "WCNS_WIDE_COLS": "1", "WCNS_WIDE_FOLD": "1"},
    {"WCNS_WIDE_MIN_COLS": "1", "WCNS_WIDE_COLS": "1", "WCNS_WIDE_FOLD": "3"},
    {"WCNS_WIDE_MIN_COLS": "1", "WCNS_WIDE_COLS": "33", "WCNS_WIDE_FOLD": "2"},
    {"WCNS_WIDE_MIN_COLS": "1", "WCNS_WIDE_COLS": "40", "WCNS_WIDE_FOLD": "8"},
    {"WCNS_WIDE_COLS": "32", "WCNS_WIDE_FOLD": "1", "WCNS_WIDE_ST": "1"},
    {"WCNS_WIDE_COLS": "288", "WCNS_WIDE_FOLD": "1", "WCNS_WIDE_ST": "3"},
], ids=lambda e: "-".join(e.values()))
@pytest.mark.parametrize("name", ["vortex", "vortex_nk8", "vortex_nk11", "vortex_rows_j", "plate"])
def test_wide_splits_equal_the_clustered_sweeps(name, env, monkeypatch):
    from wcns_b200.solver import FLAG_SWEEP_WIDE, Wcns
    case = _workload(name)
    monkeypatch.setenv("WCNS_SWEEP_CLUSTER", "4")
    ref = Wcns(case)
    assert ref.sweep_mode() == "clustered"
    href = ref.step(3)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    g = Wcns(case, flags=FLAG_SWEEP_WIDE)
    assert g.sweep_mode() == "wide"
    np.testing.assert_array_equal(g.step(3), href)
    for a, b in zip(_states(g, case), _states(ref, case)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("fold", ["1", "2"])
def test_sa_sweeps_do_not_depend_on_the_split(fold, monkeypatch):
    """The scalar sweeps over folded and single-row chunks against the
    one-CTA-per-block kernel of a clustered context."""
    from wcns_b200.solver import FLAG_SWEEP_WIDE, Wcns
    case = cases.small_channel_case()
    out = []
    for flags in (0, FLAG_SWEEP_WIDE):
        if flags:
            monkeypatch.setenv("WCNS_WIDE_MIN_COLS", "1")
            monkeypatch.setenv("WCNS_WIDE_COLS", "1")
            monkeypatch.setenv("WCNS_WIDE_FOLD", fold)
        g = Wcns(case, flags=flags)
        g.sa_setup(case.sa["timedt_turb"], case.sa["kmaxlim"])
        g.step(3)
        out.append([g.get(f, nb) for nb in range(1, case.nblocks + 1) for f in STATE + ("qke", "vist")])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dims", [(6, 258, 261), (7, 5, 300)])
def test_long_rows_match_oracle(dims):
    """Rows near the longest that one CTA takes, and a block whose rows run
    along j because k is longer."""
    from oracle.pyoracle import Oracle
    from wcns_b200.solver import FLAG_SWEEP_WIDE, Wcns
    ni, nj, nk = dims
    case = perturbed(cases.vortex_case(ni=ni, nj=nj, nk=nk, lz=25.0))
    g, o = Wcns(case, flags=FLAG_SWEEP_WIDE), Oracle(case)
    assert g.sweep_mode() == "wide"
    for gp, op in [("boundary_all", "boundary_all"), ("initial_q_dq_c_t", "initial_q_dq_c_t"), ("timestep_tgh", "timestep"),
                   ("r_h_s_invis", "rhs_invis"), ("communicate_dq_npp", "communicate_dq"), ("l_h_s_tgh", "lhs")]:
        getattr(g, gp)()
        o.phase(op)
    e = compare_fields(g, o, ["dq1", "dq2", "dq3", "dq4", "dq5", *STATE])
    assert max(e.values()) <= 1e-12, e
