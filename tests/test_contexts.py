"""Several contexts alive at once: what one is built or re-shaped with must not reach
another.  The shared-memory limit of a kernel belongs to the process, so a context
whose kernels take more than the 48 KB every kernel has is stepped for the first time
after contexts that need less were built, re-shaped and stepped; it has to give what
it gives alone, bit for bit."""
import threading

import numpy as np
import pytest

from tests.helpers import perturbed, supersonic_box_case
from wcns_b200 import cases

pytestmark = pytest.mark.gpu

STATE = ("r", "u", "v", "w", "p")


def _context(case, shape=None, bits=64):
    from wcns_b200.solver import Wcns
    g = Wcns(case)
    if case.sa:
        g.sa_setup(case.sa["timedt_turb"], case.sa["kmaxlim"])
    if bits == 32:
        g.set_precision(32)
    if shape is not None:
        g.set_shape([g.shape[q] if s is None else s for q, s in enumerate(shape)])
    return g


def _steps(g):
    h = g.step(2)
    return [h, *g.residual_curve()[:2]] + [g.get(f, nb) for nb in range(1, len(g.dims) + 1) for f in STATE]


def _box(ni, nj, nk, nvis=0, **kw):
    case = supersonic_box_case(ni, nj, nk, **kw)
    case.params.nvis = nvis
    return case


BIG = {
    # 21 lines of 5 or (in chunks of 6 half nodes, with lines enough for the chip) 16
    # points and their boundary sections: 51 KB
    "sections_5": (lambda: _box(5, 21, 9), None, 64),
    "sections_16": (lambda: _box(16, 21, 900), None, 64),
    # 32 viscous lines of 3 points, 25 of 4: 56 and 50 KB
    "viscous_3": (lambda: _box(32, 6, 3, nvis=1, nscheme=4), None, 64),
    "viscous_4": (lambda: _box(4, 25, 6, nvis=1, nscheme=4), None, 64),
    # 77 and 42 columns in a CTA's shared memory: 118 and 65 KB
    "one_cta_cluster": (lambda: perturbed(cases.small_plate_case()), (1, 0, None, None), 64),
    "fine_cluster": (lambda: perturbed(cases.small_plate_case()), (2, 1, None, None), 64),
    # whole lines of 65 and 33 points of the mixed residual: 50 to 72 KB
    "mixed": (lambda: cases.vortex_case(ni=65, nj=33, nk=17, nscheme=41, nflux=3), None, 32),
    # partial sums of more than 96 blocks
    "blocks": (lambda: cases.batch_case(ncases=130, seed=1), None, 64),
}


def _smaller():
    """Contexts that take less than any of the above, one after the other, each stepped."""
    for case, shape, bits in ((cases.vortex_case(ni=12, nj=9, nk=8, nscheme=4, nflux=1), (8, 1, 1, 1), 64),
                              (cases.vortex_case(ni=12, nj=9, nk=8, nscheme=41, nflux=3), (0, 0, 2, 2), 64),
                              (cases.small_plate_case(), (7, 0, 1, 1), 64),
                              (cases.small_plate_case(), (4, 1, 2, 2), 32),
                              (cases.batch_case(ncases=98, seed=2), (0, 0, 4, 4), 64)):
        g = _context(case, shape, bits)
        g.step(1)
        yield g


@pytest.mark.parametrize("name", BIG)
def test_a_context_steps_after_smaller_ones(name):
    make, shape, bits = BIG[name]
    alone = _context(make(), shape, bits)
    want = _steps(alone)
    alone.close()
    g = _context(make(), shape, bits)
    others = list(_smaller())
    for a, b in zip(_steps(g), want):
        np.testing.assert_array_equal(a, b)
    assert len(others) == 5


@pytest.mark.parametrize("name", ["one_cta_cluster", "mixed"])
def test_a_context_steps_after_another_was_tuned_and_refused(name):
    from wcns_b200.solver import WcnsError
    make, shape, bits = BIG[name]
    alone = _context(make(), shape, bits)
    want = _steps(alone)
    alone.close()
    g = _context(make(), shape, bits)
    other = _context(cases.small_plate_case())
    other.step(1)
    other.autotune(1)
    with pytest.raises(WcnsError):
        other.set_shape([64, 1, 32, 32])
    for a, b in zip(_steps(g), want):
        np.testing.assert_array_equal(a, b)


def test_adjoint_operators_of_two_threads():
    """Tangent and adjoint of a large and of a small block, called in turn from two
    threads: each launch needs its own context's shared memory."""
    from wcns_b200.solver import Wcns
    dims, out, fails = [(65, 33, 9), (9, 8, 7)], {}, []

    def work(q):
        try:
            ni, nj, nk = dims[q]
            g = Wcns(cases.vortex_case(ni=ni, nj=nj, nk=nk, nscheme=4, nflux=3))
            g.boundary_all()
            g.initial_q_dq_c_t()
            g.timestep_tgh()
            rng = np.random.default_rng(q)
            g.adj_set("v", 1, [rng.standard_normal((nk + 6, nj + 6, ni + 6)) for _ in range(5)])
            res = []
            for _ in range(40):
                g.rhs_invis_tangent()
                res.append(g.adj_get("rdot", 1))
            out.setdefault(q, []).append(res)
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            fails.append((q, e))

    threads = [threading.Thread(target=work, args=(q,)) for q in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not fails, fails
    for q in (0, 1):
        for res in out[q][0]:
            for a, b in zip(res, out[q][0][0]):
                np.testing.assert_array_equal(a, b)


def test_tuning_restores_dq_while_the_default_stream_is_busy():
    """The context's stream and the default stream do not wait for each other."""
    import torch
    from wcns_b200.solver import Wcns
    g = Wcns(perturbed(cases.small_plate_case()))
    g.step(1)
    before = [g.get(f"dq{m}", nb) for nb in range(1, len(g.dims) + 1) for m in range(1, 6)]
    torch.cuda._sleep(400_000_000)  # some 0.2 s
    g.autotune(1)
    torch.cuda.synchronize()
    after = [g.get(f"dq{m}", nb) for nb in range(1, len(g.dims) + 1) for m in range(1, 6)]
    for a, b in zip(before, after):
        np.testing.assert_array_equal(a, b)
