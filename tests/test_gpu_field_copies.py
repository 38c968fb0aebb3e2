"""Fields read in the reference's order, in pieces of 4 MB by several host
threads: what set_field wrote comes back bit for bit for every field, on grids
of a fraction of a piece, just under and over one, and of several; from a
thread of its own as well; and contexts that come and go give their pinned
memory back to each other."""
import threading

import numpy as np
import pytest

from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.test_gpu_spectral import boxed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 2, 3), (78, 78, 79), (80, 79, 80), (126, 62, 62), (150, 70, 60)])
def test_fields_come_back_in_reference_order(dims):
    p = boxed(*dims)
    rng = np.random.default_rng(sum(dims))
    with Simulation(p, derive=False, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL) as g:
        for which in (capi.FIELD_U, capi.FIELD_E, capi.FIELD_N, capi.FIELD_F, capi.FIELD_C):
            a = rng.standard_normal(g._shape(which))
            g.set_field(which, a)
            np.testing.assert_array_equal(g.field(which), a)
            got = []
            t = threading.Thread(target=lambda: got.append(g.field(which)))
            t.start()
            t.join()
            np.testing.assert_array_equal(got[0], a)


def test_contexts_share_kept_pinned_memory():
    p = boxed(20, 18, 16)
    ref = None
    for keep in (0, 1 << 30, 1 << 30, 0):
        capi.pool_keep(0, keep)
        sims = [Simulation(p, derive=False, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL) for _ in range(3)]
        out = []
        for s in sims:
            s.calc_distance()
            s.set_field(capi.FIELD_C, np.arange(np.prod(s._shape(capi.FIELD_C)), dtype=float).reshape(s._shape(capi.FIELD_C)) * 1e-16)
            s.bc_potentials()
            s.calc_epotential()
            out.append(s.field(capi.FIELD_U))
        for s in sims:
            s.close()
        ref = out[0] if ref is None else ref
        for u in out:
            np.testing.assert_array_equal(u, ref)
