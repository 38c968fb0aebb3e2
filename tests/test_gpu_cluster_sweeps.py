"""FP64 sweeps resident in one cluster (SOLVER_F64 on small grids): uneven
slabs, one plane per CTA, the largest planes a CTA holds, fewer CTAs than
sixteen, periodic axes of every kind, and a grid just too large for it (one
launch per sweep).

Bar: the stopping sweep of the closed-form solve and U within 1e-11 relative
L2 of it, from the same U and C (as test_gpu_spectral.py)."""
import numpy as np
import pytest

from oracle import oracle as O
from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.helpers import rel_l2
from tests.test_gpu_spectral import F64, SPEC64, blobs, boxed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,flows", [
    ((16, 16, 16), (1, 1, 1)),
    ((20, 21, 17), (1, 1, 1)),
    ((46, 46, 46), (1, 1, 1)),
    ((90, 84, 5), (1, 1, 1)),
    ((12, 10, 2), (1, 1, 0)),
    ((13, 12, 16), (0, 0, 1)),
    ((9, 1, 33), (1, 0, 0)),
    ((60, 58, 40), (1, 1, 1)),
])
def test_cluster_sweeps_equal_the_closed_form(dims, flows):
    p = boxed(*dims, xflow=flows[0], yflow=flows[1], zflow=flows[2])
    o = O.OracleState(p)
    C = blobs(o, p, seed=sum(dims), width=20.0)
    U = np.zeros_like(C)
    rng = np.random.default_rng(2)
    for axis in range(3):
        if flows[2 - axis]:
            for side in (0, -1):
                sl = [slice(1, -1)] * 3
                sl[axis] = side
                U[tuple(sl)] = 1e-3 * rng.standard_normal(U[tuple(sl)].shape)
    out = []
    for kw in (F64, SPEC64):
        with Simulation(p, derive=False, **kw) as s:
            s.set_field(capi.FIELD_C, C)
            s.set_field(capi.FIELD_U, U)
            out.append((s.calc_epotential(), s.field(capi.FIELD_U)))
    err = rel_l2(out[0][1], out[1][1])
    print(f"{dims} {flows}: {out[0][0]} sweeps, U rel L2 {err:.2e}")
    assert out[0][0] == out[1][0] and out[0][0] > 10
    assert err < 1e-11
