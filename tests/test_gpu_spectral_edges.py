"""The axis passes of SOLVER_SPECTRAL at the edges of their tiles: axes of 1, 2
and 3 nodes, one below, at and above the 64 outputs of a tile's half (127, 128,
129, 130 nodes) and the 16-element summation chunks, open and periodic, odd and
even.

Bar: the same stopping sweep as the FP64 sweep solver from the same U and C,
and U within 1e-11 relative L2 of its iterate (as test_gpu_spectral.py)."""
import numpy as np
import pytest

from oracle import oracle as O
from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.helpers import rel_l2
from tests.test_gpu_spectral import F64, SPEC64, blobs, boxed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,flows", [
    ((127, 3, 2), (1, 1, 1)),
    ((128, 2, 17), (1, 1, 0)),
    ((129, 16, 1), (1, 0, 1)),
    ((3, 130, 2), (1, 1, 1)),
    ((2, 129, 5), (0, 1, 1)),
    ((1, 2, 128), (1, 0, 1)),
    ((6, 3, 131), (0, 1, 1)),
    ((33, 32, 31), (0, 1, 0)),
])
def test_axis_passes_at_tile_edges(dims, flows):
    p = boxed(*dims, xflow=flows[0], yflow=flows[1], zflow=flows[2])
    o = O.OracleState(p)
    C = blobs(o, p, seed=sum(dims), width=30.0)
    U = np.zeros_like(C)
    rng = np.random.default_rng(1)
    for axis in range(3):  # a boundary potential on the open faces
        if flows[2 - axis]:
            for side in (0, -1):
                sl = [slice(1, -1)] * 3
                sl[axis] = side
                U[tuple(sl)] = 1e-3 * rng.standard_normal(U[tuple(sl)].shape)
    sims = [Simulation(p, derive=False, **kw) for kw in (SPEC64, F64)]
    for s in sims:
        s.set_field(capi.FIELD_C, C)
        s.set_field(capi.FIELD_U, U)
    sw = [s.calc_epotential() for s in sims]
    err = rel_l2(sims[0].field(capi.FIELD_U), sims[1].field(capi.FIELD_U))
    print(f"{dims} {flows}: spectral {sw[0]} vs FP64 sweeps {sw[1]}, U rel L2 {err:.2e}")
    assert sw[0] == sw[1] and sw[0] > 0
    assert err < 1e-11
    for s in sims:
        s.close()


@pytest.mark.parametrize("maxerr", [0.9, 1e-2, 1e-6])
@pytest.mark.parametrize("maxit", [0, 1, 2, 3, 34, 67, 100, 1100])
def test_search_stops_where_the_sweeps_stop(maxit, maxerr):
    # the on-device search at every cap that changes its evaluations: no test
    # at all (0, 1), one candidate, one and two brackets of 33, and caps above
    # and below the sweep that passes; a charge of zero takes no sweep
    p = boxed(12, 10, 9)
    o = O.OracleState(p)
    for C in (blobs(o, p, seed=4), np.zeros_like(o.C)):
        out = []
        for kw in (SPEC64, F64):
            with Simulation(p, derive=False, **kw) as s:
                s.set_field(capi.FIELD_C, C)
                s.set_field(capi.FIELD_U, np.zeros_like(C))
                n = s.calc_epotential(maxerr=maxerr, maxit=maxit)
                out.append((n, s.field(capi.FIELD_U)))
        assert out[0][0] == out[1][0]
        assert rel_l2(out[0][1], out[1][1]) < 1e-11
