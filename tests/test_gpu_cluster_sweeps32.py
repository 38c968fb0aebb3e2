"""FP32 sweeps of the refining solver on grids that one cluster can hold: the
shape the launch tuner picks (the cluster, wherever it measures faster) against
the tile kernels asked for by hand.  Odd rows, a last layer of one plane, a last
tile of one column, one row per tile layer more than a multiple of eight, the
smallest plane and the most rows a cluster takes.

Bar: the same stopping sweep and the same bits of U."""
import numpy as np
import pytest

from oracle import oracle as O
from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.test_gpu_spectral import blobs, boxed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 16, 16), (17, 9, 13), (32, 32, 32), (31, 33, 21), (33, 17, 9), (8, 8, 5),
                                  (30, 64, 64), (64, 32, 12)])
def test_tuned_shape_has_the_bits_of_the_tile_kernels(dims):
    p = boxed(*dims)
    o = O.OracleState(p)
    C = blobs(o, p, seed=sum(dims), width=20.0)
    out = []
    for by_hand in (False, True):
        with Simulation(p, derive=False, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_F32_REFINE) as s:
            if by_hand:
                s.set_option(capi.OPT_SWEEP_RESIDENT, 0)
                s.set_option(capi.OPT_SWEEP_CTAS, -1)
            s.set_field(capi.FIELD_C, C)
            s.set_field(capi.FIELD_U, np.zeros_like(C))
            out.append((s.calc_epotential(), s.field(capi.FIELD_U)))
    assert out[0][0] == out[1][0] and out[0][0] > 10
    np.testing.assert_array_equal(out[0][1], out[1][1])
