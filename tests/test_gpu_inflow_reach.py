"""The fused BCinflow gives candidates up on their position when no velocity
they could draw carries them into the domain within a step.  With time steps
from a thousandth of a cell to several cells per step, cold and hot plasmas and
a drift out of the domain, the fused loop keeps exactly the particles of the
per-subroutine loop, which generates, advances and removes every candidate
(BCinflow.f90:23-476, AdvancePosition.f90:15, BCoutflow.f90:24-83).

Bar: the same particles bit for bit (F64 layout), as sets."""
import numpy as np
import pytest

from oracle import oracle as O
from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.helpers import small_plasma, sort_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flows", [(1, 1, 1), (1, 0, 1)])
@pytest.mark.parametrize("dt_factor,kt_factor,vx", [(1.0, 1.0, 4e5), (300.0, 1.0, 4e5), (300.0, 0.0, -4e5),
                                                    (3000.0, 4.0, 4e5)])
def test_fused_inflow_keeps_what_the_plain_loop_keeps(dt_factor, kt_factor, vx, flows):
    p = small_plasma(n=9, ppc=6, seed=11, xflow=flows[0], yflow=flows[1], zflow=flows[2])
    p.dt *= dt_factor
    for s in range(8):
        p.kelvin[s] *= kt_factor
        p.v0[s][0] = vx
    p.maxit = 50  # the potential plays no part here
    p = O.derive(p)
    out = []
    for fused in (False, True):
        with Simulation(p, derive=False, layout=capi.LAYOUT_F64, solver=capi.SOLVER_SPECTRAL) as g:
            g.calc_distance()
            g.particles_initialize()
            (g.run_fused if fused else g.run)(0, 1)
            out.append(sort_particles(*g.particles()))
    assert len(out[0][1]) > 0
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][0][:, :3], out[1][0][:, :3])
