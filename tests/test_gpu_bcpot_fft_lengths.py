"""FFT BCpotentials at every transform length it has and on both sides of the
steps between them: tangential extents around powers of two (circular lengths
8 .. 1024, and 2048 along P), odd plane counts (a row pair with one row), and a
grid above the size up to which the face pairs share their launches.

Bar: 1e-12 relative L2 of the face potentials from the FP64 direct sum on the
GPU (as test_gpu_bcpot_fft.py against the oracle's)."""
import numpy as np
import pytest

from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.helpers import rel_l2
from tests.test_gpu_spectral import boxed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,flows", [
    ((1, 4, 5), (1, 1, 1)),
    ((4, 8, 3), (1, 1, 1)),
    ((9, 8, 5), (1, 1, 1)),
    ((16, 17, 9), (1, 1, 1)),
    ((33, 32, 2), (1, 0, 1)),
    ((64, 65, 3), (1, 1, 1)),
    ((129, 7, 64), (1, 1, 1)),
    ((128, 3, 129), (0, 1, 1)),
    ((257, 5, 6), (1, 1, 1)),
    ((6, 256, 257), (1, 1, 0)),
    ((513, 4, 3), (1, 1, 1)),
    ((3, 2, 512), (1, 1, 1)),
    ((1024, 2, 2), (1, 1, 1)),
    ((130, 101, 96), (1, 1, 1)),
])
def test_fft_bcpotentials_at_every_length(dims, flows):
    p = boxed(*dims, xflow=flows[0], yflow=flows[1], zflow=flows[2])
    rng = np.random.default_rng(sum(dims))
    C = np.zeros((p.nz + 2, p.ny + 2, p.nx + 2))
    C[1:-1, 1:-1, 1:-1] = 1e-13 * rng.standard_normal((p.nz, p.ny, p.nx))
    with Simulation(p, derive=False, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL) as g:
        g.calc_distance()
        g.set_field(capi.FIELD_C, C)
        out = []
        for method in (2, 0):  # FFT, direct sum
            g.set_option(capi.OPT_BCPOT_TENSOR, method)
            g.bc_potentials()
            out.append(g.field(capi.FIELD_U))
    err = rel_l2(out[0], out[1])
    print(f"{dims} {flows}: rel L2 {err:.2e}")
    assert np.abs(out[1]).max() > 0
    assert err < 1e-12
