"""The tiled CELL32 deposit (ParticlesGridify, ParticlesGridify.f90:65-123) at
the sizes where its chunks can go wrong: particle counts around a warp's chunk
of two, four and eight particles per lane, arrays with a partial last chunk,
rows that a chunk straddles (periodic and open, so that the ghost folds of both
kinds are reached), and cell-ordered arrays with far particles in them, as
BCoutflow's hole filling leaves them.

Bar: N equal bit for bit to the warp-aggregated kernel of ParticlesGridifyAll,
which sums the same fixed-point weights (integer sums are exact in any order).
"""
import numpy as np
import pytest

from picard_b200 import capi
from picard_b200 import params as P
from picard_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def _plasma(nx, ny, nz, ppc, n, seed, far, flows):
    p = P.config_plain_32(seed=seed, n=8, ppc=ppc, capacity=n)
    p.nx, p.ny, p.nz = nx, ny, nz
    p.xmin, p.xmax = -500.0 * nx, 500.0 * nx
    p.ymin, p.ymax = -500.0 * ny, 500.0 * ny
    p.zmin, p.zmax = -500.0 * nz, 500.0 * nz
    p.xflow, p.yflow, p.zflow = flows
    p = capi.params_derive(p)
    rng = np.random.default_rng(seed)
    cell = np.arange(n, dtype=np.int64) * (nx * ny * nz) // n
    at = np.stack([cell % nx, cell // nx % ny, cell // (nx * ny)], axis=1)
    t = at + rng.random((n, 3)) + 0.05 * rng.standard_normal((n, 3))
    moved = rng.random(n) < far
    t[moved] = rng.random((int(moved.sum()), 3)) * [nx, ny, nz]
    t = np.clip(t, 0.0, [nx, ny, nz])
    rp = np.zeros((n, 8))
    rp[:, :3] = t * 1000.0 + [p.xmin, p.ymin, p.zmin]
    return p, rp, (1 + np.arange(n) % 2).astype(np.int32)


@pytest.mark.parametrize("dims,n,far,flows", [
    ((7, 6, 5), 1, 0.0, (1, 1, 1)),
    ((7, 6, 5), 63, 0.0, (1, 1, 1)),
    ((7, 6, 5), 64, 0.0, (1, 0, 1)),
    ((33, 9, 4), 4099, 0.0, (0, 1, 1)),
    ((33, 9, 4), 70001, 0.02, (1, 1, 0)),
    ((80, 70, 60), 2424831, 0.0, (1, 1, 1)),    # four per lane, the last two-per-lane count and one
    ((80, 70, 60), 2424832, 0.01, (1, 0, 1)),
    ((80, 70, 60), 2600003, 0.3, (0, 1, 1)),
    ((40, 36, 30), 2424833, 0.0, (1, 1, 0)),    # eight per lane
    ((40, 36, 30), 2600001, 0.02, (0, 0, 1)),
    ((150, 40, 25), 2500127, 1.0, (1, 1, 1)),   # no order at all
])
def test_tiled_deposit_at_chunk_edges(dims, n, far, flows):
    p, rp, ip = _plasma(*dims, 4, n, seed=n % 97, far=far, flows=flows)
    with Simulation(p, derive=False, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL) as g:
        g.set_particles(rp, ip)
        g.particles_gridify()
        N_tile = g.field(capi.FIELD_N)
        g.particles_gridify_all()
        N_warp = g.field(capi.FIELD_N)
    assert np.abs(N_tile).sum() > 0
    np.testing.assert_array_equal(N_tile, N_warp)
