"""GridifyAll on the FP64 layout (ParticlesGridifyAll.f90:1-455), whose densities come
from the tiles of Gridify and whose fluxes from a pass of their own: counts around a
warp, a tile chunk and a block, particles in no order, some within half a cell outside
the domain, open and periodic axes.

Bar: N bit for bit Gridify's; every node's N within half a unit of 2^-40 per particle
(and 1e-12 for the oracle's own sums) of the oracle's, F within 1e-9 relative L2 of it (half a unit of 2^-20 m/s per weight)."""
import numpy as np
import pytest

from picard_b200 import capi
from tests.helpers import rel_l2, small_plasma
from tests.test_gpu_parity import F64, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("yflow", [1, 0])
@pytest.mark.parametrize("n", [0, 1, 31, 33, 63, 65, 255, 257, 2047, 4001])
def test_densities_and_fluxes(n, yflow):
    p, o, g = make(small_plasma(n=9, ppc=4, seed=8, yflow=yflow), **F64)
    rng = np.random.default_rng(n)
    lo, hi, d = (np.array(v) for v in ([p.xmin, p.ymin, p.zmin], [p.xmax, p.ymax, p.zmax], list(p.dxyz)))
    rp = np.zeros((n, 8))
    rp[:, :3] = rng.uniform(lo - 0.4 * d, hi + 0.4 * d, (n, 3))
    rp[:, 3:6] = 4e5 * rng.standard_normal((n, 3))
    ip = (1 + rng.integers(0, p.species, n)).astype(np.int32)
    o.set_particles(rp, ip)
    g.set_particles(rp, ip)
    o.gridify()
    o.gridify_all()
    g.particles_gridify()
    N = g.field(capi.FIELD_N)
    g.particles_gridify_all()
    np.testing.assert_array_equal(g.field(capi.FIELD_N), N)
    F = g.field(capi.FIELD_F)
    if n == 0:
        assert not N.any() and not F.any()
        return
    n2p = np.array([p.n2p[s] for s in range(p.species)])
    assert (np.abs(N - o.N).max(axis=(0, 1, 2)) <= n2p * n * 2.0 ** -41 + 1e-12 * np.abs(o.N).max()).all()
    assert rel_l2(F, o.F) < 1e-9
