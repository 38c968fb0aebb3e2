"""BCoutflow on the CELL32 layout at the counts where its blocks of 2,048
particles, its keep words of 32 and its reads of four end: particles in outer
cells on either side of every face (whose in-cell offset decides) among interior
ones, open and periodic axes.

Bar: the oracle's survivors in the oracle's order (species and velocities
exactly; positions to the layout's 2^-32 of a cell, 1e-6 here)."""
import numpy as np
import pytest

from tests.helpers import small_plasma
from tests.test_gpu_parity import C32, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zflow", [1, 0])
@pytest.mark.parametrize("n", [1, 3, 4, 31, 33, 1026, 2047, 2048, 2049, 2051, 4097])
def test_outflow_at_block_and_word_edges(n, zflow):
    p, o, g = make(small_plasma(n=9, ppc=4, seed=8, zflow=zflow), **C32)
    o.initialize()
    rp, ip = o.particles()
    rng = np.random.default_rng(n)
    pick = rng.permutation(len(ip))[:n]
    assert len(pick) == n
    rp, ip = rp[pick].copy(), ip[pick].copy()
    d = np.array(list(p.dxyz))
    lo, hi = np.array([p.xmin, p.ymin, p.zmin]), np.array([p.xmax, p.ymax, p.zmax])
    for axis in range(3 if zflow else 2):
        for face, side in ((lo, -1), (hi, 1)):
            m = rng.random(n) < 0.15
            rp[m, axis] = face[axis] + side * d[axis] * rng.uniform(-0.9, 0.9, m.sum())
    rp[:, 3:6] = rp[:, 3:6].astype(np.float32)
    o.set_particles(rp, ip)
    g.set_particles(rp, ip)
    o.bc_outflow()
    g.bc_outflow()
    assert g.num_local == o.num_local and (n < 31 or 0 < o.num_local < n)
    if o.num_local:
        (rg, ig), (ro, io) = g.particles(), o.particles()
        np.testing.assert_array_equal(ig, io)
        np.testing.assert_array_equal(rg[:, 3:6].astype(np.float32), ro[:, 3:6].astype(np.float32))
        np.testing.assert_allclose(rg[:, :3], ro[:, :3], rtol=0, atol=1e-6 * d.max())
