"""BCoutflow's fill by pointer jumping (outflow.cuh), whose rounds end when nothing
moves, and, for windows under 2^17 positions with few survivors, by following the
chains: windows of 2^14 positions and more with their survivors at the front, in the
middle, at the very end, alone, in one run, at random, or none at all -- so that the
removed positions behind the last survivor, which stand for themselves, are many, few
or none, and chains of one hop and of thousands are resolved.

Bar: the oracle's particles in the oracle's order, bit for bit."""
import numpy as np
import pytest

from tests.helpers import small_plasma
from tests.test_gpu_parity import F64, make

pytestmark = pytest.mark.gpu

KEPT = 20_000


@pytest.mark.parametrize("window", [1 << 14, 50_001, 100_000, 1 << 17, 200_003])
@pytest.mark.parametrize("where", ["none", "first", "last", "middle", "front_run", "end_run", "random", "sparse"])
def test_jumping_leaves_the_reference_order(where, window):
    pl = small_plasma(n=8, ppc=1, seed=3)
    pl.max_per_proc = 300_000
    p, o, g = make(pl, **F64)
    rng = np.random.default_rng(window)
    n = KEPT + window
    at = {"none": [], "first": [0], "last": [window - 1], "middle": [window // 2],
          "front_run": np.arange(300), "end_run": np.arange(window - 300, window),
          "random": np.sort(rng.permutation(window)[:min(window // 5, KEPT)]), "sparse": np.sort(rng.permutation(window)[:40])}[where]
    alive = np.zeros(n, bool)
    alive[:KEPT] = True
    alive[KEPT + np.asarray(at, int)] = True
    # as many holes below n' as survivors above it
    alive[rng.permutation(KEPT)[:len(at)]] = False
    lo, hi = np.array([p.xmin, p.ymin, p.zmin]), np.array([p.xmax, p.ymax, p.zmax])
    rp = np.zeros((n, 8))
    rp[:, :3] = lo + (hi - lo) * rng.uniform(0.05, 0.95, (n, 3))
    rp[~alive, 0] = hi[0] + 0.3 * p.dxyz[0]
    rp[:, 3] = np.arange(n)
    ip = 1 + (np.arange(n) % p.species).astype(np.int32)
    o.set_particles(rp, ip)
    g.set_particles(rp, ip)
    for _ in range(2):  # a second call on what is left: nothing to remove
        o.bc_outflow()
        g.bc_outflow()
        assert g.num_local == o.num_local == KEPT
        (rg, ig), (ro, io) = g.particles(), o.particles()
        np.testing.assert_array_equal(ig, io)
        np.testing.assert_array_equal(rg[:, :6], ro[:, :6])
