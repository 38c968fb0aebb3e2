"""The FP32 sweeps in one cluster, asked for by hand (PICARD_OPT_SWEEP_CLUSTER), so
that they run whatever the launch tuner measures: against the tile kernels, for
solves that stop after every one of the first sweeps (rounds whose last sums are
taken at once, behind the loop) and far later, on odd rows, partial layers and
tiles, the smallest plane and the most rows and layers a cluster takes.

Bar: the same stopping sweep and the same bits of the residual and of U."""
import numpy as np
import pytest

from oracle import oracle as O
from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.test_gpu_spectral import blobs, boxed

pytestmark = pytest.mark.gpu

REFINE = dict(layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_F32_REFINE)


def solve(s, C, maxerr):
    s.set_field(capi.FIELD_C, C)
    s.set_field(capi.FIELD_U, np.zeros_like(C))
    n = s.calc_epotential(maxerr=maxerr)
    return n, s.stats()["last_residual"], s.field(capi.FIELD_U)


@pytest.mark.parametrize("dims", [(16, 16, 16), (17, 9, 13), (32, 32, 32), (31, 33, 21), (33, 17, 9), (8, 8, 5),
                                  (1, 1, 8), (30, 64, 63), (64, 32, 12)])
def test_cluster_sweeps_have_the_bits_of_the_tile_kernels(dims):
    p = boxed(*dims)
    C = blobs(O.OracleState(p), p, seed=sum(dims), width=20.0)
    rng = np.random.default_rng(1)
    noise = 1e-12 * rng.standard_normal(C[1:-1, 1:-1, 1:-1].shape)
    rough = C.copy()
    rough[1:-1, 1:-1, 1:-1] += noise
    cases = [(rough, e) for e in 0.6 * 0.8 ** np.arange(12)] + [(C, p.maxerr), (C, 0.3)]
    with Simulation(p, derive=False, **REFINE) as s:
        s.set_option(capi.OPT_SWEEP_CLUSTER, 1)
        assert s.get_option(capi.OPT_SWEEP_CLUSTER) == 1
        cluster = [solve(s, *c) for c in cases]
        assert s.get_option(capi.OPT_SWEEP_CLUSTER) == 1
        s.set_option(capi.OPT_SWEEP_CLUSTER, 0)
        s.set_option(capi.OPT_SWEEP_CTAS, -1)
        assert s.get_option(capi.OPT_SWEEP_CLUSTER) == 0
        tiles = [solve(s, *c) for c in cases]
    stops = {t[0] for t in tiles}
    print(dims, sorted(stops))
    assert len(stops) >= 4
    for a, b in zip(cluster, tiles):
        assert a[:2] == b[:2]
        np.testing.assert_array_equal(a[2], b[2])


@pytest.mark.parametrize("dims,kw,flows", [
    ((48, 40, 33), REFINE, 1),  # 80 tile rows a layer
    ((16, 16, 4), REFINE, 1),   # one layer
    ((16, 16, 64), REFINE, 1),  # layers of eight planes
    ((16, 16, 16), REFINE, 0),
    ((16, 16, 16), dict(layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL), 1),
])
def test_a_grid_that_does_not_fit_is_refused(dims, kw, flows):
    p = boxed(*dims, zflow=flows)
    with Simulation(p, derive=False, **kw) as s:
        with pytest.raises(capi.PicardError) as e:
            s.set_option(capi.OPT_SWEEP_CLUSTER, 1)
        assert e.value.code == capi.ERR_STATE
        assert s.get_option(capi.OPT_SWEEP_CLUSTER) == 0
        s.set_option(capi.OPT_SWEEP_CLUSTER, 0)


@pytest.mark.parametrize("dims", [(16, 16, 16), (33, 17, 9), (30, 64, 63)])
def test_every_sweep_of_a_round_has_its_residual(dims, monkeypatch, capfd):
    """Rounds of 1, 3, 5 and 7 sweeps (2 maxit + 1, no stop): the solver's log of a
    round, with the sum of its residuals to the last bit, for both kernels."""
    p = boxed(*dims)
    C = blobs(O.OracleState(p), p, seed=3, width=20.0)
    monkeypatch.setenv("PICARD_SOLVE_LOG", "1")
    logs = []
    with Simulation(p, derive=False, **REFINE) as s:
        for on in (1, 0):
            s.set_option(capi.OPT_SWEEP_CLUSTER, on)
            capfd.readouterr()
            for maxit in (0, 1, 2, 3):
                s.set_field(capi.FIELD_C, C)
                s.set_field(capi.FIELD_U, np.zeros_like(C))
                assert s.calc_epotential(maxerr=1e-30, maxit=maxit) == 2 * maxit + 1
            logs.append([x for x in capfd.readouterr().err.splitlines() if x.startswith("picard solve")])
    assert len(logs[0]) == 4 and logs[0] == logs[1]
