"""A fused or batched loop that runs out of particle capacity some steps in: the
sweeps of the steps it finished are reported as a loop over those steps alone
reports them, and the context's next CalcEpotential returns its own sweeps and
residual (CalcEpotential.f90:55-96), not those of a solve the loop left behind.

Bar: equal counts, and equal bits of the residual, against a context with room."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from picard_b200 import capi
from picard_b200 import params as P
from picard_b200.simulation import Simulation
from tests.test_gpu_spectral import blobs

pytestmark = pytest.mark.gpu

STEPS = 8


def growing(capacity, seed=3):
    """A comet whose source adds particles every step."""
    p = P.config_plain_scale(seed=seed, nx=16, ny=16, nz=16, ppc_ion=4, capacity=capacity)
    p.Qn[2] = 1e29
    return O.derive(p)


def started(capacity, seed=3):
    s = Simulation(growing(capacity, seed), derive=False, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL)
    s.calc_distance()
    s.particles_initialize()
    return s


@pytest.fixture(scope="module")
def with_room():
    """Particles after each step, sweeps through each step, and a solve of its own."""
    with started(2_000_000) as s:
        nums, sweeps = [], [0]
        for it in range(STEPS):
            sweeps.append(sweeps[-1] + s.run_fused(it, it + 1))
            nums.append(s.num_local)
        assert nums[-1] > nums[2] > nums[1], nums
        charge = blobs(O.OracleState(s.p), s.p, seed=5, width=3.0)
        return nums, sweeps, charge, own_solve(s, charge)


def own_solve(s, charge):
    s.set_field(capi.FIELD_C, charge)
    s.set_field(capi.FIELD_U, np.zeros_like(charge))
    out = (s.calc_epotential(), s.stats()["last_residual"], s.stats()["last_bnorm"])
    assert out[0] > 0
    return out + (s.field(capi.FIELD_U),)


def same_solve(a, b):
    assert a[:3] == b[:3]
    np.testing.assert_array_equal(a[3], b[3])


def test_a_fused_loop_out_of_room_leaves_no_solve_behind(with_room):
    nums, sweeps, charge, own = with_room
    with started(nums[3]) as s:
        total = C.c_int64(0)
        rc = capi.lib().picard_gpu_run_fused(s._h, 0, STEPS, C.byref(total))
        assert rc == capi.ERR_CAPACITY and "capacity" in capi.last_error()
        done = s.stats()["steps"]
        assert 2 <= done < STEPS
        assert total.value == sweeps[done] == s.stats()["sweeps"]
        assert s.stats()["solves"] == done
        for _ in range(2):
            same_solve(own_solve(s, charge), own)


def test_a_batch_with_one_run_out_of_room_leaves_no_solve_behind(with_room):
    nums, sweeps, charge, own = with_room
    with started(nums[3]) as s, started(2_000_000, seed=4) as other, started(2_000_000, seed=4) as alone:
        runs = (C.c_void_p * 2)(s._h.value, other._h.value)
        totals = (C.c_int64 * 2)()
        rc = capi.lib().picard_batch_run_fused(runs, 2, 0, STEPS, totals)
        assert rc == capi.ERR_CAPACITY and "capacity" in capi.last_error()
        done = s.stats()["steps"]
        assert 2 <= done < STEPS and totals[0] == sweeps[done]
        assert totals[1] == alone.run_fused(0, other.stats()["steps"])
        for t in (s, other):
            same_solve(own_solve(t, charge), own)
