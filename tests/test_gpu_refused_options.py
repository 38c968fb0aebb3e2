"""A sweep option that picard_gpu_set_option refuses leaves the context's sweep
shape as it was, the cluster included; one that it takes replaces the cluster."""
import pytest

from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.test_gpu_spectral import boxed

pytestmark = pytest.mark.gpu

KNOBS = (capi.OPT_SWEEP_CTAS, capi.OPT_SWEEP_PDL, capi.OPT_SWEEP_STAGES, capi.OPT_SWEEP_RESIDENT,
         capi.OPT_SWEEP_PAIRS, capi.OPT_SWEEP_FUSED, capi.OPT_SWEEP_R_GLOBAL, capi.OPT_SWEEP_CLUSTER)


def knobs(s):
    return [s.get_option(k) for k in KNOBS]


def test_a_refused_value_changes_nothing():
    with Simulation(boxed(16, 16, 16), derive=False, layout=capi.LAYOUT_CELL32,
                    solver=capi.SOLVER_F32_REFINE) as s:
        s.set_option(capi.OPT_SWEEP_CLUSTER, 1)
        before = knobs(s)
        for option, value in ((capi.OPT_SWEEP_CTAS, -2), (capi.OPT_SWEEP_STAGES, 3), (capi.OPT_SWEEP_RESIDENT, 99),
                              (capi.OPT_SWEEP_CLUSTER, 2)):
            with pytest.raises(capi.PicardError):
                s.set_option(option, value)
            assert knobs(s) == before
        s.set_option(capi.OPT_SWEEP_STAGES, 1)
        assert s.get_option(capi.OPT_SWEEP_CLUSTER) == 0
