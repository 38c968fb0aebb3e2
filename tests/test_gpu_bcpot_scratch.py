"""The direct BCpotentials where the device has no room for its partial sums: the call
takes fewer plane groups in an array the context has, and gives the same potential.

A child process is started with a cudaMallocAsync that can be told to return an error,
as the driver's does when memory has run out; nothing on the device fails.

Bar: U within 1e-13 relative L2 of the call with room, and a second call's bits equal
to the first's."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int deny = 0, refused = 0;
int cudaMallocAsync(void** p, size_t n, void* stream) {
  if (deny) {
    __atomic_add_fetch(&refused, 1, __ATOMIC_RELAXED);
    *p = 0;
    return 2;  /* cudaErrorMemoryAllocation */
  }
  void* rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  int (*real)(void**, size_t, void*) = rt ? (int (*)(void**, size_t, void*))dlsym(rt, "cudaMallocAsync") : 0;
  return real ? real(p, n, stream) : 2;
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
from oracle import oracle as O
from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.test_gpu_spectral import blobs, boxed
shim = ctypes.CDLL(None)
out = {}
for n, (dims, flows) in enumerate((((20, 18, 16), (1, 1, 1)), ((3, 40, 5), (1, 1, 1)), ((1, 1, 1), (1, 1, 1)),
                                   ((33, 17, 50), (1, 0, 1)))):
    p = boxed(*dims, xflow=flows[0], yflow=flows[1], zflow=flows[2])
    C = blobs(O.OracleState(p), p, seed=4, width=9.0)
    for deny in (1, 0):
        with Simulation(p, derive=False, layout=capi.LAYOUT_F64, solver=capi.SOLVER_F64) as s:
            s.set_option(capi.OPT_BCPOT_TENSOR, 0)
            s.calc_distance()
            s.set_field(capi.FIELD_C, C)
            ctypes.c_int.in_dll(shim, "deny").value = deny
            for call in range(2):
                s.bc_potentials()
                out[f"{n} {deny} {call}"] = s.field(capi.FIELD_U)
            ctypes.c_int.in_dll(shim, "deny").value = 0
np.savez(sys.argv[1], **out)
print("refused", ctypes.c_int.in_dll(shim, "refused").value)
"""


def test_direct_sum_without_room_for_its_partials(tmp_path):
    src, so, path = tmp_path / "shim.c", tmp_path / "shim.so", str(tmp_path / "out.npz")
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"], check=True)
    run = subprocess.run([sys.executable, "-c", CHILD, path], cwd=ROOT, capture_output=True, text=True, timeout=300,
                         env=dict(os.environ, PYTHONPATH=ROOT, LD_PRELOAD=str(so)))
    assert run.returncode == 0, run.stderr[-2000:]
    assert int(run.stdout.split()[-1]) >= 8
    got = np.load(path)
    for n in range(4):
        roomy, tight = got[f"{n} 0 0"], got[f"{n} 1 0"]
        assert np.linalg.norm(roomy) > 0
        assert np.linalg.norm(roomy - tight) <= 1e-13 * np.linalg.norm(roomy)
        np.testing.assert_array_equal(tight, got[f"{n} 1 1"])
        np.testing.assert_array_equal(roomy, got[f"{n} 0 1"])
