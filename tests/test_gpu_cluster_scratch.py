"""FP64 sweeps where the device has no room for the cluster's partial sums (17 MB, on
the first solve): the solve runs with one launch per sweep, as it does on grids that
no cluster holds.

A child process is started with a cudaMallocAsync that returns an error for large
arrays, as the driver's does when memory has run out; nothing on the device fails.

Bar: the stopping sweep of the cluster and U within 1e-12 relative L2 of it."""
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
int refused = 0;
int cudaMallocAsync(void** p, size_t n, void* stream) {
  if (n >= (16u << 20)) {
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
p = boxed(20, 18, 16)
C = blobs(O.OracleState(p), p, seed=4, width=9.0)
with Simulation(p, derive=False, layout=capi.LAYOUT_F64, solver=capi.SOLVER_F64) as s:
    s.set_field(capi.FIELD_C, C)
    s.set_field(capi.FIELD_U, np.zeros_like(C))
    sweeps = [s.calc_epotential()]
    U = s.field(capi.FIELD_U)
    s.set_field(capi.FIELD_U, np.zeros_like(C))
    sweeps.append(s.calc_epotential())
np.savez(sys.argv[1], U=U, sweeps=sweeps)
shim = ctypes.CDLL(None)
print("refused", ctypes.c_int.in_dll(shim, "refused").value if hasattr(shim, "refused") else 0)
"""


def test_sweeps_without_room_for_the_partial_sums(tmp_path):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"], check=True)
    out = []
    for preload in ({}, {"LD_PRELOAD": str(so)}):
        path = str(tmp_path / f"out{len(out)}.npz")
        run = subprocess.run([sys.executable, "-c", CHILD, path], cwd=ROOT, capture_output=True, text=True, timeout=300,
                             env=dict(os.environ, PYTHONPATH=ROOT, **preload))
        assert run.returncode == 0, run.stderr[-2000:]
        refused = int(run.stdout.split()[-1])
        assert refused == (1 if preload else 0)
        out.append(np.load(path))
    a, b = out
    assert list(a["sweeps"]) == list(b["sweeps"]) and a["sweeps"][0] > 10
    assert np.linalg.norm(a["U"] - b["U"]) <= 1e-12 * np.linalg.norm(a["U"])
