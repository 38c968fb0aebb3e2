"""Fields read where the host has no pinned memory left for their pieces: they come
back through pageable memory, every bit of them, as they do with it.

A child process is started with a cudaHostAlloc that returns an error for large
blocks, as the driver's does when pinned memory has run out; nothing on the device
fails."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int refused = 0;
int cudaHostAlloc(void** p, size_t n, unsigned flags) {
  if (n >= (1u << 20)) {
    __atomic_add_fetch(&refused, 1, __ATOMIC_RELAXED);
    *p = 0;
    return 2;  /* cudaErrorMemoryAllocation */
  }
  void* rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  int (*real)(void**, size_t, unsigned) = rt ? (int (*)(void**, size_t, unsigned))dlsym(rt, "cudaHostAlloc") : 0;
  return real ? real(p, n, flags) : 2;
}
"""

CHILD = r"""
import ctypes
import numpy as np
from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.test_gpu_spectral import boxed
for dims in ((1, 2, 3), (80, 79, 80), (150, 70, 60)):
    rng = np.random.default_rng(sum(dims))
    with Simulation(boxed(*dims), derive=False, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL) as g:
        for which in (capi.FIELD_U, capi.FIELD_E, capi.FIELD_N, capi.FIELD_F, capi.FIELD_C):
            a = rng.standard_normal(g._shape(which))
            g.set_field(which, a)
            np.testing.assert_array_equal(g.field(which), a)
print("refused", ctypes.c_int.in_dll(ctypes.CDLL(None), "refused").value)
"""


def test_fields_without_pinned_memory(tmp_path):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    run = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    assert int(run.stdout.split()[-1]) >= 15  # every field's pieces met the refusal
