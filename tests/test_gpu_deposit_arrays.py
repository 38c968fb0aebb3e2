"""The tiled FP64 deposit (ParticlesGridify.f90:65-123) at the edges of its
chunks: particle counts around a warp's 64, boxes that do not fit a warp's tile
(no order, far particles, rows that a chunk straddles), positions on cell
boundaries and faces, arrays that do not start on 16 bytes, and open and
periodic folds.

Bar: N within 1e-11 (of the largest value, C within 1e-12) of a float64 sum in numpy of
the same CIC weights, whose own error is the 2^-40 rounding of each weight;
and the F64 layout's ParticlesGridify equal bit for bit to the N of its
ParticlesGridifyAll, which sums the same fixed-point weights another way."""
import ctypes as C

import numpy as np
import pytest

from picard_b200 import capi
from picard_b200.simulation import Simulation
from tests.test_gpu_deposit_tiles import _plasma

pytestmark = pytest.mark.gpu


def _numpy_deposit(p, rp, ip):
    n, lo = (p.nx, p.ny, p.nz), (p.Lx_min, p.Ly_min, p.Lz_min)
    flow = (p.xflow, p.yflow, p.zflow)
    node, frac = [], []
    for a in range(3):
        t = (rp[:, a] - lo[a]) / p.dxyz[a] + 0.5
        node.append(np.floor(t).astype(np.int64))
        frac.append(t - np.floor(t))
    acc = np.zeros((p.species, p.nz + 2, p.ny + 2, p.nx + 2))
    for q in range(8):
        w, idx = 1.0, []
        for a in range(3):
            up = q >> a & 1
            w = w * (frac[a] if up else 1.0 - frac[a])
            i = node[a] + up
            idx.append(np.clip(i, 1, n[a]) if flow[a] else (i - 1) % n[a] + 1)
        np.add.at(acc, (ip - 1, idx[2], idx[1], idx[0]), w)
    return acc


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("dims,n,far,flows", [
    ((7, 6, 5), 1, 0.0, (1, 1, 1)),
    ((7, 6, 5), 63, 0.0, (1, 0, 1)),
    ((7, 6, 5), 65, 1.0, (1, 1, 1)),
    ((33, 9, 4), 4099, 0.02, (0, 1, 1)),
    ((40, 36, 30), 200001, 0.0, (1, 1, 0)),
    ((60, 50, 40), 150000, 1.0, (0, 0, 1)),
])
def test_deposit_of_fp64_positions(dims, n, far, flows, shift):
    import torch

    p, rp, ip = _plasma(*dims, 4, n, seed=n % 89, far=far, flows=flows)
    if n > 100:  # cell boundaries, base-node boundaries and faces
        rp[0:30, 0] = p.Lx_min + p.dxyz[0] * (np.arange(30) % p.nx)
        rp[30:60, 1] = p.Ly_min + p.dxyz[1] * (np.arange(30) % p.ny + 0.5)
        rp[60, :3] = [p.xmin, p.ymin, p.zmin]
        rp[61, :3] = [p.xmax, p.ymax, p.zmax]
    want = _numpy_deposit(p, rp, ip)
    # arrays of another owner, shifted by one element: 8- instead of 16-byte alignment
    dev = torch.device("cuda", 0)
    cols = [torch.zeros(n + 1, dtype=torch.float64, device=dev)[shift:shift + n] for _ in range(3)]
    for a in range(3):
        cols[a].copy_(torch.from_numpy(rp[:, a].copy()))
    sp = torch.zeros(n + 1, dtype=torch.int32, device=dev)[shift:shift + n]
    sp.copy_(torch.from_numpy(ip))
    nodes = p.nodes
    N = torch.full((nodes * p.species,), float("nan"), dtype=torch.float64, device=dev)
    Cg = torch.full((nodes,), float("nan"), dtype=torch.float64, device=dev)
    stream = torch.cuda.current_stream(dev).cuda_stream
    capi.check(capi.lib().picard_gpu_particles_gridify_noalloc(
        C.byref(p), *(c.data_ptr() for c in cols), sp.data_ptr(), n, N.data_ptr(), Cg.data_ptr(), C.c_void_p(stream)),
        "picard_gpu_particles_gridify_noalloc")
    torch.cuda.synchronize(dev)
    got = N.cpu().numpy().reshape(p.nz + 2, p.ny + 2, p.nx + 2, p.species)
    inner = (slice(1, -1),) * 3
    for s in range(p.species):
        w = want[s][inner] * p.n2p[s]
        assert np.abs(got[inner + (s,)] - w).max() <= 1e-11 * p.n2p[s] * max(1.0, want[s].max())
    charge = sum(p.charge[s] * got[..., s] for s in range(p.species))
    scale = max(abs(p.charge[s]) * np.abs(got[..., s]).max() for s in range(p.species))
    assert np.abs(Cg.cpu().numpy().reshape(charge.shape) - charge).max() <= 1e-12 * scale
    if shift == 0:
        with Simulation(p, derive=False, layout=capi.LAYOUT_F64, solver=capi.SOLVER_SPECTRAL) as g:
            g.set_particles(rp, ip)
            g.particles_gridify()
            N_tile = g.field(capi.FIELD_N)
            g.particles_gridify_all()
            np.testing.assert_array_equal(N_tile, g.field(capi.FIELD_N))
