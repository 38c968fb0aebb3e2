"""The work that users of picard_b200 have it do, as cases that can be timed and compared.

The framework advances particle-in-cell runs: a user's program builds a run from its parameter block, advances it some
steps and reads its potential and densities.  So most cases are stretches of the main loop, each pass a few steps and the
read of the fields that follows them, over the range of grids, densities, layouts, solvers and boundary conditions that
the workloads of this repository span: the smallest served request (where launches and host round trips count), the 32^3
plain workload in both particle layouts, the reference's own default parameters, ragged and periodic boxes, the runs of
the serving stream and of the batched sweep, and the at-scale plasma of 268 million particles.  Two more are single
layers on inputs of their own: the open-boundary Poisson solve of a given charge, and the deposit of particles that the
caller holds on the device.

A loop case returns U and N of the whole grid, the particle count, the Jacobi sweeps and, where the program logs them, the
energies.  Each pass goes on from where the pass before it ended, as a run does.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from picard_b200 import capi
from picard_b200 import params as P
from picard_b200.simulation import Simulation, batch_run_fused

WARM_STEPS = 4  # steps behind a run before its first timed pass: its species have separated, its plans exist

LAYOUTS = {"cell32": capi.LAYOUT_CELL32, "f64": capi.LAYOUT_F64}
SOLVERS = {"spectral": capi.SOLVER_SPECTRAL, "refine": capi.SOLVER_F32_REFINE, "f64": capi.SOLVER_F64}


def _loop(name, plasma, nx, ny, nz, ppc, steps, **more):
    case = {"name": name, "kind": "loop", "plasma": plasma, "nx": nx, "ny": ny, "nz": nz, "ppc": ppc, "steps": steps,
            "loop": "fused", "layout": "cell32", "solver": "spectral", "tensor": False, "xflow": True, "yflow": True,
            "zflow": True, "sort_every": 0}
    case.update(more)
    return case


def listed():
    return [
        # A whole small request of the serving stream: context, distance table, plasma, steps, fields, release.  24^3
        # at 8 particles per cell is the smallest run of that stream; host work and launches decide it.
        {"name": "request_24", "kind": "request", "n": 24, "ppc": 4, "steps": 20},
        # The smallest run of the batched sweep (16^3) on its own, its fields looked at every few steps.
        _loop("small_16", "plain", 16, 16, 16, 4, 10),
        # The 32^3 plain workload, fused loop: 1.05 million particles, everything in L2.
        _loop("plain_32", "plain", 32, 32, 32, 16, 20),
        # The same workload in the reference's arithmetic: FP64 particles, FP64 sweeps, the direct boundary sum, one
        # call per subroutine with the energy log.
        _loop("plain_32_f64", "plain", 32, 32, 32, 16, 4, loop="calls", layout="f64", solver="f64"),
        # The reference's own default parameters (30^3, 128 particles per cell, electron mass, a neutral source):
        # particles cross cells every few steps, and the loop is called as the Fortran program calls it.
        _loop("default_30", "default", 30, 30, 30, 64, 10, loop="calls"),
        # A ragged box with periodic sides, as a solar-wind box has them: inflow and outflow along x only.
        _loop("periodic_60x36x30", "plain", 60, 36, 30, 12, 10, yflow=False, zflow=False),
        # The FP32 sweeps under FP64 anchors (the solver of Simulation's default) with the tensor-core boundary.
        _loop("refine_48x40x33", "plain", 48, 40, 33, 8, 2, solver="refine", tensor=True),
        # A middling run of the serving stream on an odd grid, sorted by cell now and then as long runs are.
        _loop("haser_77_sorted", "haser", 77, 77, 77, 13, 10, sort_every=10),
        # Runs of the batched parameter sweep, advanced together.
        {"name": "batch_16_runs", "kind": "batch", "runs": 16, "steps": 10},
        # The open-boundary Poisson solve of a given charge: boundary potential and Jacobi iterate.
        {"name": "poisson_120x72x56", "kind": "poisson", "nx": 120, "ny": 72, "nz": 56, "blobs": 32},
        # The deposit of particles that another runtime holds on the device, FP64 positions.
        {"name": "deposit_arrays_64", "kind": "deposit", "nx": 64, "ny": 64, "nz": 64, "particles": 8000000,
         "yflow": True},
        # The at-scale plasma with its Haser source: 268 million particles, 7.8 GB of them.
        _loop("scale_256x128x128", "haser", 256, 128, 128, 32, 20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, and sizes spread over the range that the workloads of that kind have."""
    kind = rng.choice(["request", "small", "fused", "fused", "haser", "calls", "f64", "periodic", "refine", "batch",
                       "poisson", "deposit"])
    if kind == "request":
        return {"kind": "request", "n": rng.randint(24, 56), "ppc": rng.randint(4, 12), "steps": rng.randint(8, 24)}
    if kind == "batch":
        return {"kind": "batch", "runs": rng.randint(4, 20), "steps": rng.randint(4, 12)}
    if kind == "poisson":
        return {"kind": "poisson", "nx": _log_int(rng, 20, 200), "ny": _log_int(rng, 20, 140),
                "nz": _log_int(rng, 20, 140), "blobs": rng.randint(4, 40)}
    if kind == "deposit":
        return {"kind": "deposit", "nx": rng.randint(17, 96), "ny": rng.randint(17, 96), "nz": rng.randint(17, 96),
                "particles": _log_int(rng, 100_000, 16_000_000) | 1, "yflow": rng.random() < 0.7}
    if kind == "small":
        return _named(rng, "plain", _log_int(rng, 16, 24), rng.randint(2, 6), rng.randint(6, 20))
    if kind == "fused":
        return _named(rng, "plain", _log_int(rng, 24, 128), rng.randint(4, 16), rng.randint(4, 16))
    if kind == "haser":
        return _named(rng, "haser", _log_int(rng, 24, 128), rng.randint(4, 32), rng.randint(4, 12),
                      sort_every=rng.choice([0, 4]))
    if kind == "calls":
        return _named(rng, rng.choice(["plain", "haser"]), _log_int(rng, 24, 72), rng.randint(4, 16),
                      rng.randint(3, 8), loop="calls")
    if kind == "f64":
        return _named(rng, "plain", _log_int(rng, 16, 36), rng.randint(4, 16), rng.randint(2, 4), loop="calls",
                      layout="f64", solver=rng.choice(["f64", "spectral"]))
    if kind == "periodic":
        return _named(rng, "plain", _log_int(rng, 24, 80), rng.randint(4, 16), rng.randint(4, 10),
                      yflow=rng.random() < 0.5, zflow=False)
    return _named(rng, "plain", _log_int(rng, 24, 56), rng.randint(4, 12), 2, solver="refine", tensor=True)


def _named(rng, plasma, n, ppc, steps, **more):
    """A box of about n^3 cells with uneven edges."""
    nx, ny, nz = (max(8, int(n * rng.uniform(0.8, 1.2))) for _ in range(3))
    case = _loop("", plasma, nx, ny, nz, ppc, steps, **more)
    del case["name"]
    return case


# ------------------------------------------------------------------ inputs


def _box(p, nx, ny, nz, cell=1000.0):
    p.nx, p.ny, p.nz = nx, ny, nz
    p.xmin, p.xmax = -0.5 * cell * nx, 0.5 * cell * nx
    p.ymin, p.ymax = -0.5 * cell * ny, 0.5 * cell * ny
    p.zmin, p.zmax = -0.5 * cell * nz, 0.5 * cell * nz


def _capacity(nx, ny, nz, ppc):
    """Room for the plasma, the inflow candidates of every face and what a neutral source adds over a long run."""
    face = 2 * ((ny + 2) * (nz + 2) + (nx + 2) * (nz + 2) + (nx + 2) * (ny + 2))
    return int(nx * ny * nz * ppc * 2 * 1.1 + 4 * face * ppc + 500_000)


def _solar_wind(p, seed):
    """Drift and field of one run of a sweep: 300..800 km/s along x, 1..10 nT in a random direction."""
    r = random.Random(seed)
    v = r.uniform(300e3, 800e3)
    for s in range(8):
        p.v0[s][0] = v
    u = [r.gauss(0.0, 1.0) for _ in range(3)]
    b = r.uniform(1e-9, 10e-9) / math.sqrt(sum(c * c for c in u))
    for d in range(3):
        p.B0[d] = b * u[d]


def _params(plasma, nx, ny, nz, ppc, seed):
    cap = _capacity(nx, ny, nz, ppc)
    if plasma == "default":
        p = capi.params_default()
        cell = (p.xmax - p.xmin) / p.nx
        _box(p, nx, ny, nz, cell)
        p.ppc[1] = ppc
        p.seed = seed
        p.max_per_proc = 4 * cap
        return p
    if plasma == "haser":
        p = P.config_plain_scale(seed=seed, nx=nx, ny=ny, nz=nz, ppc_ion=ppc, capacity=cap)
        p.Qn[2] = 10.0 ** random.Random(seed).uniform(25.0, 28.0)
    else:
        p = P.config_plain_32(seed=seed, n=8, ppc=ppc, capacity=cap)
        _box(p, nx, ny, nz)
    _solar_wind(p, seed)
    return p


def _start(p, layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL):
    sim = Simulation(p, layout=layout, solver=solver)
    sim.calc_distance()
    sim.particles_initialize()
    return sim


def prepare(case, seed):
    if torch.cuda.is_available():
        # contexts come and go: freed device memory stays in the pool, as in the serving loop
        capi.pool_keep(torch.cuda.current_device(), 32 << 30)
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_request(case, seed):
    n = case["n"]
    return {"kind": "request", "params": capi.params_derive(_params("haser", n, n, n, case["ppc"], seed)),
            "steps": case["steps"]}


def _prepare_loop(case, seed):
    p = _params(case["plasma"], case["nx"], case["ny"], case["nz"], case["ppc"], seed)
    p.xflow, p.yflow, p.zflow = int(case["xflow"]), int(case["yflow"]), int(case["zflow"])
    sim = Simulation(p, layout=LAYOUTS[case["layout"]], solver=SOLVERS[case["solver"]])
    if case["tensor"]:
        sim.set_option(capi.OPT_BCPOT_TENSOR, 1)
    sim.set_option(capi.OPT_SORT_EVERY, case["sort_every"])
    sim.calc_distance()
    sim.particles_initialize()
    if case["loop"] == "calls":
        sim.run(0, WARM_STEPS)
    else:
        sim.run_fused(0, WARM_STEPS)
    return {"kind": "loop", "sim": sim, "at": WARM_STEPS, "steps": case["steps"], "loop": case["loop"]}


def _batch_params(case, seed):
    # grids and densities belong to the case, the plasma to the seed
    shapes = random.Random(1000 * case["runs"] + case["steps"])
    out = []
    for r in range(case["runs"]):
        n, ppc = shapes.randint(16, 96), shapes.randint(4, 16)
        out.append((n, ppc, _params("plain", n, n, n, ppc, 1000 * seed + r)))
    return out


def _prepare_batch(case, seed):
    sims = [_start(p) for _, _, p in _batch_params(case, seed)]
    batch_run_fused(sims, 0, WARM_STEPS)
    return {"kind": "batch", "sims": sims, "at": WARM_STEPS, "steps": case["steps"]}


def _charge(case, seed):
    """Gaussian blobs of charge (sigma 4..16 cells, amplitudes N(0, 1) e per cell) and 1% noise, zero on the ghosts."""
    rng = np.random.default_rng(seed)
    dims = (case["nz"], case["ny"], case["nx"])
    C = np.zeros([n + 2 for n in dims])
    for _ in range(case["blobs"]):
        s, a = rng.uniform(4, 16), rng.standard_normal()
        g = [np.exp(-0.5 * ((np.arange(n + 2) - rng.uniform(1, n)) / s) ** 2) for n in dims]
        C += a * g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
    C += 0.01 * rng.uniform(-1, 1, C.shape)
    C[0] = C[-1] = C[:, 0] = C[:, -1] = C[:, :, 0] = C[:, :, -1] = 0.0
    return C * P.EC


def _poisson_params(case):
    p = P.config_plain_32(seed=0, n=8, ppc=1, capacity=1024)
    _box(p, case["nx"], case["ny"], case["nz"])
    return p


def _prepare_poisson(case, seed):
    sim = Simulation(_poisson_params(case), layout=capi.LAYOUT_CELL32, solver=capi.SOLVER_SPECTRAL)
    sim.calc_distance()
    sim.set_field(capi.FIELD_C, _charge(case, seed))
    sim.bc_potentials()
    return {"kind": "poisson", "sim": sim}


def _deposit_params(case):
    p = P.config_plain_32(seed=0, n=8, ppc=32, capacity=1024)
    _box(p, case["nx"], case["ny"], case["nz"])
    p.yflow = int(case["yflow"])
    return capi.params_derive(p)


def _deposit_particles(case, seed, p):
    """Positions as a run holds them: created cell by cell, then carried a tenth of a cell or so, inside the domain."""
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    n, cells = case["particles"], case["nx"] * case["ny"] * case["nz"]
    cell = torch.div(torch.arange(n, device=dev) * cells, n, rounding_mode="floor")
    at = (cell % p.nx, torch.div(cell, p.nx, rounding_mode="floor") % p.ny,
          torch.div(cell, p.nx * p.ny, rounding_mode="floor"))
    lo, hi, d = (p.xmin, p.ymin, p.zmin), (p.xmax, p.ymax, p.zmax), p.dxyz
    pos = []
    for a in range(3):
        u = torch.rand(n, generator=gen, device=dev, dtype=torch.float64)
        g = torch.randn(n, generator=gen, device=dev, dtype=torch.float64)
        pos.append((lo[a] + (at[a] + u + 0.1 * g) * d[a]).clamp_(lo[a], hi[a]))
    species = (torch.arange(n, device=dev, dtype=torch.int32) % 2) + 1
    return pos, species


def _prepare_deposit(case, seed):
    p = _deposit_params(case)
    pos, species = _deposit_particles(case, seed, p)
    nodes = (p.nx + 2) * (p.ny + 2) * (p.nz + 2)
    return {"kind": "deposit", "params": p, "pos": pos, "species": species,
            "N": torch.empty(nodes * p.species, dtype=torch.float64, device=species.device),
            "C": torch.empty(nodes, dtype=torch.float64, device=species.device)}


# -------------------------------------------------------------------- a pass


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_request(state):
    with Simulation(state["params"], derive=False, solver=capi.SOLVER_SPECTRAL) as sim:
        sim.calc_distance()
        sim.particles_initialize()
        sweeps = sim.run_fused(0, state["steps"])
        return {"sweeps": sweeps, "num": sim.num_local, "U": sim.field(capi.FIELD_U), "N": sim.field(capi.FIELD_N)}


def _run_loop(state):
    sim, a, b = state["sim"], state["at"], state["at"] + state["steps"]
    if state["loop"] == "calls":
        log = []
        sweeps = sim.run(a, b, log_interval=1, log=lambda it, t, n, up, ue, ub: log.append((up, ue, ub)))
    else:
        log = None
        sweeps = sim.run_fused(a, b)
    state["at"] = b
    out = {"sweeps": sweeps, "num": sim.num_local, "U": sim.field(capi.FIELD_U), "N": sim.field(capi.FIELD_N)}
    if log is not None:
        out["energies"] = np.array(log)
    return out


def _run_batch(state):
    sims, a, b = state["sims"], state["at"], state["at"] + state["steps"]
    sweeps = batch_run_fused(sims, a, b)
    state["at"] = b
    return {"sweeps": np.array(sweeps), "num": np.array([s.num_local for s in sims]),
            "U": [s.field(capi.FIELD_U) for s in sims]}


def _run_poisson(state):
    sim = state["sim"]
    sim.bc_potentials()
    sweeps = sim.calc_epotential()
    return {"sweeps": sweeps, "U": sim.field(capi.FIELD_U)}


def _run_deposit(state):
    p, (x, y, z), sp, N, C = state["params"], state["pos"], state["species"], state["N"], state["C"]
    stream = torch.cuda.current_stream(sp.device).cuda_stream
    capi.check(capi.lib().picard_gpu_particles_gridify_noalloc(
        ctypes.byref(p), x.data_ptr(), y.data_ptr(), z.data_ptr(), sp.data_ptr(), sp.numel(), N.data_ptr(),
        C.data_ptr(), ctypes.c_void_p(stream)), "picard_gpu_particles_gridify_noalloc")
    return {"N": N, "C": C}


# --------------------------------------------------------------- least work


def _loop_work(nx, ny, nz, particles, species, steps, f64=False, open_axes=3):
    """One step reads every particle and writes its position and velocity; it builds C from the deposit, solves for U and
    E (an FFT-based solve: 5 N log2 N forward and back, twice for the doubled boundary convolutions) and gathers E."""
    cells = nx * ny * nz
    nodes = (nx + 2) * (ny + 2) * (nz + 2)
    per = 49 + 48 if f64 else 29 + 28
    lg = math.log2(max(2, cells))
    step_bytes = particles * per + nodes * (8 * species + 8 + 8 + 24)
    step_flops = particles * 140 + 10 * cells * lg + open_axes * 2 * 5 * cells * lg
    out = nodes * 8 * (species + 1)
    return {"bytes": steps * step_bytes + out, "flops": steps * step_flops}


def work(case):
    kind = case["kind"]
    if kind == "request":
        n = case["n"]
        return _loop_work(n, n, n, 2 * case["ppc"] * n ** 3, 3, case["steps"])
    if kind == "loop":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        species = 2 if case["plasma"] == "plain" else 3
        opened = int(case["xflow"]) + int(case["yflow"]) + int(case["zflow"])
        return _loop_work(nx, ny, nz, 2 * case["ppc"] * nx * ny * nz, species, case["steps"], case["layout"] == "f64",
                          opened)
    if kind == "batch":
        runs = [_loop_work(n, n, n, 2 * ppc * n ** 3, 2, case["steps"]) for n, ppc, _ in _batch_params(case, 0)]
        return {k: sum(r[k] for r in runs) for k in ("bytes", "flops")}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells, nodes = nx * ny * nz, (nx + 2) * (ny + 2) * (nz + 2)
    if kind == "poisson":
        lg = math.log2(cells)
        return {"bytes": 16 * nodes, "flops": 10 * cells * lg + 3 * 2 * 5 * cells * lg}
    return {"bytes": case["particles"] * 28 + 24 * nodes, "flops": case["particles"] * 40}


# ------------------------------------------------------------ 64-bit values


def exact(case, seed):
    if case["kind"] == "deposit":
        return _exact_deposit(case, seed)
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    return None  # a loop's plasma comes from the framework's own counter-based generator


def _exact_deposit(case, seed):
    p = _deposit_params(case)
    pos, species = _deposit_particles(case, seed, p)
    lo, n, flow = (p.Lx_min, p.Ly_min, p.Lz_min), (p.nx, p.ny, p.nz), (p.xflow, p.yflow, p.zflow)
    node, frac = [], []
    for a in range(3):
        t = (pos[a] - lo[a]) / p.dxyz[a] + 0.5
        node.append(t.floor().long())
        frac.append(t - t.floor())
    nxp, nyp, nzp = (v + 2 for v in n)
    acc = torch.zeros(p.species, nzp * nyp * nxp, dtype=torch.float64, device=species.device)
    for corner in range(8):
        w, idx = 1.0, []
        for a in range(3):
            up = corner >> a & 1
            w = w * (frac[a] if up else 1.0 - frac[a])
            i = node[a] + up  # ghosts fold onto the first or last node (open) or wrap (periodic)
            idx.append(i.clamp(1, n[a]) if flow[a] else (i - 1) % n[a] + 1)
        flat = idx[0] + nxp * (idx[1] + nyp * idx[2])
        for s in range(p.species):
            acc[s].index_add_(0, flat, torch.where(species == s + 1, w, torch.zeros_like(w)))
    acc = acc.reshape(p.species, nzp, nyp, nxp)
    for a in range(3):  # ghost layers: zero (open) or the opposite interior layer (periodic)
        dim = 3 - a
        first, last = acc.select(dim, 0), acc.select(dim, n[a] + 1)
        if flow[a]:
            first.zero_()
            last.zero_()
        else:
            first.copy_(acc.select(dim, n[a]))
            last.copy_(acc.select(dim, 1))
    N = torch.stack([acc[s] * p.n2p[s] for s in range(p.species)], dim=-1)
    C = sum(N[..., s] * p.charge[s] for s in range(p.species))
    return {"N": N.reshape(-1), "C": C.reshape(-1)}


def _face_potential(C, d, axis):
    """Potential on the two faces normal to `axis`, one node outside the box, of the charges C (z, y, x)."""
    n = C.shape
    t1, t2 = [a for a in range(3) if a != axis]
    L1, L2 = 2 * n[t1], 2 * n[t2]

    def circular(L, m, h):
        k = torch.arange(L, device=C.device, dtype=torch.float64)
        return torch.minimum(k, L - k) * h

    r2 = circular(L1, n[t1], d[t1])[:, None] ** 2 + circular(L2, n[t2], d[t2])[None, :] ** 2
    faces = [0.0, 0.0]
    for a in range(n[axis]):
        ch = torch.fft.rfft2(C.select(axis, a), s=(L1, L2))
        for f, off in enumerate((a + 1, n[axis] - a)):
            faces[f] = faces[f] + ch * torch.fft.rfft2(1.0 / torch.sqrt(r2 + (off * d[axis]) ** 2))
    scale = 1.0 / (2.0 * P.TAU * P.EPS0)
    return [scale * torch.fft.irfft2(f, s=(L1, L2))[:n[t1], :n[t2]] for f in faces]


def _exact_poisson(case, seed):
    p = capi.params_derive(_poisson_params(case))
    dev = torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")
    C = torch.from_numpy(_charge(case, seed)).to(dev)
    d = (p.dxyz[2], p.dxyz[1], p.dxyz[0])
    inner = C[1:-1, 1:-1, 1:-1]
    n = inner.shape
    U = torch.zeros_like(C)
    for axis in range(3):
        lo, hi = _face_potential(inner, d, axis)
        U.select(axis, 0)[1:-1, 1:-1] = lo
        U.select(axis, n[axis] + 1)[1:-1, 1:-1] = hi
    b = -inner / (d[0] * d[1] * d[2] * P.EPS0)
    inv2 = [1.0 / h ** 2 for h in d]
    af = 0.5 / sum(inv2)
    r0 = b.clone()  # the residual of the starting iterate: zero inside, the face potentials outside
    for axis in range(3):
        r0.select(axis, 0).sub_(inv2[axis] * U.select(axis, 0)[1:-1, 1:-1])
        r0.select(axis, n[axis] - 1).sub_(inv2[axis] * U.select(axis, n[axis] + 1)[1:-1, 1:-1])
    omega = torch.zeros_like(b)
    modes, rh = [], r0
    for axis in range(3):
        m = torch.arange(1, n[axis] + 1, dtype=torch.float64, device=dev)
        Q = math.sqrt(2.0 / (n[axis] + 1)) * torch.sin(math.pi / (n[axis] + 1)
                                                       * (m[:, None] * m[None, :] % (2 * (n[axis] + 1))))
        modes.append(Q)
        rh = torch.movedim(torch.tensordot(Q, rh, dims=([1], [axis])), 0, axis)
        om = af * inv2[axis] * 4.0 * torch.sin(0.5 * math.pi * m / (n[axis] + 1)) ** 2
        omega = omega + om.reshape([-1 if a == axis else 1 for a in range(3)])
    g = 1.0 - omega
    tol2 = p.maxerr ** 2 * float((b * b).sum())
    lg2, rh2 = 2.0 * torch.log(g.abs()), rh * rh

    def norm2(k):
        return float((rh2 * torch.exp(k * lg2)).sum())

    hi = 1  # ||residual|| does not grow with the sweeps: double, then halve
    while norm2(hi) > tol2 and hi < p.maxit - 1:
        hi *= 2
    lo = hi // 2
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if norm2(mid) <= tol2 else (mid, hi)
    small = -torch.expm1(hi * torch.log1p(-omega.clamp(max=0.999999)))
    gd = torch.exp(0.5 * hi * lg2) * (torch.where(g < 0, -1.0, 1.0) if hi % 2 else 1.0)
    sol = -af * torch.where(omega < 0.5, small, 1.0 - gd) / omega * rh
    for axis in range(3):
        sol = torch.movedim(torch.tensordot(modes[axis].T, sol, dims=([1], [axis])), 0, axis)
    U[1:-1, 1:-1, 1:-1] += sol
    return {"sweeps": None, "U": U}
