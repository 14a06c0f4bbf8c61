"""What is timed on this framework: its work as a user's program has it done, from the smallest
gas cell to the largest, in both precision forms, alone and batched, with ions, through the host
entry point and through the MATLAB-signature drop-ins.

Each pass starts from the same population and fields (a segment of a run: load, step, read back),
so a pass does the same work however often it is repeated.  The order of electrons in memory after a
sort is arbitrary, so they are returned by identity, as a program that follows them needs them: the
loaded ones in the rows of their ids (zeros for one that has left), the secondaries in the order of
theirs, in a fixed number of rows.  The FP32 split form's values are returned in its own precision.

exact() restates the physics in 64 bits with torch alone: the axisymmetric Yee sub-cycle, the
Boris push, the shell deposit, the Philox draws and the null-collision Monte Carlo, and for the
drop-ins the reference kernels' arithmetic.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "gas-atenuator_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

QE, ME, CC, KB = 1.602176634e-19, 9.1093837015e-31, 299792458.0, 1.380649e-23
EPS0, MU0, M_ION = 8.8541878128e-12, 1.25663706212e-6, 28.0134 * 1.66053906660e-27
GRIDS = ((64, 256), (128, 512), (256, 1024), (512, 2048))


def cell(kind, n_r, n_z, delta_um, dt_fs, torr, photo, e_kev, steps, fp32, sort=20, ratio=1,
         gas_map=False, ions=0):
    """One gas cell: grid, time step, pressure, photoionizations (two electrons each)."""
    return dict(kind=kind, n_r=n_r, n_z=n_z, delta_um=delta_um, dt_fs=dt_fs, torr=torr,
                photo=photo, e_kev=e_kev, steps=steps, fp32=fp32, sort=sort, ratio=ratio,
                gas_map=gas_map, ions=ions)


def listed():
    def named(name, c):
        return dict(c, name=name)
    return [
        # the smallest cell that is run in earnest (the checks' size): launches and latency only
        named("cell tiny fp32", cell("cell", 32, 64, 5.0, 10.0, 300.0, 2_000, 8.0, 40, True)),
        # the reference's CPU-runnable case, 20,000 electrons, in the plain FP64 form
        named("cell 64x256 fp64", cell("cell", 64, 256, 10.0, 20.0, 1.0, 10_000, 8.0, 100, False)),
        # an odd grid, a ragged population and a per-cell gas density
        named("cell 151x333 fp32", cell("cell", 151, 333, 10.0, 20.0, 30.0, 150_077, 12.0, 60, True,
                                        gas_map=True)),
        # the headline: 2,000,000 electrons on 256 x 1024 cells, in both forms
        named("cell 256x1024 fp32", cell("cell", 256, 1024, 5.0, 10.0, 1.0, 1_000_000, 8.0, 60, True,
                                         sort=30)),
        named("cell 256x1024 fp64", cell("cell", 256, 1024, 5.0, 10.0, 1.0, 1_000_000, 8.0, 60, False,
                                         sort=30)),
        # the single large cascade: 16M electrons on 1024 x 4096 cells at 10 Torr
        named("cell 1024x4096 fp32", cell("cell", 1024, 4096, 5.0, 10.0, 10.0, 8_000_000, 12.0, 30,
                                          True, sort=30)),
        # electrons with N2+ ions, a run in its middle: two ion sub-cycles
        named("ions 256x1024 fp32", cell("cell", 256, 1024, 10.0, 20.0, 5.0, 1_000_000, 8.0, 100,
                                         True, sort=30, ions=1_000_000)),
        # a sweep of uneven cells stepped as one batch, both forms
        named("batch 16 fp32", dict(kind="batch", cells=16, law=2, photo_max=1_000_000, steps=50,
                                    fp32=True, sort=30)),
        named("batch 6 fp64", dict(kind="batch", cells=6, law=5, photo_max=300_000, steps=50,
                                   fp32=False, sort=30)),
        # a MATLAB host's outer step: pinned host arrays in and out
        named("host 256x1024 fp64", cell("host", 256, 1024, 5.0, 10.0, 1.0, 200_000, 8.0, 100, False)),
        # the MATLAB driver's functions: 20 particle steps of electricmagneticfield6 on its
        # 100 x 500 grid, and find_CS0 with electron_collision
        named("em6 100x500", dict(kind="em6", n_r=100, n_z=500, n_e=200_000, n_i1=50_000,
                                  n_i2=10_001, cycle=100, faithful=True)),
        named("collision 200k", dict(kind="collision", n=200_003, rmax=25, zmax=50, faithful=True)),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["cell", "cell", "cell", "cell", "ions", "batch", "host", "em6", "collision"])
    fp32 = rng.random() < 0.65
    if kind in ("cell", "ions", "host"):
        n_r, n_z = logint(20, 1024), logint(40, 4096)
        photo = logint(1_000, 4_000_000 if kind == "cell" else 500_000)
        steps = logint(10, 150)
        if photo * steps > 100_000_000:
            steps = max(10, 100_000_000 // photo)
        d = rng.choice([5.0, 10.0])
        return cell("host" if kind == "host" else "cell", n_r, n_z, d, 2 * d,
                    math.exp(rng.uniform(math.log(0.1), math.log(30.0))), photo,
                    rng.uniform(2.0, 20.0), steps, fp32 and kind != "host", sort=rng.choice([10, 20, 30, 40]),
                    ratio=rng.choice([1, 1, 1, 1, 1, 2]) if kind == "cell" else 1,
                    gas_map=rng.random() < 0.25,
                    ions=logint(10_000, 1_000_000) if kind == "ions" else 0)
    if kind == "batch":
        return dict(kind="batch", cells=rng.randint(2, 20), law=rng.randint(10, 10_000_000),
                    photo_max=logint(30_000, 500_000), steps=logint(10, 60), fp32=fp32,
                    sort=rng.choice([20, 30]))
    if kind == "em6":
        return dict(kind="em6", n_r=logint(16, 200), n_z=logint(40, 1000), n_e=logint(1_000, 600_000),
                    n_i1=logint(1, 200_000), n_i2=rng.choice([0, 1, 5_000, 20_011]),
                    cycle=5 * logint(2, 40), faithful=rng.random() < 0.7)
    return dict(kind="collision", n=logint(1_000, 2_000_000), rmax=rng.randint(10, 60),
                zmax=rng.randint(5, 100), faithful=rng.random() < 0.6)


# ------------------------------------------------------------------ inputs
def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class Draws:
    """Seeded random arrays made on the device."""

    def __init__(self, seed):
        self.dev = device()
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(int(seed))

    def u(self, *shape):
        return torch.rand(*shape, generator=self.g, device=self.dev, dtype=torch.float64)

    def n(self, *shape):
        return torch.randn(*shape, generator=self.g, device=self.dev, dtype=torch.float64)


def u_of_ev(ev):
    e = ev * QE / (ME * CC * CC)
    return CC * math.sqrt(e * (2 + e))


def births(R, n, e_kev, Rp, Lp, id_base=0):
    """Per photon a dipole photoelectron (photon energy minus 410 eV) and an isotropic 360 eV Auger
    electron at a Rayleigh(50 um) radius (at most 0.99 of the wall's), uniform azimuth and z: r, z, the local
    (r, theta, z) components of gamma v, id."""
    r = torch.clamp(50e-6 * torch.sqrt(-2 * torch.log1p(-R.u(n))), max=0.99 * Rp)
    z = R.u(n) * Lp
    phi = 2 * math.pi * R.u(n)
    x = 2 * R.u(n) - 1
    mu = torch.sign(x) * torch.abs(x) ** (1.0 / 3)
    psi = 2 * math.pi * R.u(n)
    s = torch.sqrt(torch.clamp(1 - mu * mu, min=0))
    ct = 2 * R.u(n) - 1
    pa = 2 * math.pi * R.u(n)
    st = torch.sqrt(torch.clamp(1 - ct * ct, min=0))
    cp, sp = torch.cos(phi), torch.sin(phi)
    out = torch.empty(5, n, 2, dtype=torch.float64, device=R.dev)
    out[0], out[1] = r[:, None], z[:, None]
    for k, (mag, d) in enumerate(((u_of_ev(1000 * e_kev - 410), (mu, s * torch.cos(psi), s * torch.sin(psi))),
                                  (u_of_ev(360.0), (st * torch.cos(pa), st * torch.sin(pa), ct)))):
        out[2, :, k] = mag * (d[0] * cp + d[1] * sp)
        out[3, :, k] = mag * (-d[0] * sp + d[1] * cp)
        out[4, :, k] = mag * d[2]
    ids = torch.arange(2 * n, device=R.dev, dtype=torch.int64) + id_base
    return [out[k].reshape(-1).contiguous() for k in range(5)] + [ids]


def smooth(R, ncol, nrow, amp):
    """A smooth field as MATLAB holds an ncol x nrow matrix (rows of the tensor: its columns)."""
    i = torch.arange(ncol, device=R.dev, dtype=torch.float64)[None, :] / ncol
    j = torch.arange(nrow, device=R.dev, dtype=torch.float64)[:, None] / nrow
    k = R.u(4, 5)
    f = torch.zeros(nrow, ncol, device=R.dev, dtype=torch.float64)
    for q in range(4):
        a, b, c, d, e = (k[q, m] for m in range(5))
        f += (2 * a - 1) * torch.sin(math.pi * (b * 3 * i + c)) * torch.cos(math.pi * (d * 3 * j + e))
    return (amp * f).contiguous()


def grid_fields(R, n_r, n_z, e0, h0):
    er, ez, h = smooth(R, n_r, n_z + 1, e0), smooth(R, n_r + 1, n_z, e0), smooth(R, n_r, n_z, h0)
    er[0], er[-1] = 0, 0                     # conducting ends and wall
    ez[:, -1] = 0
    return er, ez, h


def batch_cells(case):
    """The cells of a batch: pressure log-uniform in 0.1-10 Torr, one of four grids at 10 um, photon
    energy uniform in 2-20 keV, photoionizations log-uniform from 10,000."""
    rng = np.random.default_rng(case["law"])
    cells = []
    for _ in range(case["cells"]):
        n_r, n_z = GRIDS[rng.integers(len(GRIDS))]
        torr, e_kev = float(10 ** rng.uniform(-1, 1)), float(rng.uniform(2, 20))
        photo = int(round(10 ** rng.uniform(4, math.log10(case["photo_max"]))))
        cells.append(cell("cell", n_r, n_z, 10.0, 20.0, torr, photo, e_kev, case["steps"],
                          case["fp32"], sort=case["sort"]))
    return cells


def cell_inputs(c, seed, id_base=0):
    R = Draws(seed)
    n_r, n_z, d = c["n_r"], c["n_z"], c["delta_um"] * 1e-6
    inp = dict(parts=births(R, c["photo"], c["e_kev"], n_r * d, n_z * d, id_base),
               fields=grid_fields(R, n_r, n_z, 1e6, 1e3), gas=None, ions=None)
    rho = c["torr"] * 133.322368 / (KB * 300.0)
    inp["rho"] = rho
    if c["gas_map"]:
        inp["gas"] = rho * (0.25 + R.u(n_z, n_r))
    if c["ions"]:
        n, sig = c["ions"], math.sqrt(KB * 300.0 / M_ION)
        p = births(R, (n + 1) // 2, 1.0, n_r * d, n_z * d)
        inp["ions"] = [a[:n].contiguous() for a in p[:2]] + [sig * R.n(n) for _ in range(3)] + \
            [torch.arange(n, device=R.dev, dtype=torch.int64) + (1 << 40),
             (R.u(n) < 0.1).to(torch.int8) + 1]
    return inp


def wedge_inputs(case, seed):
    """Macro-particles in a 0.1 rad wedge of 1 cm radius, as the MATLAB driver holds them."""
    R = Draws(seed)
    PHIp, Rp = 0.1, 1e-2

    def species(n, Lp, vmag, cyl):
        r, phi, z = Rp * (0.02 + 0.96 * R.u(n)), PHIp * (0.02 + 0.96 * R.u(n)), Lp * (0.02 + 0.96 * R.u(n))
        d = R.n(n, 3)
        d = d / torch.linalg.norm(d, dim=1, keepdim=True)
        v = vmag * (0.3 + 0.7 * R.u(n, 1)) * d
        pos = [r, phi, z] if cyl else [r * torch.cos(phi), r * torch.sin(phi), z]
        return torch.stack(pos, 1), v

    if case["kind"] == "em6":
        n_r, n_z = case["n_r"], case["n_z"]
        delta = Rp / n_r
        Lp = n_z * delta
        f = grid_fields(R, n_r, n_z, 3e5, 300.0)
        return dict(e=species(case["n_e"], Lp, 4e7, True), i1=species(case["n_i1"], Lp, 2e3, True),
                    i2=species(case["n_i2"], Lp, 2e3, True), fields=[a.t() for a in f],
                    delta=delta, Rp=Rp, Lp=Lp, PHIp=PHIp, dt=1e-13 * 100 / n_r, FN=1e4)
    n, rmax, zmax, Lp = case["n"], case["rmax"], case["zmax"], 0.05
    delta = Rp / rmax
    k = np.arange(1, rmax + 1)
    phimax = np.ceil(k / rmax * Rp * PHIp / delta)
    sum_cell = np.cumsum(phimax)
    xy = int(sum_cell[-1])
    pos, v = species(n, Lp, 1.0, False)
    # the reference compares keV with ln(keV): above 2.5 keV its table search leaves the table
    ev = torch.exp(math.log(20.0) + R.u(n) * math.log((2500.0 if case["faithful"] else 8000.0) / 20.0))
    g = 1 + ev * 1.6022e-19 / (9.109e-31 * 9e16)
    v = v / torch.linalg.norm(v, dim=1, keepdim=True) * (3e8 * torch.sqrt(1 - 1 / g ** 2))[:, None]
    return dict(pos=pos, vel=v, kin=ev / 1000, sum_cell=sum_cell, phimax=phimax, xy=xy,
                density=3.2e22 * (0.5 + R.u(xy * zmax)), temperature=300 * (0.8 + 0.4 * R.u(xy * zmax)),
                PHIp=PHIp, dr=delta, dz=Lp / zmax, ion_pos=1e-3 * R.u(1000, 3), ion_vel=500 * R.n(1000, 3),
                draws=torch.cat([R.u(n, 4), R.n(n, 3).float().double(), torch.zeros_like(R.u(n, 1))], 1),
                dt=1e-10)


def rows_of(c):
    """Rows for a cell's electrons: room for the ionization cascade of its steps."""
    n = 2 * c["photo"]
    return int(n * math.exp(8e-6 * c["torr"] * c["steps"] * c["dt_fs"])) + 4096


def pad(a, rows):
    """The rows of `a` (its last dimension) in a fixed number of them."""
    if a.shape[-1] > rows:
        raise ValueError(f"{a.shape[-1]} rows, and room for {rows}")
    return torch.nn.functional.pad(a, (0, rows - a.shape[-1]))


# ----------------------------------------------------------------- prepare
def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def make_sim(c, inp, seed, ctx=None):
    from gasatt import abi
    from gasatt.sim import Sim
    from gasatt.workload import config
    n = 2 * c["photo"]
    cap = rows_of(c) + n
    cfg = config(c["n_r"], c["n_z"], c["delta_um"] * 1e-6, c["dt_fs"] * 1e-15, c["torr"],
                 precision=abi.FP32_SPLIT if c["fp32"] else abi.FP64, capacity=cap, seed=seed,
                 sort_period=c["sort"], fdtd_ratio=c["ratio"],
                 ion_capacity=c["ions"] + rows_of(c) - n if c["ions"] else 0)
    sim = Sim(cfg, ctx=ctx)
    sim.bind_stream()
    if inp["gas"] is not None:
        sim.set_gas_density(inp["gas"].t().cpu().numpy())
    return sim


def out_buffers(cap):
    f = torch.empty(5, cap, dtype=torch.float64, device=device())
    return f, torch.empty(cap, dtype=torch.int64, device=device())


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("em6", "collision"):
        s = dict(case=case, inp=wedge_inputs(case, seed))
        if kind == "collision":
            from gasatt.tables import N2Tables
            s["tab"] = N2Tables()
        return s
    if kind == "batch":
        from gasatt.dropin import Context
        from gasatt.sim import Batch
        ctx = Context(0)
        ctx.bind_stream()
        cells = batch_cells(case)
        inps, sims = [], []
        for i, c in enumerate(cells):
            inps.append(cell_inputs(c, seed * 1000 + i, id_base=i << 32))
            sims.append(make_sim(c, inps[i], seed * 1000 + i, ctx))
        return dict(case=case, sims=sims, inps=inps, ctx=ctx, batch=Batch(sims, sort_period=case["sort"]),
                    out=[out_buffers(int(s.cfg.capacity)) for s in sims],
                    fields=[[torch.empty_like(f) for f in i["fields"]] for i in inps])
    inp = cell_inputs(case, seed)
    sim = make_sim(case, inp, seed)
    s = dict(case=case, sims=[sim], inps=[inp], out=[out_buffers(int(sim.cfg.capacity))],
             fields=[[torch.empty_like(f) for f in inp["fields"]]])
    if case["ions"]:
        s["ion_out"] = out_buffers(int(sim.cfg.ion_capacity))
        s["ion_q"] = torch.empty(int(sim.cfg.ion_capacity), dtype=torch.int8, device=device())
    if kind == "host":
        # what a MATLAB host has: pinned n x 3 Cartesian arrays (leading dimension cap) and a copy
        # of them to start the next pass from
        r, z, ur, ut, uz, _ = inp["parts"]
        n, cap = r.numel(), int(sim.cfg.capacity)
        g = torch.sqrt(1 + (ur * ur + ut * ut + uz * uz) / CC ** 2)
        start = torch.zeros(6, n, dtype=torch.float64, device=r.device)
        start[0], start[2], start[3], start[4], start[5] = r, z, ur / g, ut / g, uz / g
        s["start"] = start.cpu().pin_memory()
        s["io"] = torch.zeros(6, cap, dtype=torch.float64).pin_memory()
        set_fields(sim, inp["fields"])
    return s


# --------------------------------------------------------------------- run
def set_fields(sim, f):
    from gasatt._lib import check, lib
    check(sim.ctx.handle, lib.gasatt_sim_set_fields(sim.h, ptr(f[0]), ptr(f[1]), ptr(f[2]), 1))


def get_fields(sim, f):
    from gasatt._lib import check, lib
    check(sim.ctx.handle, lib.gasatt_sim_get_fields(sim.h, ptr(f[0]), ptr(f[1]), ptr(f[2]), 1))


def read(sim, buf):
    """The live electrons after a sort (which drops the dead): 5 x n values and ids, on the device."""
    from gasatt._lib import check, lib
    f, ids = buf
    n = ctypes.c_int64()
    sim.sort()
    check(sim.ctx.handle, lib.gasatt_sim_read(sim.h, *[ptr(f[k]) for k in range(5)], ptr(ids),
                                              ids.numel(), ctypes.byref(n), 1))
    return f[:, :n.value], ids[:n.value]


def counts(d):
    return [d[k] for k in ("n_alive", "n_ionizations", "n_elastic", "n_excitation", "n_null",
                           "n_lost_wall", "n_ions", "status_flags")]


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "em6":
        return run_em6(state)
    if kind == "collision":
        return run_collision(state)
    if kind == "host":
        return run_host(state)
    sims, inps = state["sims"], state["inps"]
    for sim, inp in zip(sims, inps):
        sim.load(*inp["parts"])
        set_fields(sim, inp["fields"])
        if inp["ions"] is not None:
            from gasatt._lib import check, lib
            i = inp["ions"]
            check(sim.ctx.handle, lib.gasatt_sim_load_ions(sim.h, *[ptr(a) for a in i], i[0].numel(), 1))
    if kind == "batch":
        state["batch"].step(case["steps"])
    else:
        sims[0].step(case["steps"])
    dtype = torch.float32 if case["fp32"] else torch.float64
    diag = [sim.diag() for sim in sims]
    got = [read(sim, buf) for sim, buf in zip(sims, state["out"])]
    for sim, f in zip(sims, state["fields"]):
        get_fields(sim, f)
    out = electrons([g[0] for g in got], [g[1] for g in got], cells_of(case), dtype)
    out["fields"] = [torch.cat([f[k].reshape(-1) for f in state["fields"]]).to(dtype) for k in range(3)]
    out["counts"] = torch.tensor([counts(d) for d in diag])
    out["kinetic_ev"] = torch.tensor([d["kinetic_ev"] for d in diag], dtype=dtype)
    if case.get("ions"):
        from gasatt._lib import check, lib
        f, ids = state["ion_out"]
        n, sim = ctypes.c_int64(), sims[0]
        check(sim.ctx.handle, lib.gasatt_sim_read_ions(sim.h, *[ptr(f[k]) for k in range(5)], ptr(ids),
                                                       ptr(state["ion_q"]), ids.numel(), ctypes.byref(n), 1))
        # ions feel the FP32 form's fields, so they are held to its precision
        out["ion"] = ions(f[:, :n.value], ids[:n.value], dtype, int(sim.cfg.ion_capacity))
    return out


def cells_of(case):
    return batch_cells(case) if case["kind"] == "batch" else [case]


NAMES = ("r", "z", "ur", "ut", "uz")


def electrons(parts, ids, cells, dtype):
    """The electrons of all cells (cell i's loaded ones have the ids i 2^32 + 0, 1, ...)."""
    rows = sum(2 * c["photo"] for c in cells)
    loaded = torch.zeros(5, rows + 1, dtype=dtype, device=ids[0].device)      # and one row for the others
    born, born_id, at = [], [], 0
    for i, (part, k, c) in enumerate(zip(parts, ids, cells)):
        n, row = 2 * c["photo"], k - (i << 32)
        first = (row >= 0) & (row < n)
        loaded[:, torch.where(first, row + at, rows)] = part.to(dtype)
        born.append(part[:, ~first])
        born_id.append(k[~first])
        at += n
    born_id, order = torch.sort(torch.cat(born_id))
    born = torch.cat(born, 1)[:, order].to(dtype)
    room = sum(rows_of(c) for c in cells) - rows
    return dict(loaded={k: loaded[i, :rows] for i, k in enumerate(NAMES)},
                born={k: pad(born[i], room) for i, k in enumerate(NAMES)}, born_id=pad(born_id, room))


def ions(part, ids, dtype, rows):
    ids, order = torch.sort(ids)
    return dict(id=pad(ids, rows), **{k: pad(part[i][order].to(dtype), rows) for i, k in enumerate(NAMES)})


def run_host(state):
    """gasatt_sim_run_host on the pinned arrays, then the electrons back on the device for what the
    host's program does next, in the order of their radius and z (the call returns no ids)."""
    from gasatt._lib import check, lib
    case, sim = state["case"], state["sims"][0]
    start, io = state["start"], state["io"]
    n0, cap = start.shape[1], io.shape[1]
    io[:, :n0] = start
    n = ctypes.c_int64(n0)
    check(sim.ctx.handle, lib.gasatt_sim_run_host(sim.h, ptr(io), ptr(io[3]), ctypes.byref(n), cap, case["steps"]))
    p = io[:, :n.value].to(device(), non_blocking=True)
    out = host_order(p, torch.float32 if case["fp32"] else torch.float64, rows_of(case))
    get_fields(sim, state["fields"][0])
    out["fields"] = [f.to(out["pos"].dtype) for f in state["fields"][0]]
    return out


def host_order(p, dtype, rows):
    p = p[:, torch.sort(p[2], stable=True)[1]]
    p = pad(p[:, torch.sort(p[0], stable=True)[1]], rows)
    return dict(pos=p[:3].to(dtype), vel=p[3:].to(dtype))


def flags_of(case):
    from gasatt import FAITHFUL
    return FAITHFUL if case["faithful"] else 0


def run_em6(state):
    import gasatt
    i, case = state["inp"], state["case"]
    out = gasatt.electricmagneticfield6(*i["e"], *i["i1"], *i["i2"], *i["fields"], i["delta"], i["dt"],
                                        i["Rp"], i["Lp"], i["PHIp"], i["FN"], case["cycle"],
                                        flags=flags_of(case) | gasatt.POS_IN_CYL)
    return em6_rows(case, out)


def em6_rows(case, out):
    n = [case[k] for k in ("n_e", "n_e", "n_i1", "n_i1", "n_i2", "n_i2")]
    return [pad(a.t(), k) for a, k in zip(out, n)] + list(out[6:9]) + [pad(out[9], case["n_e"])]


def run_collision(state):
    import gasatt
    i, t, fl = state["inp"], state["tab"], flags_of(state["case"])
    sig = gasatt.find_CS0(t["t_el"], t["t_sel"], t["t_ion"], t["t_exc"], i["kin"], flags=fl)
    out = gasatt.electron_collision(i["pos"], i["vel"], i["ion_pos"], i["ion_vel"], t["t_el"], t["t_sel_1"],
                                    t["t_del"], t["t_sdel"], t["t_exc"], i["kin"], i["sum_cell"], i["xy"],
                                    i["density"], i["temperature"], i["PHIp"], i["phimax"], i["dr"], i["dz"],
                                    *sig, i["dt"], draws=i["draws"], flags=fl)
    return list(sig) + collision_rows(case=state["case"], out=out)


def collision_rows(case, out):
    born = case["n"] // 2 + 64
    return [pad(a.t(), k + born) for a, k in zip(out, (case["n"], case["n"], 1000, 1000))]


# -------------------------------------------------------------------- work
def work(case):
    """Per step the electrons' state read and written and the grid's fields and current; once, the
    inputs read and the outputs written."""
    kind = case["kind"]
    if kind == "em6":
        n, cells, k = case["n_e"] + case["n_i1"] + case["n_i2"], case["n_r"] * case["n_z"], case["cycle"] // 5
        return {"bytes": 96 * n + 48 * cells + k * (96 * n + 80 * cells), "flops": k * (300 * n + 220 * cells)}
    if kind == "collision":
        return {"bytes": case["n"] * (48 + 64 + 8 + 24 + 48 + 24), "flops": 200 * case["n"]}
    both = [0.0, 0.0]
    for c in cells_of(case):
        n, cells = 2 * c["photo"], c["n_r"] * c["n_z"]
        state, real = (24, 4) if c["fp32"] else (40, 8)
        once = n * (48 + 8 + 5 * real) + cells * (24 + 3 * real)
        step = 2 * state * n + cells * (6 * real + 32)
        both[0] += once + c["steps"] * step + (c["steps"] // 50) * 2 * 49 * c["ions"]
        both[1] += c["steps"] * (250 * n + 60 * cells)
    return {"bytes": both[0], "flops": both[1]}


# ------------------------------------------------------------------- exact
M32 = 0xFFFFFFFF


def shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def i64(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def philox(seed, ids, step, block):
    """Philox4x32-10 (Salmon et al., SC'11) of counter (id, step, block) and key seed."""
    c = [ids & M32, shr(ids, 32), torch.full_like(ids, step & M32), torch.full_like(ids, block)]
    k0, k1 = seed & M32, (seed >> 32) & M32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [shr(p1, 32) ^ c[1] ^ k0, p1 & M32, shr(p0, 32) ^ c[3] ^ k1, p0 & M32]
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return c


def draw2(seed, ids, step, block):
    c = philox(seed, ids, step, block)
    return [((c[2 * k] << 20) | (c[2 * k + 1] >> 12)).double() * 2.0 ** -52 + 2.0 ** -53 for k in range(2)]


def child_id(parent, step):
    z = parent + i64((0x9E3779B97F4A7C15 * (step + 1)) & (2 ** 64 - 1))
    z = (z ^ shr(z, 30)) * i64(0xBF58476D1CE4E5B9)
    z = (z ^ shr(z, 27)) * i64(0x94D049BB133111EB)
    return z ^ shr(z, 31)


def raw_tables():
    z = np.load(os.path.join(PKG, "data", "n2_tables.npz"))
    return {k: np.asarray(z[k], dtype=np.float64) for k in z.files}


def tail(x, y, q):
    s = np.log(y[-1] / y[-2]) / np.log(x[-1] / x[-2])
    return y[-1] * (q / x[-1]) ** s


def excitation(t, T, loss=False):
    """Per table row the excitation cross-section (without its constant) at T eV and its threshold;
    0 below it.  loss: with the last factor as electron_transport.cu:214-215 has it."""
    k, A, om, nu, ga = (t["t_exc"][:, j][:, None] for j in range(5))
    with np.errstate(invalid="ignore"):
        s = A / k ** 2 * (k / T) ** om * ((1 - k / T) ** ga if loss else 1 - (k / T) ** ga) ** nu
    return np.where(T > k, s, 0.0), k


def cross_sections(t, E, faithful):
    """find_CS0.m on energies E [keV]; corrected: power-law tails, 0 below threshold."""
    T = E * 1000
    el_x, el_y, sl_x, sl_y = t["t_el"][0], t["t_el"][1], t["t_sel"][:, 0], t["t_sel"][:, 1]
    io_x, io_y = t["t_ion"][:, 0], t["t_ion"][:, 1]
    hi = np.where((E > el_x[-1]) & (not faithful), tail(el_x, el_y, E), np.interp(E, el_x, el_y)) * 2.8002852e-21 * 2
    se = np.where(E >= 0.05, hi, np.interp(T, sl_x, sl_y) * 1e-20)
    si = np.where(T > io_x[-1], tail(io_x, io_y, T), np.interp(T, io_x, io_y, left=0.0)) * 1e-20
    si = np.where(T <= io_x[0], 0.0, si) if not faithful else si
    s, _ = excitation(t, T[None, :])
    return se, si, 6.542e-14 * s.sum(0) * 1e-4


def elastic_tables(t):
    s1 = t["t_sel_1"][:-1]
    y = np.concatenate([s1[:, 1] * 1e-20 / 2.8002852e-21 / 2, t["t_el"][1]])
    x = np.log(np.concatenate([t["t_sdel"][0, 1:], t["t_del"][0, 1:]]))
    V = np.log(np.concatenate([t["t_sdel"][1:, 1:], t["t_del"][1:, 1:]], 1).T)
    return x, y, V


class SimTables:
    """The resident simulation's tables on 2048 log-spaced energies from 0.1 eV to 30 keV."""

    def __init__(self, dev):
        t, G = raw_tables(), 2048
        self.ln0 = math.log(0.1)
        self.dln = (math.log(30000.0) - self.ln0) / (G - 1)
        E = np.exp(self.ln0 + np.arange(G) * self.dln)
        se, si, sx = cross_sections(t, E / 1000, False)
        x, _, V = elastic_tables(t)
        le = np.clip(np.log(E / 1000), x[0], x[-1])
        i = np.clip(np.searchsorted(x, le, side="left") - 1, 0, len(x) - 2)
        a = ((x[i + 1] - le) / (x[i + 1] - x[i]))[:, None]
        pdf = 4 * math.pi * np.sin(np.arange(181) * math.pi / 180) * np.exp(a * V[i] + (1 - a) * V[i + 1])
        cdf = np.zeros((G, 181))
        cdf[:, 1:] = np.cumsum((pdf[:, 1:] + pdf[:, :-1]) / 2, 1)
        cdf /= cdf[:, -1:]
        s, k = excitation(t, E[None, :])
        with np.errstate(invalid="ignore"):
            edep = np.where(s.sum(0) > 0, (s * k).sum(0) / s.sum(0), 0.0)
        tot = se + si + sx
        eps = np.append(E[1:], E[-1]) * QE / (ME * CC * CC)
        v = CC * np.sqrt(eps * (2 + eps)) / (1 + eps)
        self.sigv = float(np.max(np.append(np.maximum(tot, np.append(tot[1:], tot[-1])) * v, tot[-1] * CC)))
        self.G, self.kmin = G, float(k.min())
        up = lambda m: torch.tensor(m, dtype=torch.float64, device=dev)  # noqa: E731
        self.el, self.io, self.ex, self.edep, self.cdf = up(se), up(si), up(sx), up(edep), up(cdf)

    def place(self, ev):
        L = (torch.log(ev) - self.ln0) / self.dln
        i = torch.clamp(torch.floor(L), 0, self.G - 2).long()
        return L, i, torch.clamp(L - i, 0.0, 1.0)

    @staticmethod
    def mix(a, i, f):
        return a[i] + f * (a[i + 1] - a[i])


def rotate(u, st, ct, sp, cp):
    v = torch.sqrt((u * u).sum(0))
    s = torch.sqrt(u[0] ** 2 + u[1] ** 2)
    ok = s * s > 0.0001
    f = st / torch.where(ok, s, torch.ones_like(s))
    a = torch.stack([u[0] * ct + f * (u[0] * u[2] * cp - v * u[1] * sp),
                     u[1] * ct + f * (u[1] * u[2] * cp + v * u[0] * sp), u[2] * ct - s * st * cp])
    return torch.where(ok, a, torch.stack([v * st * cp, v * st * sp, v * ct]))


class Exact:
    """One gas cell in 64 bits."""

    def __init__(self, c, inp, seed):
        self.c, self.seed, self.dev = c, seed, inp["parts"][0].device
        self.nr, self.nz, self.d, self.dt = c["n_r"], c["n_z"], c["delta_um"] * 1e-6, c["dt_fs"] * 1e-15
        self.Rp, self.Lp = self.nr * self.d, self.nz * self.d
        self.x = torch.stack(inp["parts"][:2])
        self.u = torch.stack(inp["parts"][2:5])
        self.id = inp["parts"][5].clone()
        self.er, self.ez, self.h = (f.clone() for f in inp["fields"])
        i = torch.arange(self.nr, device=self.dev, dtype=torch.float64)
        self.vol = math.pi * (((i + 1) * self.d) ** 2 - (i * self.d) ** 2) * self.d
        self.T = SimTables(self.dev)
        self.gas, self.rho = inp["gas"], inp["rho"]
        self.nu = (float(inp["gas"].max()) if inp["gas"] is not None else inp["rho"]) * self.T.sigv
        self.below = int(-math.expm1(-self.nu * self.dt) * 2.0 ** 52)
        self.n = dict(ion=0, ela=0, exc=0, nul=0, lost=0)
        self.ions, self.jion = None, None
        if inp["ions"] is not None:
            p = inp["ions"]
            self.ions = [torch.stack(p[:2]), torch.stack(p[2:5]), p[5].clone(), p[6].double()]

    def drift(self, x, u, dt):
        g = torch.sqrt(1 + (u * u).sum(0) / CC ** 2)
        X, Y, Z = x[0] + 0.5 * u[0] / g * dt, 0.5 * u[1] / g * dt, x[1] + 0.5 * u[2] / g * dt
        r = torch.sqrt(X * X + Y * Y)
        pos = r > 0
        s = torch.where(pos, r, torch.ones_like(r))
        cs, sn = torch.where(pos, X / s, torch.ones_like(r)), torch.where(pos, Y / s, torch.zeros_like(r))
        uz = u[2]
        hi = Z > self.Lp
        Z, uz = torch.where(hi, 2 * self.Lp - Z, Z), torch.where(hi, -uz, uz)
        lo = Z < 0
        return (torch.stack([r, torch.where(lo, -Z, Z)]),
                torch.stack([cs * u[0] + sn * u[1], -sn * u[0] + cs * u[1], torch.where(lo, -uz, uz)]),
                r <= self.Rp)

    def corners(self, x, n, half):
        q = x / self.d - (0.5 if half else 0.0)
        a = torch.floor(q)
        w = q - a
        a = a.long()
        return torch.clamp(a, 0, n - 1), torch.clamp(a + 1, 0, n - 1), w

    def gather(self, x):
        def at(F, i, j):
            return ((1 - i[2]) * F[j[0], i[0]] + i[2] * F[j[0], i[1]]) * (1 - j[2]) + \
                ((1 - i[2]) * F[j[1], i[0]] + i[2] * F[j[1], i[1]]) * j[2]
        ih, jh = self.corners(x[0], self.nr, True), self.corners(x[1], self.nz, True)
        i, j = self.corners(x[0], self.nr + 1, False), self.corners(x[1], self.nz + 1, False)
        return at(self.er, ih, j), at(self.ez, i, jh), at(self.h, ih, jh)

    def kick(self, x, u, qm, dt):
        """Relativistic Boris push in E = (Er, 0, Ez), B = (0, mu0 H, 0); qm: charge over mass."""
        er, ez, h = self.gather(x)
        f = qm * dt / 2
        um0, um2 = u[0] + f * er, u[2] + f * ez
        t = f * MU0 * h / torch.sqrt(1 + (um0 ** 2 + u[1] ** 2 + um2 ** 2) / CC ** 2)
        p0, p2 = um0 - um2 * t, um2 + um0 * t
        s = 2 * t / (1 + t * t)
        return torch.stack([um0 - p2 * s + f * er, u[1], um2 + p0 * s + f * ez])

    def deposit(self, x, u, q):
        g = torch.sqrt(1 + (u * u).sum(0) / CC ** 2)
        i, j = self.corners(x[0], self.nr, True), self.corners(x[1], self.nz, True)
        out = []
        for v in (u[0] / g * q, u[2] / g * q):
            J = torch.zeros(self.nz * self.nr, device=self.dev, dtype=torch.float64)
            for a, wa in ((i[0], 1 - i[2]), (i[1], i[2])):
                for b, wb in ((j[0], 1 - j[2]), (j[1], j[2])):
                    J.index_add_(0, b * self.nr + a, wa * wb * v)
            out.append(J.view(self.nz, self.nr) / self.vol)
        return out

    def field_step(self):
        R = self.c["ratio"]
        dt, er, ez, h, d = self.dt / R, self.er, self.ez, self.h, self.d
        jr, jz = self.j
        if self.jion is not None:
            jr, jz = jr + self.jion[0], jz + self.jion[1]
        k = dt / 2 / EPS0
        ri = torch.arange(self.nr, device=self.dev, dtype=torch.float64) * d
        for sub in range(4 * R + 1):
            if sub % 2 == 0:
                f = (dt / 4 if sub in (0, 4 * R) else dt / 2) / (MU0 * d)
                h = h + (f * (ez[:, 1:] - ez[:, :-1]) - f * (er[1:] - er[:-1]))
                continue
            er = er.clone()
            er[1:-1] += -k * (jr[:-1] + jr[1:]) / 2 - k / d * (h[1:] - h[:-1])
            er[0], er[-1] = 0, 0
            ez = ez.clone()
            ez[:, 0] += -k * jz[:, 0] + 4 * k / d * h[:, 0]
            ez[:, 1:-1] += -k * (jz[:, :-1] + jz[:, 1:]) / 2 + k * (1 / (2 * ri[1:]) + 1 / d) * h[:, 1:] + \
                k * (1 / (2 * ri[1:]) - 1 / d) * h[:, :-1]
        self.er, self.ez, self.h = er, ez, h

    def keep(self, ok):
        if not bool(ok.all()):
            self.n["lost"] += int((~ok).sum())
            self.x, self.u, self.id = self.x[:, ok], self.u[:, ok], self.id[ok]

    def start(self):
        self.x, self.u, ok = self.drift(self.x, self.u, self.dt)
        self.keep(ok)
        self.j = self.deposit(self.x, self.u, -QE)

    def push(self, whole=True):
        self.u = self.kick(self.x, self.u, -QE / ME, self.dt)
        for _ in range(2 if whole else 1):
            self.x, self.u, ok = self.drift(self.x, self.u, self.dt)
            self.keep(ok)

    def step(self, s):
        self.field_step()
        self.push()
        self.j = self.deposit(self.x, self.u, -QE)
        c = philox(self.seed, self.id, s, 0)
        k = torch.nonzero(((c[0] << 20) | (c[1] >> 12)) < self.below)[:, 0]
        if k.numel():
            self.collide(k, s)

    def collide(self, k, s):
        T, ids, u, n = self.T, self.id[k], self.u[:, k], k.numel()
        u2 = (u * u).sum(0)
        g = torch.sqrt(1 + u2 / CC ** 2)
        ev = ME * CC * CC * ((u2 / CC ** 2) / (g + 1)) / QE
        um = torch.sqrt(u2)
        ng = torch.full_like(ev, self.rho)
        if self.gas is not None:
            i = torch.clamp(torch.floor(self.x[0, k] / self.d).long(), 0, self.nr - 1)
            j = torch.clamp(torch.floor(self.x[1, k] / self.d).long(), 0, self.nz - 1)
            ng = self.gas[j, i]
        L, i, f = T.place(ev)
        v = um / g * ng
        ne, ni, nx = T.mix(T.el, i, f) * v, T.mix(T.io, i, f) * v, T.mix(T.ex, i, f) * v
        X = draw2(self.seed, ids, s, 0)[1] * self.nu
        a, b = draw2(self.seed, ids, s, 1)
        I = 15.6
        ela = X < ne
        ion = ~ela & (X < ne + ni) & (ev > I)
        loss = T.mix(T.edep, i, f)
        exc = ~ela & ~ion & (X < ne + ni + nx) & (ev > T.kmin) & (loss > 0) & (loss < ev)
        out = u.clone()
        sp, cp = torch.sin(2 * math.pi * b), torch.cos(2 * math.pi * b)
        row = T.cdf[torch.clamp(torch.floor(L + 0.5), 0, T.G - 1).long()]
        lo = torch.clamp(torch.searchsorted(row, a[:, None], right=True)[:, 0] - 1, 0, 179)
        at = torch.arange(n, device=self.dev)
        th = (lo + (a - row[at, lo]) / (row[at, lo + 1] - row[at, lo])) * (math.pi / 180)
        out = torch.where(ela, rotate(u, torch.sin(th), torch.cos(th), sp, cp), out)
        T0, t = 4.17 - 1000 / (ev + 2 * I), 13.8 * ev / (ev + I)
        a2 = T0 / t
        E1 = T0 + t * torch.tan(a * (torch.atan(((ev - I) / 2 - T0) / t) + torch.atan(a2)) - torch.atan(a2))
        E2 = ev - E1 - I
        Ep, Es = torch.maximum(E1, E2), torch.minimum(E1, E2)
        Ee = ME * CC * CC / QE
        sp2, ss2 = (Es / ev) / ((1 - Es / ev) * ev / (2 * Ee) + 1), (1 - Es / ev) / (1 + Es / (2 * Ee))

        def speed(E):
            e = E * QE / (ME * CC * CC)
            return CC * torch.sqrt(e * (2 + e))
        d = u / um
        out = torch.where(ion, rotate(d * speed(Ep), torch.sqrt(sp2), torch.sqrt(1 - sp2), sp, cp), out)
        sec = rotate(d * speed(Es), torch.sqrt(ss2), torch.sqrt(1 - ss2), -sp, -cp)
        out = torch.where(exc, d * speed(torch.where(exc, ev - loss, ev)), out)
        self.u[:, k] = out
        for name, m in (("ion", ion), ("ela", ela), ("exc", exc), ("nul", ~(ela | ion | exc))):
            self.n[name] += int(m.sum())
        kid = child_id(ids[ion], s)
        x = self.x[:, k[ion]]
        self.x, self.u = torch.cat([self.x, x], 1), torch.cat([self.u, sec[:, ion]], 1)
        self.id = torch.cat([self.id, kid])
        if self.ions is not None:
            p, q = draw2(self.seed, ids[ion], s, 2), draw2(self.seed, ids[ion], s, 3)
            sig = math.sqrt(KB * 300.0 / M_ION)
            ra, rb = sig * torch.sqrt(-2 * torch.log(p[0])), sig * torch.sqrt(-2 * torch.log(q[0]))
            w = torch.stack([ra * torch.cos(2 * math.pi * p[1]), ra * torch.sin(2 * math.pi * p[1]),
                             rb * torch.cos(2 * math.pi * q[1])])
            self.ions = [torch.cat([self.ions[0], x], 1), torch.cat([self.ions[1], w], 1),
                         torch.cat([self.ions[2], kid]), torch.cat([self.ions[3], torch.ones_like(w[0])])]

    def push_ions(self):
        x, u, ids, q = self.ions
        dt = 50 * self.dt
        u = self.kick(x, u, q * QE / M_ION, dt)
        for _ in range(2):
            x, u, ok = self.drift(x, u, dt)
            x, u, ids, q = x[:, ok], u[:, ok], ids[ok], q[ok]
        self.ions = [x, u, ids, q]
        self.jion = self.deposit(x, u, q * QE)

    def run(self, first=0):
        self.start()
        for s in range(self.c["steps"]):
            self.step(first + s)
            if self.ions is not None and (s + 1) % 50 == 0:
                self.push_ions()
        return self

    def kinetic(self):
        u2 = (self.u * self.u).sum(0) / CC ** 2
        return float((ME * CC * CC / QE * (u2 / (torch.sqrt(1 + u2) + 1))).sum())


def exact(case, seed):
    kind = case["kind"]
    if kind == "em6":
        return exact_em6(case, wedge_inputs(case, seed))
    if kind == "collision":
        return exact_collision(case, wedge_inputs(case, seed))
    if kind == "host":
        e = Exact(case, cell_inputs(case, seed), seed)
        e.start()
        for s in range(1, case["steps"]):
            e.step(s)
        e.field_step()
        e.push(whole=False)
        v = e.u / torch.sqrt(1 + (e.u * e.u).sum(0) / CC ** 2)
        p = torch.cat([e.x[:1], torch.zeros_like(e.x[:1]), e.x[1:], v])
        return dict(host_order(p, torch.float64, rows_of(case)), fields=[e.er, e.ez, e.h])
    cells, done = cells_of(case), []
    for i, c in enumerate(cells):
        k = seed * 1000 + i if kind == "batch" else seed
        done.append(Exact(c, cell_inputs(c, k, id_base=i << 32), k).run())
    out = electrons([torch.cat([e.x, e.u]) for e in done], [e.id for e in done], cells, torch.float64)
    if case["fp32"]:
        # where the FP32 form takes one collision that 64 bits do not, all secondaries after it are
        # in other rows
        out["born"] = None
    out["born_id"] = None
    out["fields"] = [torch.cat([f[k].reshape(-1) for f in [(e.er, e.ez, e.h) for e in done]]) for k in range(3)]
    out["counts"] = None
    out["kinetic_ev"] = torch.tensor([e.kinetic() for e in done], dtype=torch.float64)
    if case.get("ions"):
        x, u, ids, _ = done[0].ions
        out["ion"] = ions(torch.cat([x, u]), ids, torch.float64, case["ions"] + rows_of(case) - 2 * case["photo"])
    return out


def exact_em6(case, inp):
    """electricmagneticfield6.m:65-188 with its kernels' arithmetic."""
    qe, c, eps, mu = 1.6e-19, 3e8, 8.854187817e-12, 4 * math.pi * 1e-7
    faith, nr, nz, d, dt = case["faithful"], case["n_r"], case["n_z"], inp["delta"], inp["dt"]
    Rp, Lp, PHIp, FN, ddt = inp["Rp"], inp["Lp"], inp["PHIp"], inp["FN"], 5 * inp["dt"]
    sp = [inp["e"], inp["i1"], inp["i2"]]
    ns = [p.shape[0] for p, _ in sp]
    P, v = torch.cat([p for p, _ in sp]).t(), torch.cat([w for _, w in sp]).t()
    dev = P.device
    x = torch.stack([P[0] * torch.cos(P[1]), P[0] * torch.sin(P[1]), P[2]])
    q, m = (torch.cat([torch.full((n,), w, device=dev, dtype=torch.float64) for n, w in zip(ns, a)])
            for a in ((-qe, qe, 2 * qe), (9.1096e-31, 4.65e-26, 4.65e-26)))
    alive = torch.ones_like(q, dtype=torch.bool)
    er, ez, h = (f.t().clone() for f in inp["fields"])
    i = torch.arange(nr, device=dev, dtype=torch.float64)
    vol = PHIp / 2 * (((i + 1) * d) ** 2 - (i * d) ** 2) * d
    cP, sP = math.cos(PHIp), math.sin(PHIp)
    kin = torch.zeros_like(q)

    def half(x, v):
        X = x + 0.5 * v * ddt
        r = torch.sqrt(X[0] ** 2 + X[1] ** 2)
        phi = torch.atan(X[1] / X[0]) if faith else torch.atan2(X[1], X[0])
        vx, vy, vz = v[0].clone(), v[1].clone(), v[2].clone()
        for sign in (1, -1):
            while True:
                out = phi < 0 if sign > 0 else phi > PHIp
                if not bool(out.any()):
                    break
                phi = torch.where(out, phi + sign * PHIp, phi)
                vx, vy = (torch.where(out, vx * cP - sign * vy * sP, vx),
                          torch.where(out, sign * vx * sP + vy * cP, vy))
        Z = X[2]
        hi = Z > Lp
        Z, vz = torch.where(hi, 2 * Lp - Z, Z), torch.where(hi, -vz, vz)
        lo = Z < 0
        Z, vz = torch.where(lo, -Z, Z), torch.where(lo, -vz, vz)
        return torch.stack([r * torch.cos(phi), r * torch.sin(phi), Z]), torch.stack([vx, vy, vz]), r, phi, r <= Rp

    def corners(a, n, shift):
        s = a / d - shift
        k = torch.floor(s)
        w = s - k
        k = k.long()
        return torch.clamp(k, 0, n - 1), torch.clamp(k + 1, 0, n - 1), w

    def at(F, i, j):
        return ((1 - i[2]) * F[j[0], i[0]] + i[2] * F[j[0], i[1]]) * (1 - j[2]) + \
            ((1 - i[2]) * F[j[1], i[0]] + i[2] * F[j[1], i[1]]) * j[2]

    k1 = dt / 2 / eps
    for _ in range(case["cycle"] // 5):
        x1, v1, r, phi, ok = half(x, v)
        x, v = torch.where(alive, x1, x), torch.where(alive, v1, v)
        alive = alive & ok
        vr = v[0] * torch.cos(phi) + v[1] * torch.sin(phi)
        z = x[2]
        ih, jh = corners(r, nr, 0.5), corners(z, nz, 0.5)
        J = []
        for w in (vr, v[2]):
            a = torch.zeros(nz * nr, device=dev, dtype=torch.float64)
            for ci, wi in ((ih[0], 1 - ih[2]), (ih[1], ih[2])):
                for cj, wj in ((jh[0], 1 - jh[2]), (jh[1], jh[2])):
                    a.index_add_(0, torch.where(alive, cj * nr + ci, 0),
                                 torch.where(alive, FN * wi * wj * q * w, 0.0))
            J.append(a.view(nz, nr) / vol)
        jr, jz = J
        for n in range(12):
            f = (-dt / 4 if n == 0 else dt / 4 if n == 11 else dt / 2) / (mu * d)
            h = h + f * (ez[:, 1:] - ez[:, :-1]) - f * (er[1:] - er[:-1])
            if n in (0, 11):
                continue
            new = er.clone()
            new[1:-1] = er[1:-1] - k1 * (jr[:-1] + jr[1:]) / 2 - k1 / d * (h[1:] - h[:-1])
            new[0], new[-1] = (er[1], er[-2]) if faith else (0, 0)
            er = new
            ri = (torch.arange(1, nr, device=dev, dtype=torch.float64) + (1 if faith else 0)) * d
            ez = ez.clone()
            ez[:, 0] += (k1 if faith else -k1) * jz[:, 0] + 4 * k1 / d * h[:, 0]
            ez[:, 1:-1] += -k1 * (jz[:, :-1] + jz[:, 1:]) / 2 + k1 * (1 / (2 * ri) + 1 / d) * h[:, 1:] + \
                k1 * (1 / (2 * ri) - 1 / d) * h[:, :-1]
        rc = torch.where(alive, r, 0.5 * Rp)
        ih = corners(rc, nr, 0.5)
        ii, jj = corners(rc, nr + 1, 0.0), corners(z, nz + 1, 0.0)
        Er, Ez, H = at(er, ih, jj), at(ez, ii, jh), at(h, ih, jh)
        g = 1 / torch.sqrt(1 - (v * v).sum(0) / c ** 2)
        cp, sn = torch.cos(phi), torch.sin(phi)
        if faith:
            Fr, Fz = q * (Er - v[2] * H * mu), q * (Ez + vr * H * mu)
            u = g * v + torch.stack([Fr * cp, Fr * sn, Fz]) / m * ddt
        else:
            f = q / m * ddt / 2
            E, B = torch.stack([Er * cp, Er * sn, Ez]), torch.stack([-mu * H * sn, mu * H * cp, torch.zeros_like(H)])
            um = g * v + f * E
            t = f / torch.sqrt(1 + (um * um).sum(0) / c ** 2) * B
            up = um + torch.linalg.cross(um, t, dim=0)
            u = um + torch.linalg.cross(up, 2 / (1 + (t * t).sum(0)) * t, dim=0) + f * E
        g = torch.sqrt(1 + (u * u).sum(0) / c ** 2)
        kin = torch.where(alive, (g - 1) * m * c * c, kin)
        x1, v1, r, phi, ok = half(x, u / g)
        x, v = torch.where(alive, x1, x), torch.where(alive, v1, v)
        alive = alive & ok
    out, at0 = [], 0
    for n in ns:
        k = torch.nonzero(alive[at0:at0 + n])[:, 0] + at0
        out += [x[:, k].t(), v[:, k].t()]
        at0 += n
    k = torch.nonzero(alive[:ns[0]])[:, 0]
    return em6_rows(case, out + [er.t(), ez.t(), h.t(), kin[k] / (1000 * qe)])


def exact_collision(case, inp):
    """find_CS0.m, then electron_collision.m around electron_transport.cu:39-229."""
    t, faith = raw_tables(), case["faithful"]
    e, c, m, m_ion, kb, I = 1.6022e-19, 3e8, 9.109e-31, 4.65e-26, 1.38064853e-23, 15.6
    pi = 3.1415926 if faith else math.pi
    kin = inp["kin"].cpu().numpy()
    sig = cross_sections(t, kin, faith)
    pos, v = inp["pos"].cpu().numpy(), inp["vel"].cpu().numpy().copy()
    U = inp["draws"].cpu().numpy()
    rho, temp = inp["density"].cpu().numpy(), inp["temperature"].cpu().numpy()
    sc = np.concatenate([[0], inp["sum_cell"]]).astype(np.int64)
    rmax, dphi = case["rmax"], inp["PHIp"] / inp["phimax"]
    ve = np.sqrt((v * v).sum(1))
    ir = np.clip(np.floor(np.hypot(pos[:, 0], pos[:, 1]) / inp["dr"]).astype(int), 0, rmax - 1)
    ip = np.floor(np.arctan(pos[:, 1] / pos[:, 0]) / dphi[ir]).astype(int)
    ip = np.maximum(np.minimum(ip, sc[ir + 1] - sc[ir] - 1), 0)
    index = np.clip(np.floor(pos[:, 2] / inp["dz"]).astype(int) * inp["xy"] + sc[ir] + ip, 0, rho.size - 1)
    p = [ve * inp["dt"] * rho[index] * s for s in sig]
    tot = p[0] + p[1] + p[2]
    a, b = p[0] / tot, (p[0] + p[1]) / tot
    k = np.nonzero(U[:, 0] < (tot if faith else -np.expm1(-tot)))[0]
    ela = k[U[k, 1] < a[k]]
    rest = k[~(U[k, 1] < a[k])]
    ision = (U[rest, 1] < b[rest]) & (kin[rest] > I / 1000)
    ion, exc = rest[ision], rest[~ision]

    def rot(w, th, ph):
        turn = [torch.tensor(f(q)) for q in (th, ph) for f in (np.sin, np.cos)]
        return rotate(torch.tensor(w.T), *turn).numpy().T
    # elastic
    x, y, V = elastic_tables(t)
    E = kin[ela] if faith else np.clip(np.log(kin[ela]), x[0], x[-1])
    i = np.clip(np.searchsorted(x, E, side="left") - 1, 0, len(x) - 2)
    fa, fb = (x[i + 1] - E) / (x[i + 1] - x[i]), (E - x[i]) / (x[i + 1] - x[i])
    tcs = (fa * y[i] + fb * y[i + 1]) * 2
    ang = np.arange(181)
    pdf = 2 * pi * np.sin(ang * pi / 180) * np.exp(fa[:, None] * V[i] + fb[:, None] * V[i + 1]) * 2 / tcs[:, None]
    n = np.arange(len(ela))
    if faith:
        S = np.concatenate([np.zeros((len(ela), 1)), np.cumsum(pdf * pi / 180, 1)], 1)
        rnd = U[ela, 2] * S[:, -1]
        j = np.argmin(rnd[:, None] > S, 1)
        i1 = S[n, j]
        i2 = i1 + pdf[n, np.minimum(j, 180)] * pi / 180
        th = ((i2 - rnd) / (i2 - i1) * (j - 1) + (rnd - i1) / (i2 - i1) * j) * pi / 180
    else:
        C = np.concatenate([np.zeros((len(ela), 1)), np.cumsum((pdf[:, 1:] + pdf[:, :-1]) / 2 * pi / 180, 1)], 1)
        rn = U[ela, 2] * C[:, -1]
        j = np.minimum((C[:, 1:] <= rn[:, None]).sum(1), 179)
        th = (j + (rn - C[n, j]) / (C[n, j + 1] - C[n, j])) * pi / 180
    out = v.copy()
    out[ela] = rot(v[ela], th, 2 * pi * U[ela, 3])
    # ionization
    T = kin[ion] * 1000
    T0, tt = 4.17 - 1000 / (T + 2 * I), 13.8 * T / (T + I)
    k1, k2 = np.arctan(((T - I) / 2 - T0) / tt), np.arctan(T0 / tt)
    k0 = T0 + tt * np.tan(U[ion, 2] * (k1 + k2) - k2)
    E1, E2 = k0, T - k0 - I
    Ep, Es = np.maximum(E1, E2), np.minimum(E1, E2)
    kk, Ee = (k0 if faith else Es), m * c * c / e
    ph = 2 * pi * U[ion, 3]
    tp = np.arcsin(np.sqrt((kk / T) / ((1 - kk / T) * T / (2 * Ee) + 1)))
    ts = np.arcsin(np.sqrt((1 - kk / T) / (1 + kk / (2 * Ee))))
    speed = lambda E: c * np.sqrt(1 - 1 / (1 + E * e / (m * c * c)) ** 2)  # noqa: E731
    out[ion] = rot(v[ion] * (speed(Ep) / ve[ion])[:, None], tp, ph)
    if faith:
        sec = np.stack([np.sin(ts) * np.cos(ph - pi), np.sin(ts) * np.sin(ph - pi), np.cos(ts)], 1)
        sec *= speed(Es)[:, None]
    else:
        sec = rot(v[ion] / ve[ion][:, None] * speed(Es)[:, None], ts, ph - pi)
    # excitation
    T = kin[exc] * 1000
    s, ks = excitation(t, T[None, :], loss=True)
    with np.errstate(invalid="ignore", divide="ignore"):
        left = T - (s * ks).sum(0) / s.sum(0)
    some = s.sum(0) > 0
    out[exc[some]] = v[exc[some]] * (speed(left[some]) / ve[exc[some]])[:, None]
    iv = U[ion, 4:7] / np.sqrt(m_ion / (kb * temp[index[ion]]))[:, None]
    cat = lambda *a: torch.tensor(np.concatenate(a))  # noqa: E731
    return [torch.tensor(w) for w in sig] + collision_rows(case, [
        cat(pos, pos[ion]), cat(out, sec), cat(inp["ion_pos"].cpu().numpy(), pos[ion]),
        cat(inp["ion_vel"].cpu().numpy(), iv)])
