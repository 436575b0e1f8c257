"""Workloads whose speed matters to a user of tracer_code_gb300, from the
smallest calls to the 1024x256 timestep, each through a public entry point.

A case is a dict of plain values.  ``prepare`` makes what a user's program
holds before the call (a handle with its state uploaded, a network with its
weights, host arrays), ``run`` makes one pass of the call and returns its
outputs, ``work`` counts the bytes and operations the path cannot do without
and ``exact`` gives outputs in 64 bits where they have a closed form.

Kinds of case:

- ``timestep``: tc_step_host on pinned host arrays, the call of a Fortran host
  that keeps the module arrays; every pass advances the state by one step;
- ``short_run``: restart from a state, a few timesteps, the state read back;
- ``ensemble``: independent cases stepped together, one graph launch a step;
- ``solve``: one streamfunction solve of a thermal state from SF = 0;
- ``advect``: energy_time with the velocities held (RK_update = 0): the
  tracer stages, the tracer-ratio step and the temperature stages;
- ``diagnostics``: compute_velocities and stats, the calls of every step;
- ``network_gradient``: loss and parameter gradient of one training batch;
- ``network_forward``: the learned guess of one or more images.
"""
from __future__ import annotations

import ctypes
import math
import os

import numpy as np
import torch

import tracer_code_gb300 as tc
from tracer_code_gb300 import learned, state
from tracer_code_gb300.ensemble import Ensemble

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(tc.__file__)), "weights", "guess_512x128.npy")

# solver arms: name -> (solver_precision, learned_guess, cycle_correction)
SOLVERS = {"fp64": (0, 0, 0), "mixed": (1, 0, 0), "window": (1, 0, 3), "learned": (1, 3, 4)}
# W-cycles of one solve to 1e-8 in ordinary use, for work() only
CYCLES = {"fp64": 45, "mixed": 48, "window": 18, "learned": 18}
# smoother visits of the levels above the coarsest in one W-cycle, by level count
VISITS = {2: [1], 3: [1, 3], 4: [1, 3, 6], 5: [1, 3, 6, 9], 6: [1, 3, 6, 10, 14]}


# ---- cases --------------------------------------------------------------------
def flow(kind, nx, nz, grids, tpc, Ra, visT, solver, aspect=4.0, **more):
    c = {"kind": kind, "nx": nx, "nz": nz, "grids": grids, "tpc": tpc, "Ra": float(Ra), "B": 0.8,
         "visT": float(visT), "solver": solver, "aspect": float(aspect)}
    c.update(more)
    return c


def listed():
    return [
        # the framework's main workload: 6.6 M tracers, learned + mixed solver
        dict(name="step_1024x256_learned", **flow("timestep", 1024, 256, 6, 25, 1e7, 1e4, "learned")),
        # the same physics with the reference's own FP64 method
        dict(name="step_1024x256_fp64", **flow("timestep", 1024, 256, 6, 25, 1e7, 1e4, "fp64")),
        # a medium production run: windowed mixed solver, an odd tracer count
        dict(name="run_512x128_window", **flow("short_run", 512, 128, 5, 13, 1e5, 100, "window", steps=2)),
        # the 128x128 isoviscous benchmark, everything at the reference's defaults
        dict(name="run_128x128_fp64", **flow("short_run", 128, 128, 6, 20, 1e5, 1, "fp64", 1.0, steps=2, B=0.5,
                                             plain=True)),
        # sizes that are no powers of two, stretched in x, mixed solver without the correction
        dict(name="run_360x88_mixed", **flow("short_run", 360, 88, 4, 7, 3e4, 30, "mixed", steps=2, gridX=1)),
        # the reference's shipped inputs: temperature tracers, repositioning, plastic viscosity
        dict(name="step_200x200_shipped", kind="shipped", nx=200, nz=200, tpc=30, threads=16, steps=1),
        # a parameter study: six cases of three sizes in one graph launch per step
        dict(name="ensemble_6", kind="ensemble", count=6, tpc=8, Ra=1e5, visT=100.0),
        # flow for a given temperature field, a small grid: latency counts
        dict(name="solve_256x64_window", **flow("solve", 256, 64, 4, 0, 1e5, 100, "window")),
        # transport with held velocities, 6.6 M tracers
        dict(name="advect_1024x256", **flow("advect", 1024, 256, 6, 25, 1e7, 1, "fp64")),
        # the smallest calls of the time loop
        dict(name="diagnostics_256x64", **flow("diagnostics", 256, 64, 4, 4, 1e5, 1, "fp64")),
        # one training batch of the learned guess, as train_guess uses it
        dict(name="gradient_8x512x128", kind="network_gradient", nb=8, H=128, W=512),
        # the learned guess at the main workload's size
        dict(name="forward_1x1024x256", kind="network_forward", nb=1, H=256, W=1024),
    ]


def log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["timestep", "short_run", "short_run", "solve", "solve", "advect", "diagnostics",
                       "ensemble", "shipped", "network_gradient", "network_forward"])
    if kind in ("network_gradient", "network_forward"):
        W = rng.choice([128, 256, 512, 1024])
        unit = {128: 64, 256: 32, 512: 16, 1024: 16}[W]
        H = unit * rng.randint(1, 256 // unit)
        most = min(8, max(1, 8 * 512 * 128 // (H * W)))
        return {"kind": kind, "nb": rng.randint(1, most), "H": H, "W": W}
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randint(2, 6), "tpc": rng.randint(3, 10),
                "Ra": float("%.3g" % log_between(rng, 2e4, 1e5)), "visT": float("%.3g" % log_between(rng, 2, 100))}
    if kind == "shipped":
        n = 8 * rng.randint(8, 25)
        return {"kind": kind, "nx": n, "nz": n, "tpc": rng.randint(10, 30), "threads": rng.randint(1, 16), "steps": 1}
    aspect = rng.choice([1.0, 2.0, 4.0])
    most = {"timestep": 512, "short_run": 512, "solve": 1024, "advect": 1024, "diagnostics": 1024}[kind]
    nz = int(log_between(rng, 32, most / 4 + 1))
    nx = max(32, min(most, int(nz * aspect * rng.uniform(0.8, 1.2))))
    tpc = int(log_between(rng, 3, 26))
    if kind == "advect" and rng.random() < 0.5:
        tpc = min(40, 2 * tpc)
    if nx * nz * tpc > 7_000_000:
        tpc = max(3, 7_000_000 // (nx * nz))
    solver = rng.choice(["fp64", "mixed", "window", "window"])
    Ra, visT = log_between(rng, 1e4, 1e5), log_between(rng, 2, 100)
    grids = 4
    while grids < 6 and ((nx >> (grids - 1)) + 2) * ((nz >> (grids - 1)) + 2) > 700:  # a small coarsest grid
        grids += 1
    if kind in ("timestep", "short_run", "solve", "diagnostics") and (nx * nz > 10_000 or rng.random() < 0.8):
        # sizes that halve down to the coarsest grid, odd multiples among them, as
        # users pick them; small grids also come as they fall (the set-up rounds
        # those, often to fewer levels)
        unit = 1 << (grids - 1)
        nx, nz = max(32, nx // unit * unit), max(32, nz // unit * unit)
    c = flow(kind, nx, nz, grids, 0 if kind == "solve" else tpc, "%.3g" % Ra, "%.3g" % visT, solver, aspect)
    if kind == "short_run":
        c["steps"] = rng.randint(1, 3)
        if rng.random() < 0.25:
            c["gridX"] = 1
    return c


# ---- parameters and inputs ---------------------------------------------------------
def params(case):
    if case["kind"] == "shipped":
        # main.f90:8-116 as shipped: ivis 3 (plastic), the non-Newtonian iteration,
        # temperature tracers, tracer repositioning, two levels
        p = tc.default_params()
        p.nx, p.nz, p.aspect, p.tpc = case["nx"], case["nz"], 1.0, case["tpc"]
        p.comp, p.ntype, p.tracer = 0, 0, 1
        p.equalize, p.equalize_threads = 1, case["threads"]
        p.ivis, p.non_Newtonian, p.grids, p.torder = 3, 1, 2, 2
        return p
    p = tc.config_1024x256(case["tpc"] or 4)
    p.nx, p.nz, p.grids, p.aspect = case["nx"], case["nz"], case["grids"], case["aspect"]
    p.RaT, p.visT = case["Ra"], case["visT"]
    p.RaC[0] = case["B"] * case["Ra"]
    p.gridX = case.get("gridX", 0)
    if case["visT"] == 1.0:
        p.ivis = 0
    if case.get("plain"):
        p.dlayer = 0.2
    else:
        p.mg_zero_coarse = 1
        p.mg_coarse_matrix = 1
    if case["tpc"] == 0:
        p.comp, p.ntype = 0, 0
        p.ivis = 1 if case["visT"] != 1.0 else 0
    p.solver_precision, p.learned_guess, p.cycle_correction = SOLVERS[case["solver"]]
    if case["kind"] == "advect":
        p.RK_update = 0
    return p


def perturbation(seed, x, z):
    """A few large-scale temperature modes drawn from the seed, zero at the top and bottom."""
    a = np.random.default_rng(seed).uniform(-0.003, 0.003, 3)
    return sum(a[m] * np.cos((m + 1) * np.pi * x) for m in range(3)) * np.sin(np.pi * z)


def start_state(p, seed):
    """The framework's conductive start with the seed's perturbation and tracers."""
    nx, nz = p.nx, p.nz
    st = state.initial_state(p, seed=1 + seed % 1000003, nx=nx, nz=nz)
    x, z = state.grid_coordinates(p, nx, nz)
    st["T"] += perturbation(seed, x[None, :], z[:, None])
    span = p.order // 2 + 1
    st["T"][span, :] = 1.0
    st["T"][span + nz, :] = 0.0
    if p.tracer == 1:
        st["Ttr"] += perturbation(seed, state.xgrid(p, st["rtr"]), state.zgrid(p, st["str"], nz))
    if p.comp == 0:
        st.pop("Cnew", None)
        if p.tracer == 0:
            for k in ("rtr", "str", "Ttype"):
                st.pop(k, None)
    return st


def cell_flow(p, seed):
    """A streamfunction of convection cells with the seed's amplitudes, zero on the walls."""
    span = p.order // 2 + 1
    a = np.random.default_rng(seed).uniform(0.5, 1.0, 3)
    x = np.arange(-span, p.nx + span + 1) * (p.aspect / p.nx)
    z = np.arange(-span, p.nz + span + 1) / p.nz
    f = sum(a[m] * np.sin((m + 1) * np.pi * x / p.aspect) for m in range(3))
    return 20.0 * np.ascontiguousarray(f[None, :] * np.sin(np.pi * z)[:, None])


def pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def simulation(p):
    """A handle, with the network attached where the solver uses one; p takes
    the grid the multigrid set-up rounds nx, nz to (optimize_grid)."""
    sim = tc.Simulation(p)
    p.nx, p.nz = sim.nx, sim.nz
    net = None
    if p.learned_guess:
        net = learned.Net(1, p.nz, p.nx)
        net.load(WEIGHTS)
        learned.attach(sim, net)
    return sim, net


def ptr(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


def download(s):
    """tc_download_state into the program's own host arrays."""
    sim, h = s["sim"], s["host"]
    sim._chk(sim.L.tc_download_state(sim.h, ptr(h["T"]), ptr(h.get("Cnew")), ptr(h["SF"]), ptr(h.get("rtr")),
                                     ptr(h.get("str")), ptr(h.get("Ttype"))), "download")
    if "Ttr" in h:
        sim._chk(sim.L.tc_download_tracer_temperature(sim.h, ptr(h["Ttr"])), "download_tracer_temperature")
    return h


def row_arrays(row):
    """A stats row as one array of its real columns and one of its integer columns."""
    real = [row[k] for k in ("time", "Tavg", "vrms", "Nu", "Nu_bot", "RaT_avg", "mobility", "strain_max", "q1", "q2",
                             "q3", "q4")] + [row["Cavg"][0], row["ent"][0]]
    whole = [row[k] for k in ("empty_cells", "tracer_min", "tracer_max", "n_eta", "n_temp")]
    return np.array(real), np.array(whole, dtype=np.int64)


def images(nb, H, W, seed, device="cuda"):
    """Smooth log10 viscosity, RHS and streamfunction images and a slightly later streamfunction."""
    g = torch.Generator().manual_seed(seed)
    y = (torch.arange(H, dtype=torch.float64) / H)[:, None]
    x = (torch.arange(W, dtype=torch.float64) / W)[None, :]

    def field(modes, sine):
        out = torch.zeros(nb, H, W, dtype=torch.float64)
        for m in range(1, modes + 1):
            a = torch.randn(nb, 1, 1, generator=g, dtype=torch.float64) / m
            ph = 0.0 if sine else 2 * math.pi * torch.rand(nb, 1, 1, generator=g, dtype=torch.float64)
            wx = torch.sin(math.pi * m * x) if sine else torch.cos(math.pi * m * x + ph)
            out += a * wx * torch.sin(math.pi * (1 + m % 2) * y)
        return out

    sf = 50.0 * field(4, True)
    raw = torch.stack([-4.0 * (1 - y + 0.1 * field(5, False)), 1e6 * field(6, False), sf], dim=1)
    new = sf + 0.5 * field(6, True)
    return raw.to(torch.float32).to(device).contiguous(), new.to(torch.float32).to(device).contiguous()


# ---- prepare -----------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("network_gradient", "network_forward"):
        net = learned.Net(case["nb"], case["H"], case["W"])
        net.load(WEIGHTS)
        raw, new = images(case["nb"], case["H"], case["W"], seed)
        out = torch.empty_like(new)
        return {"case": case, "net": net, "raw": raw, "new": new, "out": out}
    if kind == "ensemble":
        ps = []
        for i in range(case["count"]):
            c = flow("short_run", *[(256, 64, 4), (512, 128, 5), (200, 96, 4)][i % 3], case["tpc"] + i,
                     case["Ra"] / (1 + 0.3 * i), case["visT"], "window", 2.0 if i % 3 == 2 else 4.0)
            ps.append(params(c))
        e = Ensemble(ps, seeds=[1 + (seed + 17 * i) % 1000003 for i in range(len(ps))], autotune=False)
        return {"case": case, "ensemble": e}
    p = params(case)
    sim, net = simulation(p)
    st = start_state(p, seed)
    s = {"case": case, "sim": sim, "net": net}
    if kind in ("advect", "diagnostics"):
        st["SF"] = cell_flow(p, seed)
        sim.upload(st)
        sim.compute_viscosity(1)
        sim.compute_velocities()
        s["host"] = {k: pinned(v) for k, v in st.items()}
    elif kind == "timestep":
        s["host"] = {k: pinned(v) for k, v in st.items()}
        sim.upload(s["host"])
        download(s)
    else:
        s["start"] = {k: pinned(v) for k, v in st.items()}
        s["host"] = {k: pinned(v) for k, v in st.items()}
        sim.upload(s["start"])
    return s


# ---- run ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "network_gradient":
        loss = s["net"].loss_backward(s["raw"].data_ptr(), s["new"].data_ptr(), case["nb"])
        return {"loss": loss, "grads": s["net"].get_grads()}
    if kind == "network_forward":
        s["net"].forward(s["raw"].data_ptr(), case["nb"], s["out"].data_ptr())
        return {"out": s["out"]}
    if kind == "ensemble":
        e = s["ensemble"]
        rows, cycles, dts = e.step()
        rows = [row_arrays(r) for r in rows]
        return {"SF": [m.get("SF") for m in e.sims], "T": [m.get("T") for m in e.sims],
                "rows": np.stack([r[0] for r in rows]), "whole": np.stack([r[1] for r in rows]),
                "cycles": np.array(cycles), "dt": np.array(dts)}
    sim = s["sim"]
    if kind == "diagnostics":
        sim.compute_velocities()
        real, whole = row_arrays(sim.stats())
        u, w = sim.velocities()
        return {"u": u, "w": w, "row": real, "whole": whole}
    if kind == "solve":
        sim.upload(s["start"])
        q = sim.multigrid()
        return {"SF": sim.get("SF"), "cycles": q}
    if kind == "advect":
        dt = sim.energy_time()
        return {"state": download(s), "dt": np.array([dt])}
    if kind == "timestep":
        row, q, dt = sim.step_host(s["host"])
    else:
        sim.upload(s["start"])
        sim.set_clock(0, 0.0)
        for _ in range(case["steps"]):
            row, q, dt = sim.step()
        download(s)
    real, whole = row_arrays(row)
    return {"state": s["host"], "row": real, "whole": whole, "cycles": q, "dt": np.array([dt])}


# ---- work --------------------------------------------------------------------------
def conv_flops(H, W):
    """Multiply-adds x 2 of the network's forward pass on one image."""
    layers = [(3, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (128, 128, 3),
              (128, 128, 3), (256, 128, 2), (128, 128, 2), (192, 64, 1), (64, 64, 1), (96, 32, 0), (32, 32, 0)]
    return sum(2.0 * 9 * ci * co * (H >> lev) * (W >> lev) for ci, co, lev in layers)


def solve_flops(nx, nz, grids, solver):
    """Smoother multiply-adds x 2 of one solve: 70 sweeps a visit, 15 a point."""
    per_cycle = sum(v * 70.0 * 30.0 * (nx >> lev) * (nz >> lev) for lev, v in enumerate(VISITS[grids]))
    return CYCLES[solver] * per_cycle


def work(case):
    kind = case["kind"]
    if kind in ("network_gradient", "network_forward"):
        nb, H, W = case["nb"], case["H"], case["W"]
        nparam = 1.21e6
        if kind == "network_forward":
            return {"bytes": nb * H * W * 16.0 + 4 * nparam, "flops": nb * conv_flops(H, W)}
        return {"bytes": nb * H * W * 16.0 + 8 * nparam, "flops": 3.0 * nb * conv_flops(H, W)}
    if kind == "ensemble":
        sizes = [[(256, 64, 4), (512, 128, 5), (200, 96, 4)][i % 3] for i in range(case["count"])]
        total = {"bytes": 0.0, "flops": 0.0}
        for i, (nx, nz, grids) in enumerate(sizes):
            w = work(flow("timestep", nx, nz, grids, case["tpc"] + i, 1e5, 100, "window"))
            total = {k: total[k] + w[k] for k in total}
        return total
    nx, nz = case["nx"], case["nz"]
    nodes, plane = (nx + 1.0) * (nz + 1.0), (nx + 5.0) * (nz + 5.0) * 8.0
    tracers = nodes * case["tpc"]
    if kind == "diagnostics":
        return {"bytes": 5 * plane, "flops": 60.0 * nodes}
    if kind == "solve":
        return {"bytes": 3 * plane, "flops": solve_flops(nx, nz, case["grids"], case["solver"])}
    stages = 4 * (60.0 * tracers + 80.0 * nodes)
    state_bytes = 6 * plane + 36.0 * tracers
    if kind == "advect":
        return {"bytes": state_bytes, "flops": stages}
    steps = case.get("steps", 1)
    if kind == "shipped":
        n = nx * nz / 4.0
        band = 2.0 * n * nx  # one banded factorisation: n x kl x (ku + kl) multiply-adds
        return {"bytes": state_bytes, "flops": steps * (6 * (band * nx * 2 + 70 * 30.0 * nodes) + stages)}
    return {"bytes": state_bytes,
            "flops": steps * (4 * solve_flops(nx, nz, case["grids"], case["solver"]) + stages)}


# ---- exact -------------------------------------------------------------------------
def exact_velocities(p, SF):
    """u = dSF/dz, w = -dSF/dx by central differences, with the free-slip mirrors."""
    span, nx, nz = p.order // 2 + 1, p.nx, p.nz
    dr, ds = p.aspect / nx, 1.0 / nz
    u, w = np.zeros((nz + 3, nx + 3)), np.zeros((nz + 3, nx + 3))
    S = SF[span - 2:span + nz + 3, span - 2:span + nx + 3]  # rows -2..nz+2
    inner = slice(2, -2)
    uu = (S[3:-1, inner] - S[1:-3, inner]) / (2 * ds)  # nodes 0..nz x 0..nx
    ww = -(S[inner, 3:-1] - S[inner, 1:-3]) / (2 * dr)
    uu[:, 0] = uu[:, -1] = 0.0
    ww[0, :] = ww[-1, :] = 0.0
    u[1:-1, 1:-1], w[1:-1, 1:-1] = uu, ww
    u[0, 1:-1], u[-1, 1:-1] = uu[1], uu[-2]
    u[:, 0], u[:, -1] = -u[:, 2], -u[:, -3]
    w[1:-1, 0], w[1:-1, -1] = ww[:, 1], ww[:, -2]
    w[0, :], w[-1, :] = -w[2, :], -w[-3, :]
    return u, w


def exact_advection(p, st):
    """Positions after one RK4 step in the velocities of SF, and dt (stability_RK4), in 64 bits."""
    u, w = exact_velocities(p, st["SF"])
    nx, nz = p.nx, p.nz
    dr, ds = p.aspect / nx, 1.0 / nz
    inner = np.abs(u[1:-1, 1:-1]) / dr + np.abs(w[1:-1, 1:-1]) / ds
    dt = p.courant / (inner.max() / 2.8 + (4 / dr ** 2 + 4 / ds ** 2) / 2.8)

    def tables(f):
        d = np.zeros_like(f)
        d[:, 1:-1] = (f[:, 2:] - f[:, :-2]) / (2 * dr)
        return torch.from_numpy(f).cuda(), torch.from_numpy(d).cuda()

    fields = [tables(u), tables(w)]

    def velocity(r, s):
        """Taylor step in r from the nearer column, then in s from the nearer row."""
        i, k = (r / dr).long(), (s / ds).long()
        hr, hs = r - i * dr, s - k * ds
        far = hr > dr / 2
        i, hr = torch.where(far, i + 1, i), torch.where(far, hr - dr, hr)
        up = hs > ds / 2
        k, hs = torch.where(up, k + 1, k), torch.where(up, hs - ds, hs)

        def at(f, d, kk):
            return f[kk + 1, i + 1] + d[kk + 1, i + 1] * hr

        return [at(f, d, k) + (at(f, d, k + 1) - at(f, d, k - 1)) / (2 * ds) * hs for f, d in fields]

    r0, s0 = torch.from_numpy(st["rtr"]).cuda(), torch.from_numpy(st["str"]).cuda()
    r, s, ra, sa = r0, s0, 0.0, 0.0
    for weight, forward in ((1, 0.5), (2, 0.5), (2, 1.0), (1, 0.0)):
        vr, vs = velocity(r, s)
        ra, sa = ra + weight * vr, sa + weight * vs
        r, s = r0 + forward * dt * vr, s0 + forward * dt * vs
    return (r0 + dt / 6 * ra).cpu().numpy(), (s0 + dt / 6 * sa).cpu().numpy(), dt


def exact_network(case, seed):
    """The network in 64 bits (no rounding of weights or activations) by plain torch."""
    import torch.nn.functional as F
    raw, new = images(case["nb"], case["H"], case["W"], seed)
    raw, new = raw.double(), new.double()
    flat = torch.from_numpy(np.load(WEIGHTS).astype(np.float32)).double().cuda().requires_grad_(True)
    layers = [(3, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 128), (128, 128), (256, 128),
              (128, 128), (192, 64), (64, 64), (96, 32), (32, 32)]
    at, par = 0, []
    for ci, co in layers:
        w = flat[at:at + co * 9 * ci].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        at += co * 9 * ci
        par.append((w, flat[at:at + co]))
        at += co
    head, hb = flat[at:at + 32], flat[at + 32]

    def conv(l, x):
        return F.relu(F.conv2d(x, par[l][0], par[l][1], padding=1))

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3)

    c0, c1, c2 = raw[:, 0], raw[:, 1], raw[:, 2]
    mean = c0.mean((1, 2), keepdim=True)
    std = ((c0 * c0).mean((1, 2), keepdim=True) - mean * mean).sqrt()
    r1 = (c1 * c1).mean((1, 2), keepdim=True).sqrt()
    r2 = (c2 * c2).mean((1, 2), keepdim=True).sqrt()
    x = torch.stack([(c0 - mean) / std, c1 / r1, c2 / r2], 1)
    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, F.avg_pool2d(e0, 2)))
    e2 = conv(5, conv(4, F.avg_pool2d(e1, 2)))
    b3 = conv(7, conv(6, F.avg_pool2d(e2, 2)))
    d2 = conv(9, conv(8, torch.cat([up(b3), e2], 1)))
    d1 = conv(11, conv(10, torch.cat([up(d2), e1], 1)))
    d0 = conv(13, conv(12, torch.cat([up(d1), e0], 1)))
    out = (d0 * head.view(1, 32, 1, 1)).sum(1) + hb
    if case["kind"] == "network_forward":
        return {"out": out.detach()}
    d = (out - (new - c2) / r2)[:, 1:, 1:]
    loss = (d * d).sum() / (case["nb"] * (case["H"] - 1) * (case["W"] - 1))
    loss.backward()
    return {"loss": float(loss), "grads": flat.grad.detach()}


def exact(case, seed):
    if case["kind"] in ("network_gradient", "network_forward"):
        return exact_network(case, seed)
    if case["kind"] == "diagnostics":
        p = params(case)
        if p.nx % (1 << (p.grids - 1)) or p.nz % (1 << (p.grids - 1)):  # a grid the set-up may round
            return None
        u, w = exact_velocities(p, cell_flow(p, seed))
        return {"u": u, "w": w, "row": None, "whole": None}
    if case["kind"] == "advect":
        p = params(case)
        if p.nx % (1 << (p.grids - 1)) or p.nz % (1 << (p.grids - 1)):  # a grid the set-up may round
            return None
        st = start_state(p, seed)
        st["SF"] = cell_flow(p, seed)
        r, s, dt = exact_advection(p, st)
        return {"state": {"rtr": r, "str": s}, "dt": np.array([dt])}
    return None
