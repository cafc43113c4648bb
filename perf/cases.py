"""Representative calls of the library through its public entry points, with
their inputs: what a program that advances two-phase flows with it spends its
time on, from one small pressure solve to a time step of a 256^3 box.

listed()            the cases
draw(rng)           one more case of the same ranges
prepare(case, seed) what the program holds before the call
run(state)          one pass, and its outputs
work(case)          bytes and floating point operations that a pass cannot do without
exact(case, seed)   the outputs in plain 64-bit arithmetic, where one call defines them

Kinds:
  step      a simulation of `steps` time steps in 2D from host fields to host
            fields (upload, start-up, steps, download); `geometry` planar or
            axisym; `form` plain (the reference's solvers) or spectral (FFT
            preconditioner, unregularised momentum CG)
  batch     independent droplet-on-cylinder simulations advanced together, in
            the production form (single-precision stencils, warm start,
            spectral preconditioner)
  box       the same as step, in 3D
  poisson   the variable-density pressure solve alone (right-hand side,
            preconditioner, PCG), as a host code's own time loop calls it
  noalloc   the same solve on the caller's device buffers
  fft       the constant-density Poisson solve
  train     one optimiser step of the warm-start network on a batch of crops
  gradient  forward and backward of the network on one full plane
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parties-vof-ibm_b200"))

from pvof import abi, cases, cnn, runtime  # noqa: E402

DT = 1e-4


def listed():
    return [
        # the smallest calls: a host code's pressure correction on a coarse grid,
        # where launches and waits count
        {"name": "noalloc 48x96", "kind": "noalloc", "nx": 48, "ny": 96, "geometry": "planar"},
        # the direct solver on the Rayleigh-Taylor grid (a width that is no power of two)
        {"name": "fft 200x800", "kind": "fft", "nx": 200, "ny": 800},
        # the direct solver at a production size
        {"name": "fft 1024x2048", "kind": "fft", "nx": 1024, "ny": 2048},
        # the library's benchmark workload: the planar instability, plain FP64
        {"name": "step 128x512", "kind": "step", "geometry": "planar", "nx": 128, "ny": 512, "steps": 1,
         "form": "plain", "tension": False, "ratio": 1.0 / 3.0},
        # axisymmetric rising bubble with surface tension on an odd grid (grid-wide solvers)
        {"name": "bubble 241x482", "kind": "step", "geometry": "axisym", "nx": 241, "ny": 482, "steps": 1,
         "form": "plain", "tension": True, "ratio": 1e-2},
        # a production time step: density ratio 1e-3 on 1024 x 1024 in the fast form
        {"name": "step spectral 1024x1024", "kind": "step", "geometry": "planar", "nx": 1024, "ny": 1024, "steps": 1,
         "form": "spectral", "tension": False, "ratio": 1e-3},
        # a parameter study: droplets on cylinders advanced together
        {"name": "droplets 6x 64..192", "kind": "batch", "count": 6, "lo": 64, "hi": 192, "steps": 1},
        # the pressure solve alone, planes larger than the L2 cache
        {"name": "poisson 2048x2048", "kind": "poisson", "nx": 2048, "ny": 2048},
        # 3D, the reference's solvers, an odd box
        {"name": "box 120x97x104", "kind": "box", "nx": 120, "ny": 97, "nz": 104, "steps": 1, "form": "plain"},
        # 3D at production size in the fast form
        {"name": "box spectral 256x256x256", "kind": "box", "nx": 256, "ny": 256, "nz": 256, "steps": 1,
         "form": "spectral"},
        # training the warm-start network on 64 x 64 crops
        {"name": "train 64x64 b8", "kind": "train", "nx": 64, "ny": 64, "batch": 8},
        # the network on a full plane, forward and backward
        {"name": "gradient 1000x1000", "kind": "gradient", "nx": 1000, "ny": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["noalloc", "fft", "step", "step", "spectral", "batch", "poisson", "box", "box spectral", "train",
                       "gradient"])
    if kind == "noalloc":
        nx = _log(rng, 24, 200)
        ny = min(_log(rng, nx, 4 * nx), 72000 // (nx + 7) - 7, 1000)
        return {"kind": "noalloc", "nx": nx, "ny": ny, "geometry": "planar"}
    if kind == "fft":
        nx = rng.choice([2 ** rng.randint(5, 11), _log(rng, 40, 320)])
        return {"kind": "fft", "nx": nx, "ny": _log(rng, 32, 2048)}
    if kind == "step":
        nx = _log(rng, 32, 256)
        geometry = rng.choice(["planar", "axisym"])
        return {"kind": "step", "geometry": geometry, "nx": nx, "ny": _log(rng, nx, 2 * nx + 64), "steps": 1,
                "form": "plain", "tension": rng.random() < 0.5, "ratio": rng.choice([0.5, 1.0 / 3.0, 0.1, 1e-2])}
    if kind == "spectral":
        nx = rng.choice([64, 96, 128, 160, 256, 320, 384, 512, 640, 768, 1024])
        return {"kind": "step", "geometry": "planar", "nx": nx, "ny": _log(rng, 64, 1024), "steps": 1,
                "form": "spectral", "tension": rng.random() < 0.5, "ratio": rng.choice([0.1, 1e-2, 1e-3])}
    if kind == "batch":
        lo = rng.choice([64, 80, 96])
        return {"kind": "batch", "count": rng.randint(2, 8), "lo": lo, "hi": rng.choice([96, 128, 160, 192]), "steps": 1}
    if kind == "poisson":
        return {"kind": "poisson", "nx": _log(rng, 200, 1600), "ny": _log(rng, 200, 1600)}
    if kind == "box":
        return {"kind": "box", "nx": _log(rng, 16, 128), "ny": _log(rng, 16, 128), "nz": _log(rng, 16, 128), "steps": 1,
                "form": "plain"}
    if kind == "box spectral":
        return {"kind": "box", "nx": 2 ** rng.randint(4, 8), "ny": _log(rng, 24, 200), "nz": 2 ** rng.randint(4, 7),
                "steps": 1, "form": "spectral"}
    if kind == "train":
        return {"kind": "train", "nx": _log(rng, 24, 160), "ny": _log(rng, 24, 160), "batch": rng.randint(1, 12)}
    return {"kind": "gradient", "nx": _log(rng, 48, 1024), "ny": _log(rng, 48, 1024)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _stream_velocity(grid, rng, amp):
    """A divergence-free velocity of a few seeded modes that vanishes into the
    y walls (planar, x periodic), on the staggered G range."""
    NX, NY, _ = cases.dims(grid)
    Lx, Ly = grid.xmax - grid.xmin, grid.ymax - grid.ymin
    dx, dy = Lx / (NX - 1), Ly / (NY - 1)
    x, y = np.arange(NX + 1) * dx, np.arange(NY + 1) * dy
    psi = np.zeros((NY + 1, NX + 1))
    for _ in range(3):
        m, n = rng.integers(1, 4, size=2)
        a, ph = rng.uniform(0.3, 1.0), rng.uniform(0, 2 * np.pi)
        psi += a / (np.pi * max(2 * m / Lx, n / Ly)) * np.sin(np.pi * n * y / Ly)[:, None] \
            * np.cos(2 * np.pi * m * x / Lx + ph)[None, :]
    psi *= amp
    return (psi[1:, :-1] - psi[:-1, :-1]) / dy, -(psi[:-1, 1:] - psi[:-1, :-1]) / dx


def _pinned(n):
    return torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy()


class _Sim:
    """A solver, its initial fields as host blocks, and the blocks that results
    are read into."""

    def __init__(self, grid, params, fields, results, particles=None):
        self.solver = runtime.Solver(grid, params, device=0)
        if particles:
            self.solver.set_particles(particles)
        self.start = {}
        for name, arr in fields.items():
            b = _pinned(self.solver.block_count(name))
            b[:] = cases.field_to_block(grid, arr).ravel()
            self.start[name] = b
        self.out = {name: _pinned(self.solver.block_count(name)) for name in results}

    def begin(self):
        for name, block in self.start.items():
            self.solver.upload(name, block)
        self.solver.initialize()

    def end(self):
        return {name: self.solver.download(name, out=block) for name, block in self.out.items()}


def _planar_setup(case, rng, **kw):
    Ly = case["ny"] / case["nx"]
    Cn = max(0.01, 1.5 / case["nx"]) if case["nx"] < 512 else 0.005
    r = case.get("ratio", 1e-3)
    grid, params, planes = cases.rayleigh_taylor(
        case["nx"], case["ny"], Lx=1.0, Ly=Ly, Cn=Cn, amp=rng.uniform(0.02, 0.06), y0=Ly * rng.uniform(0.45, 0.55),
        atwood=(1 - r) / (1 + r), Re=rng.uniform(2000, 4000), surface_tension=case.get("tension", False),
        P_CG_MAXIT=40000, **kw)
    return grid, params, planes


def _step_state(case, seed):
    rng = np.random.default_rng(seed)
    kw = {}
    if case["form"] == "spectral":
        kw = {"pressure_preconditioner": 1, "velocity_cg_unregularized": 1}
    if case["geometry"] == "planar":
        grid, params, planes = _planar_setup(case, rng, **kw)
        planes["U"], planes["V"] = _stream_velocity(grid, rng, 0.2)
    else:
        zmax = 2.0 * case["ny"] / case["nx"]
        grid, params, planes = cases.rising_bubble(
            case["nx"], case["ny"], rmax=2.0, zmax=zmax, radius=rng.uniform(0.45, 0.55), zc=zmax * rng.uniform(0.25, 0.4),
            Cn=max(0.01, 3.0 / case["nx"]), rho_ratio=case["ratio"], mu_ratio=case["ratio"],
            Re=rng.uniform(80, 120), surface_tension=case["tension"], We=200.0, P_CG_MAXIT=40000, **kw)
        xc, yc, xu, yv = cases.cell_centres(grid)
        a, b = rng.uniform(0.05, 0.15, size=2)
        planes["U"] = a * np.sin(np.pi * xu / 2.0)[None, :] * np.sin(2 * np.pi * yc / zmax)[:, None]
        planes["V"] = b * np.cos(0.5 * np.pi * xc / 2.0)[None, :] * np.sin(np.pi * yv / zmax)[:, None]
    return _Sim(grid, params, planes, ("C_L", "U", "V", "P"))


def _batch_state(case, seed):
    rng = np.random.default_rng(seed)
    widths = cases.smooth_widths(min(case["lo"], case["hi"]), max(case["lo"], case["hi"]))
    sims = []
    for q in range(case["count"]):
        grid, params, planes, parts = cases.droplet_on_cylinder(
            widths[q % len(widths)], Rd=rng.uniform(0.3, 0.6), Rs=rng.uniform(0.2, 0.4), theta=rng.uniform(30.0, 150.0),
            P_CG_MAXIT=20000, stencil_fp32=1, pressure_warm_start=1, pressure_preconditioner=1,
            velocity_cg_unregularized=1)
        planes["U"], planes["V"] = _stream_velocity(grid, rng, 0.1)
        sims.append(_Sim(grid, params, dict(planes, C_L=planes["F"]), ("C_L", "U", "V", "P"), particles=parts))
    return sims


def _box_state(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = 2.0 / nx
    Lx, Ly, Lz = 2.0, h * ny, h * nz
    grid = cases.box_grid(nx, ny, nz, Lx, Ly, Lz)
    Cn = max(0.005, 1.5 * h)
    kw = {"pressure_preconditioner": 1, "velocity_cg_unregularized": 1} if case["form"] == "spectral" else {}
    params = cases.default_params(Re=rng.uniform(800, 1200), rho1=1.0, rho2=1e-2, mu1=1.0, mu2=1e-2, Cn=Cn,
                                  Pe_CH=1.0 / Cn, surface_tension=1, We=100.0, P_CG_MAXIT=40000, **kw)
    f64 = dict(dtype=torch.float64, device="cuda")
    NX, NY, NZ = cases.dims(grid)
    x, y, z = (torch.arange(n, **f64) for n in (NX, NY, NZ))
    xc, yc, zc = (x + 0.5) * h, (y + 0.5) * h, (z + 0.5) * h
    H = torch.full((NZ, NX), 0.5 * Ly, **f64)
    for _ in range(6):
        m, n = rng.integers(1, 4, size=2)
        H += rng.uniform(0.0, 0.02) * torch.cos(2 * np.pi * (m * xc[None, :] / Lx + n * zc[:, None] / Lz)
                                                + rng.uniform(0, 2 * np.pi))
    two = 2 * np.pi
    a = rng.uniform(0.05, 0.15, size=3)
    ph = rng.uniform(0, two, size=3)
    fields = {
        "F": 0.5 * (1.0 + torch.tanh((H[:, None, :] - yc[None, :, None]) / (math.sqrt(2.0) * Cn))),
        "U": a[0] * torch.sin(two * x * h / Lx + ph[0])[None, None, :] * torch.sin(np.pi * yc / Ly)[None, :, None]
        * torch.cos(two * zc / Lz)[:, None, None],
        "V": a[1] * torch.cos(two * xc / Lx + ph[1])[None, None, :] * torch.sin(np.pi * y * h / Ly)[None, :, None]
        * torch.cos(two * zc / Lz)[:, None, None],
        "W": a[2] * torch.cos(two * xc / Lx)[None, None, :] * torch.sin(np.pi * yc / Ly)[None, :, None]
        * torch.sin(two * z * h / Lz + ph[2])[:, None, None],
        "P": torch.zeros((NZ, NY, NX), **f64),
    }
    G = cases.G
    sim = _Sim(grid, params, {}, ("C_L", "U", "V", "W", "P"))
    for name, t in fields.items():
        b = torch.zeros(cases.block_shape(grid), dtype=torch.float64, pin_memory=True)
        b[G:G + NZ, G:G + NY, G:G + NX] = t.cpu()
        sim.start[name] = b.view(-1).numpy()
    return sim


def _poisson_setup(case, seed):
    rng = np.random.default_rng(seed)
    grid, params, planes = _planar_setup(dict(case, ratio=1e-2), rng)
    U, V = _stream_velocity(grid, rng, 0.2)
    NX, NY, _ = cases.dims(grid)
    xc, yc, xu, yv = cases.cell_centres(grid)
    Ly = grid.ymax
    # the part of the velocity that the projection removes
    m, n = rng.integers(1, 4, size=2)
    planes["U"] = U + 0.05 * np.sin(2 * np.pi * m * xu + 0.3)[None, :] * np.cos(np.pi * n * yc / Ly)[:, None]
    planes["V"] = V + 0.05 * np.cos(2 * np.pi * m * xc)[None, :] * np.sin(np.pi * n * yv / Ly)[:, None]
    return grid, params, planes


def _interior_of(grid, block):
    return cases.interior(grid, cases.block_plane(grid, block))


def _fft_setup(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    grid, params, _ = cases.rayleigh_taylor(nx, ny, Lx=1.0, Ly=ny / nx, Cn=0.02)
    x = (np.arange(nx) + 0.5) / nx
    y = (np.arange(ny) + 0.5) / ny
    rhs = 0.1 * rng.standard_normal((ny, nx))
    for _ in range(4):
        m, n = rng.integers(1, 6, size=2)
        rhs += rng.standard_normal() * np.cos(2 * np.pi * m * x + rng.uniform(0, 6.28))[None, :] \
            * np.cos(np.pi * n * y)[:, None]
    rhs -= rhs.mean()
    plane = np.zeros((ny + 1, nx + 1))
    plane[:ny, :nx] = rhs
    return grid, params, plane


def _noalloc_setup(case, seed):
    """rho and rhs on the physical cells, from a smooth interface and the
    divergence of a smooth velocity over a time step."""
    grid, params, planes = _poisson_setup(case, seed)
    rho, rhs = _poisson_planes(grid, params, planes, 0)
    return grid, params, rho, rhs


def _poisson_planes(grid, params, planes, stage):
    """Density and right-hand side on the physical cells (x periodic, walls in y)."""
    NX, NY, _ = cases.dims(grid)
    c = np.clip(planes["F"], 0.0, 1.0)[:NY - 1, :NX - 1]
    rho = c + params.rho2 / params.rho1 * (1.0 - c)
    u, v = planes["U"][:NY - 1, :NX - 1].copy(), planes["V"][:NY, :NX - 1].copy()
    v[0] = 0.0
    v[NY - 1] = 0.0
    dx = (grid.xmax - grid.xmin) / (NX - 1)
    bet = (4.0 / 15.0, 1.0 / 15.0, 1.0 / 6.0)[stage]
    rhs = (np.roll(u, -1, axis=1) - u + v[1:] - v[:-1]) / dx / (DT * 2.0 * bet)
    return rho, rhs


def _ghosted(grid, phys):
    """Physical cells into a ghosted plane, x periodic, walls in y mirrored."""
    G = cases.G
    return np.ascontiguousarray(np.pad(np.pad(phys, ((G, G + 1), (0, 0)), mode="edge"), ((0, 0), (G, G + 1)),
                                       mode="wrap"))


def _net_planes(gen, H, W, n):
    """Network inputs (density, scaled residual, scaled correction) and targets:
    smooth seeded fields plus a little noise."""
    d = dict(dtype=torch.float32, device="cuda")
    y = torch.linspace(0, 1, H, **d)[:, None]
    x = torch.linspace(0, 1, W, **d)[None, :]
    out = []
    for _ in range(n):
        r = torch.rand(8, generator=gen, device="cuda")
        rho = 0.5 + 0.5 * torch.tanh((y - 0.5 - 0.1 * torch.cos(6.28 * (x + r[0]))) * 20)
        res = torch.sin(12 * r[1] * x + 6 * y) + 0.3 * torch.randn(H, W, generator=gen, **d)
        phi = 1.4 * torch.cos(6.28 * (x + r[2])) * torch.cos(3.14 * y * (1 + r[3]))
        t = 0.2 * torch.sin(9 * (x + r[4])) * torch.cos(7 * (y + r[5])) + 0.02 * torch.randn(H, W, generator=gen, **d)
        out.append((torch.stack([rho.expand(H, W), res, phi]).contiguous().view(-1), t.contiguous().view(-1)))
    return out


def _net_params(seed):
    """Weights in mid-training: the initialisation with a last layer that is not zero."""
    p = cnn.init_params(seed)
    rng = np.random.default_rng(seed + 1)
    p = p + (0.01 * rng.standard_normal(p.size)).astype(np.float32)
    return p.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return {"case": case, "sim": _step_state(case, seed)}
    if kind == "batch":
        return {"case": case, "sims": _batch_state(case, seed)}
    if kind == "box":
        return {"case": case, "sim": _box_state(case, seed)}
    if kind == "poisson":
        grid, params, planes = _poisson_setup(case, seed)
        sim = _Sim(grid, params, planes, ("DELTAP",))
        sim.begin()
        sim.solver.set_stage(0, DT)
        return {"case": case, "sim": sim, "grid": grid}
    if kind == "fft":
        grid, params, plane = _fft_setup(case, seed)
        sim = _Sim(grid, params, {"P_RHS": plane}, ("DELTAP",))
        sim.solver.upload("P_RHS", sim.start["P_RHS"])
        return {"case": case, "sim": sim, "grid": grid}
    if kind == "noalloc":
        grid, params, rho, rhs = _noalloc_setup(case, seed)
        dev = {k: torch.from_numpy(_ghosted(grid, a)).cuda() for k, a in (("rho", rho), ("rhs", rhs))}
        dev["phi"] = torch.zeros_like(dev["rho"])
        f = runtime.load().pvof_Pressure_solve_cg_noalloc
        f.argtypes = [C.POINTER(abi.GridDesc), C.POINTER(abi.Params), C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                      C.POINTER(C.c_int), C.POINTER(C.c_double)]
        return {"case": case, "grid": grid, "params": params, "dev": dev, "solve": f,
                "stream": torch.cuda.current_stream().cuda_stream}
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    H, W = case["ny"], case["nx"]
    net = cnn.Network(H, W, params=_net_params(seed))
    if kind == "train":
        batch = _net_planes(gen, H, W, case["batch"])
        net.step = 100   # resumed training: moments of earlier steps
        net.m.copy_(1e-3 * torch.randn(net.m.numel(), generator=gen, device="cuda"))
        net.v.fill_(1e-3)
        return {"case": case, "net": net, "batch": batch}
    (x, dy), = _net_planes(gen, H, W, 1)
    return {"case": case, "net": net, "x": x, "dy": dy / (H * W)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "box"):
        sim = state["sim"]
        sim.begin()
        sim.solver.run_steps(case["steps"], DT)
        return sim.end()
    if kind == "batch":
        for sim in state["sims"]:
            sim.begin()
        runtime.run_steps_batched([sim.solver for sim in state["sims"]], case["steps"], DT)
        return [sim.end() for sim in state["sims"]]
    if kind == "poisson":
        sim = state["sim"]
        sim.solver.call("Pressure_set_RHS")
        sim.solver.call("Pressure_compute_preconditioner")
        sim.solver.call("Pressure_solve_cg", None)
        return _interior_of(state["grid"], sim.end()["DELTAP"])
    if kind == "fft":
        sim = state["sim"]
        sim.solver.call("Pressure_solve_fft")
        return _interior_of(state["grid"], sim.end()["DELTAP"])
    if kind == "noalloc":
        dev = state["dev"]
        dev["phi"].zero_()
        rc = state["solve"](C.byref(state["grid"]), C.byref(state["params"]), dev["rho"].data_ptr(),
                            dev["rhs"].data_ptr(), dev["phi"].data_ptr(), state["stream"], None, None)
        if rc < 0:
            raise RuntimeError("pvof_Pressure_solve_cg_noalloc: %d" % rc)
        return cases.interior(state["grid"], dev["phi"])
    net = state["net"]
    if kind == "train":
        loss = net.train_batch(state["batch"], 1e-3)
        return {"loss": loss, "gradient": net.g, "parameters": net.p}
    return {"gradient": net.gradient(state["x"], state["dy"]), "y": net.y}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _net_work(n, backward):
    macs = 9 * (3 * 32 + 4 * 32 * 32 + 32)
    flops = 2.0 * macs * n
    if backward:
        flops = 3.0 * flops - 2.0 * 9 * 3 * 32 * n   # no input gradient of the first layer
    return flops


def work(case):
    kind = case["kind"]
    n = float(case.get("nx", 0) * case.get("ny", 0) * case.get("nz", 1))
    if kind == "train":
        b = case["batch"]
        return {"bytes": 4.0 * 4 * n * b + 4.0 * 38000 * 8, "flops": _net_work(n, True) * b}
    if kind == "gradient":
        return {"bytes": 4.0 * 5 * n + 4.0 * 38000 * 2, "flops": _net_work(n, True)}
    if kind == "fft":
        return {"bytes": 16.0 * n, "flops": n * (5.0 * math.log2(case["nx"]) + 10.0)}
    if kind in ("poisson", "noalloc"):
        # density (or velocity and phase) in, correction out; the iteration
        # count of a PCG without a grid-dependent shortcut: about 1.5 max(nx, ny)
        return {"bytes": 8.0 * 4 * n, "flops": 30.0 * n * 1.5 * max(case["nx"], case["ny"])}
    if kind == "batch":
        widths = cases.smooth_widths(min(case["lo"], case["hi"]), max(case["lo"], case["hi"]))
        n = float(sum(2 * widths[q % len(widths)] ** 2 for q in range(case["count"])))
        return {"bytes": 8.0 * 9 * n, "flops": 3.0 * 6000.0 * n * case["steps"]}
    fields = 10 if kind == "box" else 8
    per = 6000.0   # stencils, a few momentum and biharmonic iterations, an FFT preconditioned pressure solve
    if case["form"] == "plain":
        per = 2000.0 + 30.0 * 1.5 * max(case["nx"], case["ny"])
    return {"bytes": 8.0 * fields * n, "flops": 3.0 * per * n * case["steps"]}


# ---------------------------------------------------------------------------
# the same outputs in plain 64-bit arithmetic
# ---------------------------------------------------------------------------

def _poisson_exact(grid, rho, rhs):
    """div(2/(rho+rho') grad phi) = rhs on square cells, x periodic, mirror
    walls in y, mean-free: conjugate gradients preconditioned by the
    constant-density inverse (FFT in x, even extension in y)."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    rho = torch.as_tensor(np.ascontiguousarray(rho), device=dev)
    b = torch.as_tensor(np.ascontiguousarray(rhs), device=dev)
    ny, nx = rho.shape
    i2 = (nx / (grid.xmax - grid.xmin)) ** 2
    j2 = (ny / (grid.ymax - grid.ymin)) ** 2
    cx = 2.0 / (rho + torch.roll(rho, -1, 1)) * i2
    cy = 2.0 / (rho[:-1] + rho[1:]) * j2

    def op(p):   # minus the operator: positive
        fx = cx * (torch.roll(p, -1, 1) - p)
        fy = cy * (p[1:] - p[:-1])
        r = fx - torch.roll(fx, 1, 1)
        r[:-1] += fy
        r[1:] -= fy
        return -r

    diag = cx + torch.roll(cx, 1, 1)
    diag[:-1] += cy
    diag[1:] += cy
    s = diag.rsqrt()
    kx = torch.arange(nx // 2 + 1, device=dev, dtype=torch.float64)
    ky = torch.arange(2 * ny, device=dev, dtype=torch.float64)
    lam = i2 * (2 - 2 * torch.cos(2 * np.pi * kx / nx))[None, :] + j2 * (2 - 2 * torch.cos(np.pi * ky / ny))[:, None]
    lam[0, 0] = j2

    def inverse(r):   # mirror walls: the even extension, periodic in y
        f = torch.fft.rfft2(torch.cat([r, r.flip(0)], 0)) / lam
        return torch.fft.irfft2(f, s=(2 * ny, nx))[:ny]

    phi = torch.zeros_like(b)
    r = -(b - b.mean())
    z = s * inverse(s * r)
    d = z.clone()
    g = (r * z).sum()
    r0 = float((r * r).sum()) ** 0.5
    for _ in range(400):
        ad = op(d)
        a = g / (d * ad).sum()
        phi += a * d
        r -= a * ad
        if float((r * r).sum()) ** 0.5 < 1e-14 * r0:
            break
        z = s * inverse(s * r)
        g2 = (r * z).sum()
        d = z + (g2 / g) * d
        g = g2
    return phi - phi.mean()


def _fft_exact(grid, rhs):
    """lap phi = rhs: FFT in x, a tridiagonal system in y per wave number (mirror
    walls), the mean mode zero in the first row."""
    ny, nx = rhs.shape
    i2 = (nx / (grid.xmax - grid.xmin)) ** 2
    j2 = (ny / (grid.ymax - grid.ymin)) ** 2
    f = np.fft.rfft(rhs, axis=1)
    lam = i2 * (2 - 2 * np.cos(2 * np.pi * np.arange(f.shape[1]) / nx))
    out = np.zeros_like(f)
    # elimination over all wave numbers at once
    b = np.full((ny, f.shape[1]), -2.0 * j2) - lam[None, :]
    b[0] += j2
    b[-1] += j2
    up = np.full((ny, f.shape[1]), j2)
    r = f.copy()
    b[0, 0], up[0, 0], r[0, 0] = 1.0, 0.0, 0.0
    g = np.zeros_like(b)
    bet = b[0].copy()
    out[0] = r[0] / bet
    for j in range(1, ny):
        g[j] = up[j - 1] / bet
        bet = b[j] - j2 * g[j]
        out[j] = (r[j] - j2 * out[j - 1]) / bet
    for j in range(ny - 2, -1, -1):
        out[j] -= g[j + 1] * out[j + 1]
    return np.fft.irfft(out, n=nx, axis=1)


def _net_forward64(p, x):
    """The network in 64 bits: six 3x3 convolutions, zero padding, ReLU between."""
    shapes = [(32, 3)] + [(32, 32)] * 4 + [(1, 32)]
    at, h = 0, x
    for q, (co, ci) in enumerate(shapes):
        w = p[at:at + co * ci * 9].view(co, ci, 3, 3)
        b = p[at + co * ci * 9:at + co * ci * 9 + co]
        at += co * ci * 9 + co
        # nine shifted products: no convolution library in 64 bits is needed
        hp = torch.nn.functional.pad(h, (1, 1, 1, 1))
        H, W = h.shape[1:]
        y = b[:, None] + sum(w[:, :, u, v] @ hp[:, u:u + H, v:v + W].reshape(ci, -1) for u in range(3) for v in range(3))
        h = y.view(co, H, W)
        if q < 5:
            h = torch.relu(h)
    return h.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "fft":
        grid, _, plane = _fft_setup(case, seed)
        return _fft_exact(grid, plane[:-1, :-1])
    if kind == "poisson":
        grid, params, planes = _poisson_setup(case, seed)
        return _poisson_exact(grid, *_poisson_planes(grid, params, planes, 0)).cpu().numpy()
    if kind == "noalloc":
        grid, params, rho, rhs = _noalloc_setup(case, seed)
        return _poisson_exact(grid, rho, rhs)
    if kind not in ("train", "gradient"):
        return None   # whole time steps: no short definition apart from the library's own
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    H, W = case["ny"], case["nx"]
    p = torch.tensor(_net_params(seed), device="cuda").double().requires_grad_(True)
    if kind == "train":
        batch = _net_planes(gen, H, W, case["batch"])
        loss = sum(((_net_forward64(p, x.double().view(3, H, W)) - t.double()) ** 2).mean() for x, t in batch) / len(batch)
        loss.backward()
        return {"loss": loss.detach(), "gradient": p.grad, "parameters": None}
    (x, dy), = _net_planes(gen, H, W, 1)
    y = _net_forward64(p, x.double().view(3, H, W))
    (y * (dy / (H * W)).double()).sum().backward()
    return {"gradient": p.grad, "y": y.detach()}
