"""The work a program has this framework do, as measurable cases.

Each case is one pass through the public entry points (the Python classes and
functions of the package, or the C ABI of libpfgpu with device pointers, which
it accepts wherever it accepts host ones):

  p2g       particles in, the six face fields and their 4^3 activity out
  transfer  P2G + saved copy + G2P (FLIP 0.97), the particle velocities out
  step      one whole SparseSim3DTP.step() from given particles
  project   one variable-coefficient pressure projection of given face fields
  mr        one whole MRSim3DTP.step() (2-level grid) from given particles
  train     optimiser steps of the learned coarse solve on harvested pairs

Every pass starts from the same inputs: the particles (or face velocities) are
handed over again at its beginning, as a program with new inputs does.
"""
import ctypes as C
import importlib
import math

import numpy as np
import torch

pf = importlib.import_module("adaptive-pf-flip_b200")
L = pf._lib
DEV = "cuda"

RHO_L, RHO_G = 1000.0, 1.0  # the density ratio of the repository's scenes


def listed():
    return [
        # a preview-size splat on a ragged grid, uneven particle counts in no memory order (after a splash):
        # launches and latency
        {"name": "p2g_ragged_40", "kind": "p2g", "nx": 40, "ny": 33, "nz": 27, "fill": "uneven", "order": "mixed"},
        # the transfer stress scene of the benchmark: bubble tank at 128^3, 11.3M particles
        {"name": "transfer_tank_128", "kind": "transfer", "nx": 128, "ny": 128, "nz": 128, "fill": "tank",
         "order": "cells"},
        # a unit-test-size simulation, the smallest step a program runs
        {"name": "step_rt_24", "kind": "step", "nx": 24, "ny": 24, "nz": 24, "fill": "full", "solver": "plain",
         "advect": 2, "extras": False},
        # the repository's base configuration: Rayleigh-Taylor at 48^3, reference-equivalent solver
        {"name": "step_rt_48", "kind": "step", "nx": 48, "ny": 48, "nz": 48, "fill": "full", "solver": "plain",
         "advect": 2, "extras": False},
        # every option of the step on a ragged grid with an open surface: adaptivity, surface tension, adaptive
        # timestep, volume correction, RK3
        {"name": "step_options_72", "kind": "step", "nx": 72, "ny": 58, "nz": 45, "fill": "tank", "solver": "plain",
         "advect": 3, "extras": True},
        # the largest: the Rayleigh-Taylor step at 256^3 (131M particles) with the learned pressure solver
        {"name": "step_rt_256_learned", "kind": "step", "nx": 256, "ny": 256, "nz": 256, "fill": "full",
         "solver": "learned", "advect": 2, "extras": False},
        # pressure alone, the drop-in solver to 1e-6: the ellipsoid system of the error tables
        {"name": "project_plain_64", "kind": "project", "nx": 64, "ny": 64, "nz": 64, "solver": "plain"},
        # ... and at a production size
        {"name": "project_plain_128", "kind": "project", "nx": 128, "ny": 128, "nz": 128, "solver": "plain"},
        # the learned solver on the same system
        {"name": "project_learned_128", "kind": "project", "nx": 128, "ny": 128, "nz": 128, "solver": "learned"},
        # the mixed-precision solver (FP32 inner solve) on an odd grid
        {"name": "project_mixed_51", "kind": "project", "nx": 51, "ny": 64, "nz": 45, "solver": "mixed_fp32"},
        # the multires step on a dam break refined around the free surface
        {"name": "mr_dam_128", "kind": "mr", "nx": 128, "ny": 128, "nz": 128, "dynamic": False},
        # training of the coarse network: forward, backward and Adam on pairs of a 64^3 system
        {"name": "train_64", "kind": "train", "n": 64, "steps": 4, "batch": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    n = _log(rng, lo, hi)
    if rng.random() < 0.4:
        return n, n, n
    return n, max(lo, int(n * rng.uniform(0.6, 1.0))), max(lo, int(n * rng.uniform(0.6, 1.0)))


def draw(rng):
    kind = rng.choice(["p2g", "transfer", "step", "step", "step", "project", "project", "project", "mr", "train"])
    if kind in ("p2g", "transfer"):
        nx, ny, nz = _dims(rng, 20, 128)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "fill": rng.choice(["full", "tank", "uneven"]),
                "order": rng.choice(["cells", "mixed"])}
    if kind == "step":
        solver = rng.choice(["plain", "plain", "learned"])
        nx, ny, nz = _dims(rng, 20, 112) if solver == "plain" else _dims(rng, 64, 160)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "fill": rng.choice(["full", "tank"]), "solver": solver,
                "advect": rng.choice([2, 2, 3]), "extras": rng.random() < 0.3}
    if kind == "project":
        solver = rng.choice(["plain", "plain", "learned", "mixed_fp32", "mixed_bf16"])
        nx, ny, nz = _dims(rng, 24, 112 if solver in ("plain", "learned") else 64)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "solver": solver}
    if kind == "mr":
        dynamic = rng.random() < 0.4
        nx, ny, nz = _dims(rng, 24, 96 if dynamic else 160)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "dynamic": dynamic}
    return {"kind": "train", "n": _log(rng, 40, 96), "steps": rng.choice([2, 4]), "batch": rng.choice([2, 4, 8])}


# ---------------------------------------------------------------------------
# inputs


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed + 1))


def _cells(case, fill):
    """Interior cells holding fluid, x fastest: all of them, the tank's lower 70 %, or the dam break's
    column and pool."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = torch.zeros((nz, ny, nx), dtype=torch.bool, device=DEV)
    if fill == "dam":
        m[1:nz - 1, 1:max(2, int(0.6 * ny)), 1:max(2, int(0.4 * nx))] = True
        m[1:nz - 1, 1:max(2, int(0.15 * ny)), 1:nx - 1] = True
    else:
        top = ny - 1 if fill in ("full", "uneven") else max(2, int(0.7 * ny))
        m[1:nz - 1, 1:top, 1:nx - 1] = True
    return m


def _particles(case, fill, seed):
    """Eight jittered particles per cell (one per sub-cell), or as many thrown over the cells at random
    ("uneven": none to about twenty in a cell); the heavy phase above the perturbed interface ("full"), or water
    around an air bubble ("tank"); small velocities."""
    g = _generator(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = 1.0 / max(nx, ny, nz)
    cell = _cells(case, fill).reshape(-1).nonzero().reshape(-1)
    if fill == "uneven":
        cell = cell[torch.randint(0, len(cell), (8 * len(cell),), generator=g, device=DEV).sort().values]
        sub = None
    else:
        cell = cell.repeat_interleave(8)
        sub = torch.arange(8, device=DEV).repeat(len(cell) // 8)
    n = len(cell)
    pos = torch.rand((n, 3), generator=g, device=DEV, dtype=torch.float32)
    at = cell
    for a, d in enumerate((nx, ny, nz)):
        c = (at % d).to(torch.float32)
        at = at // d
        if sub is None:
            pos[:, a] = (c + pos[:, a] * 0.999) * dx
        else:
            pos[:, a] = (c + 0.5 * ((sub >> a) & 1).to(torch.float32) + 0.499 * pos[:, a]) * dx
    del cell, at, sub
    lx, ly, lz = nx * dx, ny * dx, nz * dx
    x, y, z = pos[:, 0], pos[:, 1], pos[:, 2]
    if fill == "tank":
        r = 0.15 * min(lx, ly, lz)
        gas = (x - 0.5 * lx) ** 2 + (y - 0.3 * ly) ** 2 + (z - 0.5 * lz) ** 2 < r * r
    elif fill == "dam":
        gas = torch.zeros(n, dtype=torch.bool, device=DEV)
    else:
        gas = y < ly * (0.5 + 0.05 * torch.cos(2 * math.pi * x / lx) * torch.cos(2 * math.pi * z / lz))
    vel = torch.randn((n, 3), generator=g, device=DEV, dtype=torch.float32) * 0.1
    typ = gas.to(torch.uint8)
    vol = torch.ones(n, device=DEV, dtype=torch.float32)
    if case.get("order") == "mixed":
        q = torch.randperm(n, generator=g, device=DEV)
        pos, vel, typ = pos[q].contiguous(), vel[q].contiguous(), typ[q].contiguous()
    return {"n": n, "dx": dx, "pos": pos, "vel": vel, "typ": typ, "vol": vol}


def _phase(grid):
    pp = pf.PhaseParams(RHO_L, RHO_G)
    pp.rho_tilde_0 = pf.calibrateRhoTilde0(pp, 1.0, grid=grid)
    return pp


def _field_shapes(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return [(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)]


def _blocks(shape):
    return tuple((d + 3) // 4 for d in shape)


def _upload(lib, ctx, p):
    L.check(lib.pf_upload_particles(ctx, p["n"], p["pos"].data_ptr(), p["vel"].data_ptr(), p["typ"].data_ptr(),
                                    p["vol"].data_ptr()), ctx, "pf_upload_particles")


def _pressure_system(case, seed):
    """An all-fluid box with solid walls: random bubbles of light fluid (face raw masses 0) in heavy fluid
    (saturated masses) and a band-limited random velocity field on the faces."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng(7919 * (seed + 1))
    dx = 1.0 / max(nx, ny, nz)
    ext = np.array([nx, ny, nz]) * dx
    centres = r.uniform(0.0, 1.0, (64, 3)) * ext
    semi = r.uniform(0.02, 0.08, (64, 3))
    mk = torch.full((nz, ny, nx), 2.0, device=DEV)
    mk[1:-1, 1:-1, 1:-1] = 1.0
    k = np.arange(-8, 9)
    kz, ky, kx = np.meshgrid(k, k, k, indexing="ij")
    band = (kx ** 2 + ky ** 2 + kz ** 2 <= 64) & (kx ** 2 + ky ** 2 + kz ** 2 > 0)
    out = {"mk": mk, "dx": dx, "vel": [], "air": []}
    for a, shape in enumerate(_field_shapes(case)):
        ax = []
        for b in range(3):
            i = torch.arange(shape[2 - b], device=DEV, dtype=torch.float64)
            ax.append((i + (0.0 if b == a else 0.5)) * dx)
        coef = torch.zeros(band.shape, dtype=torch.complex128)
        m = int(band.sum())
        coef[torch.from_numpy(band)] = torch.from_numpy(r.normal(0, 1, m) + 1j * r.normal(0, 1, m)) / math.sqrt(m)
        f = coef.to(DEV)
        kk = torch.from_numpy(k).to(DEV, torch.float64)
        for b in (0, 1, 2):  # separable sum of the Fourier modes, one axis at a time (x, y, z)
            e = torch.exp(2j * math.pi * kk[:, None] * ax[b][None, :] / float(ext[b]))
            f = torch.movedim(torch.tensordot(f, e, dims=([2 - b], [0])), -1, 2 - b)
        v = f.real.to(torch.float32).contiguous()
        idx = torch.arange(shape[2 - a], device=DEV)
        wall = (idx <= 1) | (idx >= shape[2 - a] - 2)
        view = [None, None, None]
        view[2 - a] = slice(None)
        v = torch.where(wall[tuple(view)], torch.zeros_like(v), v).contiguous()
        air = torch.zeros(shape, dtype=torch.bool, device=DEV)
        for c, s in zip(centres, semi):
            d = (((ax[2] - c[2]) / s[2]) ** 2)[:, None, None] + (((ax[1] - c[1]) / s[1]) ** 2)[None, :, None] \
                + (((ax[0] - c[0]) / s[0]) ** 2)[None, None, :]
            air |= d < 1.0
        out["vel"].append(v)
        out["air"].append(air)
    return out


def _masses(sys_, rho_tilde_0):
    rmin = math.log(RHO_L / RHO_G) * RHO_G * rho_tilde_0
    full = 2.0 * (rmin + rho_tilde_0 * RHO_L)
    return [torch.where(a, 0.0, full).to(torch.float32).contiguous() for a in sys_["air"]]


def _solver(name, tol=1e-6):
    if name == "learned":
        return pf.SolverConfig(mode=pf.PF_SOLVER_LEARNED, rel_tol=tol, precond=pf.PF_PRECOND_NETWORK)
    if name == "exact_coarse":
        return pf.SolverConfig(mode=pf.PF_SOLVER_LEARNED, rel_tol=tol, precond=pf.PF_PRECOND_EXACT_COARSE)
    if name.startswith("mixed"):
        return pf.SolverConfig(mode=pf.PF_SOLVER_MIXED, rel_tol=tol, bf16_storage=int(name == "mixed_bf16"))
    return pf.SolverConfig(mode=pf.PF_SOLVER_PLAIN, rel_tol=tol)


DT_PROJECT = 1.0 / 240.0
MAX_ITER = 20000


def _set_field(lib, g, f, dense, act):
    L.check(lib.pf_grid_set_field(g.ctx, f, dense.data_ptr(), act.data_ptr()), g.ctx, "pf_grid_set_field")


def _get_field(lib, g, f, dense, act=None):
    L.check(lib.pf_grid_get_field(g.ctx, f, dense.data_ptr(), act.data_ptr() if act is not None else None), g.ctx,
            "pf_grid_get_field")


def _project_state(case, seed):
    s = _pressure_system(case, seed)
    g = pf.SparseMacGrid3D(case["nx"], case["ny"], case["nz"], s["dx"],
                            max_particles=s["mk"].numel() // 4)
    lib = pf.load()
    pp = _phase(g)
    acts = [torch.ones(_blocks(sh), dtype=torch.uint8, device=DEV) for sh in _field_shapes(case)]
    mk_act = torch.ones(_blocks(s["mk"].shape), dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    _set_field(lib, g, pf.PF_MK, s["mk"], mk_act)
    for a, m in enumerate(_masses(s, pp.rho_tilde_0)):
        _set_field(lib, g, pf.PF_MU + a, m, acts[a])
    return {"grid": g, "lib": lib, "pp": pp, "vel": s["vel"], "acts": acts,
            "p": torch.empty(s["mk"].shape, device=DEV), "out": [torch.empty_like(v) for v in s["vel"]]}


def prepare(case, seed):
    kind = case["kind"]
    lib = pf.load()
    st = {"case": case, "lib": lib}
    if kind in ("p2g", "transfer"):
        p = _particles(case, case["fill"], seed)
        g = pf.SparseMacGrid3D(case["nx"], case["ny"], case["nz"], p["dx"], max_particles=p["n"])
        st.update(grid=g, part=p, phase=_phase(g)._c())
        if kind == "transfer":
            st["vel"] = torch.empty_like(p["vel"])
        else:
            sh = _field_shapes(case)
            st["fields"] = [(torch.empty(s, device=DEV), torch.empty(_blocks(s), dtype=torch.uint8, device=DEV))
                            for s in sh + sh]
    elif kind == "step":
        p = _particles(case, case["fill"], seed)
        cap = p["n"] + p["n"] // 4 + 64 if case["extras"] else p["n"]
        sim = pf.SparseSim3DTP(case["nx"], case["ny"], case["nz"], p["dx"], max_particles=cap)
        sim.phase = _phase(sim.grid)
        sim.dt, sim.advection_order = 1.0 / 240.0, case["advect"]
        sim.alpha_liquid = sim.alpha_gas = 0.97
        sim.cg_iters, sim.cg_tol, sim.solver = MAX_ITER, 0.0, _solver(case["solver"])
        if case["solver"] == "learned":
            pf.LearnedCoarseSolver(sim.grid).load_default()
        if case["extras"]:
            sim.narrow_band_air = sim.gas_particle_coarsening = sim.liquid_particle_refill = True
            sim.surface_tension, sim.surface_tension_curvature_smoothing_radius = True, 1
            sim.adaptive_timestep = True
            sim.c_div_volume_correction = True
            sim.liquid_volume_target = float(p["n"])
        st.update(sim=sim, part=p, pos=torch.zeros((cap, 3), device=DEV), vel=torch.zeros((cap, 3), device=DEV),
                  typ=torch.zeros(cap, dtype=torch.uint8, device=DEV), vol=torch.zeros(cap, device=DEV),
                  p=torch.empty((case["nz"], case["ny"], case["nx"]), device=DEV))
    elif kind == "project":
        st.update(_project_state(case, seed))
        if case["solver"] == "learned":
            pf.LearnedCoarseSolver(st["grid"]).load_default()
    elif kind == "mr":
        p = _particles(case, "tank" if case["dynamic"] else "dam", seed)
        sim = pf.MRSim3DTP(case["nx"], case["ny"], case["nz"], p["dx"], max_particles=p["n"])
        sim.phase = _phase(sim.grid)
        sim.dt, sim.dynamic_refinement = 1.0 / 480.0, case["dynamic"]
        sim.set_levels(pf.multires.interface_levels(_cells(case, "tank" if case["dynamic"] else "dam").cpu().numpy(), 3))
        st.update(sim=sim, part=p, pos=torch.empty_like(p["pos"]), vel=torch.empty_like(p["vel"]))
    else:
        box = {"nx": case["n"], "ny": case["n"], "nz": case["n"]}
        s = _project_state(box, seed)
        g, net = s["grid"], pf.LearnedCoarseSolver(s["grid"])
        net.init(seed=seed)
        for a in range(3):
            _set_field(lib, g, pf.PF_U + a, s["vel"][a], s["acts"][a])
        net.harvest(True, stride=4, max_per_system=32, capacity_floats=1 << 22)
        pf.spProjectStepVC3D(g, s["pp"], DT_PROJECT, 128, 0.0, solver=_solver("exact_coarse"))
        net.harvest(False)
        st.update(net=net, grid=g, params=net.params(), seed=seed)
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass


def run(state):
    case, lib = state["case"], state["lib"]
    kind = case["kind"]
    if kind in ("p2g", "transfer"):
        g = state["grid"]
        ctx = g.ctx
        _upload(lib, ctx, state["part"])
        L.check(lib.pf_p2g(ctx, C.byref(state["phase"]), 1.0), ctx, "pf_p2g")
        if kind == "p2g":
            for q, (dense, act) in enumerate(state["fields"]):
                _get_field(lib, g, pf.PF_U + q, dense, act)
            return [t for pair in state["fields"] for t in pair]
        L.check(lib.pf_save_velocity(ctx), ctx, "pf_save_velocity")
        L.check(lib.pf_g2p(ctx, None, 0.97, 0.97), ctx, "pf_g2p")
        L.check(lib.pf_download_particles(ctx, None, state["vel"].data_ptr(), None, None), ctx,
                "pf_download_particles")
        return state["vel"]
    if kind == "step":
        sim = state["sim"]
        ctx = sim.grid.ctx
        sim.c_div_last = 0.0
        _upload(lib, ctx, state["part"])
        sim.step()
        L.check(lib.pf_download_particles(ctx, state["pos"].data_ptr(), state["vel"].data_ptr(),
                                          state["typ"].data_ptr(), state["vol"].data_ptr()), ctx,
                "pf_download_particles")
        _get_field(lib, sim.grid, pf.PF_P, state["p"])
        # the adaptivity may change the count: the arrays have the particle capacity, zero past the last particle
        return {"pos": state["pos"], "vel": state["vel"], "type": state["typ"], "vol": state["vol"], "p": state["p"],
                "n": sim.n}
    if kind == "project":
        g = state["grid"]
        for a in range(3):
            _set_field(lib, g, pf.PF_U + a, state["vel"][a], state["acts"][a])
        pf.spProjectStepVC3D(g, state["pp"], DT_PROJECT, MAX_ITER, 0.0, solver=_solver(case["solver"]))
        _get_field(lib, g, pf.PF_P, state["p"])
        for a in range(3):
            _get_field(lib, g, pf.PF_U + a, state["out"][a])
        return {"p": state["p"], "u": state["out"][0], "v": state["out"][1], "w": state["out"][2]}
    if kind == "mr":
        sim = state["sim"]
        _upload(lib, sim.ctx, state["part"])
        sim.n = state["part"]["n"]
        if case["dynamic"]:
            L.check(lib.pf_mr_reset_refinement(sim.ctx), sim.ctx, "pf_mr_reset_refinement")
        sim.step()
        L.check(lib.pf_download_particles(sim.ctx, state["pos"].data_ptr(), state["vel"].data_ptr(), None, None),
                sim.ctx, "pf_download_particles")
        return {"pos": state["pos"], "vel": state["vel"]}
    net = state["net"]
    net.load(state["params"])
    losses = net.train(case["steps"], case["batch"], 1e-3, state["seed"])
    return {"losses": losses, "params": net.params()}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _fluid_cells(case, fill):
    nx, ny, nz = case["nx"] - 2, case["ny"] - 2, case["nz"] - 2
    return int(nx * ny * nz * {"full": 1.0, "uneven": 1.0, "tank": 0.7, "dam": 0.33}[fill])


def work(case):
    """Inputs read once and outputs written once (29 B a particle in, 8 B a face and field pair, 4 B a
    cell value), and the arithmetic of the method: per particle 3 x 36 kernel weights at about 8 operations in
    P2G and 2 x 3 trilinear samples in G2P; per unknown and iteration about 27 operations of preconditioned CG,
    whose iterations grow with the longest axis."""
    kind = case["kind"]
    if kind == "train":
        tiles = math.ceil((case["n"] + 1) / 8) ** 3
        flops = 3.0 * 2 * 800000 * tiles * case["batch"] * case["steps"]
        return {"bytes": case["steps"] * (800000 * 4 * 6 + case["batch"] * tiles * 16), "flops": flops}
    nmax = max(case["nx"], case["ny"], case["nz"])
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "project":
        its = nmax * (46 if case["solver"] != "learned" else 14)
        return {"bytes": cells * 4.0 * (1 + 3 + 3 + 3 + 1), "flops": 27.0 * cells * its}
    fill = case.get("fill") or ("tank" if case["dynamic"] else "dam")
    fluid = _fluid_cells(case, fill)
    n = 8 * fluid
    p2g = 3 * 36 * 8.0 * n
    if kind == "p2g":
        return {"bytes": 29.0 * n + 24.0 * cells, "flops": p2g}
    if kind == "transfer":
        return {"bytes": 41.0 * n, "flops": p2g + 100.0 * n}
    if kind == "mr":
        return {"bytes": 53.0 * n, "flops": p2g + 300.0 * n + 27.0 * 160 * fluid / 4}
    its = nmax * (8 if case["solver"] == "plain" else 2)
    return {"bytes": 58.0 * n + 4.0 * cells, "flops": p2g + 300.0 * n + 27.0 * fluid * its}


# ---------------------------------------------------------------------------
# the same results in 64 bits


def _weights(p, case, a):
    """Nodes and normalised cubic weights of axis a's face field for the particles p (grid units), as a
    generator over the 4^3 window: (linear node index, weight)."""
    shape = _field_shapes(case)[a]
    gpos = [p[:, b] - (0.0 if b == a else 0.5) for b in range(3)]
    base = [torch.floor(q) for q in gpos]

    def window():
        for c in range(-1, 3):
            for b in range(-1, 3):
                for i in range(-1, 3):
                    off = (i, b, c)
                    d2, ok, lin = 0.0, None, 0
                    for q in (2, 1, 0):
                        node = base[q] + off[q]
                        size = shape[2 - q]
                        d2 = d2 + (gpos[q] - node) ** 2
                        inside = (node >= 0) & (node < size)
                        ok = inside if ok is None else ok & inside
                        lin = lin * size + node.clamp(0, size - 1).to(torch.int64)
                    w = (1.0 - d2 / 2.25).clamp_min(0.0) ** 3
                    yield lin, torch.where(ok, w, torch.zeros_like(w))

    total = sum(w for _, w in window())
    inv = torch.where(total > 0, 1.0 / total, torch.zeros_like(total))
    return window, inv


def _exact_p2g(case, part):
    shapes = _field_shapes(case)
    mom = [torch.zeros(s, dtype=torch.float64, device=DEV).reshape(-1) for s in shapes]
    mass = [torch.zeros(s, dtype=torch.float64, device=DEV).reshape(-1) for s in shapes]
    for lo in range(0, part["n"], 1 << 20):
        q = slice(lo, min(part["n"], lo + (1 << 20)))
        p = part["pos"][q].double() / part["dx"]
        m = torch.where(part["typ"][q] == 0, RHO_L, RHO_G).double() * part["vol"][q].double()
        for a in range(3):
            window, inv = _weights(p, case, a)
            for lin, w in window():
                w = w * inv * m
                mass[a].index_add_(0, lin, w)
                mom[a].index_add_(0, lin, w * part["vel"][q, a].double())
    vel = [torch.where(w > 0, u / w, torch.zeros_like(u)).reshape(s) for u, w, s in zip(mom, mass, shapes)]
    return vel, [w.reshape(s) for w, s in zip(mass, shapes)]


def _exact_g2p(case, part, fields, alpha):
    """FLIP/PIC blend on an unchanged grid: the FLIP increment is zero."""
    out = torch.empty((part["n"], 3), dtype=torch.float64, device=DEV)
    for lo in range(0, part["n"], 1 << 21):
        q = slice(lo, min(part["n"], lo + (1 << 21)))
        p = part["pos"][q].double() / part["dx"]
        for a in range(3):
            f = fields[a]
            gpos = [p[:, b] - (0.0 if b == a else 0.5) for b in range(3)]
            base = [torch.floor(t) for t in gpos]
            frac = [t - b for t, b in zip(gpos, base)]
            s = 0.0
            for c in range(8):
                w, lin = 1.0, 0
                for b in (2, 1, 0):
                    bit = (c >> b) & 1
                    w = w * (frac[b] if bit else 1.0 - frac[b])
                    lin = lin * f.shape[2 - b] + (base[b] + bit).clamp(0, f.shape[2 - b] - 1).to(torch.int64)
                s = s + w * f.reshape(-1)[lin]
            out[q, a] = alpha * part["vel"][q, a].double() + (1.0 - alpha) * s
    return out


def _beta(mass, rho_tilde_0):
    m = mass.double()
    rmin = math.log(RHO_L / RHO_G) * RHO_G * rho_tilde_0
    phi = torch.sqrt((m - rmin).clamp_min(0.0) / (rho_tilde_0 * RHO_L)).clamp_max(1.0)
    phi = torch.where(m < rmin, torch.zeros_like(phi), phi)
    return 1.0 / (phi * RHO_L + (1.0 - phi) * RHO_G)


def _exact_project(case, seed):
    """The projection of the all-fluid box: 7-point system with the first fluid cell pinned, solved by
    Jacobi-preconditioned CG to rounding."""
    s = _pressure_system(case, seed)
    # every face is either empty or saturated, so beta does not depend on the calibration
    beta = [_beta(m, 1.0) for m in _masses(s, 1.0)]
    dx, scale = s["dx"], DT_PROJECT / s["dx"] ** 2
    vel = [v.double() for v in s["vel"]]
    inner = [slice(1, -1)] * 3

    def along(f, a, lo):  # the low or high face of every interior cell
        sl = [slice(1, -1), slice(1, -1), slice(1, -1)]
        n = f.shape[2 - a]
        sl[2 - a] = slice(1, n - 2) if lo else slice(2, n - 1)
        return f[tuple(sl)].clone()

    shape = s["mk"][tuple(inner)].shape
    rhs = torch.zeros(shape, dtype=torch.float64, device=DEV)
    diag = torch.zeros_like(rhs)
    low, high = [], []
    for a in range(3):
        dim = 2 - a
        bl, bh = along(beta[a], a, True), along(beta[a], a, False)
        vl, vh = along(vel[a], a, True), along(vel[a], a, False)
        for t, at in ((bl, 0), (vl, 0), (bh, -1), (vh, -1)):  # faces on the solid walls
            t.select(dim, at).zero_()
        rhs -= (vh - vl) / dx
        diag += bl + bh
        low.append(bl)
        high.append(bh)
    free = torch.ones(shape, dtype=torch.bool, device=DEV)
    free[0, 0, 0] = False  # the pin
    rhs[0, 0, 0] = 0.0
    keep = free.double()
    d = torch.where(free, scale * diag, torch.ones_like(diag))

    def apply(x):
        y = diag * x
        xf = x * keep
        for a in range(3):
            dim, n = 2 - a, shape[2 - a]
            y.narrow(dim, 1, n - 1).sub_(low[a].narrow(dim, 1, n - 1) * xf.narrow(dim, 0, n - 1))
            y.narrow(dim, 0, n - 1).sub_(high[a].narrow(dim, 0, n - 1) * xf.narrow(dim, 1, n - 1))
        return torch.where(free, scale * y, x)

    x = torch.zeros_like(rhs)
    r = rhs.clone()
    z = r / d
    q = z.clone()
    rz = (r * z).sum()
    top = float(r.abs().max())
    for it in range(200 * max(shape)):
        w = apply(q)
        alpha = rz / (q * w).sum()
        x += alpha * q
        r -= alpha * w
        z = r / d
        new = (r * z).sum()
        q = z + (new / rz) * q
        rz = new
        if it % 64 == 63 and float(r.abs().max()) < 1e-12 * top:
            break
    p = torch.zeros(s["mk"].shape, dtype=torch.float64, device=DEV)
    p[tuple(inner)] = x
    out = []
    for a in range(3):
        dim, v = 2 - a, vel[a].clone()
        n = p.shape[dim]
        grad = p.narrow(dim, 1, n - 1) - p.narrow(dim, 0, n - 1)
        fluid = s["mk"] == 1
        lo, hi = fluid.narrow(dim, 0, n - 1), fluid.narrow(dim, 1, n - 1)
        mid = v.narrow(dim, 1, n - 1)
        upd = mid - DT_PROJECT / dx * beta[a].narrow(dim, 1, n - 1) * grad
        mid.copy_(torch.where(lo & hi, upd, torch.where(lo | hi, torch.zeros_like(upd), mid)))
        out.append(v)
    return {"p": p, "u": out[0], "v": out[1], "w": out[2]}


def exact(case, seed):
    if case["kind"] in ("p2g", "transfer"):
        part = _particles(case, case["fill"], seed)
        vel, mass = _exact_p2g(case, part)
        if case["kind"] == "transfer":
            return _exact_g2p(case, part, vel, 0.97)
        return [t for f in vel + mass for t in (f, None)]
    if case["kind"] == "project":
        return _exact_project(case, seed)
    return None  # whole steps and training chain many roundings: compared with the start's outputs alone
