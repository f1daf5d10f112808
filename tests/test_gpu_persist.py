"""The PLAIN solve at every way its work is split over the GPU, and the other modes beside it.

A system's tiles go to 148 CTAs: one to six tiles each live on chip (a kernel per
count, 5 running in the next larger one's; MIXED up to eight), more are streamed
with as many of r and x on chip as fit, and beyond about 7200 tiles three kernels run
per iteration.  The grids below take one of each, ragged ones among them, with
solid, empty and fluid cells mixed.

A few iterations are compared with the oracle's: both round every vector update
alike in FP64 and differ in the order of the inner products only, which moves
the iterate by some 1e-15 per iteration; the pressure is stored in FP32, so it
may differ by one unit in its last place (2^-23 of the value), and where a value
cancels by 1e-12 of the field's scale.
"""
import numpy as np
import pytest

import oracle as O
from gpu_helpers import to_oracle_phase

pytestmark = pytest.mark.gpu

GRIDS = [(5, 6, 4), (39, 30, 22), (46, 47, 40), (54, 55, 62), (63, 62, 56), (64, 64, 64), (70, 71, 72), (78, 79, 72),
         (80, 79, 77), (88, 86, 81), (104, 97, 90), (127, 118, 100), (160, 158, 155)]


def _system(shape, seed, solids=True):
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    mk = np.full((nz, ny, nx), 2, np.float32)
    inner = rng.choice(np.array([0, 1, 1, 1, 1, 1, 1, 2 if solids else 1], np.float32), (nz - 2, ny - 2, nx - 2))
    mk[1:-1, 1:-1, 1:-1] = inner
    f = {7: mk}
    for a, s in enumerate(((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx))):
        f[a] = rng.normal(0, 1, s).astype(np.float32)
        f[3 + a] = (rng.uniform(0, 1.2, s) * (rng.random(s) > 0.2)).astype(np.float32)
    return f


@pytest.mark.parametrize("shape", GRIDS, ids=str)
def test_iterates_match_the_oracle(pf, shape):
    its, dt, c_div = 9, 1.0 / 60, 0.01
    fields = _system(shape, sum(shape))
    pp = pf.PhaseParams(1.0, 0.01)
    g = pf.SparseMacGrid3D(*shape, 1.0 / max(shape), max_particles=int(np.prod(shape)) // 4 + 64)
    og = O.OracleGrid(*shape, 1.0 / max(shape))
    for f, v in fields.items():
        act = np.ones(g.bdims(f)[::-1], np.uint8)
        g.set_field(f, v, act)
        og.set_field(f, v, act)
    st = pf.spProjectStepVC3D(g, pp, dt, its, 0.0, c_div)
    so = O.Oracle().project(og, to_oracle_phase(pp), dt, its, 0.0, c_div)
    assert st.iterations == so.iterations == its and not st.converged
    assert st.n_cells == so.n_cells and st.pin_cell == so.pin_cell
    assert abs(st.res_final - so.res_final) <= 1e-11 * so.res_final
    p, q = g.get_field(pf.PF_P)[0].astype(np.float64), og.get_field(pf.PF_P)[0].astype(np.float64)
    scale = np.abs(q).max()
    assert scale > 0
    assert np.all(np.abs(p - q) <= 2.0 ** -23 * np.abs(q) + 1e-12 * scale)
    g.close()


@pytest.mark.parametrize("shape,bf16", [(g, i % 3) for i, g in enumerate(GRIDS[:9])], ids=str)
def test_mixed_reaches_the_plain_solution(pf, shape, bf16):
    """The mixed mode's inner solve at every number of tiles a CTA keeps (and
    the first size past them).  Both solves stop at 1e-9 of the initial
    residual; with a condition number of some 1e4 here (a hundredfold contrast,
    empty cells everywhere) the pressures agree within 1e-5.  No solid cells
    inside: a fluid cell walled in by them has no solution for c_div != 0 (the
    oracle does not converge there either)."""
    fields = _system(shape, 1 + sum(shape), solids=False)
    pp = pf.PhaseParams(1.0, 0.01)
    out = []
    for mode in (pf.PF_SOLVER_PLAIN, pf.PF_SOLVER_MIXED):
        g = pf.SparseMacGrid3D(*shape, 1.0 / max(shape), max_particles=int(np.prod(shape)) // 4 + 64)
        for f, v in fields.items():
            g.set_field(f, v, np.ones(g.bdims(f)[::-1], np.uint8))
        st = pf.spProjectStepVC3D(g, pp, 1.0 / 60, 20000, 0.0, 0.01,
                                  solver=pf.SolverConfig(mode=mode, rel_tol=1e-9, bf16_storage=bf16))
        assert st.converged and st.res_final < 1e-9 * st.res0
        out.append(g.get_field(pf.PF_P)[0].astype(np.float64))
        g.close()
    assert np.abs(out[0] - out[1]).max() <= 1e-5 * np.abs(out[0]).max()


@pytest.mark.parametrize("inner_fp32", [False, True])
@pytest.mark.parametrize("shape", [(5, 6, 4), (39, 30, 22), (71, 57, 65), (96, 89, 82)], ids=str)
def test_flexible_pcg_on_ragged_systems_reaches_the_plain_solution(pf, shape, inner_fp32):
    """The flexible PCG takes the cells in pairs of x neighbours: pairs with one
    fluid cell, pairs across tile and domain edges, one to several slots per
    CTA.  Stop and tolerance as for the mixed mode above."""
    fields = _system(shape, 2 + sum(shape), solids=False)
    pp = pf.PhaseParams(1.0, 0.01)
    out = []
    for solver in (pf.SolverConfig(rel_tol=1e-9),
                   pf.SolverConfig(mode=pf.PF_SOLVER_LEARNED, rel_tol=1e-9, precond=pf.PF_PRECOND_JACOBI,
                                   inner_fp32=inner_fp32)):
        g = pf.SparseMacGrid3D(*shape, 1.0 / max(shape), max_particles=int(np.prod(shape)) // 4 + 64)
        for f, v in fields.items():
            g.set_field(f, v, np.ones(g.bdims(f)[::-1], np.uint8))
        st = pf.spProjectStepVC3D(g, pp, 1.0 / 60, 20000, 0.0, 0.01, solver=solver)
        assert st.converged and st.res_final < 1e-9 * st.res0
        out.append(g.get_field(pf.PF_P)[0].astype(np.float64))
        g.close()
    assert np.abs(out[0] - out[1]).max() <= 1e-5 * np.abs(out[0]).max()


def test_long_solve_gives_the_bits_of_the_allocation_free_one(pf):
    """A solve of more iterations than one launch runs (2048), on a system that
    lasts that long, against the allocation-free entry point, whose three kernels
    per iteration form the same sums in the same order."""
    import ctypes as C

    import torch
    n, dt, its = 38, 1.0 / 240, 2500  # 125 tiles, all pooled by both entry points
    sc = pf.scenes.ellipsoid_pressure(n, seed=1)
    pp = pf.PhaseParams(sc["rho_l"], sc["rho_g"])
    g = pf.SparseMacGrid3D(n, n, n, 1.0 / n, max_particles=n ** 3 // 4)
    pp.rho_tilde_0 = pf.calibrateRhoTilde0(pp, 1.0, grid=g)
    named = pf.scenes.pressure_grid_fields(sc, pp.rho_tilde_0)
    fields = {f: np.ascontiguousarray(named[k], np.float32) for k, f in
              (("u", 0), ("v", 1), ("w", 2), ("mu", 3), ("mv", 4), ("mw", 5), ("mk", 7))}
    for f, v in fields.items():
        g.set_field(f, v, np.ones(g.bdims(f)[::-1], np.uint8))
    st = pf.spProjectStepVC3D(g, pp, dt, its, 0.0)
    assert st.iterations == its and not st.breakdown
    dev = {k: torch.from_numpy(fields[f]).cuda() for k, f in
           (("mk", 7), ("mu", 3), ("mv", 4), ("mw", 5), ("u", 0), ("v", 1), ("w", 2))}
    p = torch.zeros((n, n, n), device="cuda")
    s2 = pf._lib.SolveStats()
    torch.cuda.synchronize()
    rc = pf.load().pf_project_noalloc(n, n, n, 1.0 / n, *[dev[k].data_ptr() for k in ("mk", "mu", "mv", "mw", "u", "v", "w")],
                                      p.data_ptr(), C.byref(pp._c()), dt, its, 0.0, 0.0, 0.0, C.byref(s2), None)
    assert rc == 0
    assert st.iterations == s2.iterations and st.breakdown == s2.breakdown
    assert st.res_final == s2.res_final
    assert np.array_equal(g.get_field(pf.PF_P)[0], p.cpu().numpy())
    g.close()


THREADS = """
import threading
import numpy as np
from conftest import load_package
from test_gpu_persist import _system
pf = load_package()
shapes, rounds, done = [(88, 86, 81), (127, 118, 100)], 20, {}

def solve(g, shape):
    for _ in range(rounds):
        st = pf.spProjectStepVC3D(g, pf.PhaseParams(1.0, 0.01), 1.0 / 60, 1, 0.0, 0.01)
        assert st.iterations == 1
    done[shape] = True

grids = []
for s in shapes:
    g = pf.SparseMacGrid3D(*s, 1.0 / max(s), max_particles=int(np.prod(s)) // 4 + 64)
    for f, v in _system(s, sum(s)).items():
        g.set_field(f, v, np.ones(g.bdims(f)[::-1], np.uint8))
    grids.append(g)
threads = [threading.Thread(target=solve, args=a) for a in zip(grids, shapes)]
[t.start() for t in threads]
[t.join() for t in threads]
assert len(done) == 2, "a thread's solve failed"
"""


def test_two_threads_solve_side_by_side(pf, tmp_path):
    """Two contexts, a thread each, on systems whose streaming kernels take
    different amounts of shared memory; every launch is held back for 3 ms after
    it is set up, so one thread's set-up falls before the other's launch."""
    from coop_shim import run_under_shim
    run_under_shim(tmp_path, THREADS, delay_us=3000)


# one to six slots a CTA (on chip), seven and eight (PLAIN streams them, MIXED's live on
# chip), streaming with r and x kept and with part of them kept
BITS = [((39, 30, 22), (0, 1, 2)), ((46, 47, 40), ()), ((54, 55, 62), ()), ((63, 62, 56), ()), ((64, 64, 64), ()),
        ((70, 71, 72), (0, 2)), ((78, 79, 72), (1,)), ((80, 79, 77), (0, 1, 2)),
        ((88, 86, 81), ()), ((127, 118, 100), ())]


def solve_all(pf, check_every=0, its=23):
    """A few iterations of PLAIN on every system and of MIXED where the second
    entry names its storage modes; all outputs."""
    out = {}
    for shape, bf16 in BITS:
        g = pf.SparseMacGrid3D(*shape, 1.0 / max(shape), max_particles=int(np.prod(shape)) // 4 + 64)
        fields = _system(shape, 3 + sum(shape), solids=False)
        cases = [("plain", pf.SolverConfig(check_every=check_every), its)]
        cases += [(f"mixed{b}", pf.SolverConfig(mode=pf.PF_SOLVER_MIXED, bf16_storage=b, check_every=check_every,
                                                rel_tol=1e-7), 300) for b in bf16]
        for name, solver, n in cases:
            for f, v in fields.items():
                g.set_field(f, v, np.ones(g.bdims(f)[::-1], np.uint8))
            st = pf.spProjectStepVC3D(g, pf.PhaseParams(1.0, 0.01), 1.0 / 60, n, 0.0, 0.01, solver=solver)
            key = f"{shape}_{name}"
            out[key] = g.get_field(pf.PF_P)[0]
            out[key + "_stats"] = np.array([st.iterations, st.refinements, st.converged, st.breakdown, st.res_final])
        g.close()
    return out


SOLVE_ALL = """
import sys
import numpy as np
from conftest import load_package
from test_gpu_persist import solve_all
np.savez({path!r}, **solve_all(load_package(), {check_every}))
"""


def _same_bits(a, b):
    assert sorted(a) == sorted(b)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


def test_refused_launches_leave_the_work_to_the_kernels_per_iteration(pf, tmp_path):
    """A device that refuses the cooperative launches (the shim answers them as one
    without room for the grid does) solves by the kernels per iteration: the same
    bits, PLAIN at every way its slots are kept and MIXED in its three storages."""
    from coop_shim import run_under_shim
    path = str(tmp_path / "refused.npz")
    run_under_shim(tmp_path, SOLVE_ALL.format(path=path, check_every=0), refuse_every=1)
    _same_bits(solve_all(pf), dict(np.load(path)))


@pytest.mark.parametrize("mode", ["plain", "mixed"])
@pytest.mark.parametrize("shape", [(39, 30, 22), (88, 86, 81)], ids=str)
def test_check_every_is_the_iterations_of_a_launch(pf, shape, mode):
    """The host looks at the solve every check_every iterations: one launch for each."""
    g = pf.SparseMacGrid3D(*shape, 1.0 / max(shape), max_particles=int(np.prod(shape)) // 4 + 64)
    fields = _system(shape, sum(shape), solids=False)
    counts = []
    for check_every in (0, 6, 1):
        for f, v in fields.items():
            g.set_field(f, v, np.ones(g.bdims(f)[::-1], np.uint8))
        cfg = pf.SolverConfig(check_every=check_every) if mode == "plain" else pf.SolverConfig(
            mode=pf.PF_SOLVER_MIXED, check_every=check_every, inner_rel_tol=1e-30, inner_max_iter=12)
        before = g.lib.pf_launch_count(g.ctx)
        st = pf.spProjectStepVC3D(g, pf.PhaseParams(1.0, 0.01), 1.0 / 60, 12, 0.0, 0.01, solver=cfg)
        assert st.iterations == 12
        counts.append(g.lib.pf_launch_count(g.ctx) - before)
    g.close()
    if mode == "mixed" and max(shape) > 80:  # three launches per iteration, however often the host looks
        assert counts[1] == counts[0] and counts[2] == counts[0]
    else:
        assert [c - counts[0] for c in counts] == [0, 1, 11]


def test_launches_chain_with_the_same_bits(pf):
    """Seven iterations a launch against all in one, for every kernel that runs a
    solve in launches: the vectors, scalars, faces and tags pass from one to the next."""
    _same_bits(solve_all(pf), solve_all(pf, check_every=7))


def test_a_launch_refused_in_mid_solve(pf, tmp_path):
    """A solve's first launch runs seven iterations, its second is refused, and the
    kernels per iteration take over: the same bits."""
    from coop_shim import run_under_shim
    path = str(tmp_path / "taken_over.npz")
    run_under_shim(tmp_path, SOLVE_ALL.format(path=path, check_every=7), refuse_every=2)
    _same_bits(solve_all(pf), dict(np.load(path)))


def test_other_streams_run_between_the_launches(pf):
    """While a long solve runs, a small kernel on another stream waits for a launch
    of the solve at most, not for the solve: the longest wait is under half of the
    solve's device time."""
    import threading
    import time

    import torch
    n, its = 96, 3000
    sc = pf.scenes.ellipsoid_pressure(n, seed=1)
    pp = pf.PhaseParams(sc["rho_l"], sc["rho_g"])
    g = pf.SparseMacGrid3D(n, n, n, sc["dx"], max_particles=n ** 3 // 4)
    pp.rho_tilde_0 = pf.calibrateRhoTilde0(pp, 1.0, grid=g)
    names = ("u", "v", "w", "mu", "mv", "mw", "p", "mk")
    fields = pf.scenes.pressure_grid_fields(sc, pp.rho_tilde_0)
    for k, v in fields.items():
        if k in names:
            f = names.index(k)
            g.set_field(f, v, np.ones(g.bdims(f)[::-1], np.uint8))
    side, x = torch.cuda.Stream(), torch.zeros(1, device="cuda")
    with torch.cuda.stream(side):
        x += 1
    side.synchronize()
    waits = []
    for _ in range(3):  # a host that stalls may hold up one of them
        st, longest = [], 0.0
        t = threading.Thread(target=lambda: st.append(pf.spProjectStepVC3D(g, pp, 1.0 / 240, its, 0.0)))
        t.start()
        while t.is_alive():
            t0 = time.perf_counter()
            with torch.cuda.stream(side):
                x += 1
            side.synchronize()
            longest = max(longest, 1e3 * (time.perf_counter() - t0))
        t.join()
        assert st[0].iterations == its
        waits.append((longest, st[0].solve_ms))
    assert min(w / ms for w, ms in waits) < 0.5, waits
    g.close()
