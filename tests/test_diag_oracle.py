"""Interface diagnostics (src/driver/interface_diagnostics3d.cpp:363-379): the
C restatement against the compiled reference, bit for bit, on grids after
markCells and P2G of seeded two-phase scenes, and on the edge cases the
function branches on (no fluid cell, no interface cell)."""
import numpy as np
import pytest

import oracle as O

needs_ref = pytest.mark.skipif(not O.reference_available(), reason="oracle/_ref not built")


def stepped_oracle(n, seed, air=0.0, rho=(1000.0, 1.0)):
    """An oracle grid holding the markers and P2G fields of a seeded scene."""
    rng = np.random.default_rng(seed)
    dx = 1.0 / n
    pos = rng.uniform(0.6 * dx, 1 - 0.6 * dx, (30 * n ** 2, 3)).astype(np.float32).astype(np.float64)
    if air:
        pos = pos[pos[:, 1] < 1.0 - air]
    vel = rng.normal(0, 0.3, pos.shape)
    typ = (pos[:, 1] + 0.05 * np.cos(2 * np.pi * pos[:, 0]) > 0.45).astype(np.uint8)
    ps = O.Particles(pos, vel, typ, rng.uniform(0.5, 1.5, len(pos)))
    pp = O.PhaseParams(*rho)
    pp.rho_tilde_0 = O.Oracle().calibrate_rho_tilde0(pp, 1.0)
    go = O.OracleGrid(n, n, n, dx)
    o = O.Oracle()
    o.mark_cells(go, ps)
    o.p2g(go, ps, pp, 1.0)
    return go, pp


def stepped_pair(n, seed, air=0.0, rho=(1000.0, 1.0)):
    """Oracle and reference grids holding the same markers and P2G fields."""
    go, pp = stepped_oracle(n, seed, air, rho)
    gr = O.ReferenceGrid(n, n, n, 1.0 / n)
    for f in range(8):
        gr.set_field(f, *go.get_field(f))
    return go, gr, pp


@needs_ref
@pytest.mark.parametrize("n,seed,air", [(8, 1, 0.0), (12, 2, 0.3), (16, 3, 0.5), (10, 4, 0.0)])
def test_interface_diagnostics_match_reference(n, seed, air):
    go, gr, pp = stepped_pair(n, seed, air)
    so = O.Oracle().interface_diagnostics(go, pp)
    sr = O.Reference().interface_diagnostics(gr, pp)
    assert so.as_tuple() == sr.as_tuple()
    assert so.sample_cells > 0 and so.interface_cells > 0 and so.finite == 1


@needs_ref
def test_interface_diagnostics_without_fluid_or_interface():
    go, gr, pp = stepped_pair(8, 5)
    empty = np.zeros((8, 8, 8), np.float32)
    act = np.zeros(go.bdims(O.MK)[::-1], np.uint8)
    go2, gr2 = O.OracleGrid(8, 8, 8, 1 / 8), O.ReferenceGrid(8, 8, 8, 1 / 8)
    go2.set_field(O.MK, empty, act)
    gr2.set_field(O.MK, empty, act)
    assert O.Oracle().interface_diagnostics(go2, pp).as_tuple() == O.Reference().interface_diagnostics(
        gr2, pp).as_tuple() == (0, 0, 1, 0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)
    # equal phase densities: phi is 1 wherever there is mass, no interface cells
    go3, gr3, pp3 = stepped_pair(8, 6, rho=(1.0, 1.0))
    so = O.Oracle().interface_diagnostics(go3, pp3)
    assert so.as_tuple() == O.Reference().interface_diagnostics(gr3, pp3).as_tuple()


@needs_ref
@pytest.mark.parametrize("n,seed,air,strength,maxdv,radius", [
    (12, 2, 0.3, 0.07, 0.0, 0), (12, 3, 0.3, 0.07, 0.0, 1), (16, 4, 0.5, 0.2, 0.05, 2), (10, 5, 0.0, 1.0, 0.0, 3),
    (10, 6, 0.2, 0.0, 0.0, 1),  # disabled: strength 0
])
def test_surface_tension_matches_reference(n, seed, air, strength, maxdv, radius):
    """applySparseSurfaceTension3D (src/driver/interface_diagnostics3d.cpp:405-447):
    the oracle's statistics and updated face velocities equal the reference's."""
    go, gr, pp = stepped_pair(n, seed, air)
    dt = 1 / 120
    so = O.Oracle().surface_tension(go, pp, dt, strength, maxdv, radius)
    sr = O.Reference().surface_tension(gr, pp, dt, strength, maxdv, radius)
    assert so.as_tuple() == sr.as_tuple()
    if strength > 0:
        assert so.applied_cells > 0
    for f in range(8):
        a, b = go.get_field(f), gr.get_field(f)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), O.FIELD_NAMES[f]
