"""The grid-wide solvers' forms for ranges beyond one cell per resident thread,
and the biharmonic solve's two forms, against the CPU oracle solve by solve.  A
B200 keeps 148 x 512 threads resident with one block per SM and twice as many
with two, so the sizes are: the largest range of the biharmonic form on the fly
(75 776 cells) and one above it; a grid-stride momentum and single-cell pressure
solve whose threads hold one cell or two (151 552 < cells < 303 104); pressure
pairs of which some threads take two (more than 303 104 cells).  The kernel that
ran is asserted, so a change of the dispatch cannot leave a form untested."""
import ctypes as C

import pytest

from conftest import physical, rel_l2

pytestmark = pytest.mark.gpu

# the parity tests' tight set, and short fixed counts for the two solves that a
# regularised or unconverged iteration ends at its limit
TIGHT = dict(ch_tol=1e-13, ch_iter_max=600, CG_ETOL=1e-15, CG_MAXIT=40, P_CG_ETOL=1e-13, P_CG_MAXIT=60)
DT = 1e-3


def _case(nx, ny, geometry="planar", **kw):
    from pvof import cases
    kw = dict(TIGHT, velocity_seed=7, velocity_amp=0.05, **kw)
    if geometry == "planar":
        return cases.rayleigh_taylor(nx, ny, Lx=1.0, Ly=ny / nx, Cn=max(0.01, 1.5 / nx), **kw)
    return cases.rising_bubble(nx, ny, rmax=1.0, zmax=ny / nx, radius=0.3, zc=0.6, Cn=max(0.01, 1.5 / nx), rho_ratio=0.1,
                               mu_ratio=0.1, **kw)


def _pair(case, mode):
    import pyoracle as po
    from pvof import runtime
    grid, params, planes = case
    g = runtime.Solver(grid, params, device=0)
    g.set_cluster_solvers(False)
    g.set_pressure_pairs(mode)
    o = po.Oracle(grid, params)
    for s in (g, o):
        s.set_planes(planes)
        s.initialize()
        s.set_stage(0, DT)
    return g, o


def _compare(grid, g, o, fields, tol, what):
    bad = {f: rel_l2(physical(grid, g.get(f), f), physical(grid, o.get_field(f), f)) for f in fields}
    print(what, bad)
    assert all(r <= tol for r in bad.values()), (what, bad)


@pytest.mark.parametrize("nx,ny,kernel", [(27, 19, "k_cg_biharmonic_fly"), (128, 96, "k_cg_biharmonic_fly"),
                                          (296, 256, "k_cg_biharmonic_fly"), (297, 256, "k_cg_biharmonic")])
def test_biharmonic_against_oracle(nx, ny, kernel):
    """Both sides of the rule's line, at a step size whose solve takes several
    iterations.  Each side stops at a residual of 1e-13 |b|; the operator is a_dt
    plus a positive one, so it ends within 1e-13 |b| / a_dt of the solution, about
    1e-13 |C|: 1e-12 for both and the rounding of the right-hand side."""
    from pvof import abi
    case = _case(nx, ny)
    g, o = _pair(case, 0)
    assert g.solver_kernel(0) == kernel
    st = abi.Stats()
    _, so = o.routine("VOF_DIFFUSE_STEP")
    g.call("VOF_DIFFUSE_step", C.byref(st))
    assert so.ch_iters >= 5 and abs(st.ch_iters - so.ch_iters) <= 2, (st.ch_iters, so.ch_iters)
    _compare(case[0], g, o, ["C_L", "CH_RHS_N"], 1e-12, "VOF_DIFFUSE_step")
    g.close()


@pytest.mark.parametrize("geometry,nx,ny,mode,pressure", [
    ("planar", 400, 380, 0, "k_cg_pressure_fw"),     # 152 000 cells: one cell per thread, 448 threads two
    ("axisym", 391, 390, 0, "k_cg_pressure_fw"),     # odd rows, row weights
    ("planar", 552, 552, 0, "k_cg_pressure_fw"),     # 304 704: two cells, 1 600 threads three
    ("planar", 551, 553, -1, "k_cg_pressure_fwp"),   # rows that end in a single cell; 152 628 pairs, the automatic choice
])
def test_grid_stride_solves_against_oracle(geometry, nx, ny, mode, pressure):
    """A substep's solves in turn on equal inputs.  Momentum and pressure run a
    fixed number of iterations (the tolerances are not reached), so both sides
    hold the same iterate up to the rounding of 40 and 60 iterations and the order
    of the sums: 1e-12 for the converged biharmonic solve (above) and the
    velocities, 1e-11 for the unconverged pressure, the bound of the other
    comparisons between kernels of one iteration."""
    case = _case(nx, ny, geometry)
    g, o = _pair(case, mode)
    assert [g.solver_kernel(q) for q in range(3)] == ["k_cg_biharmonic", "k_cg_velocity", pressure]
    o.routine("VOF_DIFFUSE_STEP")
    g.call("VOF_DIFFUSE_step", None)
    _compare(case[0], g, o, ["C_L"], 1e-12, "VOF_DIFFUSE_step")
    for name, call in [("UPDATE_DENSITY_VISCOSITY", ("VOF_update_density_viscosity",)),
                       ("U_IMPLICIT_EXPLICIT", ("Velocity_set_implicit_explicit", b"u")),
                       ("V_IMPLICIT_EXPLICIT", ("Velocity_set_implicit_explicit", b"v")),
                       ("U_SET_RHS", ("Velocity_set_RHS", b"u")), ("V_SET_RHS", ("Velocity_set_RHS", b"v")),
                       ("ADD_GRAVITY", ("Velocity_add_gravity_2_RHS",)),
                       ("U_SOLVE_CG", ("Velocity_solve_cg", b"u", None)),
                       ("V_SOLVE_CG", ("Velocity_solve_cg", b"v", None))]:
        o.routine(name)
        g.call(*call)
    _compare(case[0], g, o, ["U", "V"], 1e-12, "Velocity_solve_cg")
    for name, call in [("U_UPDATE_BOUNDARIES", ("Velocity_update_boundaries", b"u")),
                       ("V_UPDATE_BOUNDARIES", ("Velocity_update_boundaries", b"v")),
                       ("PRESSURE_SET_RHS", ("Pressure_set_RHS",)),
                       ("PRESSURE_PRECONDITIONER", ("Pressure_compute_preconditioner",)),
                       ("PRESSURE_SOLVE_CG", ("Pressure_solve_cg", None))]:
        o.routine(name)
        g.call(*call)
    _compare(case[0], g, o, ["DELTAP"], 1e-11, "Pressure_solve_cg")
    g.close()
