"""The one-cell-per-thread solvers (ranges of at most one cell per resident
thread: k_cg_pressure_fw's resident form, k_cg_velocity_res) at the sizes
where their blocks and exchanges change: one full block, one block and a
cell, the most blocks that all poll (32) and one more, the largest range.
Against the pressure solve over pairs of cells (mode 1: another kernel, the
grid-stride passes) and, for the velocities, the CPU oracle.  Tolerances as
the other solver comparisons: fields 1e-11 relative L2 against another
kernel of the same iteration and against the oracle, solver tolerances
near machine precision."""
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TIGHT = dict(ch_tol=1e-13, ch_iter_max=600, CG_ETOL=1e-15, CG_MAXIT=400, P_CG_ETOL=1e-12, P_CG_MAXIT=20000)


def _run(grid, params, planes, mode):
    from pvof import runtime
    s = runtime.Solver(grid, params, device=0)
    s.set_cluster_solvers(False)
    s.set_pressure_pairs(mode)
    s.set_planes(planes)
    s.initialize()
    s.run_steps(1, 1e-4)
    out = {f: s.get(f) for f in ("C_L", "U", "V", "P")}
    s.close()
    return out


@pytest.mark.parametrize("nx,ny", [(16, 32), (27, 19), (128, 128), (129, 128), (296, 512)])
def test_pressure_against_pairs(nx, ny):
    from pvof import cases
    case = cases.rayleigh_taylor(nx, ny, Lx=1.0, Ly=ny / nx, Cn=max(0.01, 1.5 / nx), velocity_seed=3,
                                 velocity_amp=0.05, **TIGHT)
    one, two = _run(*case, 0), _run(*case, 1)
    errs = {f: rel_l2(one[f], two[f]) for f in one}
    assert all(e <= 1e-11 for e in errs.values()), errs


@pytest.mark.parametrize("kind,nx,ny", [("planar", 16, 32), ("planar", 27, 19), ("axisym", 40, 52)])
def test_velocity_against_oracle(kind, nx, ny):
    import pyoracle as po
    from pvof import cases
    kw = dict(velocity_seed=5, velocity_amp=0.1, Cn=0.06, **TIGHT)
    if kind == "planar":
        grid, params, planes = cases.rayleigh_taylor(nx, ny, Lx=1.0, Ly=ny / nx, **kw)
    else:
        grid, params, planes = cases.rising_bubble(nx, ny, rmax=1.0, zmax=ny / nx, radius=0.3, zc=0.6, rho_ratio=0.1,
                                                   mu_ratio=0.1, **kw)
    got = _run(grid, params, planes, 0)
    o = po.Oracle(grid, params)
    o.set_planes(planes)
    o.initialize()
    o.run_steps(1, 1e-4)
    for f in ("U", "V"):
        a, b = cases.interior(grid, got[f]), cases.interior(grid, o.get_field(f))
        assert rel_l2(a, b) <= 1e-11, (f, rel_l2(a, b))
