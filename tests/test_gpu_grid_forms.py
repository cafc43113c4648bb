"""The biharmonic solve's two forms against the CPU oracle, on both sides of the
line between them: on the fly up to a cell per thread with one block per SM
(75 776 cells on a B200), through a field above."""
import ctypes as C

import pytest

from conftest import physical, rel_l2

pytestmark = pytest.mark.gpu

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
