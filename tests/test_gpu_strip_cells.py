"""The cluster solvers' forms of 2, 4 and 8 cells per thread against the
grid-wide solvers, at strips of 1 to 8 rows (both sides of each limit, uneven
slabs, u and v of different forms): the same iteration with sums in another
order, so at tolerances near machine precision the same fields to rounding."""
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TIGHT = dict(ch_tol=1e-13, ch_iter_max=600, CG_ETOL=1e-15, CG_MAXIT=400, P_CG_ETOL=1e-12, P_CG_MAXIT=20000)


@pytest.mark.parametrize("n", [(32, 64), (128, 128), (128, 129), (100, 161), (128, 256), (128, 257), (200, 256), (256, 256)])
def test_strip_forms_match_grid_wide(n):
    from pvof import cases, runtime
    out = []
    for cluster in (False, True):
        grid, params, planes = cases.rayleigh_taylor(n[0], n[1], Lx=1.0, Ly=n[1] / n[0], Cn=0.03, velocity_seed=3,
                                                     velocity_amp=0.05, **TIGHT)
        s = runtime.Solver(grid, params, device=0)
        s.set_cluster_solvers(cluster)
        s.set_planes(planes)
        s.initialize()
        s.run_steps(1, 1e-4)
        assert s.solver_kernel(2).startswith("k_cgs_" if cluster else "k_cg_")
        out.append({f: s.get(f) for f in ("C_L", "U", "V", "P")})
        s.close()
    for f in out[0]:
        assert rel_l2(out[1][f], out[0][f]) <= 1e-10, f
