"""The spectral pressure solve where its dynamic shared memory alone is below
the default limit of 48 KB and static and dynamic together are above it."""
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# machine-precision solver stops: the two paths solve the same system
TIGHT = dict(ch_tol=1e-13, ch_iter_max=600, CG_ETOL=1e-15, CG_MAXIT=400, P_CG_ETOL=1e-12, P_CG_MAXIT=20000)


@pytest.mark.parametrize("n", [(64, 160), (128, 150), (96, 131)])
def test_spectral_near_the_default_limit(n):
    from pvof import cases, runtime
    out = []
    for pc in (0, 1):
        grid, params, planes = cases.rayleigh_taylor(n[0], n[1], Lx=1.0, Ly=n[1] / n[0], Cn=0.03,
                                                     velocity_seed=1, velocity_amp=0.05,
                                                     pressure_preconditioner=pc, **TIGHT)
        s = runtime.Solver(grid, params, device=0)
        s.set_planes(planes)
        s.initialize()
        s.run_steps(1, 1e-4)
        out.append({f: s.get(f) for f in ("C_L", "U", "V")})
        s.close()
    for f in out[0]:
        assert rel_l2(out[1][f], out[0][f]) <= 1e-9, f
