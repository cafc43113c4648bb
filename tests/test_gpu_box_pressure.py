"""The 3D pressure solve's passes at row lengths around their pairs of cells and
64-cell tiles (a row's single last cell, a tile's first and last), tile heights
of 8 rows and runs of 4 planes: the correction's residual in plain numpy.  The
solve stops at sqrt(r.Mr) < P_CG_ETOL, M the Jacobi weights, r by recurrence;
the true residual differs from it by rounding only (1e-16 of |A||phi|, some
1e-12 of the right-hand side, whose norm here is below 1e4), so 2 P_CG_ETOL
bounds it at P_CG_ETOL = 1e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(9, 8, 8), (63, 10, 9), (64, 17, 8), (65, 9, 13), (127, 8, 11), (129, 16, 12)])
def test_residual(nx, ny, nz):
    from pvof import cases, runtime
    tol = 1e-7
    grid, params, fields = cases.interface_box(nx, ny, nz, L=2.0, Cn=0.1, rho_ratio=1e-2, velocity_seed=6, velocity_amp=0.05,
                                               P_CG_ETOL=tol, P_CG_MAXIT=20000)
    s = runtime.Solver(grid, params, device=0)
    s.set_fields({k: fields[k] for k in ("F", "U", "V", "W", "P")})
    s.initialize()
    s.set_stage(0, 1e-3)
    st = s.substep()
    assert st.poisson_passes == 1 and 0 < st.p_iters < 20000
    rho, rhs, phi = (s.get_g_range(f)[:nz, :ny, :nx] for f in ("RHO", "P_RHS", "DELTAP"))
    s.close()
    i2 = (nx / 2.0) ** 2   # cells are cubes
    res, diag = rhs.copy(), np.zeros_like(rhs)
    for axis in (0, 1, 2):
        up = lambda a: np.roll(a, -1, axis)
        face = 2.0 / (rho + up(rho)) * i2
        if axis == 1:
            face[:, -1] = 0.0   # walls in y: no flux
            wall = 2.0 / (2.0 * rho) * i2   # the diagonal counts the mirrored faces
            diag[:, 0] += wall[:, 0]
            diag[:, -1] += wall[:, -1]
        flux = face * (up(phi) - phi)
        res -= flux - np.roll(flux, 1, axis)
        diag += face + np.roll(face, 1, axis)
    norm = float(np.sqrt((res * res / diag).sum()))
    print(nx, ny, nz, st.p_iters, norm)
    assert norm <= 2 * tol, norm
