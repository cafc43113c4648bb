"""Pressure_solve_fft over the sizes its passes branch on: radices 2 to 5,
larger prime factors, odd and prime x counts, odd row counts (a single last
row), columns that take the cosine transforms and columns that take the
Thomas algorithm (a prime factor above 31, more than 7000 rows).  Against the
same discrete problem solved in numpy (FFT in x, elimination in y in 64
bits), also for a right-hand side whose mean mode is not compatible, with the
tolerance of test_fft_poisson.py (1e-12 relative L2) times the longest
chain's growth, 1e-11."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _solve(rhs, i2, j2):
    ny, nx = rhs.shape
    f = np.fft.rfft(rhs, axis=1)
    lam = i2 * 4 * np.sin(np.pi * np.arange(f.shape[1]) / nx) ** 2
    out = np.zeros_like(f)
    b = np.full((ny, f.shape[1]), -2.0 * j2) - lam[None, :]
    b[0] += j2
    b[-1] += j2
    up = np.full((ny, f.shape[1]), j2)
    b[0, 0], up[0, 0], f[0, 0] = 1.0, 0.0, 0.0
    g = np.zeros_like(b)
    bet = b[0].copy()
    out[0] = f[0] / bet
    for j in range(1, ny):
        g[j] = up[j - 1] / bet
        bet = b[j] - j2 * g[j]
        out[j] = (f[j] - j2 * out[j - 1]) / bet
    for j in range(ny - 2, -1, -1):
        out[j] -= g[j + 1] * out[j + 1]
    return np.fft.irfft(out, n=nx, axis=1)


@pytest.mark.parametrize("nx,ny", [(8, 8), (9, 13), (30, 45), (31, 62), (128, 37), (97, 200), (200, 800), (1024, 296),
                                   (2048, 64), (16, 74), (16, 7040)])
def test_against_numpy(nx, ny):
    from pvof import cases, runtime
    grid, params, _ = cases.rayleigh_taylor(nx, ny, Lx=1.0, Ly=ny / nx, Cn=0.02)
    rng = np.random.default_rng(nx * ny)
    rhs = rng.standard_normal((ny, nx)) * (1.0 if ny < 2000 else 0.0)
    rhs += np.cos(2 * np.pi * np.arange(nx) / nx)[None, :] * np.cos(np.pi * (np.arange(ny) + 0.5) / ny)[:, None]
    plane = np.zeros((ny + 1, nx + 1))
    plane[:ny, :nx] = rhs
    s = runtime.Solver(grid, params, device=0)
    s.upload("P_RHS", cases.plane_to_block(grid, plane))
    s.call("Pressure_solve_fft")
    got = cases.interior(grid, s.get("DELTAP"))
    s.close()
    ref = _solve(rhs, float(nx) ** 2, float(nx) ** 2)
    assert rel_l2(got, ref) <= 1e-11, rel_l2(got, ref)
