"""The 3D spectral preconditioner's transform lengths: every power of two from 8
to 1024 in x and in z, row counts that leave the last pair of rows or block
short.  At constant density the preconditioner is the operator's exact
inverse, so a solve stops within two iterations only if the transforms and
the tridiagonal solves are right; the fields stay within 1e-10 of the Jacobi
path (the tolerances of test_gpu_box.py).  At density ratio 1e-2 with solver
tolerances near machine precision within 1e-9."""
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(8, 9, 16), (16, 13, 8), (32, 11, 64), (64, 10, 32), (128, 9, 256), (256, 9, 128),
                                      (512, 8, 8), (8, 8, 512), (1024, 9, 8), (8, 9, 1024)])
@pytest.mark.parametrize("ratio", [1.0, 1e-2])
def test_lengths(nx, ny, nz, ratio):
    from pvof import abi, cases, runtime
    L = 2.0 * nx / ny
    grid, params, fields = cases.interface_box(nx, ny, nz, L=L, Cn=0.3, rho_ratio=ratio, mu_ratio=ratio, Re=100.0, We=100.0,
                                               velocity_seed=4, velocity_amp=0.05, CG_ETOL=1e-13, CG_MAXIT=400,
                                               P_CG_ETOL=1e-10, P_CG_MAXIT=20000)
    out = []
    for pre in (0, 1):
        p = abi.Params.from_buffer_copy(params)
        p.pressure_preconditioner = pre
        s = runtime.Solver(grid, p, device=0)
        s.set_fields({k: fields[k] for k in ("F", "U", "V", "W", "P")})
        s.initialize()
        s.set_stage(0, 1e-3)
        st = s.substep()
        if pre and ratio == 1.0:
            assert st.p_iters <= 2, st.as_dict()
        out.append({f: s.get_block(f) for f in ("U", "V", "W", "P")})
        s.close()
    errs = {f: rel_l2(out[1][f], out[0][f]) for f in out[0]}
    assert all(e <= (1e-10 if ratio == 1.0 else 1e-9) for e in errs.values()), errs
