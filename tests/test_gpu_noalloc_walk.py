"""The no-allocation pressure solve where the device holds fewer threads than
the grid has cells: a walk of the range on fewer blocks, here forced by a limit
on the blocks, against the form of a cell per thread on the same inputs: the same
iteration with its sums in another order.  Both stop at sqrt(r.Mr) < 1e-12; with
M of 1 / diagonal (up to 200^2) and a smallest eigenvalue of about 10, each
correction is within 1e-12 x 200 / 10 of the solution, whose norm is at least the
0.1 that its lowest mode has: 4e-10 for the two, asserted as 1e-9.  Sizes: one
block fewer than needed, one block alone, a remainder in the last trip; planar and
axisymmetric."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometry,nx,ny,most", [("planar", 48, 85, 7), ("planar", 27, 19, 1), ("planar", 57, 90, 1),
                                                 ("axisym", 96, 192, 20)])
def test_walk_matches_a_cell_per_thread(geometry, nx, ny, most):
    import torch
    from pvof import abi, cases, runtime
    kw = dict(Cn=0.04, P_CG_ETOL=1e-12, P_CG_MAXIT=4000)
    if geometry == "planar":
        grid, params, _ = cases.rayleigh_taylor(nx, ny, Lx=1.0, Ly=ny / nx, **kw)
    else:
        grid, params, _ = cases.rising_bubble(nx, ny, rmax=1.0, zmax=ny / nx, radius=0.3, zc=0.7, rho_ratio=0.1, mu_ratio=0.1, **kw)
    rng = np.random.default_rng(nx)
    y, x = np.meshgrid((np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx, indexing="ij")
    rho = 0.55 + 0.45 * np.tanh(8 * (y - 0.5 - 0.1 * np.cos(2 * np.pi * x)))
    rhs = rng.standard_normal((ny, nx))
    weight = x if geometry == "axisym" else np.ones_like(x)   # the operator's range is orthogonal to it
    rhs -= (rhs * weight).sum() / weight.sum()
    mode = "wrap" if geometry == "planar" else "edge"
    dev = [torch.from_numpy(np.ascontiguousarray(np.pad(np.pad(a, ((3, 4), (0, 0)), mode="edge"), ((0, 0), (3, 4)), mode=mode))).cuda()
           for a in (rho, rhs)]
    f = runtime.load().pvof_noalloc_solve
    f.argtypes = [C.POINTER(abi.GridDesc), C.POINTER(abi.Params), C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                  C.POINTER(C.c_int), C.POINTER(C.c_double), C.c_int]
    assert nx * ny > 512 * most
    out = []
    for limit in (1000, most):
        phi = torch.zeros_like(dev[0])
        it, res = C.c_int(), C.c_double()
        torch.cuda.synchronize()
        rc = f(C.byref(grid), C.byref(params), dev[0].data_ptr(), dev[1].data_ptr(), phi.data_ptr(), None, C.byref(it),
               C.byref(res), limit)
        assert rc > 0 and rc < 4000, rc
        assert res.value < 1e-12
        out.append((it.value, phi.cpu().numpy()))
    (i0, a), (i1, b) = out
    print(geometry, nx, ny, i0, i1, np.linalg.norm(a - b) / np.linalg.norm(a))
    assert abs(i0 - i1) <= 4
    assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(a)
