"""The grid-wide solvers' slot exchange with blocks that fall behind: contexts
advanced together share the SMs, so a block may publish the next exchange (of
another number of sums) while others still read the last one.  Every wait must
end and the fields must be bit for bit those of each context advanced alone,
on block counts at which every block polls and at which the first gathers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("C_L", "U", "V", "P")


@pytest.mark.parametrize("sizes", [[(64, 96), (96, 160), (64, 128), (100, 150)],      # 12 to 30 blocks
                                   [(128, 200), (160, 256), (192, 384), (256, 512)]],  # 50 to 256 blocks
                         ids=["all_poll", "first_gathers"])
def test_contexts_together_equal_alone(sizes):
    from pvof import cases, runtime

    def make(q, n):
        grid, params, planes = cases.rayleigh_taylor(n[0], n[1], Lx=1.0, Ly=n[1] / n[0], Cn=0.03, velocity_seed=q,
                                                     velocity_amp=0.05, P_CG_MAXIT=5000, P_CG_ETOL=1e-5)
        s = runtime.Solver(grid, params, device=0)
        s.set_cluster_solvers(False)
        s.set_planes(planes)
        s.initialize()
        return s

    alone = [make(q, n) for q, n in enumerate(sizes)]
    for s in alone:
        s.run_steps(3, 1e-4)
    together = [make(q, n) for q, n in enumerate(sizes)]
    runtime.run_steps_batched(together, 3, 1e-4)
    for n, a, b in zip(sizes, alone, together):
        for f in FIELDS:
            assert np.array_equal(a.get(f), b.get(f)), (n, f)
        a.close()
        b.close()
