"""Device memory of a 3D context: 45 fields with their ghosts (44 and a block to
stage host copies through) and at most 32 MB of tables, partial sums and
allocation granularity beside them.  A field of 96^3 cells has 9.5 MB, so four
more fields would show."""
import pytest

pytestmark = pytest.mark.gpu


def test_box_context_memory():
    import torch
    from pvof import cases, runtime
    torch.cuda.init()

    def make(n):
        grid, params, fields = cases.interface_box(n, n, n, L=2.0, Cn=0.1, rho_ratio=1e-2)
        s = runtime.Solver(grid, params, device=0)
        s.set_fields({k: fields[k] for k in ("F", "U", "V", "W", "P")})
        s.initialize()
        s.run_steps(1, 1e-3)
        return s

    make(8).close()   # the kernels are loaded at their first launch
    before = torch.cuda.mem_get_info(0)[0]
    n = 96
    s = make(n)
    used = before - torch.cuda.mem_get_info(0)[0]
    s.close()
    N = n + 1
    pitch = (8 + N + 3 + 7) // 8 * 8   # columns of a row: i = 0 is the ninth
    field = 8 * pitch * (N + 6) * (N + 6)
    print("fields", used / field)
    assert 40 * field < used <= 45 * field + (32 << 20), used / field
