"""A destroyed system gives its device memory back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_destroy_frees_all(gpu):
    """Systems that used every buffer (a recorded assembly pattern, rows from
    segments, each layout and solver), made and destroyed three times: what is
    free after the third is what was free after the first, which also warmed
    up the driver's own pools (a recorded pattern alone is 10 MB here)."""
    import torch
    v, e = gpu.kuhn_cube(16)
    e2l, bdry, nodes = gpu.lagrange_dofs(v, e, 2)
    f = gpu.sine_source(nodes)

    def use():
        with gpu.Solver(0) as s:
            s.set_mesh(v, e)
            s.set_dof_map(2, e2l, bdry)
            for _ in range(3):   # the second build records the pattern, the third uses it
                s.build_linear_system(f=f)
            ptr, cols, vals = s.get_matrix()
            rhs = s.get_rhs()
            x, _, _ = s.solve_pcg(rtol=1e-6)
            s.adjoint_gradient(x, x + 1.0, rtol=1e-6)
            s.solve_pcg_mixed(rtol=1e-6)
            s.solve_bicgstab(rtol=1e-6)
            s.solve_gmres(rtol=1e-6)
            s.solve_flgmres(rtol=1e-6)
            s.set_spmv_plan("q16", 1)
            s.solve_pcg(rtol=1e-6)
            for layout in ("sell", "pair"):
                s.set_spmv_plan32(layout, 4)
                s.solve_pcg_mixed(rtol=1e-6)
            s.solve_block_pcg(np.stack([rhs, rhs], 1).copy(), rtol=1e-6, mixed=True)
            n = len(rhs)
            s.assemble_rows(n, np.arange(n, dtype=np.int32), ptr, cols, vals)
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    first = use()
    use()
    assert use() >= first - (1 << 20)
