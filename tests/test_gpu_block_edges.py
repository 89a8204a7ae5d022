"""Block PCG at the edges of its kernels: row counts around the 64-row chunks
its product deals to the blocks, one column to all 64 (each column tile, and
columns that pad the last one), FP64 and mixed, against the oracle's solve of
each column.  Iteration counts (FP64) within two of the oracle's; solutions
within 1e3 * rtol (relative L2), as for the single solves."""
import numpy as np
import pytest

from test_gpu_one_kernel import banded_spd, diagonal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("nrhs", [1, 8, 9, 33, 64])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000])
def test_block_edges(gpu, oracle, n, nrhs, mixed):
    ptr, cols, vals, b = banded_spd(n, 6, seed=n)
    diag = diagonal(ptr, cols, vals)
    B = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    rtol = 1e-8
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        X, nits, res = s.solve_block_pcg(B, rtol=rtol, mixed=mixed)
    for k in sorted({0, nrhs // 2, nrhs - 1}):
        bk = np.ascontiguousarray(B[:, k])
        xo, no, _, _ = oracle.pcg(ptr, cols, vals, diag, bk, rtol=rtol, btol=0.0, atol=0.0)
        if not mixed:
            assert abs(nits[k] - no) <= 2
        assert np.linalg.norm(X[:, k] - xo) <= 1e3 * rtol * np.linalg.norm(xo)
        r = np.linalg.norm(bk - oracle.spmv(ptr, cols, vals, np.ascontiguousarray(X[:, k])))
        assert abs(res[k] - r) <= 1e-13 * np.linalg.norm(bk)


def test_tile_of_each_precision(gpu):
    """The FP64 and the FP32 product have tiles of their own: the first solve
    in either precision times the four tiles of 64 columns (five launches
    each), whichever came first, and later ones keep both choices."""
    ptr, cols, vals, b = banded_spd(1000, 6, seed=9)
    B = np.random.default_rng(1).standard_normal((1000, 64))
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)

        def count(mixed):
            before = s.launch_count()
            s.solve_block_pcg(B, rtol=1e-8, mixed=mixed)
            return s.launch_count() - before, s.block_tile()
        k32, t32 = count(True)
        k64, t64 = count(False)
        assert count(True) == (k32 - 20, t32)
        assert count(False) == (k64 - 20, t64)
