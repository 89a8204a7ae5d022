"""The solvers that run as one cooperative kernel (PCG, mixed PCG, BiCGstab, GMRES)
against the
oracle at the edges of their row split: slices of 32 rows that are empty, full
or part-filled, one block and all of them, rows short and long enough to be
split among warps, rows too long for the kernel, and a product layout the
caller asked for (both solved by the other path).

The device sums in another order than the oracle's loops, so iteration counts
are compared within two and solutions by relative L2 distance 1e3 * rtol, as
everywhere for these solvers."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def banded_spd(n, half, seed, long_row=False):
    """Symmetric, diagonally dominant, `half` random off-diagonals on each
    side (those that fit), columns in random order within a row; long_row
    couples row 0 with every other."""
    rng = np.random.default_rng(seed)
    offs = [o for o in np.unique(rng.integers(1, max(2, 3 * half + 2), size=half)) if o < n] if half else []
    A = sp.csr_matrix((n, n))
    for o in offs:
        d = -rng.random(n - o)
        A = A + sp.diags([d, d], [o, -o], shape=(n, n))
    if long_row:
        d = -1e-3 * rng.random(n - 1)
        r, c = np.zeros(n - 1, int), np.arange(1, n)
        A = A + sp.csr_matrix((np.r_[d, d], (np.r_[r, c], np.r_[c, r])), shape=(n, n))
    A = sp.csr_matrix(A)
    A = sp.csr_matrix(A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 0.01 + rng.random(n)))
    A.sum_duplicates()
    ptr, cols, vals = A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data.copy()
    for i in range(0, n, 7):   # first-touch order is not column order
        p = rng.permutation(ptr[i + 1] - ptr[i])
        cols[ptr[i]:ptr[i + 1]] = cols[ptr[i]:ptr[i + 1]][p]
        vals[ptr[i]:ptr[i + 1]] = vals[ptr[i]:ptr[i + 1]][p]
    return ptr, cols, vals, rng.standard_normal(n)


def diagonal(ptr, cols, vals):
    rows = np.repeat(np.arange(len(ptr) - 1), np.diff(ptr))
    d = np.zeros(len(ptr) - 1)
    d[rows[rows == cols]] = vals[rows == cols]
    return d


def check_pcg(s, oracle, ptr, cols, vals, b, rtol, x0=None):
    diag = diagonal(ptr, cols, vals)
    xo, no, _, _ = oracle.pcg(ptr, cols, vals, diag, b, rtol=rtol, btol=0.0, atol=0.0,
                              **({} if x0 is None else {"x0": x0}))
    x, nits, res, hist = s.solve_pcg(x0=x0, rtol=rtol, btol=0.0, atol=0.0, history=True)
    assert abs(nits - no) <= 2
    assert len(hist) == nits + 1 and res == hist[-1] and res <= rtol * hist[0]
    assert np.linalg.norm(x - xo) <= 1e3 * rtol * np.linalg.norm(xo)
    return nits


SIZES = [1, 31, 32, 33, 1000, 148 * 32, 148 * 32 + 1, 40001]


@pytest.mark.parametrize("half", [0, 3, 12, 60])
@pytest.mark.parametrize("n", SIZES)
def test_pcg_row_split(gpu, oracle, n, half):
    ptr, cols, vals, b = banded_spd(n, half, seed=n + half)
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        check_pcg(s, oracle, ptr, cols, vals, b, 1e-9)
        check_pcg(s, oracle, ptr, cols, vals, b, 1e-9, x0=np.linspace(-1.0, 1.0, n))


def test_pcg_long_row_and_forced_layout(gpu, oracle):
    """A row of more entries than a lane takes, and a layout set by the caller,
    go to the launched iteration; the plan can be asked for after either."""
    ptr, cols, vals, b = banded_spd(1500, 4, seed=5, long_row=True)
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        check_pcg(s, oracle, ptr, cols, vals, b, 1e-9)
        s.spmv_plan()
    ptr, cols, vals, b = banded_spd(1000, 4, seed=6)
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        with pytest.raises(gpu.PhgGpuError):
            s.spmv_plan()
        its = [check_pcg(s, oracle, ptr, cols, vals, b, 1e-9)]
        assert s.spmv_plan()[0] in ("csr", "sell", "q16")
        for layout, param in (("csr", 8), ("sell", 4), ("q16", 1)):
            s.set_spmv_plan(layout, param)
            its.append(check_pcg(s, oracle, ptr, cols, vals, b, 1e-9))
            assert s.spmv_plan()[:2] == (layout, param)
    assert max(its) - min(its) <= 1


@pytest.mark.parametrize("half", [0, 3, 12, 60])
@pytest.mark.parametrize("n", SIZES)
def test_mixed_row_split(gpu, oracle, n, half):
    """The mixed solver on the same splits: the FP64 residual of the iterate it
    returns, recomputed by the oracle, meets the stopping rule and is the one
    reported (within the FP64 rounding of a product, 1e-13 of ||b||)."""
    ptr, cols, vals, b = banded_spd(n, half, seed=n + half)
    rtol = 1e-9
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        for x0 in (None, np.linspace(-1.0, 1.0, n)):
            r0 = b if x0 is None else b - oracle.spmv(ptr, cols, vals, x0)
            x, nits, res, nupd = s.solve_pcg_mixed(x0=x0, rtol=rtol)
            r = np.linalg.norm(b - oracle.spmv(ptr, cols, vals, x))
            slack = 1e-13 * np.linalg.norm(b)
            assert r <= rtol * np.linalg.norm(r0) + slack
            assert abs(res - r) <= slack
            assert nupd >= 1 and nits >= 1


def test_mixed_long_row_forced_layout_maxit(gpu, oracle):
    ptr, cols, vals, b = banded_spd(1500, 4, seed=5, long_row=True)
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        x, nits, res, _ = s.solve_pcg_mixed(rtol=1e-9)
        assert np.linalg.norm(b - oracle.spmv(ptr, cols, vals, x)) <= 1e-9 * np.linalg.norm(b) * (1 + 1e-6)
    ptr, cols, vals, b = banded_spd(3000, 12, seed=6)
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        x0, n0, _, _ = s.solve_pcg_mixed(rtol=1e-9)
        assert s.spmv_plan()[2]["fp32_unroll"] > 0
        for maxit in (0, 1, 3):
            x, nits, res, _ = s.solve_pcg_mixed(rtol=1e-12, maxit=maxit)
            assert nits == maxit
            r = np.linalg.norm(b - oracle.spmv(ptr, cols, vals, x))
            assert abs(res - r) <= 1e-13 * np.linalg.norm(b)
        s.set_spmv_plan32("pair", 4)
        x1, n1, _, _ = s.solve_pcg_mixed(rtol=1e-9)
        assert s.spmv_plan()[2]["fp32_layout"] == "pair"
        assert abs(n1 - n0) <= 2


@pytest.mark.parametrize("half", [3, 12, 60])
@pytest.mark.parametrize("n", SIZES)
def test_nonsymmetric_row_split(gpu, oracle, n, half):
    """BiCGstab, GMRES_r and FLGMRES_r on the same splits, the couplings to
    later rows halved so that the matrix is not symmetric.  The residuals are
    recomputed by the oracle; GMRES's estimate and BiCGstab's recurrence drift
    from them by rounding only (1e-6 of the tolerance at these condition
    numbers)."""
    ptr, cols, vals, b = banded_spd(n, half, seed=n + half)
    rows = np.repeat(np.arange(n), np.diff(ptr))
    vals = np.where(cols > rows, 0.5 * vals, vals)
    diag = diagonal(ptr, cols, vals)
    rtol, nb = 1e-9, np.linalg.norm(b)
    kw = dict(rtol=rtol, btol=0.0, atol=0.0)
    with gpu.Solver(0) as s:
        s.set_matrix(ptr, cols, vals, b)
        xo, no = oracle.bicgstab(ptr, cols, vals, diag, b, **kw)[:2]
        x, nits, res, hist = s.solve_bicgstab(history=True, **kw)
        assert abs(nits - no) <= 2 and len(hist) == nits + 1 and hist[-1] == res
        assert np.linalg.norm(b - oracle.spmv(ptr, cols, vals, x)) <= rtol * nb * (1 + 1e-6)
        assert np.linalg.norm(x - xo) <= 1e3 * rtol * np.linalg.norm(xo)
        for x0 in (None, np.linspace(-1.0, 1.0, n)):
            xo, no = oracle.gmres(ptr, cols, vals, diag, b, restart=6, x0=x0, **kw)[:2]
            x, nits, _ = s.solve_gmres(restart=6, x0=x0, **kw)
            assert abs(nits - no) <= 2
            assert np.linalg.norm(x - xo) <= 1e3 * rtol * np.linalg.norm(xo)
            xo, no = oracle.flgmres(ptr, cols, vals, diag, b, restart=4, augk=2, x0=x0, **kw)[:2]
            x, nits, _ = s.solve_flgmres(restart=4, augk=2, x0=x0, **kw)
            assert abs(nits - no) <= 2
            assert np.linalg.norm(x - xo) <= 1e3 * rtol * np.linalg.norm(xo)
