"""The solvers' launched iterations (layouts set by the caller keep them from
running as one kernel) at the ends a solve can have: a zero right-hand side,
maxit, breakdowns, BiCGstab's small s, GMRES's happy breakdown, a start from x0.
The inputs, oracles and tolerances are those of the tests of the same ends in
test_gpu_parity, test_gpu_mixed, test_gpu_bicgstab and test_gpu_gmres, whose
small systems run as one kernel."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_bicgstab import convection_diffusion
from test_gpu_one_kernel import banded_spd, diagonal

pytestmark = pytest.mark.gpu

FORCED = [("pcg", ("csr", 8)), ("pcg", ("sell", 4)), ("pcg", ("q16", 1)), ("bicgstab", ("csr", 8)),
          ("bicgstab", ("q16", 1)), ("gmres", ("csr", 8)), ("flgmres", ("csr", 8)), ("flgmres", ("sell", 4)),
          ("mixed", ("pair", 4)), ("mixed", ("q16", 1))]


def system(gpu, solver, layout, A):
    s = gpu.Solver(0)
    s.set_matrix(*A)
    if layout is not None:
        (s.set_spmv_plan32 if solver == "mixed" else s.set_spmv_plan)(*layout)
    return s


def solve(s, solver, **kw):
    """(x, iterations, residual)."""
    kw.setdefault("btol", 0.0)
    f = {"pcg": s.solve_pcg, "mixed": s.solve_pcg_mixed, "bicgstab": s.solve_bicgstab}.get(solver)
    if f is not None:
        return f(**kw)[:3]
    if solver == "gmres":
        return s.solve_gmres(restart=5, **kw)
    return s.solve_flgmres(restart=4, augk=2, **kw)


def oracle_solve(oracle, solver, A, **kw):
    ptr, cols, vals, b = A
    d = diagonal(ptr, cols, vals)
    f = {"bicgstab": oracle.bicgstab, "gmres": oracle.gmres, "flgmres": oracle.flgmres}.get(solver, oracle.pcg)
    extra = {"gmres": dict(restart=5), "flgmres": dict(restart=4, augk=2)}.get(solver, {})
    return f(ptr, cols, vals, d, b, btol=0.0, atol=0.0, **extra, **kw)[:3]


def matrix(solver):
    return banded_spd(900, 6, seed=4) if solver in ("pcg", "mixed") else convection_diffusion(9, 1.0, seed=4)


@pytest.mark.parametrize("solver,layout", FORCED)
def test_zero_rhs(gpu, solver, layout):
    ptr, cols, vals, b = matrix(solver)
    s = system(gpu, solver, layout, (ptr, cols, vals, np.zeros_like(b)))
    x, nits, res = solve(s, solver, x0=np.linspace(-1, 1, len(b)), rtol=1e-10)
    assert nits == 0 and res == 0.0 and not x.any()
    if solver in ("pcg", "bicgstab"):
        f = s.solve_pcg if solver == "pcg" else s.solve_bicgstab
        assert np.array_equal(f(history=True)[3], [0.0])
    s.close()


@pytest.mark.parametrize("solver,layout", FORCED)
def test_initial_guess(gpu, oracle, solver, layout):
    A = matrix(solver)
    x0 = np.linspace(-1, 1, len(A[3]))
    s = system(gpu, solver, layout, A)
    x, nits, res = solve(s, solver, x0=x0, rtol=1e-10)
    xo, no, _ = oracle_solve(oracle, solver, A, x0=x0, rtol=1e-10)
    if solver != "mixed":
        assert abs(nits - no) <= 2
    assert np.linalg.norm(x - xo) <= 1e-7 * np.linalg.norm(xo)
    s.close()


@pytest.mark.parametrize("maxit", [0, 1, 7])
@pytest.mark.parametrize("solver,layout", FORCED)
def test_maxit(gpu, oracle, solver, layout, maxit):
    """The iterate after maxit steps is the oracle's (FP64 solvers: 1e-8, as few
    steps round little; the mixed solver's residual is the FP64 one of its
    iterate, 1e-10 of ||b||)."""
    A = matrix(solver)
    s = system(gpu, solver, layout, A)
    x, nits, res = solve(s, solver, rtol=1e-14, maxit=maxit)
    assert nits == maxit
    if solver == "mixed":
        r = np.linalg.norm(A[3] - oracle.spmv(*A[:3], x))
        assert abs(res - r) <= 1e-10 * np.linalg.norm(A[3])
    else:
        xo, no, ro = oracle_solve(oracle, solver, A, rtol=1e-14, maxit=maxit)
        assert no == maxit
        assert np.linalg.norm(x - xo) <= 1e-8 * np.linalg.norm(xo)
        assert res == pytest.approx(ro, rel=1e-8)
    s.close()


@pytest.mark.parametrize("solver,layout", [f for f in FORCED if f[0] in ("pcg", "mixed")])
def test_breakdown(gpu, oracle, solver, layout):
    """p.Ap = 0 in the first step: counted, the warning set, x as it is."""
    b = np.array([1.0, 1.0])
    A = (np.array([0, 1, 2]), np.array([0, 1], np.int32), np.array([1.0, -1.0]), b)
    s = system(gpu, solver, layout, A)
    x, nits, res = solve(s, solver, rtol=1e-10)
    assert nits == 1 and "not be SPD" in gpu.last_warning()
    if solver == "mixed":
        assert res == np.linalg.norm(b - np.array([1.0, -1.0]) * x)
    else:
        xo, _, ro = oracle_solve(oracle, solver, A, rtol=1e-10)
        assert np.array_equal(x, xo) and res == ro
    s.close()


@pytest.mark.parametrize("layout", [("csr", 8), ("sell", 4), ("q16", 1)])
def test_bicgstab_small_s(gpu, oracle, layout):
    """The first preconditioned step is exact (s = 0): x is corrected and the
    residual recomputed from b - A x (solver-phg.c:717-729)."""
    n = 1001
    d = 2.0 ** np.random.default_rng(2).integers(-2, 4, n)
    b = np.random.default_rng(3).integers(-8, 9, n).astype(np.float64)
    b[0] = 1.0
    A = (np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), d, b)
    s = system(gpu, "bicgstab", layout, A)
    x, nits, res, hist = s.solve_bicgstab(rtol=1e-12, btol=0.0, atol=0.0, history=True)
    assert nits == 1 and res == hist[1] == 0.0 and np.array_equal(x, b / d)
    s.close()


@pytest.mark.parametrize("layout", [("csr", 8), ("sell", 4)])
def test_gmres_happy_breakdown(gpu, oracle, layout):
    """h_21 = 0 exactly: the step is dropped (solver-phg.c:1149-1153)."""
    n = 64
    d = 2.0 ** np.random.default_rng(1).integers(-2, 4, n)
    b = np.zeros(n)
    b[0] = 4.0
    A = (np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), d, b)
    s = system(gpu, "gmres", layout, A)
    x, nits, res = solve(s, "gmres", rtol=1e-12)
    assert nits == 1 and res == 0.0 and np.array_equal(x, b / d)
    s.close()


@pytest.mark.parametrize("solver,layout", FORCED + [(f, None) for f in ("pcg", "bicgstab", "gmres", "flgmres", "mixed")])
def test_nonfinite(gpu, solver, layout):
    """A zero diagonal entry is an error, the system stays usable (without a
    layout: in one kernel)."""
    ptr, cols, vals, b = matrix(solver)
    bad = np.where((cols == 5) & (np.repeat(np.arange(len(b)), np.diff(ptr)) == 5), 0.0, vals)
    s = system(gpu, solver, layout, (ptr, cols, bad, b))
    with pytest.raises(gpu.PhgGpuError) as e:
        solve(s, solver, rtol=1e-10)
    assert e.value.code == -6
    s.set_matrix(ptr, cols, vals, b)
    x, _, _ = solve(s, solver, rtol=1e-10)
    A = sp.csr_matrix((vals, cols, ptr))
    assert np.linalg.norm(b - A @ x) <= 1e-9 * np.linalg.norm(b)
    s.close()
