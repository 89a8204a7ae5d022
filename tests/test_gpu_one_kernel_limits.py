"""Which solves run as one cooperative kernel, and that those it leaves go to
the launched iteration and reach the same solution.  The path is seen in the
number of kernels the system has launched: one for a solve in one kernel."""
import numpy as np
import pytest

from test_gpu_one_kernel import banded_spd, diagonal

pytestmark = pytest.mark.gpu

SOLVERS = ("pcg", "mixed", "bicgstab", "gmres", "flgmres")


def solve(s, solver, rtol=1e-9, **kw):
    """(x, iterations) of one solve by that solver."""
    if solver == "mixed":
        return s.solve_pcg_mixed(rtol=rtol, **kw)[:2]
    kw = dict(rtol=rtol, btol=0.0, atol=0.0, **kw)
    if solver == "pcg":
        return s.solve_pcg(**kw)[:2]
    if solver == "bicgstab":
        return s.solve_bicgstab(**kw)[:2]
    if solver == "gmres":
        return s.solve_gmres(restart=6, **kw)[:2]
    return s.solve_flgmres(restart=4, augk=2, **kw)[:2]


def launches(s, f):
    """(f(), kernels launched by it)."""
    before = s.launch_count()
    out = f()
    return out, s.launch_count() - before


def check(oracle, A, solver, x, rtol=1e-9):
    """The solution of the oracle's solver (PCG for the SPD solvers), by
    relative L2 distance 1e3 * rtol as everywhere for these solvers."""
    ptr, cols, vals, b = A
    kw = dict(rtol=rtol, btol=0.0, atol=0.0)
    d = diagonal(ptr, cols, vals)
    if solver in ("pcg", "mixed"):
        xo = oracle.pcg(ptr, cols, vals, d, b, **kw)[0]
    elif solver == "bicgstab":
        xo = oracle.bicgstab(ptr, cols, vals, d, b, **kw)[0]
    else:
        xo = oracle.gmres(ptr, cols, vals, d, b, restart=6, **kw)[0]
    assert np.linalg.norm(x - xo) <= 1e3 * rtol * np.linalg.norm(xo)


def one_long_row(n, length, seed):
    """banded_spd rows of some seven entries, and row n / 2 with about `length`."""
    import scipy.sparse as sp
    ptr, cols, vals, b = banded_spd(n, 3, seed)
    A = sp.csr_matrix((vals, cols, ptr), shape=(n, n))
    rng = np.random.default_rng(seed + 1)
    r = n // 2
    c = rng.choice(np.setdiff1d(np.arange(n), [r]), length - 7, replace=False)
    v = np.full(len(c), -1e-3)
    B = sp.csr_matrix((np.r_[v, v], (np.r_[np.full(len(c), r), c], np.r_[c, np.full(len(c), r)])), shape=(n, n))
    B = B + sp.diags(np.asarray(abs(B).sum(1)).ravel())
    A = sp.csr_matrix(A + B)
    A.sum_duplicates()
    return A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data.copy(), b


@pytest.mark.parametrize("solver", SOLVERS)
@pytest.mark.parametrize("length", [20, 60, 300, 900, 1100])
def test_long_row(gpu, oracle, solver, length):
    """A row far longer than the others is one warp's serial work: the FP64
    solvers leave such a matrix to the launched products (300 entries and more
    here), the mixed one, whose launched products are no better at it, from
    1025 entries on."""
    A = one_long_row(2500, length, seed=length)
    longest = int(np.diff(A[0]).max())
    one = longest <= 1024 if solver == "mixed" else longest < 80
    with gpu.Solver(0) as s:
        s.set_matrix(*A)
        (x, _), k = launches(s, lambda: solve(s, solver))
        assert (k == 1) == one, (longest, k)
        check(oracle, A, solver, x)


@pytest.mark.parametrize("solver", SOLVERS)
def test_declined_matrix_is_remembered(gpu, solver):
    """The second solve of a matrix the kernel declined launches what a solve
    on a layout set by the caller does, no attempt before it; a new matrix is
    looked at again."""
    A = one_long_row(2500, 1100, seed=3)
    with gpu.Solver(0) as s:
        s.set_matrix(*A)
        solve(s, solver)
        layout, param, info = s.spmv_plan()
        _, second = launches(s, lambda: solve(s, solver))
        if solver == "mixed":
            s.set_spmv_plan32(info["fp32_layout"], info["fp32_unroll"])
        else:
            s.set_spmv_plan(layout, param)
        solve(s, solver)   # makes the layout's arrays and graph
        _, forced = launches(s, lambda: solve(s, solver))
        assert second == forced > 1
        s.set_matrix(*banded_spd(2000, 3, seed=4))
        assert launches(s, lambda: solve(s, solver))[1] == 1


# the launches of the one-kernel solvers, refused as the driver refuses a
# cooperative grid that cannot be resident (720, too large)
REFUSE = "".join("int %s(void) { return 720; }\n" % f for f in (
    "_ZN4phgb15launch_pcg_coopERKNS_6PcgRunEP11CUstream_st",
    "_ZN4phgb17launch_mixed_coopERKNS_8MixedRunEP11CUstream_st",
    "_ZN4phgb16launch_bicg_coopERKNS_7BicgRunEP11CUstream_st",
    "_ZN4phgb17launch_gmres_coopERKNS_8GmresRunEP11CUstream_st",
    "_ZN4phgb16launch_gear_coopERKNS_11GearBuffersERKNS_7Q16ViewEiPdP11CUstream_st"))

REFUSED_SOLVES = """
import sys
sys.path[:0] = sys.argv[1:3]
import phg_b200
from oracle import pho
import test_gpu_one_kernel_limits as t
A = t.banded_spd(3000, 6, seed=1)
for solver in t.SOLVERS:
    with phg_b200.Solver(0) as s:
        s.set_matrix(*A)
        for again in range(2):
            (x, nits), k = t.launches(s, lambda: t.solve(s, solver))
            assert k > nits, (solver, k)
            t.check(pho, A, solver, x)
        if solver == "mixed":   # the cooperative form of the q16 iterations
            s.set_spmv_plan32("q16", 1)
            (x, nits), k = t.launches(s, lambda: t.solve(s, solver))
            assert k > nits, (solver, k)
            t.check(pho, A, solver, x)
print("refused and solved")
"""


def test_refused_launch_goes_to_the_launched_path(gpu, tmp_path):
    """A program whose share of the device cannot hold the grid: every
    cooperative launch answers "too large" (a preloaded stand-in for the
    library's launch functions), and every solver still solves."""
    import os
    import subprocess
    import sys

    from conftest import ROOT
    (tmp_path / "refuse.c").write_text(REFUSE)
    lib = str(tmp_path / "refuse.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", lib, str(tmp_path / "refuse.c")], check=True)
    p = subprocess.run([sys.executable, "-c", REFUSED_SOLVES, ROOT, os.path.join(ROOT, "tests")],
                       env=dict(os.environ, LD_PRELOAD=lib), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "refused and solved" in p.stdout, (p.stdout[-2000:], p.stderr[-2000:])


def test_no_memory_for_the_matrix_copy(gpu, oracle):
    """With the product's layout made and less memory free than the kernel's
    copy of the matrix takes (12 bytes an entry), the launched iteration solves."""
    import torch
    A = banded_spd(200000, 30, seed=2)
    copy = 12 * len(A[1])
    assert copy > 96 << 20
    with gpu.Solver(0) as s:
        s.set_matrix(*A)
        s.mat_vec(A[3])
        held, chunk = [], 1 << 34
        while chunk >= 16 << 20:   # leave 32 to 48 MB
            free = torch.cuda.mem_get_info()[0]
            if free - chunk < 32 << 20:
                chunk >>= 1
                continue
            held.append(torch.empty(chunk, dtype=torch.uint8, device="cuda"))
        try:
            (x, nits), k = launches(s, lambda: solve(s, "pcg"))
        finally:
            del held
            torch.cuda.empty_cache()
        assert k > nits
        check(oracle, A, "pcg", x)
        # with the memory back, the kernel takes it
        assert launches(s, lambda: solve(s, "pcg"))[1] == 1


def test_stream_with_part_of_the_device(gpu, oracle):
    """A system on a stream that has 16 multiprocessors (a green context): the
    grids fit them, so the solves run as one kernel there too, the cooperative
    form of the q16 iterations among them."""
    import torch
    drv = pytest.importorskip("cuda.bindings.driver")

    def call(result):
        assert result[0] == drv.CUresult.CUDA_SUCCESS, result[0]
        return result[1] if len(result) == 2 else result[1:]

    torch.cuda.init()
    torch.zeros(1, device="cuda")
    dev = call(drv.cuDeviceGet(0))
    sms = call(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups = call(drv.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    desc = call(drv.cuDevResourceGenerateDesc([groups[0]], 1))
    green = call(drv.cuGreenCtxCreate(desc, dev, int(drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM)))
    stream = call(drv.cuGreenCtxStreamCreate(green, int(drv.CUstream_flags.CU_STREAM_NON_BLOCKING), 0))
    A = banded_spd(40001, 12, seed=7)
    for solver in SOLVERS:
        with gpu.Solver(0, stream=int(stream)) as s:
            s.set_matrix(*A)
            (x, _), k = launches(s, lambda: solve(s, solver))
            assert k == 1, solver
            check(oracle, A, solver, x)
            if solver == "mixed":
                s.set_spmv_plan32("q16", 1)
                check(oracle, A, solver, solve(s, solver)[0])
    drv.cuStreamDestroy(stream)
    drv.cuGreenCtxDestroy(green)


def test_mixed_solve_on_an_fp64_layout_of_the_caller(gpu, oracle):
    """phgGpuSetSpMVPlan holds for the mixed solve too, whose FP64 residuals
    take that layout: it goes to the launched iteration."""
    A = banded_spd(3000, 6, seed=8)
    with gpu.Solver(0) as s:
        s.set_matrix(*A)
        assert launches(s, lambda: solve(s, "mixed"))[1] == 1
        for layout, param in (("csr", 8), ("sell", 4), ("q16", 1)):
            s.set_spmv_plan(layout, param)
            (x, _), k = launches(s, lambda: solve(s, "mixed"))
            assert k > 5, layout
            check(oracle, A, "mixed", x)
            assert s.spmv_plan()[:2] == (layout, param)
