"""The work this framework is measured on, as a user's program has it done.

Every case is one pass through the public entry points of ``phg_b200``: a
mesh, a Lagrange P1/P2/P3 space, the assembled system and its solution.  The
meshes are Kuhn cubes of 6 m^3 tetrahedra, as everywhere in this repository;
`jitter` moves the interior vertices off the grid, so that element matrices
have no exact zeros (a mesh from a mesh generator), while `jitter = 0` is the
grid itself, whose exact zeros the assembly drops.  Data live on the GPU, as
in a program that keeps its fields there; a system works on the caller's
stream.

Kinds of cases:
  step      a new mesh: set_mesh, set_dof_map, build, solve from zero
  assemble  a new mesh: set_mesh, set_dof_map, build, the CSR and right-hand
            side read back (a program with a solver of its own)
  timestep  an implicit time step on a fixed mesh: build with a mass term on
            the pattern already recorded, solve from the last step's solution
  solve     a new right-hand side for an assembled matrix
  adjoint   one evaluation of an inverse problem: build with a coefficient,
            forward solve, adjoint gradient
  block     many right-hand sides for one matrix
  krylov    a non-symmetric matrix handed over as CSR, then BiCGstab or GMRES
  matvec    one product
"""
import functools
import math
import warnings

import numpy as np
import torch

import phg_b200 as pb

DEV = "cuda:0"
NB = {1: 4, 2: 10, 3: 20}


def listed():
    return [
        # a small problem solved many times over (a parameter study, a coarse
        # level, a unit test): latency and launches
        dict(name="step_p1_m10", kind="step", p=1, m=10, jitter=0.1, kappa=1, solver="pcg", rtol=1e-10),
        # plain P1 Poisson on 32^3 subcubes, the smallest benchmark configuration
        dict(name="step_p1_m32", kind="step", p=1, m=32, jitter=0.0, kappa=0, solver="pcg", rtol=1e-10),
        # P2 Poisson on 64^3 subcubes, mixed precision: the headline benchmark
        dict(name="step_p2_m64", kind="step", p=2, m=64, jitter=0.0, kappa=0, solver="mixed", rtol=1e-8),
        # P3 with a variable coefficient, mixed precision
        dict(name="step_p3_m20", kind="step", p=3, m=20, jitter=0.0, kappa=1, solver="mixed", rtol=1e-8),
        # the CSR of a P2 space with coefficient, mass term and boundary data
        dict(name="assemble_p2_m40", kind="assemble", p=2, m=40, jitter=0.1, kappa=1, mass=2.5, bc=1),
        # heat equation: a few iterations per step, an odd size
        dict(name="timestep_p2_m31", kind="timestep", p=2, m=31, jitter=0.1, kappa=1, mass=2000.0, rtol=1e-8),
        # FP64 solve for one more right-hand side, ordinary size
        dict(name="solve_p2_m40", kind="solve", p=2, m=40, jitter=0.1, kappa=1, solver="pcg", rtol=1e-10),
        # coefficient identification on a P1 mesh
        dict(name="adjoint_p1_m72", kind="adjoint", p=1, m=72, jitter=0.0, kappa=1, rtol=1e-10),
        # 64 right-hand sides at once, mixed precision
        dict(name="block_p2_m24_k64", kind="block", p=2, m=24, jitter=0.0, kappa=0, nrhs=64, mixed=1, rtol=1e-8),
        # convection-diffusion with the two solvers for non-symmetric matrices
        dict(name="bicgstab_m48", kind="krylov", m=48, solver="bicgstab", rtol=1e-10),
        dict(name="flgmres_m33", kind="krylov", m=33, solver="flgmres", rtol=1e-10),
        # phgMatVec on device vectors
        dict(name="matvec_p2_m48", kind="matvec", p=2, m=48, jitter=0.0, kappa=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, any order, sizes spread over their logarithm
    up to (in unknowns) about the listed cases of the kind."""
    kind = rng.choice(["step", "step", "assemble", "timestep", "solve", "adjoint", "block", "krylov", "matvec"])
    jitter = rng.choice([0.0, 0.1])
    kappa = rng.randint(0, 1)
    rtol = rng.choice([1e-8, 1e-10])
    if kind == "krylov":
        return dict(kind=kind, m=_log_int(rng, 7, 56), solver=rng.choice(["bicgstab", "gmres", "flgmres"]), rtol=1e-10)
    p = rng.choice([1, 2, 3])
    if kind == "block":
        return dict(kind=kind, p=p, m=_log_int(rng, 5, {1: 40, 2: 22, 3: 13}[p]), jitter=jitter, kappa=kappa,
                    nrhs=rng.randint(1, 64), mixed=rng.randint(0, 1), rtol=1e-8)
    m = _log_int(rng, {1: 6, 2: 4, 3: 3}[p], {1: 90, 2: 50, 3: 26}[p])
    case = dict(kind=kind, p=p, m=m, jitter=jitter, kappa=kappa)
    if kind in ("step", "solve"):
        case.update(solver=rng.choice(["pcg", "mixed"]), rtol=rtol)
    if kind == "assemble":
        # no exact zeros to drop, so that the order of the entries is known
        case.update(m=min(m, {1: 70, 2: 40, 3: 20}[p]), jitter=0.1, mass=rng.choice([0.0, 3.5]), bc=rng.randint(0, 1))
    if kind == "timestep":
        case.update(m=min(m, {1: 70, 2: 40, 3: 20}[p]), mass=rng.choice([200.0, 5000.0]), rtol=1e-8)
    if kind == "adjoint":
        case.update(m=min(m, {1: 72, 2: 32, 3: 16}[p]), kappa=1, rtol=1e-10)
    return case


# ---------------------------------------------------------------------------
# Inputs

_EDGES = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))
_FACES = ((1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2))


@functools.lru_cache(maxsize=4)
def _space(m, p):
    """Vertices, elements, element-to-DOF map, Dirichlet flags and the two to
    four vertices (with weights) each Lagrange node interpolates: the layout
    of phg_b200.lagrange_dofs (vertices, then edges, then faces), numbered on
    the GPU."""
    v, e = pb.kuhn_cube(m)
    verts = torch.from_numpy(v).to(DEV)
    elems = torch.from_numpy(e).to(DEV).long()
    nv = len(v)
    on = (verts == 0.0) | (verts == 1.0)          # nvert x 3: which coordinate planes a vertex lies on
    side = on.long() + (verts == 1.0).long()      # 0 inside, 1 low plane, 2 high plane

    def boundary(idx):                            # the points idx[i] share a face of the cube
        s = side[idx]
        return ((s == s[:, :1]).all(dim=1) & (s[:, 0] > 0)).any(dim=1)

    cols, flags = [elems], [on.any(dim=1)]
    node_v = [torch.arange(nv, device=DEV)[:, None].expand(nv, 3)]
    node_w = [torch.tensor([1.0, 0.0, 0.0], dtype=torch.float64, device=DEV).expand(nv, 3)]
    nd = nv
    if p >= 2:
        ev = elems[:, torch.tensor(_EDGES, device=DEV)]
        lo, hi = ev.amin(2), ev.amax(2)
        eu, inv = torch.unique(lo * nv + hi, return_inverse=True)
        ends = torch.stack([eu // nv, eu % nv], 1)
        eb = boundary(ends)
        third = torch.cat([ends, ends[:, :1]], 1)
        if p == 2:
            cols.append(nd + inv)
            flags.append(eb)
            node_v.append(third)
            node_w.append(torch.tensor([0.5, 0.5, 0.0], dtype=torch.float64, device=DEV).expand(len(eu), 3))
            nd += len(eu)
        else:
            low_first = (ev[:, :, 0] < ev[:, :, 1]).long()
            near = nd + 2 * inv + (1 - low_first)  # the node nearer the edge's first local vertex
            far = nd + 2 * inv + low_first
            cols.append(torch.stack([near, far], 2).reshape(len(e), 12))
            flags.append(eb.repeat_interleave(2))
            node_v.append(third.repeat_interleave(2, 0))
            w = torch.tensor([[2 / 3, 1 / 3, 0.0], [1 / 3, 2 / 3, 0.0]], dtype=torch.float64, device=DEV)
            node_w.append(w.repeat(len(eu), 1))
            nd += 2 * len(eu)
            fv = elems[:, torch.tensor(_FACES, device=DEV)].sort(2).values
            fu, finv = torch.unique((fv[..., 0] * nv + fv[..., 1]) * nv + fv[..., 2], return_inverse=True)
            corners = torch.stack([fu // (nv * nv), fu // nv % nv, fu % nv], 1)
            cols.append(nd + finv)
            flags.append(boundary(corners))
            node_v.append(corners)
            node_w.append(torch.full((len(fu), 3), 1 / 3, dtype=torch.float64, device=DEV))
    e2l = torch.cat(cols, 1).int().contiguous()
    bdry = torch.cat(flags).to(torch.uint8)
    return verts, elems.int().contiguous(), e2l, bdry, torch.cat(node_v), torch.cat(node_w)


class State:
    pass


def _fields(case, seed):
    """Mesh, space, coefficient, source and boundary data of a case."""
    gen = torch.Generator(device=DEV).manual_seed(1000003 * seed + 17)
    d = State()
    m, p = case["m"], case["p"]
    verts, d.elems, d.e2l, d.bdry, nv, nw = _space(m, p)
    inside = ((verts > 0.0) & (verts < 1.0)).all(dim=1, keepdim=True)
    move = 2.0 * torch.rand(verts.shape, generator=gen, device=DEV, dtype=torch.float64) - 1.0
    d.verts = (verts + torch.where(inside, case["jitter"] / m * move, torch.zeros_like(move))).contiguous()
    nodes = (d.verts[nv] * nw[:, :, None]).sum(1)
    d.n, ne = len(d.bdry), len(d.elems)
    amp = 0.5 + 1.5 * torch.rand(4, generator=gen, device=DEV, dtype=torch.float64)
    s1 = torch.sin(math.pi * nodes).prod(1)
    s2 = torch.sin(2 * math.pi * nodes).prod(1)
    d.f = amp[0] * 3 * math.pi ** 2 * s1 + 0.2 * amp[1] * 12 * math.pi ** 2 * s2
    z = torch.randn(ne, generator=gen, device=DEV, dtype=torch.float64)
    d.kappa = torch.exp(0.5 * z) if case["kappa"] else None
    d.g = (amp[2] * nodes[:, 0] + amp[3] * nodes[:, 1] * nodes[:, 2]).contiguous() if case.get("bc") else None
    d.noise = torch.randn(d.n, generator=gen, device=DEV, dtype=torch.float64)
    d.s1 = s1
    d.gen = gen
    return d


def _convection(case, seed):
    """Convection-diffusion on an m^3 grid, upwind differences, 7 entries per
    inner row, Dirichlet outside: CSR (int64 pointers) and right-hand side."""
    gen = torch.Generator(device=DEV).manual_seed(1000003 * seed + 29)
    m = case["m"]
    n = m ** 3
    i = torch.arange(n, device=DEV)
    c = [i % m, i // m % m, i // (m * m)]
    h = 1.0 / (m + 1)
    speed = 20.0 + 20.0 * torch.rand(3, generator=gen, device=DEV, dtype=torch.float64)
    b = [speed[k] * torch.sin(math.pi * h * (c[(k + 1) % 3] + 1).double()) for k in range(3)]
    diag = 6.0 + h * (b[0].abs() + b[1].abs() + b[2].abs())
    # columns ascending: -m^2, -m, -1, 0, +1, +m, +m^2
    cols, vals, ok = [], [], []
    for k in (2, 1, 0):
        cols.append(i - m ** k); vals.append(-1.0 - h * b[k].clamp(min=0)); ok.append(c[k] > 0)
    cols.append(i); vals.append(diag); ok.append(torch.ones_like(i, dtype=torch.bool))
    for k in (0, 1, 2):
        cols.append(i + m ** k); vals.append(-1.0 - h * (-b[k]).clamp(min=0)); ok.append(c[k] < m - 1)
    ok, cols, vals = torch.stack(ok, 1), torch.stack(cols, 1), torch.stack(vals, 1)
    d = State()
    d.n = n
    d.ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), ok.sum(1).cumsum(0)])
    d.cols = cols[ok].int().contiguous()
    d.vals = vals[ok].contiguous()
    d.rhs = torch.randn(n, generator=gen, device=DEV, dtype=torch.float64)
    return d


def prepare(case, seed):
    kind = case["kind"]
    d = _convection(case, seed) if kind == "krylov" else _fields(case, seed)
    d.case = case
    d.stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    d.solver = pb.Solver(0, d.stream.cuda_stream)
    if kind in ("timestep", "solve", "adjoint", "block", "matvec"):
        d.solver.set_mesh(d.verts, d.elems)
        d.solver.set_dof_map(case["p"], d.e2l, d.bdry)
    if kind in ("solve", "block", "matvec"):
        d.solver.build_linear_system(kappa=d.kappa, f=d.f)
    if kind == "solve":
        free = (d.bdry == 0).double()
        d.rhs = free * (d.s1 / case["m"] ** 3 + 1e-3 * d.noise / case["m"] ** 3)
    if kind == "timestep":   # two steps taken: the pattern of the rows is recorded
        for _ in range(2):
            d.solver.build_linear_system(kappa=d.kappa, f=d.f, mass=case["mass"])
        d.u0 = d.f / (3 * math.pi ** 2 + case["mass"])
    if kind == "adjoint":
        free = (d.bdry == 0).double()
        d.u_obs = free * (0.8 * d.f / (3 * math.pi ** 2) + 0.01 * d.noise)
    if kind == "block":
        free = (d.bdry == 0).double()
        d.B = (free[:, None] * torch.randn(d.n, case["nrhs"], generator=d.gen, device=DEV,
                                           dtype=torch.float64)).contiguous()
    if kind == "matvec":
        d.y = torch.empty(d.n, dtype=torch.float64, device=DEV)
    torch.cuda.synchronize()
    return d


# ---------------------------------------------------------------------------
# One pass

def _solve(s, case, x):
    if case["solver"] == "mixed":
        s.solve_pcg_mixed(rtol=case["rtol"], out=x)
    else:
        s.solve_pcg(rtol=case["rtol"], btol=0.0, out=x)
    return x


def _zeros(d):
    return torch.zeros(d.n, dtype=torch.float64, device=DEV)


def _matrix(s):
    """The assembled CSR and right-hand side, copied into device tensors
    through the C ABI."""
    L, h = pb.load_library(), s._h
    n, nnz, _ = s.sizes()
    ptr = torch.empty(n + 1, dtype=torch.int64, device=DEV)
    cols = torch.empty(nnz, dtype=torch.int32, device=DEV)
    vals = torch.empty(nnz, dtype=torch.float64, device=DEV)
    rhs = torch.empty(n, dtype=torch.float64, device=DEV)
    for rc in (L.phgGpuGetMatrix(h, ptr.data_ptr(), cols.data_ptr(), vals.data_ptr()),
               L.phgGpuGetRHS(h, rhs.data_ptr())):
        if rc < 0:
            raise RuntimeError(L.phgGpuLastError().decode())
    return ptr, cols, vals, rhs


def run(d):
    case, s = d.case, d.solver
    kind = case["kind"]
    here = torch.cuda.current_stream()
    d.stream.wait_stream(here)
    with torch.cuda.stream(d.stream):
        if kind in ("step", "assemble"):
            s.set_mesh(d.verts, d.elems)
            s.set_dof_map(case["p"], d.e2l, d.bdry)
            s.build_linear_system(kappa=d.kappa, f=d.f, g=d.g, mass=case.get("mass", 0.0))
            out = _solve(s, case, _zeros(d)) if kind == "step" else _matrix(s)
        elif kind == "timestep":
            s.build_linear_system(kappa=d.kappa, f=d.f, mass=case["mass"])
            x = d.u0.clone()
            s.solve_pcg(rtol=case["rtol"], btol=case["rtol"], out=x)
            out = x
        elif kind == "solve":
            s.set_rhs(d.rhs)
            out = _solve(s, case, _zeros(d))
        elif kind == "adjoint":
            s.build_linear_system(kappa=d.kappa, f=d.f)
            u = _zeros(d)
            s.solve_pcg(rtol=case["rtol"], btol=0.0, out=u)
            grad = torch.empty(len(d.elems), dtype=torch.float64, device=DEV)
            _, J, _ = s.adjoint_gradient(u, d.u_obs, rtol=case["rtol"], out=grad)
            out = (u, grad, J)
        elif kind == "block":
            X = torch.empty_like(d.B)
            s.solve_block_pcg(d.B, rtol=case["rtol"], mixed=bool(case["mixed"]), out=X)
            out = X
        elif kind == "krylov":
            s.set_matrix(d.ptr, d.cols, d.vals, d.rhs)
            solve = {"bicgstab": s.solve_bicgstab, "gmres": s.solve_gmres, "flgmres": s.solve_flgmres}[case["solver"]]
            out, _, _ = solve(rtol=case["rtol"], btol=0.0, out=_zeros(d))
        else:
            out = s.mat_vec(d.f, d.y)
    here.wait_stream(d.stream)
    return out


# ---------------------------------------------------------------------------
# What a pass cannot do without

# Jacobi-CG iterations per subcube and decade of the residual, by order (the
# meshes' condition grows with m); matrix entries per row by order, on the
# grid and off it.
_ITS = {1: 0.4, 2: 0.9, 3: 2.3}
_ROW = {1: (7, 14), 2: (26, 27), 3: (42, 44)}


def work(case):
    kind, m = case["kind"], case["m"]
    if kind == "krylov":
        n, nnz = m ** 3, 7 * m ** 3
        its = 2.2 * m if case["solver"] == "bicgstab" else 6.4 * m
        products = 2 * its if case["solver"] == "bicgstab" else its
        return {"bytes": products * (12 * nnz + 24 * n) + 12 * nnz, "flops": products * (2 * nnz + 10 * n)}
    p = case["p"]
    ne, n, N = 6 * m ** 3, (p * m + 1) ** 3, NB[p]
    nnz = _ROW[p][1 if case["jitter"] else 0] * n
    build = ne * (16 + 4 * N + 8 * case["kappa"]) + 24 * (m + 1) ** 3 + 12 * nnz + 33 * n
    build_flops = ne * N * N * 8
    if kind == "matvec":
        return {"bytes": 12 * nnz + 20 * n, "flops": 2 * nnz}
    if kind == "assemble":
        return {"bytes": build, "flops": build_flops}
    its = _ITS[p] * m * -math.log10(case["rtol"])
    if kind == "timestep":
        its = 45
    if kind == "block":
        k, w = case["nrhs"], 4 if case["mixed"] else 8
        return {"bytes": its * ((4 + w) * nnz + 4 * w * n * k) + 16 * n * k, "flops": its * k * (2 * nnz + 10 * n)}
    w = 4 if case.get("solver") == "mixed" else 8
    solve, solve_flops = its * ((4 + w) * nnz + 8 * w * n), its * (2 * nnz + 12 * n)
    if kind == "solve":
        return {"bytes": solve, "flops": solve_flops}
    if kind == "adjoint":
        return {"bytes": build + 2 * solve + 8 * ne, "flops": build_flops + 2 * solve_flops + 2 * ne * N * N}
    return {"bytes": build + solve, "flops": build_flops + solve_flops}


# ---------------------------------------------------------------------------
# The same in plain torch, 64 bits

def _poly_mul(a, b):
    out = {}
    for ea, ca in a.items():
        for eb, cb in b.items():
            e = tuple(x + y for x, y in zip(ea, eb))
            out[e] = out.get(e, 0.0) + ca * cb
    return out


def _poly_diff(a, c):
    out = {}
    for e, v in a.items():
        if e[c]:
            f = list(e)
            f[c] -= 1
            out[tuple(f)] = out.get(tuple(f), 0.0) + v * e[c]
    return out


def _poly_mean(a):
    """Integral over a tetrahedron, divided by its volume."""
    t = 0.0
    for e, v in a.items():
        num = 6.0
        for x in e:
            num *= math.factorial(x)
        t += v * num / math.factorial(sum(e) + 3)
    return t


@functools.lru_cache(maxsize=3)
def _reference(p):
    """S[c, d, a, b] = mean of dphi_a/dlambda_c dphi_b/dlambda_d and
    M[a, b] = mean of phi_a phi_b on a tetrahedron."""
    def lin(i, c1, c0):                            # c1 lambda_i + c0
        e = [0, 0, 0, 0]
        e[i] = 1
        return {tuple(e): c1, (0, 0, 0, 0): c0}

    def prod(scale, *fs):
        r = {(0, 0, 0, 0): scale}
        for f in fs:
            r = _poly_mul(r, f)
        return r

    if p == 1:
        phi = [lin(i, 1.0, 0.0) for i in range(4)]
    elif p == 2:
        phi = [prod(1.0, lin(i, 1, 0), lin(i, 2, -1)) for i in range(4)]
        phi += [prod(4.0, lin(i, 1, 0), lin(j, 1, 0)) for i, j in _EDGES]
    else:
        phi = [prod(0.5, lin(i, 1, 0), lin(i, 3, -1), lin(i, 3, -2)) for i in range(4)]
        for i, j in _EDGES:
            phi.append(prod(4.5, lin(i, 1, 0), lin(j, 1, 0), lin(i, 3, -1)))
            phi.append(prod(4.5, lin(i, 1, 0), lin(j, 1, 0), lin(j, 3, -1)))
        phi += [prod(27.0, *(lin(v, 1, 0) for v in f)) for f in _FACES]
    N = len(phi)
    dphi = [[_poly_diff(f, c) for c in range(4)] for f in phi]
    S = np.array([[[[_poly_mean(_poly_mul(dphi[a][c], dphi[b][e])) for b in range(N)] for a in range(N)]
                   for e in range(4)] for c in range(4)])
    M = np.array([[_poly_mean(_poly_mul(phi[a], phi[b])) for b in range(N)] for a in range(N)])
    return torch.from_numpy(S).to(DEV), torch.from_numpy(M).to(DEV)


def _element_matrices(d, p, mass):
    """Stiffness (kappa and mass included) and right-hand side per element."""
    S, M = _reference(p)
    x = d.verts[d.elems.long()]
    A = torch.cat([x, torch.ones_like(x[..., :1])], 2)
    grad = torch.linalg.inv(A)[:, :3].transpose(1, 2)          # row c: gradient of lambda_c
    vol = torch.linalg.det(x[:, 1:] - x[:, :1]).abs() / 6.0
    gg = torch.einsum("ecx,edx->ecd", grad, grad) * vol[:, None, None]
    if d.kappa is not None:
        gg = gg * d.kappa[:, None, None]
    N = NB[p]
    Ke = (gg.reshape(-1, 16) @ S.reshape(16, N * N)).reshape(-1, N, N)
    if mass:
        Ke += mass * vol[:, None, None] * M
    Re = vol[:, None] * (d.f[d.e2l.long()] @ M)
    return Ke, Re


def _system(d, p, mass):
    """Assembled rows as (ptr, cols, vals, rhs): boundary columns moved to the
    right-hand side, entries in the order the elements first touch them."""
    Ke, Re = _element_matrices(d, p, mass)
    n, N = d.n, NB[p]
    e2l = d.e2l.long()
    isb = d.bdry.bool()
    rhs = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, e2l.reshape(-1), Re.reshape(-1))
    g = d.g if d.g is not None else torch.zeros(n, dtype=torch.float64, device=DEV)
    lift = torch.einsum("eab,eb->ea", Ke, (g * isb)[e2l])
    rhs.index_add_(0, e2l.reshape(-1), -lift.reshape(-1))
    mult = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(
        0, e2l.reshape(-1), torch.ones(e2l.numel(), dtype=torch.float64, device=DEV))
    rhs = torch.where(isb, mult * g, rhs)
    rows = e2l[:, :, None].expand(-1, N, N).reshape(-1)
    colx = e2l[:, None, :].expand(-1, N, N).reshape(-1)
    keep = ~isb[rows] & ~isb[colx]
    key = (rows * n + colx)[keep]
    order = torch.nonzero(keep)[:, 0]
    bd = torch.nonzero(isb)[:, 0]
    key = torch.cat([key, bd * n + bd])
    order = torch.cat([order, torch.zeros_like(bd)])
    val = torch.cat([Ke.reshape(-1)[keep], mult[bd]])
    del rows, colx, keep, Ke
    uniq, inv = torch.unique(key, return_inverse=True)
    del key
    vals = torch.zeros(len(uniq), dtype=torch.float64, device=DEV).index_add_(0, inv, val)
    first = torch.full((len(uniq),), 2 ** 62, dtype=torch.int64, device=DEV).scatter_reduce_(0, inv, order, "amin")
    del inv, order, val
    r, c = uniq // n, uniq % n
    by_touch = torch.argsort(first)
    by_touch = by_touch[torch.argsort(r[by_touch], stable=True)]
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), torch.bincount(r, minlength=n).cumsum(0)])
    return ptr, c[by_touch], vals[by_touch], rhs, mult


def _csr(ptr, cols, vals, n):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return torch.sparse_csr_tensor(ptr, cols, vals, size=(n, n), check_invariants=False)


def _cg(A, diag, b, x, tol=1e-14, maxit=4000):
    """Jacobi-CG, column by column if b has several, started anew from the
    true residual until that is at rounding level."""
    norm = b.norm(dim=0).clamp(min=1e-300)
    if b.dim() == 2:
        diag = diag[:, None]
    for _ in range(3):
        r = b - A @ x
        z = r / diag
        q = z.clone()
        rz = (r * z).sum(0)
        for it in range(maxit):
            Aq = A @ q
            pap = (q * Aq).sum(0)
            a = torch.where(pap > 0, rz / pap.clamp(min=1e-300), torch.zeros_like(pap))
            x = x + a * q
            r = r - a * Aq
            if it % 10 == 0 and bool((r.norm(dim=0) <= tol * norm).all()):
                break
            z = r / diag
            new = (r * z).sum(0)
            q = z + torch.where(rz > 0, new / rz.clamp(min=1e-300), torch.zeros_like(rz)) * q
            rz = new
    return x


def _bicgstab(A, diag, b, tol=1e-14, maxit=2000):
    x = torch.zeros_like(b)
    for _ in range(4):
        r = b - A @ x
        if float(r.norm()) <= 10 * tol * float(b.norm()):
            break
        rh, q = r.clone(), r.clone()
        rho = float(rh @ r)
        goal = tol * float(b.norm())
        for _ in range(maxit):
            ph = q / diag
            v = A @ ph
            alpha = rho / float(rh @ v)
            s = r - alpha * v
            sh = s / diag
            t = A @ sh
            tt = float(t @ t)
            if tt == 0.0:
                x = x + alpha * ph
                break
            om = float(t @ s) / tt
            x = x + alpha * ph + om * sh
            r = s - om * t
            if float(r.norm()) <= goal:
                break
            rho_new = float(rh @ r)
            if rho_new == 0.0 or om == 0.0:
                break
            q = r + (rho_new / rho) * (alpha / om) * (q - om * v)
            rho = rho_new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "krylov":
        d = _convection(case, seed)
        rows = torch.repeat_interleave(torch.arange(d.n, device=DEV), d.ptr[1:] - d.ptr[:-1])
        diag = d.vals[rows == d.cols]
        return _bicgstab(_csr(d.ptr, d.cols.long(), d.vals, d.n), diag, d.rhs)
    d = _fields(case, seed)
    p = case["p"]
    ptr, cols, vals, rhs, mult = _system(d, p, case.get("mass", 0.0))
    if kind == "assemble":
        return None, None, vals, rhs
    rows = torch.repeat_interleave(torch.arange(d.n, device=DEV), ptr[1:] - ptr[:-1])
    diag = torch.zeros(d.n, dtype=torch.float64, device=DEV).index_add_(0, rows[rows == cols], vals[rows == cols])
    del rows
    A = _csr(ptr, cols, vals, d.n)
    free = (d.bdry == 0).double()
    if kind == "matvec":
        return A @ d.f
    if kind == "solve":
        rhs = free * (d.s1 / case["m"] ** 3 + 1e-3 * d.noise / case["m"] ** 3)
    if kind == "block":
        B = free[:, None] * torch.randn(d.n, case["nrhs"], generator=d.gen, device=DEV, dtype=torch.float64)
        return _cg(A, diag, B, torch.zeros_like(B))
    x = _cg(A, diag, rhs, torch.zeros_like(rhs))
    if kind == "adjoint":
        u_obs = free * (0.8 * d.f / (3 * math.pi ** 2) + 0.01 * d.noise)
        lam = _cg(A, diag, free * (x - u_obs), torch.zeros_like(x))
        del A
        Ke, _ = _element_matrices(d, p, 0.0)
        e2l = d.e2l.long()
        grad = -torch.einsum("ea,eab,eb->e", lam[e2l], Ke, x[e2l])
        return x, grad, 0.5 * float(((x - u_obs) ** 2).sum())
    return x
