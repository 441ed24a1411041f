"""The calls whose speed this framework stands for: Krylov solves of nodal and
edge-element systems with their preconditioners, at the sizes that scripts use
them.

Nodal systems are separable 7-point operators c_x L_x + c_y L_y + c_z L_z + s
(seeded positive coefficients, a complex shift for the complex ones) on ragged
grids. Edge systems are lowest-order Nedelec curl-curl + mass matrices on the
Kuhn mesh of the unit cube with a seeded reluctivity of the core and seeded
right-hand sides, boundary edges constrained. Their mass weights keep the
solution determined by the data to many more digits than it is solved for, so
two correct solves agree closely.

Host cases call the Python classes with numpy arrays, as the scripts written
for the reference do (every solve then re-reads the matrix values). Device
cases keep the right-hand side and the solution in HBM and go through the C
ABI's ``_dev`` entry points, as a C++ host program does.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ngsolve-sparsesolv_b200"))

import sparsesolv_ngsolve as ss  # noqa: E402
from sparsesolv_ngsolve import _capi, hcurl, problems  # noqa: E402

TOL = 1e-10
MAXITER = 1000


def listed():
    return [
        # a small nodal solve with the default options: latency and launches are everything
        dict(name="iccg_small", kind="nodal", method="ICCG", abmc=False, cplx=False, masked=False, host=True,
             nx=16, ny=16, nz=16),
        # the default options (level-scheduled IC) on an ordinary ragged nodal system
        dict(name="iccg_levels", kind="nodal", method="ICCG", abmc=False, cplx=False, masked=False, host=True,
             nx=61, ny=53, nz=57),
        # the colour-ordered form at the size of the nodal benchmark, vectors resident
        dict(name="iccg_abmc", kind="nodal", method="ICCG", abmc=True, cplx=False, masked=False, host=False,
             nx=64, ny=64, nz=64),
        # a complex-symmetric nodal system, colour-ordered
        dict(name="iccg_abmc_complex", kind="nodal", method="ICCG", abmc=True, cplx=True, masked=False, host=True,
             nx=41, ny=37, nz=45),
        # the Gauss-Seidel MRTR method with constrained boundary nodes
        dict(name="sgsmrtr", kind="nodal", method="SGSMRTR", abmc=False, cplx=False, masked=True, host=True,
             nx=40, ny=40, nz=40),
        # shifted ICCG on an edge-element matrix: about 16 entries a row, factorised in each call
        dict(name="iccg_edge", kind="edge", abmc=False, host=True, nc=24),
        # restarted GMRES with symmetric Gauss-Seidel
        dict(name="gmres_sgs", kind="gmres", cplx=False, restart=30, nx=33, ny=31, nz=29),
        # the magnetostatic benchmark's size: Compact AMS + CG, vectors resident
        dict(name="ams_cg", kind="ams", precision="fp64", host=False, nc=40),
        # the FP32-preconditioner form on a small odd mesh
        dict(name="ams_cg_fp32", kind="ams", precision="fp32", host=True, nc=23),
        # one Newton step: Update() on new values, then the solve
        dict(name="newton_step", kind="newton", nc=20),
        # the eddy-current benchmark's size: Complex Compact AMS + COCR, vectors resident
        dict(name="eddy_cocr", kind="eddy", host=False, nc=64),
        # a frequency family solved together, four sources per frequency
        dict(name="eddy_batch", kind="batch", freqs=6, nrhs=4, nc=24),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["nodal", "nodal", "nodal", "edge", "gmres", "ams", "newton", "eddy", "batch"])
    if kind in ("nodal", "gmres"):
        top = 56 if kind == "nodal" else 34
        c = dict(kind=kind, nx=_log_int(rng, 11, top), ny=_log_int(rng, 11, top), nz=_log_int(rng, 11, top),
                 cplx=rng.random() < 0.4)
        if kind == "gmres":
            return dict(c, restart=rng.choice([20, 30, 50]))
        c["method"] = rng.choice(["ICCG", "ICCG", "ICCG", "SGSMRTR"])
        c["abmc"] = c["method"] == "ICCG" and rng.random() < 0.5
        return dict(c, masked=rng.random() < 0.3, host=rng.random() < 0.6)
    if kind == "edge":
        return dict(kind=kind, abmc=rng.random() < 0.3, host=rng.random() < 0.6, nc=_log_int(rng, 8, 24))
    if kind == "ams":
        return dict(kind=kind, precision=rng.choice(["fp64", "fp32"]), host=rng.random() < 0.5,
                    nc=_log_int(rng, 12, 40))
    if kind == "newton":
        return dict(kind=kind, nc=_log_int(rng, 10, 22))
    if kind == "eddy":
        return dict(kind=kind, host=rng.random() < 0.5, nc=_log_int(rng, 14, 56))
    return dict(kind=kind, freqs=rng.choice([2, 3, 4, 6]), nrhs=rng.choice([1, 4]), nc=_log_int(rng, 10, 22))


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------

def _rng(seed, *more):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, *more])


@functools.lru_cache(maxsize=4)
def _grid_pattern(nx, ny, nz):
    A = problems.laplacian_7pt(nx, ny, nz)
    rows = np.repeat(np.arange(nx * ny * nz, dtype=np.int64), np.diff(A.indptr))
    gap = np.abs(A.indices - rows)
    return A, gap


def _nodal_parts(case, seed):
    """Coefficients (c_x, c_y, c_z, shift) and the right-hand side [z][y][x]."""
    r = _rng(seed, 1)
    c = r.uniform(0.5, 2.0, 3)
    s = r.uniform(0.01, 0.05)
    shape = (case["nz"], case["ny"], case["nx"])
    b = r.uniform(-1.0, 1.0, shape)
    if case["cplx"]:
        b = b + 1j * r.uniform(-1.0, 1.0, shape)
        return c, s + 1j * r.uniform(0.1, 0.5), b
    return c, s, b


def _nodal_matrix(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    base, gap = _grid_pattern(nx, ny, nz)
    c, s, b = _nodal_parts(case, seed)
    A = base.astype(np.complex128 if case["cplx"] else np.float64)
    A.data[gap == 0] = 2.0 * c.sum() + s
    A.data[gap == 1] = -c[0]
    A.data[gap == nx] = -c[1]
    A.data[gap == nx * ny] = -c[2]
    return A, b.ravel()


def _free_nodes(case):
    """1 for interior nodes, 0 for the outermost layer of the grid."""
    f = np.zeros((case["nz"], case["ny"], case["nx"]), dtype=np.uint8)
    f[1:-1, 1:-1, 1:-1] = 1
    return f


def _on_gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@functools.lru_cache(maxsize=3)
def _mesh(nc):
    """The Kuhn mesh of hcurl.kuhn_mesh without its element gradients, built on
    the GPU (the host form takes seconds at the largest sizes)."""
    n1 = nc + 1
    dev = "cuda"
    g = torch.arange(n1, dtype=torch.float64) / nc
    zz, yy, xx = torch.meshgrid(g, g, g, indexing="ij")
    coords = torch.stack([xx.ravel(), yy.ravel(), zz.ravel()], 1).to(dev)
    a = torch.arange(nc, device=dev)
    ii, jj, kk = (t.ravel() for t in torch.meshgrid(a, a, a, indexing="ij"))
    v0 = ii + n1 * (jj + n1 * kk)
    unit = (1, n1, n1 * n1)
    tets = []
    for p in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        v1 = v0 + unit[p[0]]
        v2 = v1 + unit[p[1]]
        tets.append(torch.stack([v0, v1, v2, v2 + unit[p[2]]], 1))
    tets = torch.cat(tets)
    lo = tets[:, [0, 0, 0, 1, 1, 2]]  # vertex numbers grow along a path, so every local edge runs low -> high
    hi = tets[:, [1, 2, 3, 2, 3, 3]]
    key, inv = torch.unique((lo * n1 ** 3 + hi).ravel(), return_inverse=True)
    edges = torch.stack([key // n1 ** 3, key % n1 ** 3], 1)
    tet_edges = inv.reshape(-1, 6)
    cen = coords[tets].mean(1)
    core = ((cen > 0.3) & (cen < 0.7)).all(1)
    m = hcurl.KuhnMesh(nc, coords.cpu().numpy(), tets.cpu().numpy(), edges.cpu().numpy(), tet_edges.cpu().numpy(),
                       np.ones(tuple(tet_edges.shape)), cen.cpu().numpy(), None, None)
    return m, core.cpu().numpy(), hcurl.boundary_freedofs(m)


#: mass weights (core, outside) of each kind of edge system
MASS = {"edge": (1.0, 1.0), "ams": (1.0, 1.0), "newton": (1.0, 1.0), "eddy": (1.0, 0.1), "batch": (1.0, 0.1)}


def _edge_parts(case, seed):
    """K (curl-curl), M (weighted mass), G, the mesh and its free edges."""
    m, core, fd = _mesh(case["nc"])
    r = _rng(seed, 2)
    nu = np.where(core, r.uniform(0.1, 0.8), r.uniform(0.9, 1.1))
    inside, outside = MASS[case["kind"]]
    K, M, G = hcurl.assemble_on_device(m, nu, np.where(core, inside, outside))
    return K, M, G, m, fd


def _edge_rhs(case, seed, n, fd, cplx, shape=()):
    r = _rng(seed, 3)
    b = r.uniform(-1.0, 1.0, shape + (n,))
    if cplx:
        b = b + 1j * r.uniform(-1.0, 1.0, shape + (n,))
    return b * fd


def _same_pattern(A, data):
    """A matrix of A's pattern with other values."""
    B = A.astype(data.dtype)
    B.data[:] = data
    return B


def _omegas(case):
    return np.logspace(-0.5, 0.5, case["freqs"])


# ---------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------

def _ams(cls, A, G, m, fd, **kw):
    c = m.coords
    return cls(A, G, freedofs=fd, coord_x=c[:, 0].copy(), coord_y=c[:, 1].copy(), coord_z=c[:, 2].copy(), **kw)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, host=case.get("host", True))
    if kind in ("nodal", "gmres"):
        A, b = _nodal_matrix(case, seed)
        if kind == "gmres":
            st["b"] = b
            st["pre"] = ss.SGSPreconditioner(A)
            st["solver"] = ss.GMRESSolver(A, st["pre"], maxiter=MAXITER, tol=TOL, restart=case["restart"])
            return st
        fd = _free_nodes(case).ravel() if case["masked"] else None
        st["solver"] = ss.SparseSolvSolver(A, method=case["method"], freedofs=fd, tol=TOL, maxiter=MAXITER,
                                           use_abmc=case["abmc"])
    elif kind == "edge":
        K, M, _, m, fd = _edge_parts(case, seed)
        A = _same_pattern(K, K.data + M.data)
        b = _edge_rhs(case, seed, m.ne, fd, False)
        st["solver"] = ss.SparseSolvSolver(A, method="ICCG", freedofs=fd, tol=TOL, maxiter=MAXITER,
                                           use_abmc=case["abmc"])
    elif kind in ("ams", "newton"):
        K, M, G, m, fd = _edge_parts(case, seed)
        A = _same_pattern(K, K.data + M.data)
        b = _edge_rhs(case, seed, m.ne, fd, False)
        if kind == "newton":
            st["pre"] = _ams(ss.CompactAMSPreconditioner, _same_pattern(K, 0.9 * K.data + M.data), G, m, fd)
            return dict(st, A=A, b=b, fd=fd)
        st["pre"] = _ams(ss.CompactAMSPreconditioner, A, G, m, fd, precision=case["precision"])
        if st["host"]:
            st["solver"] = ss.PCGSolver(A, st["pre"], freedofs=fd, maxiter=MAXITER, tol=TOL)
        else:
            st["mat"] = ss._Matrix(A)
            st["fd"] = _on_gpu(fd)
            st["cfg"] = _capi.default_config(tolerance=TOL, max_iterations=MAXITER)
    elif kind == "eddy":
        K, M, G, m, fd = _edge_parts(case, seed)
        A = _same_pattern(K, K.data + 1j * M.data)
        b = _edge_rhs(case, seed, m.ne, fd, True)
        st["pre"] = _ams(ss.ComplexCompactAMSPreconditioner, _same_pattern(K, K.data + M.data), G, m, fd)
        if st["host"]:
            st["solver"] = ss.COCRSolver(A, st["pre"], freedofs=fd, maxiter=MAXITER, tol=TOL)
        else:
            st["mat"] = ss._Matrix(A)
            st["fd"] = _on_gpu(fd)
    else:
        K, M, G, m, fd = _edge_parts(case, seed)
        om = _omegas(case)
        st["pre"] = [_ams(ss.ComplexCompactAMSPreconditioner, _same_pattern(K, K.data + w * M.data), G, m, fd)
                     for w in om]
        st["solver"] = ss.BatchedCOCRSolver(K, M, om, st["pre"], nrhs=case["nrhs"], freedofs=fd, maxiter=MAXITER,
                                            tol=TOL)
        st["b"] = _on_gpu(_edge_rhs(case, seed, m.ne, fd, True, (case["freqs"], case["nrhs"])))
        st["x"] = torch.zeros_like(st["b"])
        return st
    if st["host"]:
        st["b"] = b
    else:
        st["b"] = _on_gpu(b)
        st["x"] = torch.zeros_like(st["b"])
    return st


def _zeroed(x):
    """The initial guess, in place before the library's own stream reads it."""
    x.zero_()
    torch.cuda.current_stream().synchronize()
    return ctypes.c_void_p(x.data_ptr())


def run(st):
    kind = st["kind"]
    if kind == "batch":
        st["solver"].solve_dev(st["b"].data_ptr(), st["x"].data_ptr())
        return st["x"]
    if kind == "newton":
        st["pre"].Update(st["A"])
        x = np.zeros(st["A"].shape[0])
        ss.PCGSolver(st["A"], st["pre"], freedofs=st["fd"], maxiter=MAXITER, tol=TOL).Solve(st["b"], x)
        return x
    if st["host"]:
        return st["solver"] * st["b"]
    lib = _capi.load()
    b, x = ctypes.c_void_p(st["b"].data_ptr()), _zeroed(st["x"])
    res = _capi.ssv_result()
    if kind in ("nodal", "edge"):
        s = st["solver"]
        _capi.check(lib.ssv_solver_solve_dev(s._h, s.method.encode(), ctypes.byref(s._cfg), b, x, ctypes.byref(res),
                                             None, 0))
        return st["x"]
    fd = ctypes.cast(st["fd"].data_ptr(), _capi.PU8)
    if kind == "ams":
        _capi.check(lib.ssv_pcg_solve_dev(st["mat"].h, st["pre"]._h, fd, ctypes.byref(st["cfg"]), b, x,
                                          ctypes.byref(res), None, 0))
    else:
        it = ctypes.c_int32()
        _capi.check(lib.ssv_cocr_solve_dev(st["mat"].h, st["pre"]._h, fd, MAXITER, TOL, 0, b, x, ctypes.byref(it)))
    return st["x"]


# ---------------------------------------------------------------------------
# work, exact
# ---------------------------------------------------------------------------

def work(case):
    """The matrix and the right-hand sides read once, the solutions written once,
    two operations an entry: what one application cannot do without (an iterative
    solve does it once an iteration)."""
    if case["kind"] in ("nodal", "gmres"):
        n = case["nx"] * case["ny"] * case["nz"]
        nnz, sb, cols = 7 * n, 16 if case["cplx"] else 8, 1
    else:
        nc = case["nc"]
        n = 7 * nc ** 3 + 9 * nc ** 2 + 3 * nc  # edges of the Kuhn mesh
        nnz, cols = 16 * n, case.get("freqs", 1) * case.get("nrhs", 1)
        sb = 16 if case["kind"] in ("eddy", "batch") else 8
    return {"bytes": float(nnz * (4 + sb) + 4 * n + 2 * n * sb * cols),
            "flops": float(2 * nnz * cols * (4 if sb == 16 else 1))}


def _sine(n):
    k = np.arange(1, n + 1)
    return math.sqrt(2.0 / (n + 1)) * np.sin(np.pi * np.outer(k, k) / (n + 1)), 2.0 - 2.0 * np.cos(np.pi * k / (n + 1))


def _nodal_exact(case, seed):
    """The separable operator diagonalised by sine transforms in each direction."""
    c, s, b = _nodal_parts(case, seed)
    inner = case.get("masked", False)
    if inner:
        b = b[1:-1, 1:-1, 1:-1]
    (Sz, lz), (Sy, ly), (Sx, lx) = (_sine(k) for k in b.shape)

    def transform(v):
        v = np.tensordot(Sz, v, (1, 0))
        v = np.swapaxes(np.tensordot(Sy, np.swapaxes(v, 0, 1), (1, 0)), 0, 1)
        return np.tensordot(v, Sx, (2, 0))

    lam = c[0] * lx[None, None, :] + c[1] * ly[None, :, None] + c[2] * lz[:, None, None] + s
    x = transform(transform(b) / lam)
    if inner:
        x = np.pad(x, 1)
    return x.ravel()


def _cocg(A, diag, b, tol=1e-14, most=6000):
    """Conjugate gradients (unconjugated for complex-symmetric systems) with the
    diagonal as preconditioner, restarted from the true residual until that has
    reached `tol`, in torch's own sparse products."""
    x = torch.zeros_like(b)
    nb = float(torch.linalg.vector_norm(b))
    for _ in range(4):
        r = b - A(x)
        if float(torch.linalg.vector_norm(r)) <= tol * nb:
            break
        start = float(torch.linalg.vector_norm(r))
        z = r / diag
        p = z.clone()
        rho = (r * z).sum()
        for k in range(most):
            q = A(p)
            alpha = rho / (p * q).sum()
            x = x + alpha * p
            r = r - alpha * q
            if k % 20 == 19 and float(torch.linalg.vector_norm(r)) <= max(1e-7 * start, 0.3 * tol * nb):
                break
            z = r / diag
            new = (r * z).sum()
            p = z + (new / rho) * p
            rho = new
    return x


def _edge_exact(case, seed):
    K, M, _, m, fd = _edge_parts(case, seed)
    kind = case["kind"]
    cplx = kind in ("eddy", "batch")
    free = _on_gpu(fd.astype(np.float64))
    ip, ix = (_on_gpu(a.astype(np.int64)) for a in (K.indptr, K.indices))

    def csr(d):
        return torch.sparse_csr_tensor(ip, ix, _on_gpu(d), size=K.shape, device="cuda")

    Kd, Md = csr(K.data), csr(M.data)
    dk, dm = _on_gpu(K.diagonal()), _on_gpu(M.diagonal())

    def solve(b, w):
        if not cplx:
            A = csr(K.data + M.data)
            return _cocg(lambda v: free * (A @ v), dk + dm, b)

        def mult(v):
            u = torch.view_as_real(v).contiguous()
            k, s = Kd @ u, w * (Md @ u)
            return free * torch.complex(k[:, 0] - s[:, 1], k[:, 1] + s[:, 0])

        return _cocg(mult, torch.complex(dk, w * dm), b)

    if kind == "batch":
        b = _on_gpu(_edge_rhs(case, seed, m.ne, fd, True, (case["freqs"], case["nrhs"])))
        return torch.stack([torch.stack([solve(b[f, r], float(w)) for r in range(case["nrhs"])])
                            for f, w in enumerate(_omegas(case))])
    x = solve(_on_gpu(_edge_rhs(case, seed, m.ne, fd, cplx)), 1.0)
    return x if not case.get("host", True) else x.cpu().numpy()


def exact(case, seed):
    if case["kind"] in ("nodal", "gmres"):
        x = _nodal_exact(case, seed)
        return x if case.get("host", True) else torch.from_numpy(x)
    return _edge_exact(case, seed)
