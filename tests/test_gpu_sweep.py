"""The one-launch triangular sweeps (csrc/sweep.cu) where they can go wrong:
partial slices, rows longer than the entries held in registers, more levels than
one chunk holds, levels too narrow and wide enough for several rounds of a
cluster of 16. SGSPreconditioner applies are compared with scipy's triangular
solves; the matrices are diagonally dominant with ratio 2 or more, so the sweeps
do not amplify and the bar of 1e-13 of the largest entry is some 1e3 roundings.
Solves through the IC and MRTR forms of the sweeps are compared with the oracle
(same iterations, 1e-8)."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import spsolve_triangular

pytestmark = pytest.mark.gpu


def _dominant(P, seed, cplx):
    """Symmetric values on the symmetric pattern P, diagonal twice the row's sum."""
    rng = np.random.default_rng(seed)
    U = sp.triu(P, 1).tocsr()
    U.data = -rng.uniform(0.1, 1.0, U.nnz)
    if cplx:
        U = U.astype(np.complex128)
        U.data = U.data * np.exp(1j * rng.uniform(-0.5, 0.5, U.nnz))
    A = (U + U.T).tocsr()
    d = 2.0 * np.asarray(abs(A).sum(axis=1)).ravel() + rng.uniform(0.5, 1.0, P.shape[0])
    A = (A + sp.diags(d * (1.0 + 0.2j if cplx else 1.0))).tocsr()
    A.sort_indices()
    return A


def _band(n, hb):
    return sp.diags([np.ones(n - abs(k)) for k in range(-hb, hb + 1)], list(range(-hb, hb + 1))).tocsr()


def _grid(nx, ny, nz):
    from sparsesolv_ngsolve import problems
    return problems.laplacian_7pt(nx, ny, nz)


def _scattered(n, m, seed):
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), m)
    j = rng.integers(0, n, n * m)
    P = sp.coo_matrix((np.ones(n * m), (i, j)), shape=(n, n)).tocsr()
    return (P + P.T + sp.identity(n)).tocsr()


PATTERNS = {
    "1": lambda: _band(1, 0), "31 band 1": lambda: _band(31, 1), "33 diagonal": lambda: _band(33, 0),
    "1300 levels": lambda: _band(1300, 1), "700 band 19": lambda: _band(700, 19),
    "grid 17x5x3": lambda: _grid(17, 5, 3), "grid 45x47x49": lambda: _grid(45, 47, 49),
    "scattered 3000x6": lambda: _scattered(3000, 6, 1), "scattered 20000x2": lambda: _scattered(20000, 2, 2),
}


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("name", list(PATTERNS))
def test_sgs_apply_equals_triangular_solves(name, cplx):
    import sparsesolv_ngsolve as ss
    A = _dominant(PATTERNS[name](), 3, cplx)
    n = A.shape[0]
    x = np.random.default_rng(5).uniform(-1, 1, n) + (0.5j if cplx else 0.0)
    t = spsolve_triangular(sp.tril(A).tocsr(), x, lower=True)
    ref = spsolve_triangular(sp.triu(A).tocsr(), A.diagonal() * t, lower=False)
    y = ss.SGSPreconditioner(A) * x
    assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("method", ["ICCG", "SGSMRTR"])
@pytest.mark.parametrize("name", ["31 band 1", "1300 levels", "700 band 19", "grid 45x47x49", "scattered 3000x6"])
def test_solves_through_the_sweeps(name, method, precision):
    import sparsesolv_ngsolve as ss
    from oracle import oracle as O
    if method == "SGSMRTR" and precision == "fp32":
        pytest.skip("the FP32 form is the IC preconditioner's")
    A = _dominant(PATTERNS[name](), 4, False)
    b = np.random.default_rng(6).uniform(-1, 1, A.shape[0])
    s = ss.SparseSolvSolver(A, method=method, maxiter=300)
    s.precision = precision
    x = np.zeros(A.shape[0])
    r = s.Solve(b, x)
    xo, ro, _ = O.solve(A, b, method, O.default_config(max_iterations=300))
    assert r.converged and abs(r.iterations - ro.iterations) <= (1 if precision == "fp32" else 0)
    assert np.abs(x - xo).max() <= 1e-8 * np.abs(xo).max()


def test_matrix_values_changed_without_update():
    """Without a FreeDofs mask the sweeps use the matrix's current off-diagonals and
    the diagonal of the last Update()."""
    import sparsesolv_ngsolve as ss
    from sparsesolv_ngsolve import _capi
    A = _dominant(_grid(9, 8, 7), 7, False)
    p = ss.SGSPreconditioner(A)
    x = np.random.default_rng(8).uniform(-1, 1, A.shape[0])
    p * x
    B = A.copy()
    off = B.indices != np.repeat(np.arange(B.shape[0]), np.diff(B.indptr))
    B.data[off] *= 0.5
    _capi.check(_capi.load().ssv_matrix_update_values(p._mat.h, _capi.vptr(B.data)))
    y = p * x
    t = spsolve_triangular(sp.tril(B).tocsr(), x, lower=True)
    ref = spsolve_triangular(sp.triu(B).tocsr(), B.diagonal() * t, lower=False)
    assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()
