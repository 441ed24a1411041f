"""The rows that the ABMC aggregation leaves over (csrc/block_sweep.cu) when one of them is
long: rows without couplings use up the blocks, so a whole arrow matrix is left over, its hub
coupled to every other row. Padding all rows to the longest one took 12 bytes for every pair
of rows. Solves have the oracle's iterations (one more or less: the hub's sum runs over
hundreds of terms in another order) and its solution to 1e-8."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _arrow(alone, rows, hub_last, cplx):
    """`alone` uncoupled rows, then `rows` in chains of five, each coupled to the hub."""
    n = alone + rows
    rng = np.random.default_rng(rows)
    hub = n - 1 if hub_last else alone
    others = np.setdiff1d(np.arange(alone, n), [hub])
    chain = others[1:][np.arange(1, others.size) % 5 != 0]
    i = np.concatenate([others, chain])
    j = np.concatenate([np.full(others.size, hub), chain - 1])
    keep = (j != hub) | (np.arange(i.size) < others.size)
    i, j = i[keep], j[keep]
    v = -rng.uniform(0.1, 1.0, i.size)
    A = sp.coo_matrix((v, (i, j)), shape=(n, n))
    A = (A + A.T).tocsr()
    d = 1.5 * np.asarray(abs(A).sum(axis=1)).ravel() + rng.uniform(0.5, 1.0, n)
    A = (A.astype(np.complex128 if cplx else np.float64) + sp.diags(d * (1.0 + 0.3j if cplx else 1.0))).tocsr()
    A.sort_indices()
    return A


def _solve(A, precision):
    import sparsesolv_ngsolve as ss
    from oracle import oracle as O
    n = A.shape[0]
    b = np.random.default_rng(n).uniform(-1, 1, n).astype(A.dtype)
    s = ss.SparseSolvSolver(A, method="ICCG", use_abmc=True, maxiter=200)
    s.precision = precision
    x = np.zeros(n, dtype=A.dtype)
    r = s.Solve(b, x)
    xo, ro, _ = O.solve(A, b, "ICCG", O.default_config(use_abmc=1, max_iterations=200))
    assert r.converged and abs(r.iterations - ro.iterations) <= 1
    assert np.abs(x - xo).max() <= 1e-8 * np.abs(xo).max()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("hub_last", [False, True])
@pytest.mark.parametrize("rows", [2, 40, 1500])
def test_a_long_row_among_the_rows_left_over(rows, hub_last, cplx, precision):
    _solve(_arrow(max(2, rows // 2), rows, hub_last, cplx), precision)


@pytest.mark.parametrize("hub_last", [False, True])
def test_rows_left_over_past_the_shared_memory_take_their_own_size(hub_last):
    """12,000 rows left over with a hub of 8000 entries: nothing near 96 million entries."""
    from sparsesolv_ngsolve import _capi
    A = _arrow(8000, 8000, hub_last, False)
    lib = _capi.load()
    lib.ssv_set_alloc_budget(64 << 20)
    try:
        _solve(A, "fp64")
    finally:
        lib.ssv_set_alloc_budget(-1)
