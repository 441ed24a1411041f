"""The give-up path of the one-launch triangular sweeps (csrc/sweep.cu). Every
wait inside them is bounded; with a limit of no tries at all
(ssv_set_sweep_wait(0)) each warp gives up at its first wait, the copies in
flight land, the kernel ends and the call returns SSV_ERR_TIMEOUT. Nothing
hangs, and the context and the handles stay usable."""
from __future__ import annotations

import numpy as np
import pytest

from sparsesolv_ngsolve import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture()
def no_tries():
    from sparsesolv_ngsolve import _capi
    lib = _capi.load()

    def limit(tries):
        lib.ssv_set_sweep_wait(tries)
    yield limit
    lib.ssv_set_sweep_wait(-1)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("method", ["ICCG", "SGSMRTR"])
def test_a_solve_whose_sweeps_give_up(no_tries, method, cplx):
    import sparsesolv_ngsolve as ss
    A = P.laplacian_7pt(12, 11, 13)
    if cplx:
        A = P.complex_shifted(A, 0.3j)
    b = P.random_rhs(A.shape[0], 0).astype(A.dtype)
    good = np.zeros_like(b)
    r0 = ss.SparseSolvSolver(A, method=method, maxiter=200).Solve(b, good)
    no_tries(0)
    with pytest.raises(RuntimeError):
        ss.SparseSolvSolver(A, method=method, maxiter=200).Solve(b, np.zeros_like(b))
    no_tries(-1)
    x = np.zeros_like(b)
    r = ss.SparseSolvSolver(A, method=method, maxiter=200).Solve(b, x)
    assert r.converged and r.iterations == r0.iterations
    assert np.abs(x - good).max() <= 1e-9 * np.abs(good).max()
