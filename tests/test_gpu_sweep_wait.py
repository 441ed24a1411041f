"""The give-up path of the one-launch triangular sweeps (csrc/sweep.cu). Every
wait inside them is bounded; after ssv_set_sweep_wait(0) each warp counts its
waits as given up from the start, the kernel ends and the call returns
SSV_ERR_TIMEOUT. Nothing hangs, and the context and the handles stay usable."""
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


def _systems():
    A = P.laplacian_7pt(12, 11, 13)
    return A, P.random_rhs(A.shape[0], 0)


def _solver(kind, A):
    import sparsesolv_ngsolve as ss
    if kind in ("ICCG", "SGSMRTR"):
        s = ss.SparseSolvSolver(A, method=kind, maxiter=200)
        return lambda b: s * b
    pre = ss.SGSPreconditioner(A) if kind.endswith("SGS") else ss.ICPreconditioner(A)
    if "*" not in kind:
        return lambda b: pre * b
    s = {"PCG": ss.PCGSolver, "COCR": ss.COCRSolver, "GMRES": ss.GMRESSolver}[kind.split("*")[0]](
        A, pre, maxiter=200, tol=1e-10)
    return lambda b: s * b


@pytest.mark.parametrize("kind", ["ICCG", "SGSMRTR", "IC", "SGS", "PCG*IC", "PCG*SGS", "COCR*IC", "COCR*SGS",
                                  "GMRES*IC", "GMRES*SGS"])
def test_a_report_is_not_raised_by_a_later_call(no_tries, kind):
    """The call that gave up reports it; the same handle's next calls are right and say so."""
    A, b = _systems()
    call = _solver(kind, A)
    good = np.array(call(b))
    no_tries(0)
    with pytest.raises(RuntimeError):
        call(b)
    no_tries(-1)
    for _ in range(2):
        assert np.abs(np.array(call(b)) - good).max() <= 1e-9 * np.abs(good).max()
