"""Column-split products of blocks of columns at odd sizes: the AMS cycle of four
real or complex columns against the cycle of each column alone, and the batch's
product of 1 to 4 frequencies with 1 or 4 right-hand sides against single solves.
A cycle is some twenty products of rows of at most a few hundred entries, so two
summation orders differ by a few thousand roundings at most: the bar is 1e-12 of
the largest entry in FP64 and 1e-3 in the FP32 form. Five unpreconditioned COCR
steps amplify a rounding by the condition of their small Krylov space: 1e-9."""
from __future__ import annotations

import numpy as np
import pytest

from sparsesolv_ngsolve import hcurl as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-12), ("fp32", 1e-3)])
@pytest.mark.parametrize("nc", [2, 3, 7, 13])
@pytest.mark.parametrize("cplx", [False, True])
def test_cycle_of_four_columns(cplx, nc, precision, bar):
    import sparsesolv_ngsolve as ss
    rng = np.random.default_rng(nc)
    if cplx:
        d = H.eddy_current(nc, freq=1e3, nu_r_core=0.1, mass_eps=1.0)
        cls, A = ss.ComplexCompactAMSPreconditioner, d["a_real"]
    else:
        d = H.magnetostatic(nc, nu_iron=1.0, mass_eps=1.0)
        cls, A = ss.CompactAMSPreconditioner, d["A"]
    p = cls(A, d["G"], freedofs=d["freedofs"], coord_x=d["coords"][0], coord_y=d["coords"][1],
            coord_z=d["coords"][2], precision=precision)
    n = A.shape[0]
    X = rng.standard_normal((4, n)) + (1j * rng.standard_normal((4, n)) if cplx else 0.0)
    Y = p.MultBlock(X)
    for r in range(4):
        y = p.MultBlock(X[r:r + 1])[0]
        assert np.abs(Y[r] - y).max() <= bar * np.abs(y).max(), r


@pytest.mark.parametrize("nrhs", [1, 4])
@pytest.mark.parametrize("F", [1, 2, 3, 4])
def test_batch_product(F, nrhs):
    import sparsesolv_ngsolve as ss
    d = H.eddy_family(5, freqs=[1e2 * 4 ** k for k in range(F)], nrhs=4, nu_r_core=0.1, mass_eps=1.0)
    B = d["B"][:, :nrhs].copy()
    X = ss.BatchedCOCRSolver(d["K"], d["M"], d["omegas"], [None] * F, nrhs=nrhs, freedofs=d["freedofs"], maxiter=5,
                             tol=1e-14).Solve(B)
    for f in range(F):
        for r in range(nrhs):
            x = ss.COCRSolver(d["A"][f], None, freedofs=d["freedofs"], maxiter=5, tol=1e-14) * B[f, r]
            assert np.linalg.norm(X[f, r] - x) <= 1e-9 * np.linalg.norm(x), (f, r)
