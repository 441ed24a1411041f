"""The colour-by-colour block sweeps of the ABMC form (csrc/block_sweep.cu) on
grids large enough to take them (small ones go through the one-launch sweeps):
every sub-warp width, blocks that do not fill it, rows with more entries than
are read ahead, the oversized leftover block, real and complex, both storage
forms. Solves have the oracle's iteration counts (one more or less in the FP32
form) and its solution to 1e-8."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _grid(cplx):
    from sparsesolv_ngsolve import problems
    A = problems.laplacian_7pt(43, 41, 37)
    return problems.complex_shifted(A, 0.05 + 0.3j) if cplx else A


def _edge():
    from sparsesolv_ngsolve import hcurl as H
    m = H.kuhn_mesh(18)
    Ke, Me = H.element_matrices(m)
    return H.assemble(m, np.ones(m.tets.shape[0]), Ke + 4.0 * Me)


def _solve(A, bs, colors=4, precision="fp64"):
    import sparsesolv_ngsolve as ss
    from oracle import oracle as O
    from sparsesolv_ngsolve import _capi
    n = A.shape[0]
    rng = np.random.default_rng(n + bs)
    b = rng.uniform(-1, 1, n) + (1j * rng.uniform(-1, 1, n) if np.iscomplexobj(A.data) else 0.0)
    s = ss.SparseSolvSolver(A, method="ICCG", use_abmc=True, abmc_block_size=bs, abmc_num_colors=colors, maxiter=600)
    s.precision = precision
    x = np.zeros(n, dtype=A.dtype)
    r = s.Solve(b, x)
    prof = _capi.ssv_phase_profile()
    _capi.check(_capi.load().ssv_solver_profile(s._h, b"ICCG", ctypes.byref(s._cfg), 1, ctypes.byref(prof)))
    assert {q["name"]: q["kernels"] for q in prof.as_list()}["ic_backward"] > 1  # the block path
    xo, ro, _ = O.solve(A, b, "ICCG", O.default_config(use_abmc=1, abmc_block_size=bs, abmc_num_colors=colors,
                                                       max_iterations=600))
    assert r.converged and abs(r.iterations - ro.iterations) <= (1 if precision == "fp32" else 0)
    assert np.abs(x - xo).max() <= 1e-8 * np.abs(xo).max()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("bs", [1, 2, 3, 4, 7, 16, 32])
def test_block_widths(bs, cplx):
    _solve(_grid(cplx), bs)


@pytest.mark.parametrize("cplx", [False, True])
def test_fp32_storage(cplx):
    _solve(_grid(cplx), 4, precision="fp32")


def test_long_rows():
    _solve(_edge(), 4)
