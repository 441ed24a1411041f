"""GMRESSolver's fused Gram-Schmidt step at the edges of its blocks, and its work
vectors kept between calls: other restart lengths, both value types and two
threads on one matrix. The matrices are I + E with ||E|| <= 0.25, so the residual
that the Givens rotations report (below tol = 1e-11) is the true one to a few
hundred roundings: the bar is 2e-11 of ||b||."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _near_identity(n, cplx):
    rng = np.random.default_rng(n)
    d = [rng.uniform(-0.1, 0.1, max(n - k, 0)) for k in (1, 7)]
    A = sp.eye(n, format="csr") * 1.0
    for k, v in zip((1, 7), d):
        if len(v):
            A = A + sp.diags(v, k, shape=(n, n)) - sp.diags(0.1 * v, -k, shape=(n, n))
    A = sp.csr_matrix(A, dtype=np.complex128 if cplx else np.float64)
    if cplx:
        A.data = A.data * np.exp(0.3j)
    A.sort_indices()
    return A


def _rhs(n, cplx, seed):
    rng = np.random.default_rng(seed)
    b = rng.standard_normal(n)
    return b + 1j * rng.standard_normal(n) if cplx else b


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 4099, 300001])
def test_sizes_and_restarts(n, cplx):
    import sparsesolv_ngsolve as ss
    A = _near_identity(n, cplx)
    for seed, restart in enumerate((4, 9, 3)):
        b = _rhs(n, cplx, seed)
        x = ss.GMRESSolver(A, None, maxiter=200, tol=1e-11, restart=restart) * b
        assert np.linalg.norm(b - A @ x) <= 2e-11 * np.linalg.norm(b), (n, restart)


def test_two_threads_on_one_matrix():
    import ctypes

    import torch
    import sparsesolv_ngsolve as ss
    n = 20011
    A = _near_identity(n, False)
    inv = ss.GMRESSolver(A, None, maxiter=200, tol=1e-11, restart=5)
    inv * _rhs(n, False, 0)
    bs = [[torch.as_tensor(_rhs(n, False, 100 * t + k + 1), device="cuda") for k in range(10)] for t in range(2)]
    xs = [[torch.zeros_like(b) for b in row] for row in bs]
    torch.cuda.synchronize()
    codes = [[], []]

    def work(t):
        it = ctypes.c_int32(0)
        for b, x in zip(bs[t], xs[t]):
            codes[t].append(inv._lib.ssv_gmres_solve_dev(inv._mat.h, None, None, 200, 1e-11, 5, b.data_ptr(),
                                                         x.data_ptr(), ctypes.byref(it)))

    ts = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert codes == [[0] * 10] * 2
    for row, out in zip(bs, xs):
        for b, x in zip(row, out):
            b, x = b.cpu().numpy(), x.cpu().numpy()
            assert np.linalg.norm(b - A @ x) <= 2e-11 * np.linalg.norm(b)
