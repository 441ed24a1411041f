"""The device set-up's numeric products where a row of the product has more columns than are
summed in shared memory (256 in k_prod_num, csrc/amg_device.cu): one edge coupled to 400 others
makes such rows in the Galerkin products of all four subspaces. Every level matrix equals the
oracle's bit for bit, as in the ordinary case."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O
from sparsesolv_ngsolve import hcurl as H

pytestmark = pytest.mark.gpu


def _with_hub(A, free, seed):
    rng = np.random.default_rng(seed)
    inner = np.flatnonzero(free)
    hub = inner[inner.size // 2]
    to = rng.choice(np.setdiff1d(inner, [hub]), 400, replace=False)
    v = rng.uniform(-1.0, 1.0, to.size) * 1e-3 * abs(A.diagonal()).max()
    C = sp.coo_matrix((v, (np.full(to.size, hub), to)), shape=A.shape)
    B = (A + C + C.T + sp.diags(np.asarray(abs(C + C.T).sum(axis=1)).ravel())).tocsr()
    B.sum_duplicates()
    B.sort_indices()
    B.indptr, B.indices = B.indptr.astype(np.int32), B.indices.astype(np.int32)
    return B


@pytest.mark.parametrize("seed", [1, 2])
def test_long_rows_equal_the_oracle_bitwise(seed):
    import sparsesolv_ngsolve as ss
    d = H.magnetostatic(8, nu_iron=1.0, mass_eps=1.0)
    A = _with_hub(d["A"], d["freedofs"], seed)
    o = O.AmsOracle(A, d["G"], d["freedofs"], *d["coords"])
    longest = [max(int(np.diff(o.level_matrix(s, l, 0).indptr).max()) for l in range(len(o.levels(s)))) for s in range(4)]
    assert min(longest) > 256, longest
    p = ss.CompactAMSPreconditioner(A, d["G"], freedofs=d["freedofs"], coord_x=d["coords"][0],
                                    coord_y=d["coords"][1], coord_z=d["coords"][2])
    for s in range(4):
        assert p.levels(s) == o.levels(s)
        for l in range(len(o.levels(s))):
            for what in (0, 1) if l + 1 < len(o.levels(s)) else (0,):
                M, Mo = p.level_matrix(s, l, what), o.level_matrix(s, l, what)
                assert p.on_device
                assert np.array_equal(M.indptr, Mo.indptr) and np.array_equal(M.indices, Mo.indices)
                assert np.array_equal(M.data, Mo.data), (s, l, what)
