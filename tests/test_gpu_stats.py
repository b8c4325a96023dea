"""Statistics of the last setup (Handle.stats): the same before and after other
calls on the handle."""
import numpy as np
import pytest
import scipy.sparse as sp

import mspai_b200 as mb

pytestmark = pytest.mark.gpu


def problem(n, sizes, seed):
    """Diagonally dominant columns of 12 entries; patterns of the given sizes."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.choice(n, 12, replace=False) for _ in range(n)])
    A = sp.csc_matrix((rng.standard_normal(rows.size), (rows, np.repeat(np.arange(n), 12))),
                      shape=(n, n))
    A = sp.csc_matrix(A + sp.diags(2.0 * np.asarray(abs(A).sum(axis=0)).ravel()))
    A.sort_indices()
    J = [np.sort(np.append(rng.choice(np.delete(np.arange(n), k), sizes[k % len(sizes)] - 1,
                                      replace=False), k)) for k in range(n)]
    P = sp.csc_matrix((np.ones(sum(map(len, J))), np.concatenate(J),
                       np.concatenate([[0], np.cumsum([len(j) for j in J])])), shape=(n, n))
    return A, P


@pytest.mark.parametrize("sizes", [(4, 9, 30, 60, 150), (30, 60), (3, 450)])
@pytest.mark.parametrize("gbar", [False, True])
def test_an_adjoint_leaves_the_statistics(sizes, gbar):
    n = 700
    A, P = problem(n, sizes, seed=len(sizes))
    h = mb.Handle(0)
    h.setup(A, P, options=mb.Options(ns=0, prec="mixed"))
    before, columns = h.stats(), h.solver_columns()
    # every column belongs to one bucket
    assert sum(before["bucket_flops"]) == pytest.approx(before["flops"], rel=1e-12)
    h.adjoint(A, None, gbar=np.ones(P.nnz) if gbar else None)
    after = h.stats()
    assert np.allclose(after["bucket_flops"], before["bucket_flops"], rtol=1e-12)
    assert after["bucket_columns"] == before["bucket_columns"]
    assert h.solver_columns() == columns
    h.close()
