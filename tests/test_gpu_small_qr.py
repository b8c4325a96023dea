"""The small QR (small_qr.cu: at most eight unknowns and 64 entries of C(:, J),
eight lanes per column) against the oracle: every number of unknowns up to its
limit and beyond, row counts on both sides of 32 (its two launches), ranks that
fail, targets of several rows.  Tolerances per entry as for every fixed-pattern
column: 1e-8 in mixed mode, 1e-10 in FP64 (helpers.max_rel_diff)."""
import numpy as np
import pytest
import scipy.sparse as sp

import mspai_b200 as mb
from helpers import max_rel_diff, same_pattern
from mspai_b200 import workloads as W
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "mixed": 1e-8}


@pytest.fixture(scope="module")
def h():
    handle = mb.Handle(0)
    yield handle
    handle.close()


def check(h, A, P, prec, B=None, **kw):
    h.setup(A, P, B=B, options=mb.Options(ns=0, prec=prec, **kw))
    M = h.result()
    res, steps, status = h.column_info()
    o = O.spai_scalar(A, P, B=B, ns=0)
    assert same_pattern(M, o.M)
    assert np.all(steps == 1) and np.all(status == 0)
    assert max_rel_diff(M, o.M) < TOL[prec]
    assert np.allclose(res, o.res, rtol=1e-9, atol=1e-14)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("per_col", [1, 3, 6, 8])
def test_sizes(h, prec, per_col):
    """|J| 1 to 9 of columns with up to 9 entries: 1 to 72 rows."""
    n = 300
    rng = np.random.default_rng(per_col)
    rows = np.concatenate([rng.choice(n, per_col, replace=False) for _ in range(n)])
    A = sp.csc_matrix((rng.standard_normal(rows.size), (rows, np.repeat(np.arange(n), per_col))),
                      shape=(n, n)) + sp.diags(4.0 + rng.random(n))
    A = sp.csc_matrix(A)
    A.sort_indices()
    pr, pc = [], []
    for k in range(n):
        J = {k}
        while len(J) < 1 + k % 9:
            J.add(int(rng.integers(n)))
        pr += sorted(J)
        pc += [k] * len(J)
    check(h, A, sp.csc_matrix((np.ones(len(pr)), (pr, pc)), shape=(n, n)), prec)


@pytest.mark.parametrize("rho", [1.0, 100.0])
def test_probing_targets(h, rho):
    w = W.aniso2d_probing(17, kinds=("ones", "alt"), rho=rho)
    C, B = mb.assemble_probing(w.A, w.Ce, w.Be, rho)
    check(h, C, w.P, "mixed", B=B, probing=1, rho=rho)


def test_singular_and_unseen_columns(h):
    """A zero column in J (status 1: x = (Q^T b)(0:n)), more unknowns than rows,
    an empty column of P, a column that does not see its own row."""
    n = 40
    A = sp.lil_matrix(sp.identity(n) * 2.0)
    A[:, 3] = 0.0
    A = sp.csc_matrix(A)
    A = sp.csc_matrix((np.where(np.arange(n) == 3, 0.0, 2.0), np.arange(n), np.arange(n + 1)),
                      shape=(n, n))
    P = sp.lil_matrix((n, n))
    for k in range(n):
        P[[k, (k + 1) % n], k] = 1.0
    P[:, 10] = 0.0
    P[:, 20] = 0.0
    P[25, 20] = 1.0
    P = sp.csc_matrix(P)
    h.setup(A, P, options=mb.Options(ns=0, prec="fp64"))
    M = h.result()
    res, _, status = h.column_info()
    hit = np.array([3 in P.indices[P.indptr[k]:P.indptr[k + 1]] for k in range(n)])
    assert np.array_equal(status == 1, hit) and set(status) <= {0, 1}
    o = O.spai_scalar(A, P, ns=0)
    ok = ~hit
    for k in np.flatnonzero(ok):
        a, b = P.indptr[k], P.indptr[k + 1]
        assert np.array_equal(M.indices[M.indptr[k]:M.indptr[k + 1]], P.indices[a:b])
        ov = o.M[:, k].toarray().ravel()[P.indices[a:b]]
        assert np.allclose(M.data[M.indptr[k]:M.indptr[k + 1]], ov, rtol=1e-12, atol=1e-15)
    assert np.allclose(res[ok], o.res[ok], rtol=1e-12, atol=1e-15)
