"""The solvers on the sparse normal equations (fixed_cg.cu) against the oracle:
column sizes on and next to the limits of the launches (36: a warp per column;
144, 272 and 400: four warps), columns that the certificate or the data leave to
the dense factorizations, targets with several rows or outside of I, and
repeated setups.  Tolerances per entry as for every fixed-pattern column: 1e-8
in mixed mode, 1e-10 in FP64 (helpers.max_rel_diff)."""
import numpy as np
import pytest
import scipy.sparse as sp

import mspai_b200 as mb
from helpers import max_rel_diff, same_pattern
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "mixed": 1e-8}


@pytest.fixture(scope="module")
def h():
    handle = mb.Handle(0)
    yield handle
    handle.close()


def matrix(n, per_col, dominance, seed):
    """per_col random off-diagonal entries a column, diagonal `dominance` times
    their absolute sum."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.choice(n, per_col, replace=False) for _ in range(n)])
    cols = np.repeat(np.arange(n), per_col)
    A = sp.csc_matrix((rng.standard_normal(rows.size), (rows, cols)), shape=(n, n))
    A.setdiag(0.0)
    A.eliminate_zeros()
    A = sp.csc_matrix(A + sp.diags(dominance * np.asarray(abs(A).sum(axis=0)).ravel() + 0.1))
    A.sort_indices()
    return A


def pattern(n, sizes, seed, own=True):
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for k in range(n):
        J = {k} if own else set()
        while len(J) < sizes[k % len(sizes)]:
            j = int(rng.integers(n))
            if own or j != k:
                J.add(j)
        rows += sorted(J)
        cols += [k] * len(J)
    return sp.csc_matrix((np.ones(len(rows)), (rows, cols)), shape=(n, n))


def check(h, A, P, prec, B=None, **kw):
    h.setup(A, P, B=B, options=mb.Options(ns=0, prec=prec, **kw))
    M = h.result()
    res, _, status = h.column_info()
    o = O.spai_scalar(A, P, B=B, ns=0)
    assert np.all(status == 0)
    assert same_pattern(M, o.M)
    assert max_rel_diff(M, o.M) < TOL[prec]
    assert np.allclose(res, o.res, rtol=1e-9, atol=1e-13)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n,sizes", [(150, (1, 2, 17, 31, 32, 33, 36, 37)),
                                     (700, (143, 144, 145, 160)),
                                     (900, (271, 272, 273, 300, 400, 401))])
def test_sizes_at_the_limits(h, prec, n, sizes):
    A = matrix(n, 6, 3.0, seed=n)
    check(h, A, pattern(n, sizes, seed=n + 1), prec)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("dominance", [0.0, 0.3, 1.0])
def test_columns_without_certificate(h, prec, dominance):
    """Weak diagonals: the small columns are eliminated, of the others the
    certificate refuses some or all."""
    A = matrix(500, 8, dominance, seed=7)
    check(h, A, pattern(500, (20, 33, 60, 90), seed=8), prec)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_targets(h, prec):
    """Probing rows (a row that every column of J shares, several target rows),
    and columns that do not see their own row (b = 0 on I, or one entry)."""
    n = 400
    A = matrix(n, 5, 2.0, seed=3)
    P = pattern(n, (12, 30, 50), seed=4)
    E = np.ones((1, n))
    C, B = mb.assemble_probing(A, sp.csr_matrix(E @ A), sp.csr_matrix(E), 0.05)
    check(h, C, P, prec, B=B, probing=1, rho=0.05)
    check(h, A, pattern(n, (5, 18, 40), seed=5, own=False), prec)


@pytest.mark.parametrize("size", [20, 60])
def test_zero_column_values_and_repeats(h, size):
    """A column of C whose stored values are zero makes R singular (status 1);
    the other columns and repeated setups are unaffected, bit for bit."""
    n = 300
    A = matrix(n, 6, 3.0, seed=11)
    P = pattern(n, (size,), seed=12)
    h.setup(A, P, options=mb.Options(ns=0, prec="mixed"))
    M0 = h.result()
    h.setup(A, P, options=mb.Options(ns=0, prec="mixed"))
    assert np.array_equal(M0.data, h.result().data)
    Z = A.copy()
    Z.data[Z.indptr[5]:Z.indptr[6]] = 0.0
    h.setup(Z, P, options=mb.Options(ns=0, prec="mixed"))
    _, _, status = h.column_info()
    sees = np.array([5 in P.indices[P.indptr[k]:P.indptr[k + 1]] for k in range(n)])
    assert np.all(status[sees] == 1) and np.all(status[~sees] == 0)
    M1 = h.result()
    for k in np.flatnonzero(~sees):
        assert np.array_equal(M0.data[M0.indptr[k]:M0.indptr[k + 1]],
                              M1.data[M1.indptr[k]:M1.indptr[k + 1]])
