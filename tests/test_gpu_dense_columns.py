"""The dense factorizations of fixed patterns (fixed_solve.cuh) on columns that do
come to them, which Handle.solver_columns shows: setups that keep the factors, and
columns without a certificate (weak diagonal) for the sparse solvers.  Column
sizes on both sides of the Cholesky's blocks of 16; re-setups and the adjoint's
gbar term that start from the kept R.  Tolerances per entry as for every
fixed-pattern column: 1e-8 in mixed mode, 1e-10 in FP64 (helpers.max_rel_diff)."""
import numpy as np
import pytest
import scipy.sparse as sp

import mspai_b200 as mb
from helpers import max_rel_diff, same_pattern
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "mixed": 1e-8}
SIZES = (17, 31, 32, 33, 47, 48, 49, 64, 65, 96, 97)


@pytest.fixture
def h():
    handle = mb.Handle(0)
    yield handle
    handle.close()


def problem(n, dominance, seed, sizes=SIZES):
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.choice(n, 10, replace=False) for _ in range(n)])
    A = sp.csc_matrix((rng.standard_normal(rows.size), (rows, np.repeat(np.arange(n), 10))),
                      shape=(n, n))
    A.setdiag(0.0)
    A.eliminate_zeros()
    A = sp.csc_matrix(A + sp.diags(dominance * np.asarray(abs(A).sum(axis=0)).ravel() + 0.1))
    A.sort_indices()
    J = [np.sort(np.append(rng.choice(np.delete(np.arange(n), k), sizes[k % len(sizes)] - 1,
                                      replace=False), k)) for k in range(n)]
    P = sp.csc_matrix((np.ones(sum(map(len, J))), np.concatenate(J),
                       np.concatenate([[0], np.cumsum([len(j) for j in J])])), shape=(n, n))
    return A, P


def check(h, A, P, prec):
    M = h.result()
    _, _, status = h.column_info()
    o = O.spai_scalar(A, P, ns=0)
    assert np.all(status == 0)
    assert same_pattern(M, o.M)
    assert max_rel_diff(M, o.M) < TOL[prec]


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("dominance,keep", [(1.5, True), (0.2, True), (0.2, False)])
def test_block_boundaries(h, prec, dominance, keep):
    n = 260
    A, P = problem(n, dominance, seed=21, sizes=SIZES if keep else SIZES[6:])
    h.setup(A, P, options=mb.Options(ns=0, prec=prec, keep_factors=keep))
    assert h.solver_columns()["fixed"] > 0.95 * n
    check(h, A, P, prec)


def test_fallback_of_nearly_parallel_columns(h):
    """C^T C is not positive definite to FP32 (kappa 1e4): the Householder QR."""
    n = 260
    A, P = problem(n, 1.5, seed=22)
    A = A.tolil()
    c = A[:, 0].toarray().ravel()
    c[np.flatnonzero(c)[0]] *= 1.0 + 1e-3
    A[:, 1] = c.reshape(-1, 1)
    A = sp.csc_matrix(A)
    A.sort_indices()
    P = P.tolil()
    P[:2, 2::9] = 1.0
    P = sp.csc_matrix(P)
    P.sort_indices()
    h.setup(A, P, options=mb.Options(ns=0, prec="mixed", keep_factors=True))
    assert h.solver_columns()["fixed"] == n
    check(h, A, P, "mixed")


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_resetup_and_gradient_from_the_kept_factors(h, prec):
    n = 300
    A, P = problem(n, 0.2, seed=23, sizes=(49, 64, 97))
    h.setup(A, P, options=mb.Options(ns=0, prec=prec, keep_factors=True))
    rng = np.random.default_rng(24)
    again = mb.Options(ns=0, prec=prec, keep_factors=True, reuse_factors=8)
    gbar = rng.standard_normal(P.nnz)
    for _ in range(2):
        A.data *= 1.0 + 1e-5 * rng.standard_normal(A.nnz)
        h.setup(A, P, options=again)
        assert h.solver_columns()["fixed"] > 0.95 * n
        assert h.stats()["factor_reuse_columns"] > 0.9 * n
        check(h, A, P, prec)
        kept = h.adjoint(A, None, gbar=gbar)
        other = mb.Handle(0)
        other.setup(A, P, options=mb.Options(ns=0, prec="fp64"))
        ref = other.adjoint(A, None, gbar=gbar)
        other.close()
        assert np.max(np.abs(kept[0] - ref[0])) <= TOL[prec] * np.max(np.abs(ref[0]))
        assert abs(kept[2] - ref[2]) <= TOL[prec] * abs(ref[2])
