"""What becomes of the columns that a solver does not take: which solvers they
come to (Handle.solver_columns), and their values against the oracle or a dense
computation in numpy.  Tolerances per entry as for every column: 1e-8 in mixed
mode, 1e-10 in FP64 (helpers.max_rel_diff)."""
import numpy as np
import pytest
import scipy.sparse as sp

import mspai_b200 as mb
from helpers import max_rel_diff, same_pattern
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "mixed": 1e-8}
SPARSE = ("sparse_25k", "sparse_42k", "sparse_104k")


@pytest.fixture
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


def pattern(n, sizes, seed):
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for k in range(n):
        s = sizes[k % len(sizes)]
        J = np.sort(np.append(rng.choice(np.delete(np.arange(n), k), s - 1, replace=False), k))
        rows += J.tolist()
        cols += [k] * s
    return sp.csc_matrix((np.ones(len(rows)), (rows, cols)), shape=(n, n))


def column(M, k):
    return M.indices[M.indptr[k]:M.indptr[k + 1]]


def spectral_radius(A, J):
    """Of D^-1/2 |G - D| D^-1/2, G = A_J^T A_J: no certificate above 0.9."""
    X = np.abs(A[:, J].toarray())
    X /= np.sqrt((X ** 2).sum(axis=0))
    return np.linalg.eigvalsh(X.T @ X)[-1] - 1.0


def check(h, A, P, prec):
    M = h.result()
    res, _, status = h.column_info()
    o = O.spai_scalar(A, P, ns=0)
    assert np.all(status == 0)
    assert same_pattern(M, o.M)
    assert max_rel_diff(M, o.M) < TOL[prec]
    assert np.allclose(res, o.res, rtol=1e-9, atol=1e-13)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_no_certificate_means_the_dense_solver_at_once(h, prec):
    n = 250
    A = matrix(n, 10, 0.2, seed=2)
    P = pattern(n, (40, 55), seed=3)
    for k in range(n):
        assert spectral_radius(A, column(P, k)) > 0.95
    for _ in range(2):
        h.setup(A, P, options=mb.Options(ns=0, prec=prec))
        c = h.solver_columns()
        assert [c[s] for s in SPARSE] == [n, 0, 0]
        assert c["fixed"] == n
    check(h, A, P, prec)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_only_columns_that_do_not_fit_go_to_the_next_slot(h, prec):
    """Certified columns of up to 144, 272 and 400 unknowns, and larger ones:
    those fit no slot."""
    n, sizes = 1200, (60, 120, 200, 380, 410)
    A = matrix(n, 3, 30.0, seed=4)
    P = pattern(n, sizes, seed=5)
    h.setup(A, P, options=mb.Options(ns=0, prec=prec))
    c = h.solver_columns()
    assert [c[s] for s in SPARSE] == [n, 2 * n // 5, n // 5]
    assert c["fixed"] == n // 5
    check(h, A, P, prec)
    M0 = h.result()
    h.setup(A, P, options=mb.Options(ns=0, prec=prec))
    assert np.array_equal(M0.data, h.result().data)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("keep", [False, True])
def test_gradient_of_columns_without_certificate(h, prec, keep):
    """gbar . M at columns that the adjoint's iteration refuses (with and without
    a kept factor), and at certified ones, against lambda from numpy."""
    n = 200
    A = matrix(n, 6, 0.8, seed=6)
    P = pattern(n, (40, 60), seed=7)
    rho = np.array([spectral_radius(A, column(P, k)) for k in range(n)])
    assert np.any(rho > 0.95) and np.any(rho < 0.8)
    gbar = np.random.default_rng(8).standard_normal(P.nnz)
    h.setup(A, P, options=mb.Options(ns=0, prec=prec, keep_factors=keep))
    dC, _, loss = h.adjoint(A, None, gbar=gbar, residual_weight=0.0)
    D = A.toarray()
    g = np.zeros_like(D)
    value = 0.0
    for k in range(n):
        J = column(P, k)
        gb = gbar[P.indptr[k]:P.indptr[k + 1]]
        CJ = D[:, J]
        e = np.zeros(n)
        e[k] = 1.0
        m = np.linalg.lstsq(CJ, e, rcond=None)[0]
        lam = np.linalg.solve(CJ.T @ CJ, gb)
        g[:, J] += np.outer(e - CJ @ m, lam) - np.outer(CJ @ lam, m)
        value += gb @ m
    ref = g[A.indices, np.repeat(np.arange(n), np.diff(A.indptr))]
    assert np.max(np.abs(dC - ref)) <= TOL[prec] * np.max(np.abs(ref))
    assert abs(loss - value) <= TOL[prec] * np.sqrt(n) * abs(value)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_resetup_far_from_the_previous_values(h, prec):
    """Certified columns whose values have changed too much for a start from the
    previous solution start from zero: no dense factorization, none reused."""
    n = 500
    A = matrix(n, 5, 2.0, seed=9)
    P = pattern(n, (40, 90), seed=10)
    h.setup(A, P, options=mb.Options(ns=0, prec=prec, keep_factors=True))
    assert h.solver_columns()["fixed"] == n  # the factors are made here
    again = mb.Options(ns=0, prec=prec, keep_factors=True, reuse_factors=4)
    rng = np.random.default_rng(11)
    far = A.copy()
    far.data = A.data * np.where(rng.random(A.nnz) < 0.5, -1.0, 1.5)
    near = far.copy()
    near.data = far.data * (1.0 + 1e-5 * rng.standard_normal(A.nnz))
    for k in range(n):
        assert max(spectral_radius(M, column(P, k)) for M in (far, near)) < 0.8
    h.setup(far, P, options=again)
    c = h.solver_columns()
    assert sum(c[s] for s in SPARSE) >= n and c["fixed"] == 0
    assert h.stats()["factor_reuse_columns"] == 0
    check(h, far, P, prec)
    h.setup(near, P, options=again)  # from the solution made from zero
    assert h.solver_columns()["fixed"] == 0
    assert h.stats()["factor_reuse_columns"] == n
    check(h, near, P, prec)


def block_problem(nb, bs, blocks, seed, diag=6.0):
    """Random block matrix, four block entries a block column, and a block pattern
    of `blocks` blocks a column."""
    rng = np.random.default_rng(seed)
    J = lambda m: [sorted({k} | set(rng.choice(np.delete(np.arange(nb), k), m - 1,
                                               replace=False).tolist())) for k in range(nb)]
    A = np.zeros((bs * nb, bs * nb))
    for k, rows in enumerate(J(4)):
        for b in rows:
            A[bs * b:bs * b + bs, bs * k:bs * k + bs] = rng.standard_normal((bs, bs))
    A = sp.csc_matrix(A + diag * np.eye(bs * nb))
    A.sort_indices()
    rows = J(blocks)
    P = sp.csc_matrix((np.ones(blocks * nb), np.concatenate(rows),
                       np.arange(nb + 1) * blocks), shape=(nb, nb))
    return A, P


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("bs,blocks,solver", [(3, 1, "block_small"), (3, 4, "block_64"),
                                              (2, 20, "block_256")])
def test_block_columns_above_the_tolerance(h, prec, bs, blocks, solver):
    """A block column that is solved at its start pattern and needs an update comes
    to no other solver of the start pattern."""
    nb = 60
    A, P = block_problem(nb, bs, blocks, seed=blocks)
    h.setup(A, P, options=mb.Options(ns=1, mn=2, ep=1e-3, bs=bs, prec=prec))
    c = h.solver_columns()
    after = {"block_small": ("block_64", "block_256"), "block_64": ("block_256",),
             "block_256": ()}[solver]
    assert c[solver] == nb and c["general"] == nb
    assert all(c[s] == 0 for s in after)
    o = O.spai_block(A, P, bs, ns=1, mn=2, ep=1e-3)
    M = h.result()
    assert same_pattern(M, o.M)
    assert max_rel_diff(M, o.M) < TOL[prec]



@pytest.mark.parametrize("prec,powers", [("fp64", range(507, 513)), ("mixed", range(58, 64))])
@pytest.mark.parametrize("bs,blocks,keep", [(3, 1, False), (3, 4, False), (3, 14, False),
                                            (1, 50, True)])
def test_normal_matrix_that_overflows(h, prec, powers, bs, blocks, keep):
    """C times powers of two around the one where the squares overflow (FP64, or
    the FP32 of the mixed mode's larger columns): a column is flagged, or it is M
    times the inverse power."""
    nb = 60
    if bs > 1:
        A, P = block_problem(nb, bs, blocks, seed=blocks)
    else:
        A, P = matrix(nb * 3, 6, 3.0, seed=1), pattern(nb * 3, (blocks,), seed=2)
    o = mb.Options(ns=0, bs=bs, prec=prec, keep_factors=keep)
    h.setup(A, P, options=o)
    M0 = h.result()
    S = A.copy()
    for power in powers:
        S.data = np.ldexp(A.data, power)
        h.setup(S, P, options=o)
        M = h.result()
        _, _, status = h.column_info()
        assert same_pattern(M, M0)
        for k in np.flatnonzero(status == 0):
            a, b = M0.indptr[k], M0.indptr[k + 1]
            assert np.allclose(np.ldexp(M.data[a:b], power), M0.data[a:b], rtol=0,
                               atol=TOL[prec] * np.max(np.abs(M0.data[a:b])))


def scattered_blocks(nb, bs, per_col, blocks, seed):
    """Columns of per_col random entries and a strong diagonal, a random block
    pattern: nearly every row of C(:, J) has one entry."""
    rng = np.random.default_rng(seed)
    n = nb * bs
    A = matrix(n, per_col, 0.0, seed) + 3.0 * np.sqrt(per_col) * sp.identity(n)
    A = sp.csc_matrix(A)
    A.sort_indices()
    rows = [np.sort(np.append(rng.choice(np.delete(np.arange(nb), k), blocks - 1, replace=False),
                              k)) for k in range(nb)]
    P = sp.csc_matrix((np.ones(nb * blocks), np.concatenate(rows), np.arange(nb + 1) * blocks),
                      shape=(nb, nb))
    return A, P


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("bs,per_col,blocks", [(2, 25, 20), (2, 27, 20),  # 1,024 entries, more
                                               (2, 60, 20), (2, 100, 50), (3, 40, 8)])
def test_block_columns_of_more_rows_than_the_arena_holds(h, prec, bs, per_col, blocks):
    nb = 1500
    A, P = scattered_blocks(nb, bs, per_col, blocks, seed=per_col)
    cols = np.arange(0, nb, nb // 12)
    h.setup(A, P, options=mb.Options(ns=0, bs=bs, prec=prec))
    M = h.result()
    D = A.toarray()
    for k in cols:
        J = (bs * column(P, k)[:, None] + np.arange(bs)).ravel()
        x = np.linalg.lstsq(D[:, J], np.eye(nb * bs)[:, bs * k:bs * k + bs], rcond=None)[0]
        got = M[:, bs * k:bs * k + bs].toarray()
        assert np.allclose(got[J], x, rtol=0, atol=TOL[prec] * np.max(np.abs(x)))


def test_block_columns_of_many_rows_are_given_up_early(h):
    """A column with far more rows than the arena holds costs little beside its
    solution by the general solver (a setup without refinement uses that alone):
    before its row table stopped at the first row too many it took 4.5 times that."""
    A, P = scattered_blocks(4000, 2, 60, 20, seed=9)
    ms = {}
    for refine in (0, 4):
        o = mb.Options(ns=0, bs=2, prec="mixed", refine=refine)
        h.setup(A, P, options=o)
        h.setup(A, P, options=o)
        ms[refine] = h.stats()["setup_ms"]
    assert h.solver_columns()["general"] == 4000
    assert ms[4] < 2.0 * ms[0]


def test_small_block_columns_beside_large_ones_in_fp64(h):
    """Mixed mode solves a bucket of at most 32 unknowns a column in FP64, whatever
    the other bucket holds: nearly dependent columns (a relative 1e-8) that the
    normal equations refuse, 18 unknowns, beside columns of 120.  The residual of
    a backward stable solution is the smallest one up to 1e-16 times a modest
    factor, the FP32 factor's is not."""
    nb, bs = 60, 3
    A, _ = block_problem(nb, bs, 1, seed=5)
    A = A.toarray()
    rng = np.random.default_rng(6)
    A[:, 1::3] = A[:, 0::3] * (1.0 + 1e-8 * rng.standard_normal(A[:, 0::3].shape))
    A = sp.csc_matrix(A)
    A.sort_indices()
    P = pattern(nb, (40,) + (6,) * 9, seed=7)
    h.setup(A, P, options=mb.Options(ns=0, bs=bs, prec="mixed"))
    res, _, _ = h.column_info()
    o = O.spai_block(A, P, bs, ns=0)
    small = np.repeat(np.diff(P.indptr) == 6, bs)
    assert h.solver_columns()["general"] >= 54
    assert np.allclose(res[small], np.asarray(o.res).ravel()[small], rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("near,refused", [(0.0, False), (3e-2, True)])
def test_small_fp64_columns_by_condition(h, near, refused):
    """FP64 without refinement: elimination takes well-conditioned columns of 20
    unknowns and leaves those with two nearly parallel columns to the QR.  The
    residual norm does not change to first order in the solution's error, so that
    rounding leaves it within 1e-12 of the smallest one at condition 1e3."""
    n = 300
    A = matrix(n, 4, 6.0, seed=13)
    if near:
        D = A.toarray()
        noise = np.random.default_rng(14).standard_normal(D[:, 0::2].shape)
        D[:, 1::2] = D[:, 0::2] * (1.0 + near * noise)
        A = sp.csc_matrix(D)
        A.sort_indices()
    P = pattern(n, (20,), seed=15).tolil()
    P[:2] = 1.0
    P = sp.csc_matrix(P)
    P.sort_indices()
    h.setup(A, P, options=mb.Options(ns=0, prec="fp64"))
    c = h.solver_columns()
    assert c["sparse_small"] == n and c["fixed"] == (n if refused else 0)
    res, _, status = h.column_info()
    assert np.all(status == 0)
    assert np.allclose(res, O.spai_scalar(A, P, ns=0).res, rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("sizes", [(4,), (7, 3)])
@pytest.mark.parametrize("cs", [0, 100])
def test_small_dependent_columns(h, sizes, cs):
    """Two equal columns in every J of at most eight: rounding decides whether a QR
    meets an exact zero.  What the small QR does not solve is the warp solver's,
    with its values and its status bit for bit (a setup that keeps the factors
    uses the warp solver alone)."""
    n = 300
    D = matrix(n, 6, 3.0, seed=16).toarray()
    D[:, 1::3] = D[:, 0::3]
    D[:, 2] = 0.0
    A = sp.csc_matrix(D)
    # an explicit zero column: a zero on the diagonal whatever the rounding
    A = sp.csc_matrix(A + sp.csc_matrix(([1.0], ([5], [2])), shape=A.shape))
    A.data[A.indptr[2]:A.indptr[3]] = 0.0
    P = pattern(n, sizes, seed=17).toarray()
    both = np.maximum(P[0::3], P[1::3])
    P[0::3], P[1::3] = both, both
    P[2, 30:40] = 1.0
    P = sp.csc_matrix(P)
    P.sort_indices()
    assert P.getnnz(axis=0).max() <= 15
    small = P.getnnz(axis=0) <= 8
    h.setup(A, P, options=mb.Options(ns=0, prec="fp64", cs=cs))
    M, c = h.result(), h.solver_columns()
    res, steps, status = h.column_info()
    assert c["small_qr"] > 0 and 0 < c["warp"]
    ref = mb.Handle(0)
    ref.setup(A, P, options=mb.Options(ns=0, prec="fp64", keep_factors=True))
    N = ref.result()
    rres, _, rstatus = ref.column_info()
    ref.close()
    assert np.array_equal(status[small], rstatus[small])
    zero = np.flatnonzero(small & (P[2].toarray().ravel() != 0))
    assert zero.size > 0 and np.all(status[zero] == 1)
    same = 0
    for k in np.flatnonzero(small):
        a, b = M.indptr[k], M.indptr[k + 1]
        if np.array_equal(M.data[a:b], N.data[a:b]) and res[k] == rres[k]:
            same += 1
    assert same >= (c["warp"] if cs == 0 else 1) - np.count_nonzero(~small)
