"""Adaptive scalar columns whose slot lies in shared memory (warp_adaptive_kernel)
against the oracle: columns that end inside it, columns that outgrow it (unknowns,
entries, rows of the folded matrix, candidates, a full candidate table) and start
again in global memory, columns of more than eight entries, and more unknowns per
update than it takes.  Same pattern and steps; 1e-10 per entry, as for every FP64
column."""
import numpy as np
import pytest
import scipy.sparse as sp

import mspai_b200 as mb
from helpers import max_rel_diff, same_pattern
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    handle = mb.Handle(0)
    yield handle
    handle.close()


def matrix(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    rows, cols, vals = [], [], []
    for k in range(n):
        off = rng.choice(n - 1, int(rng.integers(lo, hi + 1)), replace=False)
        v = rng.standard_normal(off.size)
        rows += (off + (off >= k)).tolist() + [k]
        cols += [k] * (off.size + 1)
        vals += v.tolist() + [1.2 * np.abs(v).sum() + 0.1]
    A = sp.csc_matrix((vals, (rows, cols)), shape=(n, n))
    A.sort_indices()
    return A


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,lo,hi,ns,mn", [
    (33, 0, 2, 5, 1),       # within the slot
    (400, 2, 6, 3, 5),      # up to 16 unknowns, 112 entries
    (300, 2, 6, 6, 5),      # up to 31 unknowns: outgrown
    (300, 7, 11, 2, 5),     # on both sides of eight entries a column
    (1500, 12, 18, 2, 5),   # more candidates than the list, or the table, holds
    (300, 2, 5, 1, 16),     # the most unknowns per update, and one more
    (300, 2, 5, 1, 17),
])
def test_sizes(h, prec, n, lo, hi, ns, mn):
    A = matrix(n, lo, hi, n + mn)
    P = sp.identity(n, format="csc")
    o = O.spai_scalar(A, P, ep=0.05, ns=ns, mn=mn)
    for _ in range(2):  # the second from the handle's kept workspace
        h.setup(A, P, options=mb.Options(ep=0.05, ns=ns, mn=mn, prec=prec))
        M = h.result()
        res, steps, status = h.column_info()
        assert np.all(status == 0) and np.array_equal(steps, o.steps)
        assert same_pattern(M, o.M)
        assert max_rel_diff(M, o.M) < 1e-10
        assert np.allclose(res, o.res, rtol=1e-8, atol=1e-14)
