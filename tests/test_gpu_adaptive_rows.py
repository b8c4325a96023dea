"""Adaptive scalar columns whose candidates come from long rows of C: more of
them than the shared-memory slot's list (192) and its hash table (512) hold,
just as many, and one more, against the oracle.  Same pattern and steps, 1e-10
per entry, as for every FP64 column."""
import numpy as np
import pytest
import scipy.sparse as sp

import mspai_b200 as mb
from helpers import max_rel_diff, same_pattern
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def matrix(n, long_rows, length, seed):
    """Tridiagonal, diagonally dominant; `long_rows` rows with `length` entries."""
    rng = np.random.default_rng(seed)
    A = sp.diags([rng.uniform(-1, 0, n - 1), rng.uniform(2, 3, n), rng.uniform(-1, 0, n - 1)],
                 [-1, 0, 1]).tolil()
    for r in long_rows:
        at = np.sort(rng.choice(n, length, replace=False))
        A[r, at] = 0.1 * rng.standard_normal(at.size)
        A[r, r] = 2.5
    A = sp.csc_matrix(A)
    A.sort_indices()
    return A


@pytest.mark.parametrize("n,long_rows,length", [
    (700, (350,), 191), (700, (350,), 192), (700, (350,), 193),  # the list's length
    (700, (10, 200), 150),        # two rows fill the list together
    (2000, (1000,), 700),         # more than the table holds
    (6000, (0, 3000), 6000),      # every column sees two full rows
])
def test_long_rows(n, long_rows, length):
    A = matrix(n, long_rows, length, seed=n + length)
    P = sp.identity(n, format="csc")
    o = O.spai_scalar(A, P, ep=0.1, ns=2, mn=3)
    h = mb.Handle(0)
    for _ in range(2):
        h.setup(A, P, options=mb.Options(ep=0.1, ns=2, mn=3, prec="fp64"))
        M = h.result()
        res, steps, status = h.column_info()
        assert np.all(status == 0) and np.array_equal(steps, o.steps)
        assert same_pattern(M, o.M)
        assert max_rel_diff(M, o.M) < 1e-10
        assert np.allclose(res, o.res, rtol=1e-8, atol=1e-14)
    h.close()
