"""Block columns at their start pattern (block_solve.cu) against the oracle:
sizes on both sides of its two launches, columns that it leaves to the general
solver (too large, above the tolerance: pattern updates), targets with probing
rows.  Tolerances per entry as for every block column: 1e-8 in mixed mode, 1e-10
in FP64 (helpers.max_rel_diff)."""
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


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("bs,sizes", [(2, (1, 2, 4, 5, 9)), (3, (1, 2, 3, 6, 11)),
                                      (8, (1, 2, 7)), (3, (40, 86))])
def test_sizes(h, prec, bs, sizes):
    """|J| from one block to more than the 255 columns that fit."""
    nb = 100
    n = bs * nb
    rng = np.random.default_rng(bs)
    rows, cols = [], []
    for k in range(nb):
        for b in {k} | set(rng.choice(nb, 3, replace=False).tolist()):
            for i in range(bs):
                for j in range(bs):
                    rows.append(bs * b + i)
                    cols.append(bs * k + j)
    vals = rng.standard_normal(len(rows))
    A = sp.csc_matrix((vals, (rows, cols)), shape=(n, n)) + 6.0 * sp.identity(n)
    A = sp.csc_matrix(A)
    A.sort_indices()
    pr, pc = [], []
    for k in range(nb):
        J = {k}
        while len(J) < sizes[k % len(sizes)]:
            J.add(int(rng.integers(nb)))
        pr += sorted(J)
        pc += [k] * len(J)
    P = sp.csc_matrix((np.ones(len(pr)), (pr, pc)), shape=(nb, nb))
    h.setup(A, P, options=mb.Options(ns=0, bs=bs, prec=prec))
    M = h.result()
    res, steps, status = h.column_info()
    o = O.spai_block(A, P, bs, ns=0)
    assert np.all(status == 0) and np.all(steps == 1)
    assert same_pattern(M, o.M)
    assert max_rel_diff(M, o.M) < TOL[prec]
    assert np.allclose(res, o.res, rtol=1e-9, atol=1e-13)


@pytest.mark.parametrize("ep", [0.5, 0.2, 0.05])
def test_updates_after_the_start_pattern(h, ep):
    """Some columns end at the start pattern, the others update theirs."""
    w = W.block27(5, rho=10.0, probing=True)
    C, B = mb.assemble_probing(w.A, w.Ce, w.Be, 10.0)
    P = sp.identity(w.n // 3, format="csc")
    h.setup(C, P, B=B, options=mb.Options(ns=3, mn=3, ep=ep, bs=3, prec="mixed"))
    M = h.result()
    _, steps, status = h.column_info()
    o = O.spai_block(C, P, 3, B=B, ns=3, mn=3, ep=ep)
    assert np.all(status == 0)
    assert np.array_equal(steps[::3], np.asarray(o.steps).ravel()[::3])
    assert same_pattern(M, o.M)
    assert max_rel_diff(M, o.M) < TOL["mixed"]
