"""Triangular solves of systems whose fronts have rows with many children.

p unknowns couple to k others and not to one another: each of the k rows of the
centre has nearly p contributions (the analysis merges one or two leaves with it).
Up to 32 are added one after another, more through sums of 32 and sums of those; the
centre is solved by one warp (k <= 32), by a narrow item (k <= 128) or by slabs.  In
the second system two such stars, with centres of m, share a top of q: the rows
below the first centre's block have the many contributions.  Tolerance as in
test_gpu_flow.py (dominant systems)."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import mpir_b200 as mp
from helpers import rel_norm_diff

pytestmark = pytest.mark.gpu


def _assemble(blocks, n, rng):
    """Dense couplings between index ranges, made dominant."""
    K = sp.csc_matrix((n, n))
    for a, b in blocks:
        v = rng.uniform(-1.0, 1.0, size=(len(a), len(b)))
        K = K + sp.csc_matrix((v.ravel(), (np.repeat(a, len(b)), np.tile(b, len(a)))), shape=(n, n))
    K = K + K.T
    d = np.asarray(abs(K).sum(axis=1)).ravel() + 1.0
    U = sp.csc_matrix(sp.triu(K + sp.diags(np.where(np.arange(n) % 3 == 2, -d, d))))
    U.sort_indices()
    return U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data


def _check(Ap, Ai, Ax, levels):
    n = len(Ap) - 1
    solver = mp.GmresLDLIR()
    solver.analyze(Ap, Ai, Ax, ordering=mp.ORDER_NATURAL)
    assert solver.factor(Ax) == 0 and solver.info()["levels"] == levels
    Lp, Li, Lx, _, dinv = solver.export_factor()
    cols = np.repeat(np.arange(n), np.diff(Lp))
    L = (sp.csr_matrix((Lx.astype(np.float64), (Li, cols)), shape=(n, n)) + sp.identity(n)).tocsr()
    Lt = L.T.tocsr()
    rng = np.random.default_rng(n)
    for nrhs in (1, 3, 8, 16):
        Z = rng.standard_normal((nrhs, n))
        Y = solver.apply_factor(Z)
        np.testing.assert_array_equal(Y, solver.apply_factor(Z))
        y = spla.spsolve_triangular(L, Z.T, lower=True) * dinv.astype(np.float64)[:, None]
        y = spla.spsolve_triangular(Lt, y, lower=False).T
        for k in range(nrhs):
            assert rel_norm_diff(Y[k], y[k]) <= 2e-11, (nrhs, k)
    solver.close()


@pytest.mark.parametrize("k", [1, 30, 100, 140])
@pytest.mark.parametrize("p", [33, 34, 35, 36, 258, 260, 1026, 1028, 8400])
def test_star(p, k):
    if p * k > 300000:
        pytest.skip("covered by the smaller centres")
    n = p + k
    centre = np.arange(p, n)
    _check(*_assemble([(np.arange(p), centre), (centre, centre)], n, np.random.default_rng(p + k)), 2)


@pytest.mark.parametrize("p,m,q", [(40, 20, 40), (300, 20, 300), (300, 60, 40), (1100, 130, 30), (33, 200, 200)])
def test_two_stars(p, m, q):
    n = 2 * (p + m) + q
    a, ca = np.arange(p), np.arange(p, p + m)
    b, cb = np.arange(p + m, 2 * p + m), np.arange(2 * p + m, 2 * (p + m))
    top = np.arange(2 * (p + m), n)
    pairs = [(top, top)]
    for leaf, centre in ((a, ca), (b, cb)):
        pairs += [(leaf, centre), (leaf, top), (centre, centre), (centre, top)]
    _check(*_assemble(pairs, n, np.random.default_rng(n)), 3)
