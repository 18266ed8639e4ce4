"""Triangular solves at the edges of their work items (through the C ABI).

K has two dense diagonal blocks, of wa and 20 unknowns, that both couple to a
dense tail of r unknowns and not to each other; in natural order the first
block is a front of wa columns and wa + r rows, and the other block and the
tail make up the root.  wa and r walk over the bounds between the kinds of work
items: fronts solved by one warp (32 columns, 256 rows), narrow fronts (32 and
128 columns; 512 rows an item), super-blocks of 512 columns with slabs of 32,
and chunks of 512 rows.

One to sixteen vectors are compared with a float64 solve with the exported
factor.  Tolerance: K is strongly diagonally dominant, so the condition of L
is below 10; a triangular solve of order n, block products with inverses
included, is within about 3 n u cond(L) (u = 1.1e-16), two of them at n = 2,200
within 2e-11 normwise."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import mpir_b200 as mp
from helpers import rel_norm_diff

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 255), (1, 600), (16, 240), (16, 241), (31, 33), (32, 224), (32, 225), (32, 512),
         (33, 31), (33, 513), (64, 129), (65, 1100), (127, 1), (128, 512), (128, 513), (129, 0),
         (129, 31), (160, 128), (161, 129), (511, 40), (512, 512), (513, 513), (545, 1025)]


def _system(wa, r, wb=20):
    n = wa + wb + r
    rng = np.random.default_rng(1000 * wa + r)
    K = np.zeros((n, n))
    blocks = [np.arange(wa), np.arange(wa, wa + wb)]
    tail = np.arange(wa + wb, n)
    for b in blocks:
        i = np.concatenate([b, tail])
        K[np.ix_(i, i)] += rng.uniform(-1.0, 1.0, size=(len(i), len(i)))
    K = K + K.T
    d = np.abs(K).sum(axis=1) + 1.0
    K[np.arange(n), np.arange(n)] = np.where(np.arange(n) % 3 == 2, -d, d)
    U = sp.csc_matrix(np.triu(K))
    U.sort_indices()
    return n, U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data


@pytest.mark.parametrize("wa,r", SIZES)
def test_solves_at_item_edges(wa, r):
    n, Ap, Ai, Ax = _system(wa, r)
    solver = mp.GmresLDLIR()
    solver.analyze(Ap, Ai, Ax, ordering=mp.ORDER_NATURAL)
    assert solver.factor(Ax) == 0
    Lp, Li, Lx, D, Dinv = solver.export_factor()
    cols = np.repeat(np.arange(n), np.diff(Lp))
    L = (sp.csr_matrix((Lx.astype(np.float64), (Li, cols)), shape=(n, n)) + sp.identity(n)).tocsr()
    Lt = L.T.tocsr()
    rng = np.random.default_rng(n)
    for nrhs in (1, 3, 7, 16):
        X = rng.standard_normal((nrhs, n))
        # twice: the second application finds what the first one left behind
        Y = solver.apply_factor(X)
        np.testing.assert_array_equal(Y, solver.apply_factor(X))
        for k in range(nrhs):
            y = spla.spsolve_triangular(L, X[k], lower=True) * Dinv.astype(np.float64)
            y = spla.spsolve_triangular(Lt, y, lower=False)
            assert rel_norm_diff(Y[k], y) <= 2e-11, (nrhs, k)
    solver.close()
