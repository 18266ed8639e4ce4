"""Diagonal blocks and small fronts of the factorization at the edges of their tiles.

K has a dense leading block of w unknowns and one of 20, both coupled to a dense
tail of 65 and not to each other; in natural order the first is a front of w
columns and w + 65 rows: a diagonal block of w and, through the inverse of its
unit-lower factor, 65 rows below.  K is quasi-definite with unit |diagonal|.

Tolerance (u = 6e-8): each entry of L D L^T adds up to w products, each with up
to 4 u of a reciprocal good to 2 units, so the block's residual is within
2 (w + 10) u |L| |D| |L^T|.  The rows below are F X^T D^{-1} with X = L^{-1} to
(w + 4) u |X| |L| |X|, the product in three TF32 terms (2^-20 < 17 u): their
residual is within 4 (w + 16) u |F| (|X^T| |L^T|)^2."""
import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse as sp

import mpir_b200 as mp

pytestmark = pytest.mark.gpu


def _quasi_definite(n, seed):
    rng = np.random.default_rng(seed)
    sign = np.where(np.arange(n) % 3 == 2, -1.0, 1.0)
    M = rng.standard_normal((n, 4 * n))
    M /= np.linalg.norm(M, axis=1)[:, None]
    C = M @ M.T
    A = rng.standard_normal((n, n)) / np.sqrt(n)
    K = np.where(np.equal.outer(sign, sign), np.outer(sign, sign) * C * sign[:, None], A + A.T)
    K = K.astype(np.float32).astype(np.float64)
    K[np.arange(n), np.arange(n)] = sign
    return K


def _factor(K):
    n = len(K)
    U = sp.csc_matrix(np.triu(K))
    U.sort_indices()
    solver = mp.GmresLDLIR()
    solver.analyze(U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data,
                   ordering=mp.ORDER_NATURAL)
    assert solver.factor(U.data) == 0
    Lp, Li, Lx, D, _ = solver.export_factor()
    cols = np.repeat(np.arange(n), np.diff(Lp))
    L = sp.csr_matrix((Lx.astype(np.float64), (Li, cols)), shape=(n, n)).toarray() + np.eye(n)
    solver.close()
    return L, D.astype(np.float64)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64])
def test_small_front(n):
    """One front in shared memory (at most 64 rows): the block's bound above."""
    K = _quasi_definite(n, 100 + n)
    L, D = _factor(K)
    res = np.abs(K - (L * D) @ L.T)
    assert (res <= 2 * (n + 10) * 2.0 ** -24 * ((np.abs(L) * np.abs(D)) @ np.abs(L.T))).all()


@pytest.mark.parametrize("w", [33, 63, 64, 65, 95, 96, 97, 127, 128])
def test_diagonal_block(w):
    r, wb = 65, 20
    n = w + wb + r
    K = _quasi_definite(n, w)
    K[:w, w:w + wb] = K[w:w + wb, :w] = 0.0
    L, D = _factor(K)
    L1, D1 = L[:w, :w], D[:w]
    u = 2.0 ** -24
    res = np.abs(K[:w, :w] - (L1 * D1) @ L1.T)
    assert (res <= 2 * (w + 10) * u * ((np.abs(L1) * np.abs(D1)) @ np.abs(L1.T))).all()
    F = K[w + wb:, :w]
    LX = np.abs(sl.solve_triangular(L1, np.eye(w), lower=True).T) @ np.abs(L1.T)
    res = np.abs(F - (L[w + wb:, :w] * D1) @ L1.T)
    assert (res <= 4 * (w + 16) * u * (np.abs(F) @ LX @ LX)).all()


@pytest.mark.parametrize("r", [255, 511, 512, 777, 1300])
def test_extend_add_rows(r):
    """Two dense blocks of 70 and 33 add to a dense tail of r (its rows split over
    thread blocks from 512 on).  Products in three TF32 terms are within 17 u as
    above, so the residual is within 4 (n + 16) u |L| |D| |L^T|."""
    n = 103 + r
    K = _quasi_definite(n, r)
    K[:70, 70:103] = K[70:103, :70] = 0.0
    L, D = _factor(K)
    res = np.abs(K - (L * D) @ L.T)
    assert (res <= 4 * (n + 16) * 2.0 ** -24 * ((np.abs(L) * np.abs(D)) @ np.abs(L.T))).all()
