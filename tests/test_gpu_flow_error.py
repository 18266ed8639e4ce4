"""Triangular solves against their error bound, and 16-bit panels at the edges of the work items.

The blocks of the diagonal are applied through their inverses.  With X = L^-1 the
computed y of L y = z is within 3 n u |X| |L| |X| |z| entry by entry (n u for the
inverse's columns, for its product and for the blocks before it; Higham, Accuracy and
Stability of Numerical Algorithms, ch. 14; u = 2^-53), x of L^T x = D^-1 y likewise,
and D^-1 adds u: for both together 4 n u times the two bounds.  Systems with
delta = 1e-8 give L entries of 1e4 (scaled) to 1e8 (unscaled); the exact solutions come
from substitution in 80-bit arithmetic."""
import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse as sp

import mpir_b200 as mp
from helpers import rel_norm_diff
from mpir_b200 import kkt
from test_gpu_arnoldi import _backward
from test_gpu_arnoldi import _system as _banded
from test_gpu_flow import _system as _two_blocks

pytestmark = pytest.mark.gpu


def _upper(K):
    U = sp.csc_matrix(np.triu(K))
    U.sort_indices()
    return U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data


def _dense_kkt(n1, m, seed):
    """Dense quasi-definite, delta = 1e-8, five pivots -delta first, then in random order."""
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n1, n1)) / np.sqrt(n1)
    A = rng.standard_normal((m, n1))
    K = np.block([[G @ G.T + np.eye(n1), A.T], [A, -1e-8 * np.eye(m)]])
    p = np.concatenate([n1 + np.arange(5), rng.permutation(np.r_[:n1, n1 + 5:n1 + m])])
    return _upper(K[np.ix_(p, p)])


def _dense_l(n, Lp, Li, Lx):
    cols = np.repeat(np.arange(n), np.diff(Lp))
    return sp.csr_matrix((Lx.astype(np.float64), (Li, cols)), shape=(n, n)).toarray() + np.eye(n)


def _exact(L, dinv, Z):
    y = Z.T.astype(np.longdouble)
    n = len(L)
    for k in range(n):
        y[k + 1:] -= L[k + 1:, k, None].astype(np.longdouble) * y[k]
    y *= dinv.astype(np.longdouble)[:, None]
    for k in range(n - 1, 0, -1):
        y[:k] -= L[k, :k, None].astype(np.longdouble) * y[k]
    return y.T


def _bound(L, dinv, Z):
    n, u = len(L), 2.0 ** -53
    aL, aX = np.abs(L), np.abs(sl.solve_triangular(L, np.eye(n), lower=True, unit_diagonal=True))
    aZ, d = np.abs(Z.T), np.abs(dinv.astype(np.float64))[:, None]
    y = aX @ aZ
    return 4 * n * u * (aX.T @ (d * (aX @ (aL @ y))) + aX.T @ (aL.T @ (aX.T @ (d * y)))).T


SYSTEMS = {
    "dense600": lambda: _dense_kkt(400, 200, 1),
    "dense1100": lambda: _dense_kkt(700, 400, 2),
    "kkt2d": lambda: (lambda s: (s.Ap, s.Ai, s.Ax))(kkt.make(32, 2, 256, 4, 1e-8, diag_range=(1e-6, 1e2), seed=3)),
    "kkt3d": lambda: (lambda s: (s.Ap, s.Ai, s.Ax))(
        kkt.make(10, 3, 250, 8, 1e-8, shift=1e-8, scaled_range=(1e-3, 1e3), seed=4)),
}


@pytest.mark.parametrize("name", SYSTEMS)
def test_unrefined_error_bound(name):
    Ap, Ai, Ax = SYSTEMS[name]()
    n = len(Ap) - 1
    rng = np.random.default_rng(5)
    solver = mp.GmresLDLIR()
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    Lp, Li, Lx, _, dinv = solver.export_factor()
    L = _dense_l(n, Lp, Li, Lx)
    for nrhs in (1, 3, 8, 16):
        Z = rng.standard_normal((nrhs, n))
        assert (np.abs(solver.apply_factor(Z) - _exact(L, dinv, Z)) <= _bound(L, dinv, Z)).all(), nrhs
    solver.close()
    # the QDLDL functions: natural order, not scaled
    total, Lnz, etree = mp.QDLDL_etree(n, Ap, Ai)
    npos, Lp, Li, Lx, _, dinv = mp.QDLDL_factor(n, Ap, Ai, Ax, Lnz, etree)
    assert total == len(Lx) and npos > 0
    L = _dense_l(n, Lp, Li, Lx)
    assert np.abs(L).max() > (1e6 if name.startswith("dense") else 1.0)
    Z = rng.standard_normal((1, n))
    x = mp.QDLDL_solve(n, Lp, Li, Lx, dinv, Z[0].copy())
    assert (np.abs(x - _exact(L, dinv, Z)[0]) <= _bound(L, dinv, Z)[0]).all()


def _bf16(x):
    b = x.astype(np.float32).view(np.uint32).astype(np.uint64)
    return ((b + 0x7FFF + (b >> 16 & 1)) >> 16 << 16).astype(np.uint32).view(np.float32)


def _apart(wa, r):
    """As the systems of test_gpu_flow.py, with one more unknown between their blocks: the
    first block's parent is then not next to it, and the analysis keeps their fronts apart."""
    wb, n = 20, wa + 1 + 20 + r
    rng = np.random.default_rng(1000 * wa + r + 1)
    K = np.zeros((n, n))
    tail = np.arange(wa + 1 + wb, n)
    for b in (np.arange(wa), np.array([wa]), np.arange(wa + 1, wa + 1 + wb)):
        i = np.concatenate([b, tail])
        K[np.ix_(i, i)] += rng.uniform(-1.0, 1.0, size=(len(i), len(i)))
    K = K + K.T
    d = np.abs(K).sum(axis=1) + 1.0
    K[np.arange(n), np.arange(n)] = np.where(np.arange(n) % 3 == 2, -d, d)
    return (n, *_upper(K))


def _check_solves(system, uf, fronts, wa, r):
    """Against substitution with the exported factor.  The bfloat16 tier keeps L in bfloat16
    outside the blocks of the diagonal (512 columns at most) and the fronts that one
    warp solves; those stay float32.  The tolerance is that of test_gpu_flow.py."""
    n, Ap, Ai, Ax = system
    solver = mp.GmresLDLIR(uf=uf)
    solver.analyze(Ap, Ai, Ax, ordering=mp.ORDER_NATURAL)
    assert solver.factor(Ax) == 0
    assert solver.info()["supernodes"] in fronts
    Lp, Li, Lx, _, dinv = solver.export_factor()
    L = _dense_l(n, Lp, Li, Lx)
    if uf == "bf16":
        i = np.arange(n)
        # the front and, in it, the block of the diagonal that an index belongs to
        front = i >= (wa if solver.info()["supernodes"] == 2 else n)
        block = np.where(front, i - wa, i) // 512
        same = (front[:, None] == front[None, :]) & (block[:, None] == block[None, :])
        if front.any() and wa <= 32 and wa + r <= 256:
            same |= ~front[None, :]
        L = np.where(same, L, _bf16(L.astype(np.float32)).astype(np.float64))
    rng = np.random.default_rng(n)
    for nrhs in (1, 3, 8, 16):
        Z = rng.standard_normal((nrhs, n))
        Y = solver.apply_factor(Z)
        y = sl.solve_triangular(L, Z.T, lower=True, unit_diagonal=True) * dinv.astype(np.float64)[:, None]
        y = sl.solve_triangular(L.T, y, lower=False, unit_diagonal=True).T
        for k in range(nrhs):
            assert rel_norm_diff(Y[k], y[k]) <= 2e-11, (nrhs, k)
    solver.close()


@pytest.mark.parametrize("wa,r", [(20, 100), (33, 513), (100, 600), (128, 40), (129, 300), (160, 129), (513, 40),
                                  (545, 700)])
def test_bfloat16_panels(wa, r):
    _check_solves(_two_blocks(wa, r), "bf16", (1, 2), wa, r)


@pytest.mark.parametrize("uf", ["f32", "bf16"])
@pytest.mark.parametrize("wa,r", [(1, 1), (1, 255), (1, 256), (16, 241), (17, 30), (32, 224), (32, 225), (32, 513),
                                  (33, 31), (33, 513), (64, 128), (65, 1100), (127, 1), (128, 512), (128, 513),
                                  (129, 1), (129, 129), (160, 512), (161, 513), (512, 128), (513, 31), (545, 1025)])
def test_two_fronts_at_item_edges(wa, r, uf):
    _check_solves(_apart(wa, r), uf, (2,), wa, r)


@pytest.mark.parametrize("n", [19999, 20000, 20001])
def test_solves_at_the_edge_of_dependent_launches(n):
    """Up to 20,000 unknowns a solve's kernels are launched before the one ahead is done."""
    K, Ap, Ai, Ax = _banded(n)
    B = np.random.default_rng(n).standard_normal((3, n))
    solver = mp.GmresLDLIR()
    solver.analyze(Ap, Ai, Ax)
    first = None
    for _ in range(6):  # plain, recorded and replayed factorizations between the solves
        assert solver.factor(Ax) == 0
        got = [solver.Solve(b) for b in B] + list(solver.SolveBatch(B))
        first = first or got
        for k, x in enumerate(got):
            np.testing.assert_array_equal(x, first[k])
            assert _backward(K, x, B[k % 3]) <= 3.6e-15
    solver.close()
