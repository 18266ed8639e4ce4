"""Triangular solves with many leaves of at most 64 rows, which one vector takes by
kernels of their own (from 888 work items of them on, 16 leaves of up to 32 columns
an item), alone and below a common front, beside leaves that are larger.  Tolerance as
in test_gpu_flow.py (dominant systems, blocks of at most 150)."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import mpir_b200 as mp
from helpers import rel_norm_diff

pytestmark = pytest.mark.gpu


def _system(sizes, top, large=0, seed=0):
    """Dense blocks of the sizes; each couples to all of a top front's unknowns."""
    rng = np.random.default_rng(seed)
    rows, cols, at = [], [], 0
    n = int(sum(sizes)) + 150 * large + top
    t = np.arange(n - top, n)
    for b in list(sizes) + [150] * large:
        i = np.arange(at, at + b)
        rows += [np.repeat(i, b), np.repeat(i, top)]
        cols += [np.tile(i, b), np.tile(t, b)]
        at += b
    rows.append(np.repeat(t, top))
    cols.append(np.tile(t, top))
    r, c = np.concatenate(rows), np.concatenate(cols)
    K = sp.csc_matrix((rng.uniform(-1.0, 1.0, len(r)), (r, c)), shape=(n, n))
    K = K + K.T
    d = np.asarray(abs(K).sum(axis=1)).ravel() + 1.0
    U = sp.csc_matrix(sp.triu(K + sp.diags(np.where(np.arange(n) % 3 == 2, -d, d))))
    U.sort_indices()
    return n, U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data


CASES = {
    "narrow": lambda: _system([33 + k % 32 for k in range(950)], 0),
    "below_the_line": lambda: _system([33 + k % 32 for k in range(880)], 0),
    "with_rows": lambda: _system([33 + k % 12 for k in range(950)], 20),
    "tiny": lambda: _system([1 + k % 3 for k in range(15000)], 2, large=5),
    "dependent_launches": lambda: _system([1] * 14600, 3),  # (n of at most 20,000)
    "mixed": lambda: _system([1 + k % 64 for k in range(1800)], 0, large=7),
}


def _factors(n, Lp, Li, Lx):
    cols = np.repeat(np.arange(n), np.diff(Lp))
    L = (sp.csr_matrix((Lx.astype(np.float64), (Li, cols)), shape=(n, n)) + sp.identity(n)).tocsr()
    return L, L.T.tocsr()


@pytest.mark.parametrize("name", CASES)
def test_many_leaves(name):
    n, Ap, Ai, Ax = CASES[name]()
    solver = mp.GmresLDLIR()
    solver.analyze(Ap, Ai, Ax, ordering=mp.ORDER_NATURAL)
    assert solver.factor(Ax) == 0
    Lp, Li, Lx, _, dinv = solver.export_factor()
    L, Lt = _factors(n, Lp, Li, Lx)
    rng = np.random.default_rng(n)
    for nrhs in (1, 3):
        Z = rng.standard_normal((nrhs, n))
        Y = solver.apply_factor(Z)
        np.testing.assert_array_equal(Y, solver.apply_factor(Z))
        y = spla.spsolve_triangular(L, Z.T, lower=True) * dinv.astype(np.float64)[:, None]
        y = spla.spsolve_triangular(Lt, y, lower=False).T
        for k in range(nrhs):
            assert rel_norm_diff(Y[k], y[k]) <= 2e-11, (nrhs, k)
    b = rng.standard_normal(n)
    for uf in ("f32", "bf16"):
        other = solver if uf == "f32" else mp.GmresLDLIR(uf=uf)
        if other is not solver:
            other.analyze(Ap, Ai, Ax, ordering=mp.ORDER_NATURAL)
            assert other.factor(Ax) == 0
        other.Solve(b)
        assert other.last_report["status"] == 0 and other.last_report["backward_error"] <= 3.6e-15
        other.close()


def test_phases_of_leaves():
    """The QDLDL functions' forward and backward solves by themselves."""
    n, Ap, Ai, Ax = CASES["with_rows"]()
    _, Lnz, etree = mp.QDLDL_etree(n, Ap, Ai)
    _, Lp, Li, Lx, _, dinv = mp.QDLDL_factor(n, Ap, Ai, Ax, Lnz, etree)
    L, Lt = _factors(n, Lp, Li, Lx)
    z = np.random.default_rng(3).standard_normal(n)
    for call, ref in ((lambda x: mp.QDLDL_Lsolve(n, Lp, Li, Lx, x), spla.spsolve_triangular(L, z, lower=True)),
                      (lambda x: mp.QDLDL_Ltsolve(n, Lp, Li, Lx, x), spla.spsolve_triangular(Lt, z, lower=False))):
        assert rel_norm_diff(call(z.copy()), ref) <= 2e-11
