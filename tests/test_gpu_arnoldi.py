"""The inner GMRES steps at the sizes where their kernels change.

One vector is spread over a thread-block cluster: one CTA up to 8,192 unknowns,
8 up to 65,536, 16 beyond, with 8,192 entries a CTA in registers and the rest in
memory (from 131,073 unknowns on).  A banded quasi-definite system is
factored in bfloat16, so that the inner loops take several steps, and solved
for one and three right-hand sides; with a tolerance of zero an inner
loop runs to its 40 steps (rotations are applied 32 at a time).

Tolerance: refinement stops on an update of at most 10 u |x|, so the residual
is at most 10 u |A| |x| and its own rounding, (nnz a row + 1) u |A| |x|, here 6 u:
a normwise backward error below 16 u = 3.6e-15."""
import numpy as np
import pytest
import scipy.sparse as sp

import mpir_b200 as mp

pytestmark = pytest.mark.gpu


def _system(n):
    rng = np.random.default_rng(n)
    d = np.where(np.arange(n) % 3 == 2, -1.0, 1.0) * rng.uniform(2.0, 3.0, n)
    offs = [(k, rng.uniform(-1.0, 1.0, n - k)) for k in (1, 2) if n > k]
    K = sp.diags([d] + [v for _, v in offs] + [v for _, v in offs],
                 [0] + [k for k, _ in offs] + [-k for k, _ in offs], format="csc")
    U = sp.csc_matrix(sp.triu(K))
    U.sort_indices()
    return K, U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data


def _backward(K, x, b):
    r = np.abs(b - K @ x).max()
    return r / (np.abs(K).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())


@pytest.mark.parametrize("n", [1, 2, 31, 511, 512, 513, 8191, 8192, 8193, 65535, 65536, 65537,
                               131072, 131073, 140001])
def test_inner_steps_at_cluster_edges(n):
    K, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR(uf="bf16")
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    B = np.random.default_rng(n + 1).standard_normal((3, n))
    for k in range(3):
        x = solver.Solve(B[k])
        rep = solver.last_report
        assert rep["status"] == 0 and _backward(K, x, B[k]) <= 3.6e-15
        assert rep["precond_applies"] == rep["gmres_iterations"] + 1 + rep["ir_iterations"]
        if n > 100:
            assert rep["gmres_iterations"] > rep["ir_iterations"] + 1
    X = solver.SolveBatch(B)
    for k in range(3):
        assert _backward(K, X[k], B[k]) <= 3.6e-15
        assert solver.last_reports[k]["status"] == 0
    solver.close()


@pytest.mark.parametrize("n", [513, 70000])
def test_inner_steps_beyond_convergence(n):
    K, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR(uf="bf16")
    solver.SetMaxGmresIterations(40)
    solver.SetTolerance(0.0)
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    b = np.random.default_rng(n + 1).standard_normal(n)
    x = solver.Solve(b)
    rep = solver.last_report
    assert rep["gmres_iterations"] == 40 * (rep["ir_iterations"] + 1)
    assert rep["spmv_count"] == rep["gmres_iterations"] + rep["ir_iterations"] + 1
    assert _backward(K, x, b) <= 3.6e-15
    solver.close()
