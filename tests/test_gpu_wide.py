"""Inner GMRES steps of long vectors, which the whole chip sweeps (more than 200,000
unknowns, up to 4 vectors), beside those of clusters (more vectors).  The systems are
tridiagonal in blocks of 8 (small fronts), factored in bfloat16; the bounds are those of
test_gpu_arnoldi.py."""
import numpy as np
import pytest
import scipy.sparse as sp

import mpir_b200 as mp
from test_gpu_arnoldi import _backward

pytestmark = pytest.mark.gpu


def _system(n):
    rng = np.random.default_rng(n)
    d = np.where(np.arange(n) % 3 == 2, -1.0, 1.0) * rng.uniform(2.0, 3.0, n)
    o = rng.uniform(-1.0, 1.0, n - 1) * (np.arange(n - 1) % 8 != 7)
    K = sp.diags([d, o, o], [0, 1, -1], format="csc")
    K.eliminate_zeros()
    U = sp.csc_matrix(sp.triu(K))
    U.sort_indices()
    return K, U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data


@pytest.mark.parametrize("n", [200000, 200001, 303111, 500003])
def test_long_vectors(n):
    K, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR(uf="bf16")
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    B = np.random.default_rng(n).standard_normal((6, n))
    B[1] *= 1e-200  # squares beyond float64's range (and a norm below the tolerance)
    B[2] *= 1e180
    single = []
    for k, b in enumerate(B[:3]):
        x = solver.Solve(b)
        rep = solver.last_report
        assert rep["status"] == 0 and _backward(K, x, b) <= 3.6e-15
        assert rep["precond_applies"] == rep["gmres_iterations"] + (k != 1) + rep["ir_iterations"]
        assert rep["gmres_iterations"] > rep["ir_iterations"]
        np.testing.assert_array_equal(solver.Solve(b), x)
        single.append(rep["gmres_iterations"])
    for nrhs in (3, 4, 6):
        X = solver.SolveBatch(B[:nrhs])
        for k, (x, b) in enumerate(zip(X, B)):
            assert solver.last_reports[k]["status"] == 0 and _backward(K, x, b) <= 3.6e-15
            if k < 3:  # the same steps, but for roundings at a stop test
                assert abs(solver.last_reports[k]["gmres_iterations"] - single[k]) <= 2
    solver.close()


@pytest.mark.parametrize("nrhs", [1, 2])
def test_long_vectors_beyond_convergence(nrhs):
    """40 steps an inner loop with a tolerance of zero (rotations are applied 32 at a time)."""
    n = 250007
    K, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR(uf="bf16")
    solver.SetMaxGmresIterations(40)
    solver.SetTolerance(0.0)
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    B = np.random.default_rng(n).standard_normal((nrhs, n))
    X = solver.SolveBatch(B) if nrhs > 1 else [solver.Solve(B[0])]
    reps = solver.last_reports if nrhs > 1 else [solver.last_report]
    for x, b, rep in zip(X, B, reps):
        assert rep["gmres_iterations"] == 40 * (rep["ir_iterations"] + 1)
        assert _backward(K, x, b) <= 3.6e-15
    solver.close()


@pytest.mark.parametrize("n", [200000, 250007])
def test_second_sweep(n):
    """A diagonal K: the first step's vector is all but the basis vector already, and what
    is left of it is orthogonalised again."""
    rng = np.random.default_rng(n)
    d = np.where(np.arange(n) % 3 == 2, -1.0, 1.0) * rng.uniform(2.0, 3.0, n)
    K = sp.diags([d], [0], format="csc")
    solver = mp.GmresLDLIR()
    solver.SetMaxGmresIterations(3)
    solver.SetTolerance(0.0)
    solver.analyze(np.arange(n + 1), np.arange(n), d)
    assert solver.factor(d) == 0
    B = rng.standard_normal((2, n))
    for X, reps in (([solver.Solve(B[0])], [solver.last_report]), (solver.SolveBatch(B), None)):
        for x, b, rep in zip(X, B, reps or solver.last_reports):
            assert rep["reorth_count"] > 0 and rep["status"] == 0
            assert _backward(K, x, b) <= 3.6e-15
    solver.close()
