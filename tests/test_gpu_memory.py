"""A solver whose vectors did not fit solves on once it is asked for fewer.

The GMRES basis of n = 200,001 unknowns and as many steps is 320 GB, that of 16
vectors and 20,000 steps 512 GB: both allocations are refused.  With the former
number of steps the solver gives what it gave before."""
import numpy as np
import pytest

import mpir_b200 as mp
from test_gpu_arnoldi import _backward, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs,steps", [(1, 200001), (16, 20000)])
def test_solver_after_refused_allocation(nrhs, steps):
    n = 200001
    _, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR()
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    B = np.random.default_rng(7).standard_normal((nrhs, n))
    solve = (lambda: solver.SolveBatch(B)) if nrhs > 1 else (lambda: solver.Solve(B[0]))
    X = np.array(solve())
    solver.SetMaxGmresIterations(steps)
    with pytest.raises(mp.MpirError, match="nomem"):
        solve()
    solver.SetMaxGmresIterations(10)
    np.testing.assert_array_equal(np.array(solve()), X)
    solver.close()


def test_many_steps_for_sixteen_vectors():
    """12,000 steps: the vectors' states lie 1.4e8 words apart, the last one's flag past 2^31."""
    n = 12100
    K, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR()
    solver.SetMaxGmresIterations(12000)
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    B = np.random.default_rng(8).standard_normal((16, n))
    X = solver.SolveBatch(B)
    for x, b in zip(X, B):
        assert _backward(K, x, b) <= 3.6e-15
    solver.close()
