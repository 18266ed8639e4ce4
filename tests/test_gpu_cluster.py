"""Inner GMRES steps on clusters of 8 and 16 thread blocks, over and over.

The reductions pass partial sums between the blocks' shared memory in a fixed
order, so every solve of the same system has the same bits and counts; one that
lost a partial sum would not."""
import numpy as np
import pytest

import mpir_b200 as mp
from test_gpu_arnoldi import _backward, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8193, 65537, 140001])
def test_cluster_solves_repeat(n):
    K, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR(uf="bf16")
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    b = np.random.default_rng(n).standard_normal(n)
    x = solver.Solve(b)
    steps = solver.last_report["gmres_iterations"]
    assert _backward(K, x, b) <= 3.6e-15  # the bound of test_gpu_arnoldi
    for _ in range(20):
        np.testing.assert_array_equal(solver.Solve(b), x)
        assert solver.last_report["gmres_iterations"] == steps
    solver.close()
