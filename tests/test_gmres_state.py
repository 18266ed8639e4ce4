"""The state of the inner GMRES steps is laid out for 512 of them and grows with those taken."""
import subprocess

import numpy as np
import pytest

_MAIN = r"""
#include "arnoldi.hpp"
using mpir::Arnoldi;
int main() {
  // Up to 512 steps all of it; more cost nothing until they are taken.
  if (Arnoldi::bytes_for(10, 1) != 8 * (4 + 55 + 20 + 11 + 10 + 12)) return 1;
  for (int64_t m : {int64_t{513}, int64_t{12000}, int64_t{138240}, int64_t{2000000000}})
    for (int v : {1, 4, 16})
      if (Arnoldi::bytes_for(m, v) != Arnoldi::bytes_for(512, v) || Arnoldi::bytes_for(m, v) > (size_t{2} << 20) * v)
        return 2;
  return 0;
}
"""


def test_state_bytes(tmp_path):
    from mpir_b200 import build
    src, exe = tmp_path / "state.cu", tmp_path / "state"
    src.write_text(_MAIN)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", f"-I{build.CSRC}", f"-I{build.INCLUDE}", str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n,steps", [(1500, 511), (1500, 512), (1500, 513), (1500, 1300), (9000, 1025)])
def test_steps_beyond_the_first_layout(n, steps):
    """With a tolerance of zero an inner loop runs to its last step (the bounds are those
    of test_gpu_arnoldi)."""
    import mpir_b200 as mp
    from test_gpu_arnoldi import _backward, _system
    K, Ap, Ai, Ax = _system(n)
    solver = mp.GmresLDLIR(uf="bf16")
    solver.SetMaxGmresIterations(steps)
    solver.SetTolerance(0.0)
    solver.analyze(Ap, Ai, Ax)
    assert solver.factor(Ax) == 0
    B = np.random.default_rng(n).standard_normal((3, n))
    for X, reps in (([solver.Solve(B[0])], [solver.last_report]), (solver.SolveBatch(B), None)):
        reps = reps or solver.last_reports
        for x, b, rep in zip(X, B, reps):
            assert rep["gmres_iterations"] == steps * (rep["ir_iterations"] + 1)
            assert _backward(K, x, b) <= 3.6e-15
    solver.close()
