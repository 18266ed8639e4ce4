"""Kernel attributes are set on every device that a kernel runs on.

An attribute belongs to a kernel on one device, so what guards it must count
devices.  The guard is plain C++ and is compiled here; with two GPUs a solver on
each is run in one process."""
import glob
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mpir_b200", "csrc")

_MAIN = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.hpp"
int main() {
  mpir::OncePerDevice once;
  std::atomic<int> calls[66] = {};
  for (int turn = 0; turn < 3; turn++)
    for (int d = 0; d < 66; d++) once.run(d, [&] { calls[d]++; });
  for (int d = 0; d < 66; d++)
    if (calls[d] != (d < 64 ? 1 : 3)) return std::printf("device %d: %d\n", d, calls[d].load()), 1;
  mpir::OncePerDevice failing;  // a call that throws is made again
  int tries = 0;
  for (int k = 0; k < 2; k++)
    try { failing.run(1, [&] { if (tries++ == 0) throw 1; }); } catch (int) {}
  if (tries != 2) return 2;
  mpir::OncePerDevice shared;  // nobody goes on before its device is done
  std::atomic<int> value[8] = {}, bad{0};
  std::vector<std::thread> t;
  for (int k = 0; k < 16; k++)
    t.emplace_back([&] {
      for (int d = 0; d < 8; d++) {
        shared.run(d, [&] { value[d] = 1; });
        if (value[d] != 1) bad++;
      }
    });
  for (auto &x : t) x.join();
  return bad ? 3 : 0;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(_MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_shared_memory_limits_go_through_the_guard():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            assert not re.search(r"cudaFuncAttributeMaxDynamicSharedMemorySize", f.read()), path


@pytest.mark.gpu
def test_two_devices_in_one_process():
    import torch

    import mpir_b200 as mp
    from mpir_b200 import kkt
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    s = kkt.make(24, 2, 144, 4, 1e-4)
    for device in (0, 1):
        solver = mp.GmresLDLIR(device=device)
        solver.analyze(s.Ap, s.Ai, s.Ax)
        assert solver.factor(s.Ax) == 0
        for X in (solver.Solve(s.b)[None], solver.SolveBatch(np.stack([s.b, s.b]))):
            for x in X:
                assert kkt.backward_error(s.n, s.Ap, s.Ai, s.Ax, x, s.b) <= 1e-14
        solver.close()
