"""`bench.py --impl reference` where the reference's compiled harness is missing: one
JSON line that says so, and exit code 0."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_RUN = ("import runpy, sys, oracle\n"
        "oracle.have_reference = lambda: False\n"
        "sys.argv = ['bench.py', '--impl', 'reference', '--config', sys.argv[1], '--steps', '1', '--warmup', '1']\n"
        "runpy.run_path('bench.py', run_name='__main__')\n")


@pytest.mark.parametrize("config", ["stream", "grid3d", "small2d"])
def test_reference_arm_without_its_library(config):
    out = subprocess.run([sys.executable, "-c", _RUN, config], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = out.stdout.strip().splitlines()
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and "libmpir_ref.so" in d["unavailable"]
