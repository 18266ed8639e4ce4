"""Front-vector entries are numbered up to 2^32 - 2 (host code, compiled here)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpir_b200", "csrc")

_MAIN = r"""
#define __host__
#define __device__
#include "flow.cuh"
int main() {
  const int64_t ok[] = {0, 1, 0x7ffffffe, 0x7fffffff, 0x80000000ll, 0xfffffffell};
  for (int64_t i : ok)
    if (static_cast<int64_t>(mpir::flow_entry(i)) != i) return 1;
  for (int64_t i : {int64_t{-1}, int64_t{0xffffffffll}, int64_t{1} << 32}) {
    bool threw = false;
    try { mpir::flow_entry(i); } catch (const std::invalid_argument &) { threw = true; }
    if (!threw) return 2;
  }
  return sizeof(mpir::FlowGather) == 8 && alignof(mpir::FlowGather) == 8 ? 0 : 3;
}
"""


def test_entries_beyond_2_31(tmp_path):
    src, exe = tmp_path / "entry.cpp", tmp_path / "entry"
    src.write_text(_MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
    with open(os.path.join(CSRC, "flow_plan.cu")) as f:
        plan = f.read()
    assert "INT32_MAX" not in plan and "flow_entry(S.z_elems)" in plan
