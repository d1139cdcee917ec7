"""What the launchers do once (csrc/per_device.h): once per device, not per process, and again after a failure.  The header is plain C++, so it is
compiled and run here; that the launchers of kernels which always need an attribute use it is read from their sources."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torchao_fork_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
  static ao::OncePerDevice once;
  static ao::NumberPerDevice number;
  int calls[70] = {}, bad = 0;
  auto set = [&](int d, int status) { return once.run(d, [&] { ++calls[d]; return status; }); };
  bad += set(0, 7) != 7 || set(0, 0) != 0 || set(0, 9) != 0 || calls[0] != 2;   // a failure is not remembered
  for (int d = 1; d < 4; ++d) bad += set(d, 0) != 0 || set(d, 5) != 0 || calls[d] != 1;
  bad += set(69, 0) != 0 || set(69, 3) != 3 || calls[69] != 2;                  // beyond the table: every time
  for (int d = 0; d < 4; ++d) bad += number.get(d, [&] { return 10 + d; }) != 10 + d || number.get(d, [] { return 99; }) != 10 + d;
  bad += number.get(5, [] { return -1; }) != -1 || number.get(5, [] { return 99; }) != -1;
  std::vector<std::thread> threads;
  std::atomic<int> wrong{0};
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&] {
      for (int i = 0; i < 1000; ++i)
        if (number.get(10 + i % 20, [&] { return 1 + i % 20; }) != 1 + i % 20) ++wrong;
    });
  for (auto& t : threads) t.join();
  std::printf("%d %d\n", bad, (int)wrong);
  return bad || wrong;
}
"""


def test_once_is_once_per_device(tmp_path):
    (tmp_path / "once.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(tmp_path / "once.cpp"), "-o", str(tmp_path / "once")], check=True)
    r = subprocess.run([str(tmp_path / "once")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("source", ["gemv_int4_fused.cu", "gemv_int8_fused.cu", "gemm_wq_tc.cu", "gemv_stage.cuh", "lm/lm_window_attention_tc.cu"])
def test_launchers_keep_no_flag_for_all_devices(source):
    text = open(os.path.join(CSRC, source)).read()
    assert not re.findall(r"static (?:bool|int) \w*(?:done|set|at_once)\w*(?:\[[^\]]*\])? *=", text)
    assert text.count("cudaFuncAttributeMaxDynamicSharedMemorySize") == 0
