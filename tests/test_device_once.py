"""Per-device settings of a process (csrc/tmk_once.h), compiled for the host: set
once on each device, again until it succeeds, and safe from several threads."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "tmk_once.h"
#include <thread>
#include <vector>
int main() {
  tmk::DeviceOnce once;
  int calls = 0;
  auto good = [&] { ++calls; return 0; };
  auto bad = [&] { ++calls; return 7; };
  if (once(0, bad) != 7 || calls != 1) return 1;          // a failure is handed on
  if (once(0, good) != 0 || calls != 2) return 2;         // and not kept
  if (once(0, bad) != 0 || calls != 2) return 3;          // success is
  if (once(1, good) != 0 || calls != 3) return 4;         // for its device alone
  if (once(1, good) != 0 || once(0, good) != 0 || calls != 3) return 5;
  if (once(63, good) != 0 || once(63, good) != 0 || calls != 4) return 6;
  if (once(64, good) != 0 || once(64, good) != 0 || calls != 6) return 7;   // beyond those kept: every time
  std::atomic<int> n{0};
  tmk::DeviceOnce both;
  std::vector<std::thread> t;
  for (int k = 0; k < 8; ++k)
    t.emplace_back([&, k] { for (int i = 0; i < 1000; ++i) both(k & 3, [&] { ++n; return 0; }); });
  for (auto& x : t) x.join();
  return n >= 4 && n <= 8 ? 0 : 8;
}
"""


def test_settings_are_made_once_per_device(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "once.cpp", str(tmp_path / "once")
    src.write_text(PROGRAM)
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-pthread", "-I",
                        os.path.join(ROOT, "tetemoko_gb300", "csrc"), str(src), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert subprocess.run([exe]).returncode == 0


def test_no_other_state_says_that_a_device_is_configured():
    """Every shared memory limit above the default goes through that class or is set on each call."""
    csrc = os.path.join(ROOT, "tetemoko_gb300", "csrc")
    for f in os.listdir(csrc):
        text = open(os.path.join(csrc, f)).read()
        assert "configured" not in text, f
        if f != "tmk_device.cuh":
            assert "cudaFuncSetAttribute" not in text, f
