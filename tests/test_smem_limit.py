"""The record of how much dynamic shared memory a kernel was allowed (csrc/smem_limit.h), with a driver that only counts:
two devices in one process, a limit that grows, a refusal, and threads that ask for different sizes at once."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cassert>
#include <thread>
#include <vector>
#include "smem_limit.h"
int main() {
  cdeep::SmemLimit limit;
  int given[3] = {0, 0, 0}, asked = 0, fail = 0;
  auto raise = [&](int device, int bytes) {
    return limit.raise(device, bytes, [&](int n) {
      ++asked;
      if (fail) return fail;
      given[device < 2 ? device : 2] = n;
      return 0;
    });
  };
  assert(raise(0, 70000) == 0 && given[0] == 70000 && asked == 1);
  assert(raise(0, 60000) == 0 && given[0] == 70000 && asked == 1);   // already allowed
  assert(raise(1, 60000) == 0 && given[1] == 60000 && asked == 2);   // another device has a limit of its own
  assert(raise(0, 80000) == 0 && given[0] == 80000 && asked == 3);
  fail = 7;
  assert(raise(1, 90000) == 7 && asked == 4);
  fail = 0;
  assert(raise(1, 90000) == 0 && given[1] == 90000 && asked == 5);   // a refusal is not remembered
  assert(raise(1000, 50000) == 0 && raise(1000, 50000) == 0 && given[2] == 50000 && asked == 7);
  cdeep::SmemLimit shared;
  int last = 0;                                                       // written under the record's lock
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int i = 0; i < 2000; ++i) {
        const int want = 1 + (i * 37 + t * 101) % 5000;
        assert(shared.raise(0, want, [&](int n) { assert(n > last); last = n; return 0; }) == 0);
      }
    });
  for (auto& t : threads) t.join();
  assert(last == 5000 || last > 4900);
  return 0;
}
"""


def test_limits_are_kept_by_device(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "limit.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "limit")
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "complexity_deep_b200", "csrc"), str(src), "-o", exe],
                   check=True)
    subprocess.run([exe], check=True, timeout=60)


def test_no_kernel_keeps_its_limit_for_the_whole_process():
    """Whoever asks the driver itself does so at every launch or by device; a flag of the process would be true on the
    second device before it was asked."""
    csrc = os.path.join(ROOT, "complexity_deep_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        if name.endswith((".cu", ".cuh", ".h")):
            text = open(os.path.join(csrc, name)).read()
            assert "static bool attr" not in text and "static std::atomic<int> allowed" not in text, name
