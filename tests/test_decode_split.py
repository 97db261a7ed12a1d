"""How decode attention shares out a cache (csrc/decode_split.h), compiled for the host: every block counted has rows, whole row
steps but for the last one's, never more blocks than a launch sized for a longer cache, more than eight only where all of
them have the least rows, on devices (here ones that only answer) that hold such a cluster, and one of a short cache whose pairs fill the device."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cassert>
#include <thread>
#include <vector>
#include "decode_split.h"
using namespace cdeep;
static void check(const DecodeSplit& rule, int most, int rows) {
  assert(rule.blocks(0) == 1 && rule.bound(0) == 1);
  int before = 1;
  for (int L = 1; L <= rows; ++L) {
    const int bound = rule.bound(L), chunk = rule.chunk(L), blocks = rule.blocks(L);
    assert(bound >= before && bound <= most && blocks >= 1 && blocks <= bound);
    assert(chunk % 16 == 0 && (blocks - 1) * chunk < L && L <= blocks * chunk);
    before = bound;
  }
  assert(before == most);
}
int main() {
  for (int most = 1; most <= kMaxSplits; ++most) {
    DecodeSplit rule;
    rule.most = most;
    rule.large_from = 48 * most;
    check(rule, most, 6000);
    for (int L = 1; L <= 6000; ++L) assert(rule.bound(L) <= kPortable || (rule.bound(L) == most && L > 48 * (most - 1)));
    rule.many = 40;
    rule.many_from = 3000;
    check(rule, 40, 6000);
  }
  const short active[] = {592, 296, 187, 142, 112};
  for (int pairs = 297; pairs <= 3000; ++pairs) {
    const DecodeSplit rule = split_of_waves(pairs, active);
    check(rule, rule.most, 1 << 16);
    assert(rule.most <= 5 && rule.bound(64) == 1);
  }
  assert(split_of_waves(384, active).bound(2064) == 1 && split_of_waves(768, active).bound(2064) == 2 && split_of_waves(640, active).bound(4096) == 4);
  DeviceNumber number;
  int asked = 0, holds = 16;
  auto most = [&](int device) { return number.get(device, [&] { return largest_cluster([&](int n) { ++asked; return n <= holds; }); }); };
  assert(most(0) == 16 && asked == 1);
  holds = 8;
  assert(most(0) == 16 && asked == 1);          // of a device that was asked
  assert(most(1) == 8 && asked == 3);           // another one
  assert(most(1) == 8 && asked == 3);
  holds = 14;
  assert(most(2) == 13 && most(1000) == 13 && most(-1) == 13);
  DeviceNumber none;                            // nothing at all is an answer, too
  for (int i = 0; i < 2; ++i) assert(none.get(3, [&] { ++asked; return 0; }) == 0);
  assert(asked == 10);
  DeviceNumber shared;
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&] {
      for (int i = 0; i < 2000; ++i) assert(shared.get(i % 64, [] { return 13; }) == 13);
    });
  for (auto& t : threads) t.join();
  return 0;
}
"""


def test_every_block_has_rows(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "split.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "split")
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "complexity_deep_b200", "csrc"), str(src), "-o", exe],
                   check=True)
    subprocess.run([exe], check=True, timeout=60)
