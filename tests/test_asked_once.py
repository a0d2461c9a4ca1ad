"""bf_once.h: a query of the device that fails once is not remembered as its answer."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "bf_once.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
  bf::AskedOnce<int> clusters;
  int asked = 0, n = -1;
  auto fails = [&](int *k) { ++asked; *k = 0; return 2; };
  auto works = [&](int *k) { ++asked; *k = 76; return 0; };
  if (clusters.get(&n, fails) != 2 || n != -1) return 1;    // reported, and no answer given
  if (clusters.get(&n, fails) != 2 || asked != 2) return 2;  // asked again
  if (clusters.get(&n, works) != 0 || n != 76) return 3;
  if (clusters.get(&n, fails) != 0 || n != 76 || asked != 3) return 4;  // kept from here on
  bf::AskedOnce<int> shared;
  int count = 0;
  std::vector<std::thread> th;
  std::vector<int> got(8, -1);
  for (int i = 0; i < 8; ++i)
    th.emplace_back([&, i] { shared.get(&got[i], [&](int *k) { ++count; *k = 5; return 0; }); });
  for (auto &t : th) t.join();
  for (int g : got) if (g != 5) return 5;
  return count == 1 ? 0 : 6;
}
"""


def test_a_failed_query_is_asked_again(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I",
                    os.path.join(ROOT, "beamforming_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_device_queries_go_through_it():
    """No count of SMs or clusters is kept in a function's static of its own."""
    for name in ("bf_api.cu", "bf_tc.cu", "bf_tc_pair.cu"):
        text = open(os.path.join(ROOT, "beamforming_gb300", "csrc", name)).read()
        assert "static const int" not in text, name
