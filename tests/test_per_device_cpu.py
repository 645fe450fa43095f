"""Kernel attributes are set per device: a process with one context per device
(a replica per GPU, one host thread each) needs them on every device it uses.

The table that keeps track (csrc/per_device.h, plain C++) is compiled and run
here with made-up device numbers; the sources are read for attributes that are
set once per process instead."""

import pathlib
import re
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "algebra_linear_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
  alg::PerDevice p;
  int v = 0, runs[3] = {0, 0, 0};
  auto on = [&](int d) { return p.get(d, v, [&](int& value) { ++runs[d]; value = 100 + d; return 0; }); };
  // each of two devices once, each with its own value
  for (int i = 0; i < 3; ++i) {
    CHECK(on(0) == 0 && v == 100);
    CHECK(on(1) == 0 && v == 101);
  }
  CHECK(runs[0] == 1 && runs[1] == 1);
  // a failure is handed on and tried again
  alg::PerDevice q;
  int tries = 0;
  CHECK(q.get(1, v, [&](int&) { ++tries; return 7; }) == 7);
  CHECK(q.get(1, v, [&](int&) { ++tries; return 0; }) == 0 && v == 1);
  CHECK(q.get(1, v, [&](int&) { ++tries; return 7; }) == 0 && tries == 2);
  // devices past the table's end: every call
  int far = 0;
  for (int i = 0; i < 2; ++i) CHECK(q.get(100000, v, [&](int&) { ++far; return 0; }) == 0);
  CHECK(far == 2);
  // several threads on two devices: once each
  alg::PerDevice r;
  std::atomic<int> n{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&, t] {
      int w = 0;
      for (int i = 0; i < 1000; ++i) r.get(t % 2, w, [&](int&) { ++n; return 0; });
    });
  for (auto& t : ts) t.join();
  CHECK(n == 2);
  return 0;
}
"""


def test_once_per_device(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-pthread", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_no_attribute_is_set_once_per_process(src):
    text = (CSRC / src).read_text()
    # (a function-local static that holds a CUDA result or an occupancy figure)
    assert not re.search(r"static\s+(const\s+)?cudaError_t", text)
    for m in re.finditer(r"static\s+(?:const\s+)?int\s+(\w+)\s*=", text):
        body = text[m.end():m.end() + 600]
        assert "cudaOccupancy" not in body.split("\n}")[0], m.group(1)
