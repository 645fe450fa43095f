"""Row numbers that a timed-out panel may leave unset or stale are checked
where they become an index, so that the launch ends and the call reports the
timeout. The check (csrc/index_guard.h, plain C++) is compiled and run here on
labels left by a larger matrix; that the kernels use it is read from the source."""

import pathlib
import re
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "algebra_linear_b200" / "csrc"
KERNELS = re.sub(r"//[^\n]*", "", (CSRC / "dense_kernels.cuh").read_text())

PROGRAM = r"""
#include <climits>
#include <cstdio>
#include "index_guard.h"

int main() {
  using alg::index_or;
  const int n = 300, k0 = 128;
  const int stale[] = {INT_MIN, -1, 0, 127, 128, 200, 299, 300, 301, 16383, 1 << 20, INT_MAX};
  for (int label : stale)
    for (int r = k0; r < n; ++r) {
      const int s = index_or(label, k0, n, r);
      if (s < k0 || s >= n) return 1;                            // stays among the rows that move
      if (s != (label >= k0 && label < n ? label : r)) return 2;  // and changes no valid label
    }
  return 0;
}
"""


def test_index_or(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


def _kernel(name):
    body = KERNELS[KERNELS.index(name + "("):]
    return body[:body.index("__global__")]


@pytest.mark.parametrize("kernel,uses", [
    ("laswp_outside_kernel", r"(\w+)\(lab\[r\], k0, n, r\)"),
    ("compose_swaps_kernel", r"(\w+)\(lab\[\(size_t\)b \* n \+ s\], b \* nb, n, s\)"),
    ("panel_cluster_kernel", r"loc_s\[r\] = (\w+)\(loc_s\[r\], p\.c0, p\.n, p\.c0 \+ rb \+ r\)"),
])
def test_labels_are_checked_before_they_index(kernel, uses):
    found = re.findall(uses, _kernel(kernel))
    assert found == ["index_or"]


def test_panel_positions_and_slots_are_checked():
    # a record that another CTA sent out of step: its slot before it addresses
    # the tile, the rows' positions before the rows are written there
    body = _kernel("panel_reg_kernel")
    assert re.findall(r"slot = ok_wait \? (\w+)\(\(int\)wr\.slot, 0, ldt, 0\)", body) == ["index_or"]
    check = re.search(r"pos\[k\] = index_or\(pos\[k\], 0, m, rb \+ r\)", body)
    assert check
    for use in (r"side_dst\[s\] = p\.c0 \+ pos\[k\]", r"p\.a \+ \(size_t\)\(p\.c0 \+ pos\[k\]\)", r"p\.lab\[p\.c0 \+ pos\[k\]\]"):
        assert re.search(use, body).start() > check.start()
