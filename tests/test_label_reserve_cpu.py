"""The label workspace that a sparse handle reserves for its lanes is a
convenience: short of memory the factorization takes two labels a row, block by
block, so neither the reservation nor the larger buffer may end the call. Read
from the source: an allocation that fails in the middle of a handle's creation
cannot be arranged on a shared device."""

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "algebra_linear_b200" / "csrc"


def test_reservation_failures_are_not_returned():
    init = (CSRC / "sparse_numeric.cu").read_text()
    init = init[init.index("int DeviceLu::init"):]
    init = init[:init.index("\n}\n")]
    uses = re.findall(r"^.*WS_LAB.*$", init, re.M)
    assert uses and not any("ALG_TRY" in u for u in uses)


def test_the_factorization_falls_back_to_two_labels_a_row():
    lu = (CSRC / "dense.cu").read_text()
    lu = lu[lu.index("int lu_factor_partial_dev"):]
    first, second = [m for m in re.finditer(r"^.*WS_LAB.*$", lu, re.M)][:2]
    assert "ALG_TRY" not in first.group() and "lu_label_bytes" in first.group()
    assert "if (!at_end) ALG_TRY" in second.group() and "2 * sizeof(int)" in second.group()
