"""cta_leaf sends the warps without rows through a loop of their own, so its
barrier is met at two places in the code: that has to be the numbered barrier,
not __syncthreads, which the whole block must meet at one place. Read from the
source."""

import pathlib
import re

SRC = (pathlib.Path(__file__).resolve().parent.parent / "algebra_linear_b200" / "csrc" / "pivot.cuh").read_text()
CODE = re.sub(r"//[^\n]*", "", SRC)


def test_cta_leaf_uses_the_numbered_barrier():
    leaf = CODE[CODE.index("int cta_leaf("):]
    assert "__syncthreads" not in leaf
    # once per column in each of the two loops, the barrier of all NT threads
    assert leaf.count("cta_barrier<NT>()") == 2
    assert re.search(r"cta_barrier\(\) \{\s*asm volatile\(\"barrier\.sync\.aligned 1, %0;\" ::\"n\"\(NT\) : \"memory\"\)", CODE)
