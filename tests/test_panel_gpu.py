"""The block panel kernel at the edges of its range: the rows a CTA, a thread
and the cluster hold, ragged leaves and blocks, and entries that take its rare
branches. The exact form must give the oracle's pivots and factors bit for bit
(it performs the same rounded operations on every entry, so the tolerance is
zero)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (rows, columns): one CTA of 128 / 256 threads; the first clusters; odd row
# counts per CTA; two rows per thread; a block that no longer fits (leaf by
# leaf); three rows per thread; the shared-memory slab beyond 16 384 rows
SHAPES = [(1, 1), (16, 16), (17, 17), (128, 64), (129, 65), (256, 63), (257, 64), (1031, 129), (4096, 20), (4097, 64),
          (6128, 66), (6160, 64), (8193, 17), (16384, 16), (16385, 18)]


def same_bits(x, y):
    return np.array_equal(x.view(np.uint64), y.view(np.uint64))


def check(oracle, a, rows, cols):
    from algebra_linear_b200.lapack import dgetrf_rect

    ra = a.copy()
    rc, rpiv = oracle.dgetrf_rect(ra, rows, cols)
    assert rc == 0
    ipiv = [0] * cols
    dgetrf_rect(a, rows, cols, ipiv)
    assert ipiv == list(rpiv)
    assert same_bits(a, ra)


@pytest.mark.parametrize("rows,cols", SHAPES)
def test_panel_edges_bit_identical(gpu, oracle, rows, cols):
    a = np.random.default_rng(rows * 131 + cols).uniform(-1.0, 1.0, rows * cols)
    check(oracle, a, rows, cols)


@pytest.mark.parametrize("rows,cols", [(100, 40), (700, 64), (4500, 70)])
def test_panel_ties_zeros_and_extreme_exponents(gpu, oracle, rows, cols):
    """Few distinct values (exact pivot ties between rows of different CTAs),
    zeros of both signs, and entries whose quotients leave the fast division's
    exponent range."""
    rng = np.random.default_rng(rows)
    a = rng.choice([0.0, -0.0, 0.5, -0.5, 1.0, -1.0, 2.0], rows * cols)
    scale = rng.choice([1.0, 1.0, 1.0, 1.0, 1e-160, 1e155], rows)
    a = (a.reshape(cols, rows) * scale).reshape(-1)
    check(oracle, a, rows, cols)


@pytest.mark.parametrize("nb", [48, 128])
def test_blocks_wider_and_narrower_than_a_launch(gpu, oracle, monkeypatch, nb):
    """Block panels of 128 columns take two launches, whose interchanges also
    move the other half; 48 is a ragged number of leaves."""
    monkeypatch.setenv("ALG_NB", str(nb))
    rows = cols = 523
    a = np.random.default_rng(nb).uniform(-1.0, 1.0, rows * cols)
    check(oracle, a, rows, cols)
