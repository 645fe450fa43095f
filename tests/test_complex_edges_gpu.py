"""Complex panels and sweeps where their kernels change: the most rows a panel
holds in shared memory and the first beyond it, in the first block and in a
later one, a zero pivot inside such a panel, and solves at the edges of the
sweeps' blocks. Bit for bit against the oracle (the tolerance is zero)."""

import numpy as np
import pytest

from algebra_linear_b200.lapack import LapackError, zgesv, zgetrf, zgetrf_rect

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oz(oracle):
    from oracle import complex as oz

    return oz


def rand(count, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(count) + 1j * rng.standard_normal(count)


def same(x, y):
    return np.array_equal(x.view(np.float64), y.view(np.float64), equal_nan=True)


@pytest.mark.parametrize("rows,cols", [(880, 16), (881, 16), (900, 40), (939, 15), (17, 17), (385, 33)])
def test_panel_in_and_beyond_shared_memory(gpu, oz, rows, cols):
    a = rand(rows * cols, rows + cols)
    rc, lu_ref, ipiv_ref = oz.zgetrf_rect(a, rows, cols)
    assert rc == oz.OK
    ipiv = [0] * cols
    zgetrf_rect(a, rows, cols, ipiv)
    assert ipiv == [int(v) for v in ipiv_ref]
    assert same(a, lu_ref)


def test_zero_pivot_inside_a_panel_in_shared_memory(gpu, oz):
    n = 60
    a = rand(n * n, 5).reshape(n, n)
    a[37] = 0.0  # column 37
    a = a.reshape(-1).copy()
    rc, lu_ref, _ = oz.zgetrf(a, n)
    assert rc != oz.OK
    with pytest.raises(LapackError):
        zgetrf(a, n)
    assert same(a, lu_ref)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 129])
def test_sweeps_at_block_edges(gpu, oz, n):
    a, b = rand(n * n, n), rand(n, n + 1)
    rc, lu_ref, x_ref, _ = oz.zgesv(a, b)
    assert rc == oz.OK
    zgesv(a, b)
    assert same(a, lu_ref) and same(b, x_ref)
