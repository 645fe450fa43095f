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


@pytest.mark.parametrize("nb,n", [(17, 90), (31, 95), (32, 1200), (33, 150), (65, 200), (97, 1300), (127, 400)])
def test_triangular_solve_edges(gpu, oracle, monkeypatch, nb, n):
    """Block rows of every row-group count with ragged last groups, few and
    many columns right of the block."""
    monkeypatch.setenv("ALG_NB", str(nb))
    check(oracle, np.random.default_rng(nb + n).uniform(-1.0, 1.0, n * n), n, n)


@pytest.mark.parametrize("rows,cols", [(129, 129), (193, 193), (400, 257), (1031, 1031), (22000, 300)])
def test_left_columns_permuted_at_the_end(gpu, oracle, rows, cols):
    """Three and more blocks with many interchanges: the columns left of a
    block are permuted after the last one, from the blocks' composed labels (a
    last block of one column, square and tall; nearly the most rows an FP64
    panel takes)."""
    rng = np.random.default_rng(rows + cols)
    a = rng.uniform(-1.0, 1.0, (cols, rows)) * rng.permutation(np.geomspace(1.0, 2.0**20, rows))
    check(oracle, a.reshape(-1).copy(), rows, cols)


@pytest.mark.parametrize("lda_off,a_off", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 65, 15), (64, 32, 16), (65, 33, 17), (200, 130, 64), (2100, 2051, 40),
                                   (4200, 1100, 129)])
def test_fused_update_edges(gpu, m, n, k, lda_off, a_off):
    """C -= A B at the tile edges of both tile shapes, with aligned operands
    (16-byte copies) and not. Bound: k + 1 roundings of the entry's terms,
    gamma_{k+1} (|C| + |A| |B|)."""
    import torch

    from algebra_linear_b200 import _lib
    from algebra_linear_b200.device import Context

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    lda = m + (m & 1) + lda_off
    ldb = k + (k & 1) + lda_off
    u = lambda cnt: torch.rand(cnt, generator=g, dtype=torch.float64, device="cuda") * 2 - 1  # noqa: E731
    A, B, Cm = u(lda * k + a_off), u(ldb * n + a_off), u(m * n)
    ref_a = A[a_off:].as_strided((k, m), (lda, 1))
    ref_b = B[a_off:].as_strided((n, k), (ldb, 1))
    C0 = Cm.view(n, m).clone()
    with Context() as ctx:
        rc = _lib.load().alg_gemm_dmma_sub_dev(ctx.handle, m, n, k, A.data_ptr() + 8 * a_off, lda,
                                               B.data_ptr() + 8 * a_off, ldb, Cm.data_ptr(), m)
        assert rc == 0
    gamma = (k + 2) * 2.0**-53
    bound = 2 * gamma * (C0.abs() + ref_b.abs() @ ref_a.abs())
    assert ((Cm.view(n, m) - (C0 - ref_b @ ref_a)).abs() <= bound + 1e-300).all()


@pytest.mark.parametrize("n", [130, 1999])
def test_exact_update_with_odd_strides_bit_identical(gpu, oracle, n):
    """The exact update's element-wise copies (odd leading dimension) and its
    16-byte ones (even) give the oracle's bits; n = 1999 has both tile shapes."""
    import torch

    from algebra_linear_b200 import _lib
    from algebra_linear_b200.device import Context

    a = np.random.default_rng(n).uniform(-1.0, 1.0, n * n)
    ra = a.copy()
    rc, rpiv, _, _ = oracle.dgetrf(ra, n)
    assert rc == 0
    for lda in (n, n + 1):
        A = torch.zeros(lda * n, dtype=torch.float64, device="cuda")
        A.view(n, lda)[:, :n] = torch.from_numpy(a).cuda().view(n, n)
        ipiv = torch.empty(n, dtype=torch.int32, device="cuda")
        with Context() as ctx:
            assert _lib.load().alg_dgetrf_dev(ctx.handle, 0, A.data_ptr(), n, lda, ipiv.data_ptr(), None) == 0
        assert ipiv.cpu().tolist() == list(rpiv)
        got = A.view(n, lda)[:, :n].contiguous().view(-1).cpu().numpy()
        assert same_bits(got, ra)
