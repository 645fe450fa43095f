"""The small-front kernel at the edges of its panel (16 columns), tile and row
classes (64, 128, 256 rows): dense patterns (one front without a contribution
block) and bordered block diagonals (fronts that pass one up), with values that
make the pivots move rows.

The bound is the repository's FP64 backward error 10 n 2^-53 (Gaussian
elimination with partial pivoting at moderate growth); the FP32 form refines to
it without falling back to FP64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csc(mask):
    c, r = np.nonzero(mask.T)
    cp = np.concatenate([[0], np.cumsum(mask.sum(axis=0))]).astype(np.uint64)
    return cp, r.astype(np.uint64), c


def _solve(mask, seed, precision):
    from algebra_linear_b200.sparse import LuMethod, SparseLu

    n = mask.shape[0]
    rng = np.random.default_rng(seed)
    A = np.where(mask, rng.uniform(-1.0, 1.0, (n, n)), 0.0)
    A[np.arange(n), rng.permutation(n)] += np.where(mask.all(), np.sqrt(n), 0.0)
    A[np.arange(n), np.arange(n)] += 0.0 if mask.all() else 2.0
    cp, r, c = _csc(mask)
    b = A @ rng.uniform(-1.0, 1.0, n)
    lu = SparseLu.analyze(cp, r, LuMethod.supernodal())
    lu.set_precision(precision)
    outs = []
    for _ in range(2):  # a refactorization repeats the bits
        lu.factorize(cp, r, A[r.astype(int), c])
        x = b.copy()
        lu.solve(x)
        outs.append(x)
    assert np.array_equal(outs[0].view(np.uint64), outs[1].view(np.uint64))
    eta = np.abs(b - A @ x).max() / (np.abs(A).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())
    assert eta <= 10 * n * 2.0**-53
    if precision != "fp64":
        assert not lu.last_solve()["fell_back"]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [1, 3, 15, 16, 17, 33, 63, 64, 65, 127, 128, 129, 191, 255, 256, 257])
def test_dense_patterns(gpu, n, precision):
    _solve(np.ones((n, n), bool), n, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("blocks,border", [((20, 33), 7), ((50, 64, 65), 30), ((100, 90, 128), 61), ((16, 16, 16, 16), 190)])
def test_bordered_blocks(gpu, blocks, border, precision):
    n = sum(blocks) + border
    mask = np.zeros((n, n), bool)
    k = 0
    for w in blocks:
        mask[k:k + w, k:k + w] = True
        k += w
    mask[k:, :] = True
    mask[:, k:] = True
    _solve(mask, n, precision)
