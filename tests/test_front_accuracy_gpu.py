"""Small fronts whose contribution block is much larger than the products
subtracted from it: identity blocks bordered by rows and columns, with border
rows of p = 0.4 ulp(1.5) and border columns of ones, so that the Schur
complement is 1.5 I - S p J (S block columns, J all ones).

Each product alone is less than half a unit of 1.5: subtracted one by one,
every one is lost. The front's bound is one rounding of an entry per panel of
16 columns: with u the unit roundoff (1.5 has rounding unit u, in absolute terms)
an entry is off by at most `panels` u, and a component of the border's x, of
size at most one, by panels u / 1.5 plus the solve's own few roundings (the
quotient, the tiny off-diagonal terms, the assembled residual): 8 u."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,unit", [("fp64", 2.0**-53), ("fp32", 2.0**-24)])
@pytest.mark.parametrize("blocks,border", [((48, 33), 5), ((100, 90), 30), ((60, 64, 65), 17), ((100, 60), 90)])
def test_contribution_block_rounds_once_per_panel(gpu, blocks, border, precision, unit):
    from algebra_linear_b200.sparse import LuMethod, SparseLu

    S = sum(blocks)
    n = S + border
    mask = np.zeros((n, n), bool)
    k = 0
    for w in blocks:
        mask[k:k + w, k:k + w] = True
        k += w
    mask[S:, :] = True
    mask[:, S:] = True
    p = float(np.float32(0.8)) * unit  # 0.4 ulp(1.5), exact in either precision
    A = np.zeros((n, n))
    A[np.arange(S), np.arange(S)] = 1.0
    A[:S, S:] = 1.0
    A[S:, :S] = p
    A[np.arange(S, n), np.arange(S, n)] = 1.5
    c, r = np.nonzero(mask.T)
    cp = np.concatenate([[0], np.cumsum(mask.sum(axis=0))]).astype(np.uint64)
    r = r.astype(np.uint64)

    lu = SparseLu.analyze(cp, r, LuMethod.supernodal())
    assert sorted(lu.symbolic()["col_perm"][S:]) == list(range(S, n))  # the border is eliminated last
    lu.set_precision(precision, tol=1.0)  # FP32: the first solution, unrefined
    lu.factorize(cp, r, A[r.astype(int), c])
    assert lu.plan()["max_front_rows"] <= 256
    b = np.zeros(n)
    b[S:] = np.linspace(0.5, 1.0, border).astype(np.float32)
    x = b.copy()
    lu.solve(x)

    bl = b[S:].astype(np.longdouble)
    d = S * np.longdouble(p)
    want = (bl + d * bl.sum() / (np.longdouble(1.5) - border * d)) / np.longdouble(1.5)
    panels = sum(-(-w // 16) for w in (*blocks, border))
    err = float(np.abs(x[S:] - want).max())
    assert err <= (panels / 1.5 + 8.0) * unit, err / unit
