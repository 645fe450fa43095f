"""Tournament pivoting where it runs: panels of more than 8 192 rows (shorter
ones fit one cluster, whose partial pivoting is a tree of one node). n = 8300:
the first 108 columns, so the tree hands over to the cluster's 64-column panel
inside the first block; n = 9001: several blocks by the tree, then the
hand-over inside the fourth (FP32: the seventh); n = 8200: one leaf.

The bars are those of the mixed form: plain refinement, at most 8 steps, to the
FP64 backward error 10 n 2^-53. That the tree runs shows in the solution's
bits, which depend on the FP32 factors: they differ from partial pivoting's
where it runs, and at 8 192 rows, where it does not, they are the same."""

import pytest

pytestmark = pytest.mark.gpu


def _system(ctx, n):
    a, s = ctx.larnv(2, [3, 1, 4, 1], n * n)
    xt, _ = ctx.larnv(2, s, n)
    return a.clone(), a.view(n, n).t() @ xt


def _solve(ctx, a, b, n, prec, pivoting):
    from algebra_linear_b200 import mixed

    x = b.clone()
    rep = mixed.dgesv_mixed_dev(ctx, a, x, n, 1, precision=prec, pivoting=pivoting, no_gmres=True, no_fallback=True)
    return x, rep


@pytest.mark.parametrize("prec", ["fp32", "tf32x3"])
@pytest.mark.parametrize("n", [8192, 8200, 8300, 9001])
def test_tree_and_hand_over(gpu, n, prec):
    import torch

    from algebra_linear_b200 import device

    with device.Context() as ctx:
        a, b = _system(ctx, n)
        x, rep = _solve(ctx, a, b, n, prec, "tournament")
        assert rep["tournament"] and rep["path"] == "ir" and rep["ir_iterations"] <= 8, rep
        m = a.view(n, n).t()
        eta = (b - m @ x).abs().max() / (m.abs().sum(dim=1).max() * x.abs().max() + b.abs().max())
        assert float(eta) <= 10 * n * 2.0**-53
        again, _ = _solve(ctx, a, b, n, prec, "tournament")
        assert torch.equal(x.view(torch.int64), again.view(torch.int64))
        part, prep = _solve(ctx, a, b, n, prec, "partial")
        assert not prep["tournament"]
        assert torch.equal(x.view(torch.int64), part.view(torch.int64)) == (n == 8192)


def test_tree_on_columns_in_need_of_interchanges(gpu):
    """The large entry of each column sits in a row of its own, in random order:
    the tree has to find it among all the groups' candidates."""
    import torch

    from algebra_linear_b200 import device

    n = 9001
    g = torch.Generator(device="cuda").manual_seed(7)
    a = torch.rand((n, n), generator=g, dtype=torch.float64, device="cuda") * 2.0 - 1.0
    a[torch.arange(n, device="cuda"), torch.randperm(n, generator=g, device="cuda")] = n**0.5
    xt = torch.rand(n, generator=g, dtype=torch.float64, device="cuda") * 2.0 - 1.0
    b = a.t() @ xt  # (a: column-major storage)
    with device.Context() as ctx:
        x, rep = _solve(ctx, a.reshape(-1), b, n, "tf32x3", "tournament")
    assert rep["tournament"] and rep["path"] == "ir" and rep["ir_iterations"] <= 8, rep
    m = a.t()
    eta = (b - m @ x).abs().max() / (m.abs().sum(dim=1).max() * x.abs().max() + b.abs().max())
    assert float(eta) <= 10 * n * 2.0**-53
