"""The mixed batched form (FP32 factors, FP64 refinement) on systems whose rows
move: U(-1, 1) with one entry of size sqrt(n) per column in a row of its own,
rows in random order, so that the factors need interchanges in every panel and
FP32 is precise enough to refine from. A wrong row order, though repeatable,
would not converge to the right solution.

Bars: info 0, the plan's normwise backward error 10 n 2^-53 (its own residual
and this file's differ by at most the rounding of a residual, (n + 2) 2^-53), and
interchanges that really move rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 95, 97, 128, 129, 160, 161, 255, 256, 257, 289, 511, 512]


@pytest.mark.parametrize("threads,panel", [(None, None), (128, 16), (128, 32), (256, 16), (256, 32), (512, 16), (512, 32)])
def test_interchanged_systems_refine(gpu, threads, panel):
    import torch

    from algebra_linear_b200.batched import BatchPlan
    from algebra_linear_b200.device import Context

    rng = np.random.default_rng(11)
    with Context() as ctx:
        plan = BatchPlan(ctx, ORDERS, mixed=True)
        if threads is not None:
            for i in range(len(plan.info()["buckets"])):
                assert plan._lib.alg_batch_set_config(plan.handle, i, threads, panel) == 0
        a0, b0 = np.empty(plan.a_total), np.empty(plan.b_total)
        mats = []
        for k, n in enumerate(ORDERS):
            m = rng.uniform(-1.0, 1.0, (n, n))
            m[rng.permutation(n), np.arange(n)] = 2.0 * np.sqrt(n)
            mats.append(m)
            a0[plan.a_off[k]:plan.a_off[k] + n * n] = m.T.reshape(-1)
            b0[plan.b_off[k]:plan.b_off[k] + n] = m @ rng.uniform(-1.0, 1.0, n)
        a, b = torch.from_numpy(a0).cuda(), torch.from_numpy(b0).cuda()
        info = torch.full((len(ORDERS),), -7, dtype=torch.int32, device="cuda")
        plan.solve(a, b, info)
        torch.cuda.synchronize()
        x, piv, eta = b.cpu().numpy(), plan.ipiv(), plan.eta()
        assert np.array_equal(a.cpu().numpy(), a0)  # the mixed form leaves A
        assert (info.cpu().numpy() == 0).all()
        bo = plan.b_off.copy()
        plan.close()
    u = 2.0**-53
    for k, n in enumerate(ORDERS):
        sl = slice(bo[k], bo[k] + n)
        p = piv[sl]
        assert ((p >= np.arange(n)) & (p < n)).all()
        if n >= 15:
            assert (p != np.arange(n)).sum() >= n // 2
        m, xk, bk = mats[k], x[sl], b0[sl]
        e = np.abs(bk - m @ xk).max() / (np.abs(m).sum(axis=1).max() * np.abs(xk).max() + np.abs(bk).max())
        assert eta[k] <= 10 * n * u and e <= (11 * n + 2) * u, (n, e / u, eta[k] / u)


def test_repeated_runs_report_success(gpu):
    import torch

    from algebra_linear_b200.batched import BatchPlan
    from algebra_linear_b200.device import Context

    rng = np.random.default_rng(3)
    orders = rng.integers(60, 200, 300)
    with Context() as ctx:
        plan = BatchPlan(ctx, orders, mixed=True)
        a0, b0 = np.empty(plan.a_total), rng.uniform(-1.0, 1.0, plan.b_total)
        for k, n in enumerate(orders):
            m = rng.uniform(-1.0, 1.0, (n, n))
            m[rng.permutation(n), np.arange(n)] = 2.0 * np.sqrt(n)
            a0[plan.a_off[k]:plan.a_off[k] + n * n] = m.T.reshape(-1)
        a = torch.from_numpy(a0).cuda()
        first = None
        for _ in range(3):
            b = torch.from_numpy(b0).cuda()
            info = torch.full((len(orders),), -7, dtype=torch.int32, device="cuda")
            plan.solve(a, b, info)
            assert int(info.abs().max()) == 0
            if first is None:
                first = b
            assert torch.equal(b.view(torch.int64), first.view(torch.int64))
        plan.close()
