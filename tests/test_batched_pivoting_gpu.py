"""Batched dgesv on systems whose pivots move rows in every panel (no diagonal
shift): the same bits on every run, and P A = L U with LAPACK's bound. Orders at
the edges of the leaf (16), the panel (32), the tile (32 x 32), the column
chunk and the CTA shapes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 95, 97, 128, 129, 160, 161, 255, 256, 257, 289, 511, 512]


def _run(ctx, orders, mixed, threads=None, panel=None, seed=5):
    import torch

    from algebra_linear_b200.batched import BatchPlan

    plan = BatchPlan(ctx, orders, mixed=mixed)
    if threads is not None:
        for i in range(len(plan.info()["buckets"])):
            assert plan._lib.alg_batch_set_config(plan.handle, i, threads, panel) == 0
    rng = np.random.default_rng(seed)
    a0, b0 = rng.uniform(-1, 1, plan.a_total), rng.uniform(-1, 1, plan.b_total)
    a, b = torch.from_numpy(a0).cuda(), torch.from_numpy(b0).cuda()
    info = torch.empty(len(orders), dtype=torch.int32, device="cuda")
    plan.solve(a, b, info)
    torch.cuda.synchronize()
    out = a.cpu().numpy(), b.cpu().numpy(), info.cpu().numpy(), plan.ipiv()
    offs = plan.a_off.copy(), plan.b_off.copy()
    plan.close()
    return a0, b0, offs, out


def _check_lu(a0, b0, n, lu, x, piv):
    A, F = a0.reshape(n, n).T, lu.reshape(n, n).T
    perm = np.arange(n)
    for k, p in enumerate(piv):
        perm[[k, p]] = perm[[p, k]]
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    assert np.abs(L).max() <= 1.0  # partial pivoting
    # |P A - L U| <= gamma_n |L| |U| entry by entry (Higham, Accuracy and
    # Stability, Theorem 9.3), gamma_n = n u / (1 - n u)
    u = 2.0 ** -53
    gamma = n * u / (1 - n * u)
    assert (np.abs(A[perm] - L @ U) <= 2 * gamma * (np.abs(L) @ np.abs(U)) + 1e-300).all()
    # the solve adds two triangular sweeps: (A + E) x = b, |E| <= 3 gamma_n |L||U|
    r = np.abs(A @ x - b0)[perm]
    assert (r <= 4 * gamma * (np.abs(L) @ np.abs(U) @ np.abs(x)) + 1e-300).all()


@pytest.mark.parametrize("threads,panel", [(None, None), (128, 16), (128, 32), (256, 16), (256, 32), (512, 16), (512, 32)])
def test_unshifted_systems_factor_backward_stably(gpu, threads, panel):
    from algebra_linear_b200.device import Context

    with Context() as ctx:
        a0, b0, (ao, bo), (lu, x, info, piv) = _run(ctx, ORDERS, False, threads, panel)
    assert (info == 0).all()
    for k, n in enumerate(ORDERS):
        sa, sb = slice(ao[k], ao[k] + n * n), slice(bo[k], bo[k] + n)
        _check_lu(a0[sa], b0[sb], n, lu[sa], x[sb], piv[sb])


@pytest.mark.parametrize("mixed", [False, True])
def test_unshifted_batch_repeats_bit_for_bit(gpu, mixed):
    from algebra_linear_b200.device import Context

    orders = list(np.random.default_rng(1).integers(60, 200, 600))
    with Context() as ctx:
        runs = [_run(ctx, orders, mixed)[3] for _ in range(3)]
    for r in runs[1:]:
        for x, y in zip(r, runs[0]):
            assert np.array_equal(x.view(np.uint8), y.view(np.uint8))
