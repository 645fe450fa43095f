"""dgesv on singular matrices with several right-hand sides: the answer is
Singular whatever their number, b stays as it was, the factors are dgetrf's, and
many right-hand sides cost a singular matrix no solve."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _singular(n):
    rng = np.random.default_rng(n)
    a = rng.integers(-3, 4, (n, n)).astype(np.float64)
    a[:, n // 2] = 0.0  # stays exactly zero through every update
    return np.ascontiguousarray(a.T).reshape(-1)


@pytest.mark.parametrize("update", [0, 1], ids=["exact", "fma"])
@pytest.mark.parametrize("n,nrhs", [(40, 1), (40, 4), (40, 5), (300, 16), (300, 17), (300, 64), (300, 65), (3, 70000)])
def test_host_call(gpu, n, nrhs, update):
    from algebra_linear_b200.lapack import LapackError, dgesv_nrhs, dgetrf

    a0 = _singular(n)
    rng = np.random.default_rng(nrhs)
    b0 = rng.uniform(-1.0, 1.0, n * nrhs)
    a, b = a0.copy(), b0.copy()
    with pytest.raises(LapackError) as e:
        dgesv_nrhs(a, b, n, nrhs, update=update)
    assert e.value.kind == "Singular"
    assert np.array_equal(b.view(np.uint64), b0.view(np.uint64))
    if update == 0:
        f = a0.copy()
        with pytest.raises(LapackError):
            dgetrf(f, n)
        assert np.array_equal(a.view(np.uint64), f.view(np.uint64))


@pytest.mark.parametrize("update", [0, 1], ids=["exact", "fma"])
def test_device_call_and_its_launches(gpu, update):
    import torch

    from algebra_linear_b200.device import Context
    from algebra_linear_b200.lapack import LapackError

    n = 300
    with Context() as ctx:
        launches = {}
        for nrhs in (1, 64, 640):
            a = torch.as_tensor(_singular(n), device="cuda")
            b0 = torch.rand(n * nrhs, dtype=torch.float64, device="cuda")
            b = b0.clone()
            before = gpu.alg_kernel_launch_count()
            with pytest.raises(LapackError) as e:
                ctx.dgesv(a, b, n, nrhs, update)
            launches[nrhs] = gpu.alg_kernel_launch_count() - before
            assert e.value.kind == "Singular"
            assert torch.equal(b.view(torch.int64), b0.view(torch.int64))
        assert launches[640] <= launches[1]
        # the context goes on to solve (a second call, a regular matrix)
        a = torch.rand(n * n, dtype=torch.float64, device="cuda")
        a += n * torch.eye(n, dtype=torch.float64, device="cuda").view(-1)  # condition number near 1
        x = torch.rand(n * 64, dtype=torch.float64, device="cuda")
        lu, b = a.clone(), (x.view(64, n) @ a.view(n, n)).reshape(-1)
        ctx.dgesv(lu, b, n, 64, update)
        assert float((b - x).abs().max()) <= 1e-9
