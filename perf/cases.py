"""The calls that this library is used for, as cases that can be timed.

Each case is one solve through the public Python API, whole: the factors (where
the call leaves them to its caller), the solution and the pivots come back.

Kinds:
  dense    Context.dgesv on device tensors (exact or fused updates)
  host     lapack.dgesv on numpy arrays, the drop-in of the crate's function
  zhost    lapack.zgesv on numpy arrays, the complex twin
  mixed    dgesv_mixed_dev: low-precision LU with FP64 refinement
  batch    BatchPlan.solve: many small systems of uneven order
  grid     SparseLu on a convection-diffusion grid, values and b on the device
  lattice  SparseLu on a finite-element lattice through the host API
"""

from __future__ import annotations

import numpy as np
import torch

from algebra_linear_b200 import _lib
from algebra_linear_b200.batched import BatchPlan
from algebra_linear_b200.device import Context
from algebra_linear_b200.lapack import dgesv, zgesv
from algebra_linear_b200.mixed import dgesv_mixed_dev
from algebra_linear_b200.sparse import LuMethod, SparseLu

_ctx = None


def _context() -> Context:
    """The one context (stream and workspace) that a program keeps."""
    global _ctx
    if _ctx is None:
        _ctx = Context()
    return _ctx


def listed():
    return [
        # a small system inside a larger device program: launch latency
        {"name": "dense_small", "kind": "dense", "update": "exact", "n": 96, "nrhs": 1},
        # the crate's own call on host arrays, order 1024 (the plain FP64 configuration)
        {"name": "host_1024", "kind": "host", "n": 1024},
        # the drop-in arithmetic (bit for bit the crate's) at an ordinary, odd order
        {"name": "exact_5001", "kind": "dense", "update": "exact", "n": 5001, "nrhs": 1},
        # the FP64 form that the mixed one is measured against, at its largest order
        {"name": "fma_16384", "kind": "dense", "update": "fma", "n": 16384, "nrhs": 1},
        # the headline: mixed precision at its largest order
        {"name": "mixed_16384", "kind": "mixed", "precision": "tf32x3", "n": 16384, "nrhs": 1},
        # several load cases against one matrix, ragged order
        {"name": "mixed_rhs64", "kind": "mixed", "precision": "tf32x3", "n": 5000, "nrhs": 64},
        # the batched configuration: 20 000 uneven systems, FP64
        {"name": "batch_fp64", "kind": "batch", "mixed": False, "count": 20000, "lo": 8, "hi": 512},
        # a smaller batch in FP32 factors with FP64 refinement
        {"name": "batch_mixed", "kind": "batch", "mixed": True, "count": 3000, "lo": 8, "hi": 512},
        # the crate's own sparse benchmark: a new value set on a small pattern, host API
        {"name": "lattice_192", "kind": "lattice", "mx": 4, "my": 4, "mz": 4},
        # the sparse configuration: refactorize + solve on the 48^3 grid, FP64
        {"name": "grid_48", "kind": "grid", "precision": "fp64", "nx": 48, "ny": 48, "nz": 48},
        # the serving mix's 2-D pattern, low-precision fronts with refinement
        {"name": "grid_300x300", "kind": "grid", "precision": "tf32x3", "nx": 300, "ny": 300, "nz": 1},
        # the complex twin on host arrays, odd order
        {"name": "zhost_777", "kind": "zhost", "n": 777},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["dense", "dense", "host", "zhost", "mixed", "mixed", "batch", "batch", "grid", "grid", "lattice"])
    if kind == "dense":
        if rng.random() < 0.5:
            return {"kind": kind, "update": "exact", "n": _log_int(rng, 24, 6000), "nrhs": rng.choice([1, 1, 3])}
        return {"kind": kind, "update": "fma", "n": _log_int(rng, 500, 14000), "nrhs": rng.choice([1, 1, 5, 64])}
    if kind == "host":
        return {"kind": kind, "n": _log_int(rng, 40, 2500)}
    if kind == "zhost":
        return {"kind": kind, "n": _log_int(rng, 30, 1500)}
    if kind == "mixed":
        return {"kind": kind, "precision": rng.choice(["tf32x3", "tf32x3", "fp32"]), "n": _log_int(rng, 700, 14000),
                "nrhs": rng.choice([1, 1, 7, 64])}
    if kind == "batch":
        lo = rng.choice([1, 8, 30])
        return {"kind": kind, "mixed": rng.random() < 0.5, "count": _log_int(rng, 300, 12000), "lo": lo,
                "hi": _log_int(rng, 2 * lo + 30, 512)}
    if kind == "grid":
        prec = rng.choice(["fp64", "tf32x3", "fp32"])
        if rng.random() < 0.5:
            return {"kind": kind, "precision": prec, "nx": rng.randint(10, 44), "ny": rng.randint(10, 44),
                    "nz": rng.randint(10, 40)}
        return {"kind": kind, "precision": prec, "nx": _log_int(rng, 40, 320), "ny": _log_int(rng, 40, 320), "nz": 1}
    return {"kind": kind, "mx": rng.randint(2, 8), "my": rng.randint(2, 8), "mz": rng.randint(2, 7)}


# ---- inputs -------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(shape, gen, dtype=torch.float64):
    """U(-1, 1)."""
    return torch.rand(shape, generator=gen, dtype=dtype, device="cuda").mul_(2.0).sub_(1.0)


def _dense_system(case, seed):
    """(T, B): T[j, i] = A[i, j] (column-major storage of A), B[r, i] the
    right-hand sides, b = A x_true with x_true U(-1, 1). A is iid U(-1, 1); for
    the mixed and the fused forms, whose results are not bit for bit the
    crate's, each column also has one entry of size sqrt(n) in a row of its own
    (rows in random order, so the rows still have to be interchanged), which
    bounds the condition number: the solution's digits are then fixed by A and
    b at every order, and by refinement to the default target."""
    n, nrhs = case["n"], case["nrhs"]
    g = _gen(seed)
    T = _uniform((n, n), g)
    if case["kind"] == "mixed" or case["update"] == "fma":
        rows = torch.randperm(n, generator=g, device="cuda")
        T[torch.arange(n, device="cuda"), rows] += float(n) ** 0.5
    X = _uniform((nrhs, n), g)
    return T, X @ T


def _host_system(case, seed):
    n = case["n"]
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1.0, 1.0, (n, n))
    x = rng.uniform(-1.0, 1.0, n)
    if case["kind"] == "zhost":
        A = A + 1j * rng.uniform(-1.0, 1.0, (n, n))
        x = x + 1j * rng.uniform(-1.0, 1.0, n)
    return A, A @ x


def _orders(case):
    """Log-uniform orders: the plan's shape, the same for every set of values."""
    rng = np.random.default_rng(case["count"])
    lo, hi = case["lo"], case["hi"]
    return np.clip(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), case["count"])).astype(np.int32), lo, hi)


def _batch_systems(case, seed):
    """Yields (members, T, b) per order: T[k, j, i] = A_k[i, j], A_k iid
    U(-1, 1) + n I as in the batched configuration, b = A_k x."""
    orders = _orders(case)
    g = _gen(seed)
    for n in np.unique(orders):
        members = np.nonzero(orders == n)[0]
        n = int(n)
        T = _uniform((len(members), n, n), g)
        T.diagonal(dim1=1, dim2=2).add_(float(n))
        x = _uniform((len(members), 1, n), g)
        yield members, T, torch.bmm(x, T)[:, 0]


def _packed(offsets, length):
    return torch.as_tensor(offsets, device="cuda")[:, None] + torch.arange(length, device="cuda")[None, :]


def _grid_pattern(nx, ny, nz):
    """CSC pattern of the 5- or 7-point stencil; kind per entry: 0 diagonal,
    1 the row's west neighbour, 2 its east neighbour, 3 the others."""
    n = nx * ny * nz
    i = np.arange(n, dtype=np.int64)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    parts = [(i, i, 0), (i[x > 0] - 1, i[x > 0], 2), (i[x < nx - 1] + 1, i[x < nx - 1], 1),
             (i[y > 0] - nx, i[y > 0], 3), (i[y < ny - 1] + nx, i[y < ny - 1], 3)]
    if nz > 1:
        parts += [(i[z > 0] - nx * ny, i[z > 0], 3), (i[z < nz - 1] + nx * ny, i[z < nz - 1], 3)]
    r = np.concatenate([p[0] for p in parts])
    c = np.concatenate([p[1] for p in parts])
    k = np.concatenate([np.full(p[0].size, p[2], np.int8) for p in parts])
    o = np.lexsort((r, c))
    cp = np.concatenate([[0], np.cumsum(np.bincount(c, minlength=n))]).astype(np.uint64)
    return cp, r[o], c[o], k[o]


def _lattice_pattern(mx, my, mz):
    """mx my mz nodes, three unknowns each, coupled to the (up to) 26 nodes around."""
    node = np.arange(mx * my * mz)
    i, j, k = node % mx, (node // mx) % my, node // (mx * my)
    near = (np.abs(i[:, None] - i) <= 1) & (np.abs(j[:, None] - j) <= 1) & (np.abs(k[:, None] - k) <= 1)
    full = np.kron(near, np.ones((3, 3), bool))
    c, r = np.nonzero(full)
    cp = np.concatenate([[0], np.cumsum(np.bincount(c, minlength=3 * node.size))]).astype(np.uint64)
    return cp, r.astype(np.int64), c.astype(np.int64)


def _sparse_system(case, seed):
    """(col_ptr, rows, values, b, x_true)."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "lattice":
        cp, r, c = _lattice_pattern(case["mx"], case["my"], case["mz"])
        off = np.bincount(c, minlength=len(cp) - 1) - 1.0
        v = np.where(r == c, 10.0 + off[c], -1.0) * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, r.size))
    else:
        cp, r, c, k = _grid_pattern(case["nx"], case["ny"], case["nz"])
        u = rng.uniform(0.0, 1.0, r.size)
        v = np.where(k == 0, 6.0 + 0.1 * u, np.where(k == 2, -1.0 + 0.3 * u, np.where(k == 1, -1.0 - 0.3 * u, -1.0)))
        v *= 1.0 + 0.01 * rng.uniform(-1.0, 1.0, r.size)
    x = rng.uniform(-1.0, 1.0, len(cp) - 1)
    return cp, r.astype(np.uint64), v, np.bincount(r, weights=v * x[c], minlength=x.size), x


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("dense", "mixed"):
        T, B = _dense_system(case, seed)
        s["a"], s["b"] = T.view(-1), B.reshape(-1)
        s["ctx"] = _context()
    elif kind in ("host", "zhost"):
        A, b = _host_system(case, seed)
        s["a"], s["b"] = np.ascontiguousarray(A.T).reshape(-1), b
    elif kind == "batch":
        s["ctx"] = _context()
        plan = BatchPlan(s["ctx"], _orders(case), mixed=case["mixed"])
        a = torch.empty(plan.a_total, dtype=torch.float64, device="cuda")
        b = torch.empty(plan.b_total, dtype=torch.float64, device="cuda")
        for members, T, rhs in _batch_systems(case, seed):
            n = T.shape[1]
            a[_packed(plan.a_off[members], n * n)] = T.view(len(members), -1)
            b[_packed(plan.b_off[members], n)] = rhs
        s.update(plan=plan, a=a, b=b, work_a=torch.empty_like(a), work_b=torch.empty_like(b),
                 info=torch.empty(case["count"], dtype=torch.int32, device="cuda"))
    else:
        cp, r, v, b, _ = _sparse_system(case, seed)
        s["lu"] = lu = SparseLu.analyze(cp, r, LuMethod.supernodal() if kind == "grid" else LuMethod.auto())
        if kind == "grid":
            s["ctx"] = _context()
            lu.bind(s["ctx"])
            lu.set_precision(case["precision"])
            s["v"], s["b"] = torch.as_tensor(v, device="cuda"), torch.as_tensor(b, device="cuda")
        else:
            s.update(cp=cp, r=r, v=v, b=b)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "dense":
        a, b = s["a"].clone(), s["b"].clone()
        update = _lib.UPDATE_FMA if case["update"] == "fma" else _lib.UPDATE_EXACT
        ipiv = s["ctx"].dgesv(a, b, case["n"], case["nrhs"], update)
        return {"lu": a, "x": b, "ipiv": ipiv}
    if kind == "mixed":  # reads A, leaves it as it is
        b = s["b"].clone()
        dgesv_mixed_dev(s["ctx"], s["a"], b, case["n"], case["nrhs"], precision=case["precision"])
        return {"x": b}
    if kind in ("host", "zhost"):
        a, b = s["a"].copy(), s["b"].copy()
        (dgesv if kind == "host" else zgesv)(a, b)
        return {"lu": a, "x": b}
    if kind == "batch":
        s["work_b"].copy_(s["b"])
        if case["mixed"]:  # the mixed form leaves A as it is
            s["plan"].solve(s["a"], s["work_b"], s["info"])
            return {"x": s["work_b"], "info": s["info"]}
        s["work_a"].copy_(s["a"])
        s["plan"].solve(s["work_a"], s["work_b"], s["info"])
        return {"lu": s["work_a"], "x": s["work_b"], "info": s["info"]}
    if kind == "grid":
        x = s["b"].clone()
        s["lu"].factorize_dev(s["v"])
        s["lu"].solve_dev(x)
        return {"x": x}
    x = s["b"].copy()
    s["lu"].factorize(s["cp"], s["r"], s["v"])
    s["lu"].solve(x)
    return {"x": x}


def work(case):
    """Bytes: the matrix (or the values) and the right-hand sides read once,
    the factors that come back and the solutions written once. Flops: the LU
    and its sweeps. A sparse case counts the values it reads and, for the
    work, the classical nested-dissection counts of its grid."""
    kind = case["kind"]
    if kind in ("dense", "host", "zhost", "mixed"):
        n, nrhs = float(case["n"]), float(case.get("nrhs", 1))
        word, mult = (16.0, 4.0) if kind == "zhost" else (8.0, 1.0)
        passes = 1.0 if kind == "mixed" else 2.0
        return {"bytes": word * (passes * n * n + 2 * n * nrhs), "flops": mult * (2 / 3 * n ** 3 + 2 * n * n * nrhs)}
    if kind == "batch":
        n = _orders(case).astype(np.float64)
        passes = 1.0 if case["mixed"] else 2.0
        return {"bytes": float(8 * (passes * n * n + 2 * n).sum()), "flops": float((2 / 3 * n ** 3 + 2 * n * n).sum())}
    if kind == "lattice":
        n = 3.0 * case["mx"] * case["my"] * case["mz"]
        return {"bytes": 8 * (n * min(n, 81.0) + 2 * n), "flops": 20.0 * (n / 3) ** 2 * 27}
    nx, ny, nz = float(case["nx"]), float(case["ny"]), float(case["nz"])
    n = nx * ny * nz
    if nz == 1:
        return {"bytes": 8 * 7 * n, "flops": 20.0 * n ** 1.5}
    return {"bytes": 8 * 9 * n, "flops": 20.0 * n ** 2}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dense", "mixed"):
        T, B = _dense_system(case, seed)
        if kind == "mixed":
            return {"x": torch.linalg.solve(T.t(), B.t()).t().reshape(-1)}
        LU, piv = torch.linalg.lu_factor(T.t())
        return {"lu": LU.t().reshape(-1), "x": torch.linalg.lu_solve(LU, piv, B.t()).t().reshape(-1), "ipiv": None}
    if kind in ("host", "zhost"):
        A, b = _host_system(case, seed)
        A, b = torch.as_tensor(A, device="cuda"), torch.as_tensor(b, device="cuda")
        LU, piv = torch.linalg.lu_factor(A)
        x = torch.linalg.lu_solve(LU, piv, b[:, None])[:, 0]
        return {"lu": np.ascontiguousarray(LU.cpu().numpy().T).reshape(-1), "x": x.cpu().numpy()}
    if kind == "batch":
        orders = _orders(case).astype(np.int64)
        a_off = np.concatenate([[0], np.cumsum(orders ** 2)])
        b_off = np.concatenate([[0], np.cumsum(orders)])
        x = torch.empty(int(b_off[-1]), dtype=torch.float64, device="cuda")
        lu = None if case["mixed"] else torch.empty(int(a_off[-1]), dtype=torch.float64, device="cuda")
        for members, T, rhs in _batch_systems(case, seed):
            n = T.shape[1]
            LU, piv = torch.linalg.lu_factor(T.transpose(1, 2))
            x[_packed(b_off[members], n)] = torch.linalg.lu_solve(LU, piv, rhs[:, :, None])[:, :, 0]
            if lu is not None:
                lu[_packed(a_off[members], n * n)] = LU.transpose(1, 2).reshape(len(members), -1)
        return {"x": x, "info": None} if lu is None else {"lu": lu, "x": x, "info": None}
    # b = A x_true in 64 bits and a well-conditioned A: x_true, to rounding
    x = _sparse_system(case, seed)[-1]
    return {"x": torch.as_tensor(x, device="cuda") if kind == "grid" else x}
