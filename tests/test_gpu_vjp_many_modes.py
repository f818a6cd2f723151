"""The averages' vector-Jacobian product with more modes than a 48 KB matrix-vector kernel holds."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from oracle import averages_torch as AT  # noqa: E402

pytestmark = pytest.mark.gpu


def _problem(n, N):
    """n modes in blocks of up to 80, the identity and one orthogonal operation."""
    rng = np.random.default_rng(n)
    dims = [80] * (n // 80) + ([n % 80] if n % 80 else [])
    start = np.concatenate([[0], np.cumsum(dims)])
    deg = [np.arange(start[b], start[b + 1], dtype=np.int32) for b in range(len(dims))]
    ids = np.repeat(np.arange(len(dims), dtype=np.int32), dims)
    tables = [np.stack([np.eye(d), np.linalg.qr(rng.standard_normal((d, d)))[0]]) for d in dims]
    w = np.repeat(1e-3 * (1 + 0.05 * np.arange(len(dims))), dims)
    X, Y = rng.standard_normal((2, N, n))
    rho = 0.5 + rng.random(N)
    R1, fb = rng.standard_normal((2, n))
    Y1, Db = rng.standard_normal((2, n, n))
    return X, Y, rho, w, tables, deg, ids, R1, Y1 + Y1.T, fb, Db + Db.T


# 2304 modes are the last that fit 48 KB (2 n + 1536 doubles).  FP64: sums of up to 2.7 million products in another order,
# relative to the largest output; split modes: the tolerances of the other VJP tests (1e-4, 2e-5) and four times the
# random walk of 2.7 million / 32 roundings to 24 bits in the sums over pairs (7e-5)
@pytest.mark.parametrize("n", [2304, 2305, 2320])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("bf16x3", 2e-4), ("tf32x3", 1e-4)])
def test_vjp_past_the_default_shared_memory(cuda, n, prec, tol):
    from tdscha_b200 import _native
    X, Y, rho, w, tables, deg, ids, R1, Y1, fb, Db = _problem(n, 3)
    Yt = torch.tensor(Y, requires_grad=True)
    rt = torch.tensor(rho, requires_grad=True)
    S = AT.full_symmetries(tables, deg, n)
    t = torch.as_tensor
    f, D = AT.perturb_average(t(X), Yt, w, rt, t(R1), t(Y1), 300.0, 1, S)
    gY, gr = torch.autograd.grad((t(fb) * f).sum() + (t(Db) * D).sum(), (Yt, rt))
    ens = _native.DeviceEnsemble(X, Y, w, rho, 300.0, tables, deg, ids)
    c = lambda a: torch.as_tensor(a, device="cuda").contiguous()   # noqa: E731
    Yb = torch.full(Y.shape, float("nan"), dtype=torch.float64, device="cuda")
    rb = torch.full(rho.shape, float("nan"), dtype=torch.float64, device="cuda")
    ens.perturb_average_vjp(c(R1[None]), c(Y1[None]), c(fb[None]), c(Db[None]), Yb, rb, precision=prec)
    Yb, rb = Yb.cpu().numpy(), rb.cpu().numpy()
    ens.close()
    assert np.abs(Yb - gY.numpy()).max() <= tol * np.abs(gY.numpy()).max()
    assert np.abs(rb - gr.numpy()).max() <= tol * np.abs(gr.numpy()).max()
