"""Edges of the symmetry transform / fold kernels' block classes, and of the VJP's element kernels past 192 modes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# blocks of 1 to 80 modes: every padded size (multiples of 16), a mode below and at its limit; random orthogonal tables
# are not a group, so the averages take the general path.  The two variants form the same products in the same order:
# bits are compared
@pytest.mark.parametrize("dims", [(64, 50, 49, 33), (80, 65, 17, 1), (48, 32, 16, 15, 2)])
@pytest.mark.parametrize("nb", [1, 5, 9])
@pytest.mark.parametrize("precision", ["bf16x3", "tf32x3"])
def test_column_kernels_equal_the_double_buffered_ones(cuda, monkeypatch, dims, nb, precision):
    torch = cuda
    from tdscha_b200 import _native
    rng = np.random.default_rng(sum(dims))
    n, N, n_sym = sum(dims), 12, 3
    start = np.concatenate([[0], np.cumsum(dims)])
    deg = [np.arange(start[b], start[b + 1], dtype=np.int32) for b in range(len(dims))]
    ids = np.repeat(np.arange(len(dims), dtype=np.int32), dims)
    tables = [np.stack([np.linalg.qr(rng.standard_normal((d, d)))[0] for _ in range(n_sym)]) for d in dims]
    w = np.repeat(1e-3 * (1 + np.arange(len(dims))), dims)
    X, Y = rng.standard_normal((2, N, n))
    ens = _native.DeviceEnsemble(X, Y, w, np.ones(N), 300.0, tables, deg, ids)
    R = torch.as_tensor(rng.standard_normal((nb, n)), device="cuda")
    Y1 = torch.as_tensor(rng.standard_normal((nb, n, n)), device="cuda")
    Y1 = (Y1 + Y1.transpose(1, 2)).contiguous()
    out = []
    for lean in (None, "0"):
        if lean:
            monkeypatch.setenv("TDSCHA_SYM_LEAN", lean)
        else:
            monkeypatch.delenv("TDSCHA_SYM_LEAN", raising=False)
        f = torch.full((nb, n), float("nan"), dtype=torch.float64, device="cuda")
        d = torch.full((nb, n, n), float("nan"), dtype=torch.float64, device="cuda")
        ens.perturb_average_device(R, Y1, f, d, 1, precision)
        torch.cuda.synchronize()
        out.append((f, d))
    assert torch.isfinite(out[0][1]).all()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    ens.close()


# 381 modes: the matrix-vector kernel's column ranges past the first, and configurations that do not fill a thread's eight.
# FP64 against the VJP over every symmetry row: two orders of the same sums; split modes with the tolerances of
# their contractions (2^-22 relative a product)
@pytest.mark.parametrize("N", [3, 9])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-11), ("bf16x3", 1e-4), ("tf32x3", 2e-5)])
def test_vjp_past_192_modes(cuda, monkeypatch, N, prec, tol):
    torch = cuda
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(4, N, seed=N)
    ens = _native.DeviceEnsemble(s.X, s.Y, s.w, s.rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)
    n = s.X.shape[1]
    rng = np.random.default_rng(N)
    t = lambda *shape: torch.as_tensor(rng.standard_normal(shape), device="cuda")   # noqa: E731
    R1, fb, Ys, Db = t(1, n), t(1, n), t(1, n, n), t(1, n, n)
    Ys, Db = (Ys + Ys.transpose(1, 2)).contiguous(), (Db + Db.transpose(1, 2)).contiguous()

    def vjp(precision, rows):
        if rows:
            monkeypatch.setenv("TDSCHA_VJP_FREQ", "0")
        else:
            monkeypatch.delenv("TDSCHA_VJP_FREQ", raising=False)
        Yb = torch.full((N, n), float("nan"), dtype=torch.float64, device="cuda")
        rb = torch.full((N,), float("nan"), dtype=torch.float64, device="cuda")
        ens.perturb_average_vjp(R1, Ys, fb, Db, Yb, rb, precision=precision)
        torch.cuda.synchronize()
        return Yb, rb

    (Y0, r0), (Yc, rc) = vjp("fp64", True), vjp(prec, False)
    assert float((Yc - Y0).abs().max()) < tol * float(Y0.abs().max())
    assert float((rc - r0).abs().max()) < tol * float(r0.abs().max())
    ens.close()
