"""The rotations into and out of the rotated basis (tiles of whole blocks) through the averages, against the general path
on the unrotated basis."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 2x2x2: several blocks share a tile of 24 modes (one output per thread); 3x3x3 and 4x4x4: one block a tile and tiles of mixed
# blocks (4 x 4 outputs per thread, sizes that are not multiples of 4).  The ensemble without factorised symmetries has
# no rotated basis.  Both sides are FP64 sums of at most a few thousand terms in different orders: 1e-12 of the result
@pytest.mark.parametrize("L,N,nb", [(2, 30, 1), (2, 30, 5), (3, 9, 2), (4, 3, 1)])
def test_rotated_basis_equals_the_basis_as_given(cuda, monkeypatch, L, N, nb):
    torch = cuda
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(L, N, seed=L + N)
    args = (s.X, s.Y, s.w, s.rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)
    rot = _native.DeviceEnsemble(*args)
    # a group without one of its elements does not factorise
    plain = _native.DeviceEnsemble(*args[:5], [np.ascontiguousarray(b[:-1]) for b in s.symmetries], *args[6:])
    last = _native.DeviceEnsemble(*args[:5], [np.ascontiguousarray(b[-1:]) for b in s.symmetries], *args[6:])
    assert rot.classes()["n_class"] > 0
    n, n_sym = s.X.shape[1], s.symmetries[0].shape[0]
    rng = np.random.default_rng(N)
    R = torch.as_tensor(rng.standard_normal((nb, n)), device="cuda")
    Y1 = torch.as_tensor(rng.standard_normal((nb, n, n)), device="cuda")
    Y1 = (Y1 + Y1.transpose(1, 2)).contiguous()

    def averages(ens):
        f = torch.full((nb, n), float("nan"), dtype=torch.float64, device="cuda")
        d = torch.full((nb, n, n), float("nan"), dtype=torch.float64, device="cuda")
        ens.perturb_average_device(R, Y1, f, d, 1, "fp64")
        torch.cuda.synchronize()
        return f, d

    (f, d), (f1, d1), (f2, d2) = averages(rot), averages(plain), averages(last)
    # averages over the group: (n - 1) / n of the one, 1 / n of the other
    f0, d0 = ((n_sym - 1) * f1 + f2) / n_sym, ((n_sym - 1) * d1 + d2) / n_sym
    assert float((f - f0).abs().max()) <= 1e-12 * float(f0.abs().max())
    assert float((d - d0).abs().max()) <= 1e-12 * float(d0.abs().max())
    for e in (rot, plain, last):
        e.close()
