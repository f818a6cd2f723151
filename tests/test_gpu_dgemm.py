"""The grouped FP64 contraction of the character classes against the contractions over every symmetry row
(TDSCHA_SYM_FREQ=0, library products)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 48 representatives a vector: 32-row tiles (1, 3 vectors) and 64-row tiles (4, 5), rows past the last tile; a single
# configuration, contractions over the configurations unsplit (40) and in many slices (3000), ragged columns.  Both sides
# sum at most 6000 FP64 products in different orders: 6000 x 1.1e-16 bounds the difference of a sum, 1e-12 of the result
@pytest.mark.parametrize("L,N,nb", [(2, 1, 1), (2, 40, 3), (2, 3000, 1), (2, 1201, 5), (3, 33, 4), (3, 700, 1), (4, 21, 1)])
def test_grouped_contractions_equal_the_symmetry_rows(cuda, monkeypatch, L, N, nb):
    torch = cuda
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(L, N, seed=L + N)
    ens = _native.DeviceEnsemble(s.X, s.Y, s.w, s.rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)
    rng = np.random.default_rng(N)
    n = s.X.shape[1]
    R = torch.as_tensor(rng.standard_normal((nb, n)), device="cuda")
    Y1 = torch.as_tensor(rng.standard_normal((nb, n, n)), device="cuda")
    Y1 = (Y1 + Y1.transpose(1, 2)).contiguous()

    def averages(d4):
        f = torch.full((nb, n), float("nan"), dtype=torch.float64, device="cuda")
        d = torch.full((nb, n, n), float("nan"), dtype=torch.float64, device="cuda")
        ens.perturb_average_device(R, Y1, f, d, d4, "fp64")
        torch.cuda.synchronize()
        return f, d

    for d4 in (1, 0):
        monkeypatch.delenv("TDSCHA_SYM_FREQ", raising=False)
        f, d = averages(d4)
        f2, d2 = averages(d4)   # the slices are added in a fixed order
        assert torch.equal(f, f2) and torch.equal(d, d2)
        monkeypatch.setenv("TDSCHA_SYM_FREQ", "0")
        f0, d0 = averages(d4)
        assert float((f - f0).abs().max()) <= 1e-12 * float(f0.abs().max())
        assert float((d - d0).abs().max()) <= 1e-12 * float(d0.abs().max())
    ens.close()
