"""The averages' weights formed in the [a|b] contraction's epilogue against the separate [c|d] contraction
and weights kernel (TDSCHA_FREQ_FUSED_CD=0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# configurations: multiples of 4 (fp32 weights) and not (FP64 weights), below and past a tile, few and many
# vectors (either operand on the tile's 128-row side); 3x3x3 and 4x4x4 mix real and complex classes
@pytest.mark.parametrize("L,N,nb", [(2, 37, 1), (2, 512, 7), (3, 129, 2), (3, 260, 9), (4, 131, 1), (4, 68, 4)])
@pytest.mark.parametrize("precision", ["bf16x3", "tf32x3", "tf32", "bf16"])
def test_fused_weights_are_bit_identical(cuda, L, N, nb, precision, monkeypatch):
    torch = cuda
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(L, N, seed=L + N)
    rng = np.random.default_rng(N)
    rho = rng.uniform(0.5, 1.5, N)
    ens = _native.DeviceEnsemble(s.X, s.Y, s.w, rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)
    n = s.X.shape[1]
    R = torch.as_tensor(rng.standard_normal((nb, n)), device="cuda")
    Y1 = torch.as_tensor(rng.standard_normal((nb, n, n)), device="cuda")
    for d4 in (1, 0):
        out = []
        for env in ("0", None):
            if env:
                monkeypatch.setenv("TDSCHA_FREQ_FUSED_CD", env)
            else:
                monkeypatch.delenv("TDSCHA_FREQ_FUSED_CD")
            f = torch.full((nb, n), float("nan"), dtype=torch.float64, device="cuda")
            d = torch.full((nb, n, n), float("nan"), dtype=torch.float64, device="cuda")
            ens.perturb_average_device(R, Y1, f, d, d4, precision)
            torch.cuda.synchronize()
            out.append((f, d))
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]), (d4, precision)
        assert torch.isfinite(out[1][1]).all()
    ens.close()
