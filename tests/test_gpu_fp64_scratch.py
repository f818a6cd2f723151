"""The FP64 class contractions' scratch inside the averages' workspace: calls of other formats and sizes write over it in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# each call's bits are those of the same call on an ensemble that has seen nothing else
@pytest.mark.parametrize("L,N", [(2, 700), (3, 150)])
def test_calls_of_all_formats_in_turn_keep_their_bits(cuda, L, N):
    torch = cuda
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(L, N, seed=N)
    new = lambda: _native.DeviceEnsemble(s.X, s.Y, s.w, s.rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)   # noqa: E731
    n = s.X.shape[1]
    rng = np.random.default_rng(N)
    R = torch.as_tensor(rng.standard_normal((6, n)), device="cuda")
    Y1 = torch.as_tensor(rng.standard_normal((6, n, n)), device="cuda")
    Y1 = (Y1 + Y1.transpose(1, 2)).contiguous()

    def call(ens, what):
        kind, nb, precision = what
        if kind == "vjp":
            a, b = torch.full((N, n), float("nan"), dtype=torch.float64, device="cuda"), torch.full((N,), float("nan"), dtype=torch.float64, device="cuda")
            ens.perturb_average_vjp(R[:nb], Y1[:nb], R[:nb], Y1[:nb], a, b, precision=precision)
        else:
            a, b = torch.full((nb, n), float("nan"), dtype=torch.float64, device="cuda"), torch.full((nb, n, n), float("nan"), dtype=torch.float64, device="cuda")
            ens.perturb_average_device(R[:nb], Y1[:nb], a, b, 1, precision)
        torch.cuda.synchronize()
        return a, b

    calls = [("av", 1, "fp64"), ("av", 4, "bf16x3"), ("av", 1, "fp64"), ("vjp", 1, "fp64"), ("av", 6, "fp64"), ("vjp", 2, "tf32x3"),
             ("vjp", 1, "fp64"), ("av", 2, "tf32x3"), ("av", 1, "fp64"), ("av", 6, "fp64")]
    ens, alone = new(), {}
    for what in calls:
        if what not in alone:
            fresh = new()
            alone[what] = call(fresh, what)
            fresh.close()
        got = call(ens, what)
        assert torch.isfinite(got[0]).all() and torch.isfinite(got[1]).all()
        assert torch.equal(got[0], alone[what][0]) and torch.equal(got[1], alone[what][1]), what
    ens.close()
