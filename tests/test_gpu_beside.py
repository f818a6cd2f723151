"""The F contraction on the ensemble's second stream (few tiles in Z) in chains of calls on several streams and under graph
capture: the bits of calls that are waited for one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Z on few SMs (no symmetries; one vector with symmetries) and on most of them (F stays on the caller's stream); bits are
# compared, so no tolerance is needed
@pytest.mark.parametrize("sym,N,nb", [(False, 1531, 3), (False, 130, 1), (True, 500, 1), (True, 2000, 16)])
def test_queued_and_captured_calls_keep_their_bits(cuda, sym, N, nb):
    torch = cuda
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(2, N, seed=N, with_symmetries=sym)
    ens = _native.DeviceEnsemble(s.X, s.Y, s.w, s.rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)
    rng = np.random.default_rng(N)
    n, calls = s.X.shape[1], 6
    R = torch.as_tensor(rng.standard_normal((calls, nb, n)), device="cuda")
    Y1 = torch.as_tensor(rng.standard_normal((calls, nb, n, n)), device="cuda")
    Y1 = (Y1 + Y1.transpose(2, 3)).contiguous()

    def outputs():
        return (torch.full((calls, nb, n), float("nan"), dtype=torch.float64, device="cuda"),
                torch.full((calls, nb, n, n), float("nan"), dtype=torch.float64, device="cuda"))

    f0, d0 = outputs()
    for i in range(calls):
        ens.perturb_average_device(R[i], Y1[i], f0[i], d0[i], 1, "tf32x3")
        torch.cuda.synchronize()
    f, d = outputs()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    _native.set_error_check(False)   # calls are queued without a wait
    try:
        with torch.cuda.stream(stream):
            for i in range(calls):
                ens.perturb_average_device(R[i], Y1[i], f[i], d[i], 1, "tf32x3")
        torch.cuda.synchronize()
        assert torch.equal(f, f0) and torch.equal(d, d0)
        f, d = outputs()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):   # whose scratch the calls above allocated
            for i in range(calls):
                ens.perturb_average_device(R[i], Y1[i], f[i], d[i], 1, "tf32x3")
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(f, f0) and torch.equal(d, d0)
    finally:
        _native.set_error_check(True)
    ens.close()
