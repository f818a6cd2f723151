"""When the averages make and use the ensemble's second stream (F beside a Z of few tiles)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ensemble(sym, N=500):
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(2, N, seed=N, with_symmetries=sym)
    return _native.DeviceEnsemble(s.X, s.Y, s.w, s.rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)


def _vectors(torch, ens, nb):
    rng = np.random.default_rng(nb)
    R = torch.as_tensor(rng.standard_normal((nb, ens.n)), device="cuda")
    Y = torch.as_tensor(rng.standard_normal((nb, ens.n, ens.n)), device="cuda")
    return R, (Y + Y.transpose(1, 2)).contiguous()


def _call(torch, ens, v, precision):
    f, d = torch.full_like(v[0], float("nan")), torch.full_like(v[1], float("nan"))
    ens.perturb_average_device(v[0], v[1], f, d, 1, precision)
    torch.cuda.synchronize()
    return f, d


# FP64, and a Z on most SMs, never fork: they make no stream and queue no event; otherwise the first call makes
# the stream and each call forks once
@pytest.mark.parametrize("sym,nb,precision,forks", [(True, 2, "fp64", 0), (False, 3, "fp64", 0), (True, 16, "bf16x3", 0),
                                                    (False, 3, "tf32x3", 1), (True, 1, "bf16x3", 1)])
def test_made_by_the_first_fork(cuda, sym, nb, precision, forks):
    ens = _ensemble(sym)
    assert ens.side_stream() == dict(made=False, marks=0, forks=0)
    v = _vectors(cuda, ens, nb)
    for call in (1, 2):
        _call(cuda, ens, v, precision)
        assert ens.side_stream() == dict(made=forks > 0, marks=call * forks, forks=call * forks)
    ens.close()


# a profile holds events of the launching stream only, so F stays there while it is taken; the contraction is the
# same launch on either stream, so the bits are the same
@pytest.mark.parametrize("sym,nb,precision", [(False, 3, "tf32x3"), (False, 32, "bf16x3"), (True, 1, "bf16x3")])
def test_profiled_calls_stay_on_the_launching_stream(cuda, sym, nb, precision):
    ens = _ensemble(sym)
    v = _vectors(cuda, ens, nb)
    f0, d0 = _call(cuda, ens, v, precision)
    assert ens.side_stream()["forks"] == 1
    ens.set_profiling(True)
    f1, d1 = _call(cuda, ens, v, precision)
    assert ens.side_stream()["forks"] == 1
    assert ens.read_profile()["gemm_f"][0] > 0.0
    ens.set_profiling(False)
    f2, d2 = _call(cuda, ens, v, precision)
    assert ens.side_stream()["forks"] == 2
    assert cuda.equal(f1, f0) and cuda.equal(d1, d0) and cuda.equal(f2, f0) and cuda.equal(d2, d0)
    ens.close()
