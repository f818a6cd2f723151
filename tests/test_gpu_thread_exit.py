"""A host thread that called the library may end while another thread captures a graph in the default (global) mode, in which a
call that CUDA counts as unsafe ends the capture with an error."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_thread_ends_during_a_capture(cuda):
    torch = cuda
    from tdscha_b200 import _native
    from tdscha_b200 import rocksalt as RS
    s = RS.make_ensemble(2, 24, seed=1, with_symmetries=False)
    ens = _native.DeviceEnsemble(s.X, s.Y, s.w, s.rho, s.T, s.symmetries, s.deg_space, s.blocks_ids)
    rng = np.random.default_rng(1)
    Y = rng.standard_normal((ens.n, ens.n))
    called, leave = threading.Event(), threading.Event()

    def worker():
        ens.perturb_average(rng.standard_normal(ens.n), Y + Y.T)   # a call that reads the error word
        called.set()
        leave.wait(60)

    thread = threading.Thread(target=worker)
    thread.start()
    assert called.wait(120)
    torch.cuda.synchronize()
    x = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x.add_(1.0)
        leave.set()
        thread.join()
        time.sleep(0.5)             # the thread's own destructors run after the join
        x.add_(1.0)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 16.0
    # a later thread works with what the first one left
    out = []
    for _ in range(2):
        thread = threading.Thread(target=lambda: out.append(ens.perturb_average(np.ones(ens.n), Y + Y.T)))
        thread.start()
        thread.join()
    assert np.array_equal(out[0][1], out[1][1]) and np.isfinite(out[0][1]).all()
    ens.close()
