"""A refused launch is reported by the call that made it and by no later one.

The launch is refused by the runtime, before anything reaches the GPU: the
legacy default stream takes no work while a blocking stream is being captured."""
import ctypes as C

import pytest

from asteriy_2d_gb300 import problems, solver

pytestmark = pytest.mark.gpu


def test_refused_launch_is_reported_once():
    import torch
    cfg = problems.blast_config(64, 32)
    dev = torch.device("cuda:0")
    s, u = (torch.tensor(v, device=dev) for v in solver.fill_blast(cfg))
    s2, u2 = torch.empty_like(s), torch.empty_like(u)
    clock = torch.tensor([1e7, cfg.dt_first, 0.0], dtype=torch.float64, device=dev)
    count = torch.zeros(1, dtype=torch.int32, device=dev)
    T = [clock.data_ptr() + 8 * k for k in range(3)]

    def step():
        solver.step_raw(s.data_ptr(), u.data_ptr(), s2.data_ptr(), u2.data_ptr(), *T, cfg)

    step()
    torch.cuda.synchronize()
    cu = C.CDLL("libcuda.so.1")
    stream, graph = C.c_void_p(), C.c_void_p()
    assert cu.cuStreamCreate(C.byref(stream), 0) == 0
    try:
        assert cu.cuStreamBeginCapture_v2(stream, 2) == 0     # relaxed: only the implicit dependency is refused
        with pytest.raises(solver.AstError):
            step()
        cu.cuStreamEndCapture(stream, C.byref(graph))
        assert not graph.value                                # the capture was ended by the refusal
    finally:
        cu.cuStreamDestroy_v2(stream)
    solver.funk_time(*T, count.data_ptr())                    # its launch succeeds: no error of the other's
    step()
    torch.cuda.synchronize()
    assert int(count) == 1
